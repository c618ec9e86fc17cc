"""Cylinder-plane batches: the memory that a batch of many small matrices takes is bounded (4 GB of matrices, 4 GB of
workspace), and the values of its parts are those of the whole."""
import subprocess
import sys
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
sys.path.insert(0, %r)
import numpy as np, torch
import caps_gb300 as cg
q = np.linspace(0.02, 15, 16384) / 2e-6
cg.capc_logdet(4e-6, 1e-6, q[:1], "N", %d)
before = torch.cuda.mem_get_info()[0]
cg.capc_logdet(4e-6, 1e-6, q, "N", %d)
print(before - torch.cuda.mem_get_info()[0])
"""


@pytest.mark.parametrize("n", [1, 25, 64, 65])
def test_memory(n):
    p = subprocess.run([sys.executable, "-c", CHILD % (ROOT, n, n)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    # matrices and tables of 16384 wave numbers stay below 1.5 GB at these sizes; buffers grow by a quarter at most
    assert int(p.stdout) <= 1.25 * (4 << 30) + (3 << 29), p.stdout


@pytest.mark.parametrize("boundary", ["D", "N"])
def test_parts(boundary):
    import caps_gb300 as cg
    q = np.linspace(0.02, 15, 16384) / 2e-6
    got = cg.capc_logdet(4e-6, 1e-6, q, boundary, 25)
    for k in (0, 8000, 8700, 8800, 16383):
        assert got[k] == cg.capc_logdet(4e-6, 1e-6, q[k], boundary, 25)
