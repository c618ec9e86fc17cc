"""The automatic path of the FP64 form where device memory is short: dense from dimension 4000 on only where one matrix and
its workspace fit.  Buffers that the library holds from an earlier batch of another shape count as free, so that the
path does not depend on what ran before.  In a process of its own whose memory is taken up to a given rest."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
sys.path.insert(0, %r)
import numpy as np, torch
import caps_gb300 as cg

def large():
    c = cg.Caps(500e-6, 1e-6, ldim=4000)
    c.set_drude(9.0, 0.0)
    before = cg.work()["factor_flops"]
    v, s = c.logdetD_batch([300.0], [1])
    return cg.work()["factor_flops"] > before, v[0], s[0]

def mixed(n):
    c = cg.Caps(150e-6, 1e-6, ldim=1050)
    c.set_precision(cg.PREC_MIXED)
    v, s = c.logdetD_batch(np.linspace(30.0, 90.0, n), np.full(n, 2))
    assert (s < 16).all()

mixed(2)  # kernels and small buffers are loaded
plain = large()
mixed(2)  # and what it held is given back
free, _ = torch.cuda.mem_get_info()
filler = torch.empty(free - %d, dtype=torch.uint8, device="cuda")
if %r:
    mixed(100)
short = large()
print(plain[0], short[0], plain[2], short[2], plain[1] - short[1])
"""


@pytest.mark.parametrize("rest,before,dense", [(2200, False, True), (2200, True, True), (800, False, False), (800, True, False)])
def test_path(rest, before, dense):
    """dimension 8000: the matrix takes 0.51 GB, its workspace 0.28 GB, so 1.13 GB is where the path changes"""
    p = subprocess.run([sys.executable, "-c", CHILD % (ROOT, rest << 20, before)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    plain, short, s0, s1, diff = p.stdout.split()
    assert (plain, short) == ("True", str(dense))
    assert int(s0) < 16 and int(s1) < 16 and abs(float(diff)) <= (0.0 if dense else 1e-10)
