"""The calls whose speed is looked after, with their inputs and, where it is cheap, their values.

A case is one call of the Python binding as a user's program makes it.  The geometry follows
the tests and the benchmark of this repository: separation L = 1 um, a sphere of radius R, a
window of ldim = 7 R/L multipoles (matrices of dimension 2 ldim), gold-like Drude metals,
plasma metals (gamma = 0) or perfect reflectors, room temperature.  The seed moves the radius,
the frequencies and the metal by a few per cent, so that no two inputs are alike.

  kind        call                                   options
  single      Caps.logdetD(xi, m)                    rl, ldim, metal, mixed
  batch       Caps.logdetD_batch(xi[], m[])          rl, ldim, metal, mixed, nxi, nm
  energy      Caps.free_energy(T)                    rl, ldim, metal, mixed, T, learned
  t0          Caps.free_energy_T0()                  rl, ldim, metal, mixed
  spheres     Caps.logdetD2_batch(xi[], m[])         rl, ldim, metal, nxi, nm
  cylinder    capc_logdet(R, d, q[])                 rd, lmax, boundary, nq
  mlp         MLP.loss_grad(X, y), MLP.predict(X)    n
"""
import math

import numpy as np
import torch

import caps_gb300 as cg
from caps_gb300 import learned

SEP = 1e-6                        # sphere-plane separation L in metres
HBAR, KB, CL = 1.0545718e-34, 1.38064852e-23, 299792458.0
CUTOFF, EPSREL = 1e-9, 1e-6       # truncation of the sums over m and over the frequencies (the defaults)


def listed():
    return [
        # one matrix, the reference's own call: a program that links the library as a drop-in
        # asks for one (xi, m) at a time; the smallest work there is
        dict(name="single", kind="single", rl=20.0, ldim=140, metal="drude", mixed=False),
        # a few frequencies with their first m, perfect reflectors, default (FP64) form
        dict(name="batch-350", kind="batch", rl=50.0, ldim=350, metal="perfect", mixed=False, nxi=4, nm=8),
        # the same at the benchmark's geometry: matrices of dimension 2100
        dict(name="batch-1050", kind="batch", rl=150.0, ldim=1050, metal="drude", mixed=False, nxi=3, nm=8),
        # free energies at room temperature in the default form, small and ordinary
        dict(name="energy-rl20", kind="energy", rl=20.0, ldim=140, metal="drude", mixed=False, T=300.0, learned=False),
        dict(name="energy-rl100", kind="energy", rl=100.0, ldim=700, metal="drude", mixed=False, T=300.0, learned=False),
        # the benchmark's free energy: mixed form with learned truncation
        dict(name="energy-learned-rl150", kind="energy", rl=150.0, ldim=1050, metal="drude", mixed=True, T=300.0, learned=True),
        # T = 0: the adaptive frequency integral, many dependent batches of small matrices
        dict(name="t0-rl10", kind="t0", rl=10.0, ldim=70, metal="drude", mixed=False),
        # large aspect ratio: a few matrices of dimension 5000 and 6000
        dict(name="large-2500", kind="batch", rl=357.0, ldim=2500, metal="plasma", mixed=False, nxi=2, nm=2),
        dict(name="large-3000-mixed", kind="batch", rl=428.0, ldim=3000, metal="drude", mixed=True, nxi=3, nm=2),
        # sphere-sphere: log det(1 - M^2)
        dict(name="spheres-140", kind="spheres", rl=20.0, ldim=140, metal="perfect", nxi=6, nm=8),
        # cylinder-plane: the nodes of one step of its energy integral
        dict(name="cylinder-300", kind="cylinder", rd=50.0, lmax=300, boundary="D", nq=30),
        # one step of training of the truncation network on a set of the usual size, and its predictions
        dict(name="mlp-2600", kind="mlp", n=2600),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["single", "batch", "batch", "batch", "energy", "energy", "t0", "spheres", "cylinder", "mlp"])
    metal = rng.choice(["drude", "drude", "plasma", "perfect"])
    mixed = rng.random() < 0.4
    if kind == "mlp":
        return dict(kind=kind, n=int(_log(rng, 40, 20000)))
    if kind == "cylinder":
        rd = _log(rng, 3, 100)
        return dict(kind=kind, rd=rd, lmax=max(25, int(6 * rd)), boundary=rng.choice("DN"), nq=rng.randint(1, 45))
    if kind == "single":
        ldim = int(_log(rng, 20, 1050))
        return dict(kind=kind, rl=max(1.0, ldim / 7), ldim=ldim, metal=metal, mixed=mixed)
    if kind == "spheres":
        ldim = int(_log(rng, 20, 350))
        return dict(kind=kind, rl=max(1.0, ldim / 7), ldim=ldim, metal=metal, nxi=rng.randint(1, 6), nm=rng.randint(1, 8))
    if kind == "t0":
        rl = rng.uniform(2, 12)
        return dict(kind=kind, rl=rl, ldim=max(20, int(7 * rl)), metal=metal, mixed=mixed)
    if kind == "energy":
        rl = _log(rng, 4, 150) if mixed else _log(rng, 4, 80)
        return dict(kind=kind, rl=rl, ldim=max(20, math.ceil(7 * rl)), metal=metal, mixed=mixed, T=rng.uniform(250, 600),
                    learned=mixed and rng.random() < 0.5)
    ldim = int(_log(rng, 20, 3000))
    most = 24 if ldim < 1200 else 6   # matrices of one call
    nxi = rng.randint(1, 3)
    return dict(kind=kind, rl=max(1.0, ldim / 7), ldim=ldim, metal=metal, mixed=mixed, nxi=nxi, nm=rng.randint(1, most // nxi))


# ---- inputs ----

def _metal(case, r):
    """(omega_p, gamma) in eV, None for perfect reflectors"""
    wp, ga = 9.0 * (1 + 0.1 * r.uniform(-1, 1)), 0.035 * (1 + 0.2 * r.uniform(-1, 1))
    return {"perfect": None, "plasma": (wp, 0.0), "drude": (wp, ga)}[case["metal"]]


def _inputs(case, seed):
    r = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "mlp":
        n = case["n"]
        # the ranges of learned.training_set, and targets that fall off like log|logdetD| does
        X = np.stack([np.log(r.uniform(10, 50, n)) / 5, np.exp(r.uniform(np.log(0.01), np.log(14), n)) / 8, r.uniform(0, 1.8, n),
                      r.choice([5.0, 0.7, 1.0, 0.8], n), r.choice([0.0, 0.4, 1.0, 0.9], n)], axis=1).astype(np.float32)
        y = (2 * X[:, 0] - 8 * X[:, 1] - 12 * X[:, 2] + 0.1 * r.standard_normal(n)).astype(np.float32)
        return dict(X=X, y=y, net=int(r.integers(1 << 30)))
    if kind == "cylinder":
        # wave numbers as the energy integral over x = 2 d q visits them
        d = 1e-6 * (1 + 0.05 * r.uniform(-1, 1))
        return dict(R=case["rd"] * d, d=d, q=np.sort(np.exp(r.uniform(math.log(0.02), math.log(15), case["nq"]))) / (2 * d))
    R = case["rl"] * SEP * (1 + 0.03 * r.uniform(-1, 1))
    got = dict(R=R, metal=_metal(case, r))
    if kind == "energy":
        got["T"] = case["T"] * (1 + 0.02 * r.uniform(-1, 1))
    elif kind != "t0":
        # frequencies in the range of a Matsubara sum: decay exponent 2 xi L/c from 0.3 to 8
        n = case.get("nxi", 1)
        xi = np.sort(np.exp(r.uniform(math.log(0.3), math.log(8.0), n))) * (1 + R / SEP) / 2
        first = int(r.integers(0, 3))
        ms = np.arange(first, first + case.get("nm", 1))
        got.update(xi=np.repeat(xi, len(ms)), m=np.tile(ms, n).astype(np.int32))
    return got


def prepare(case, seed):
    i = _inputs(case, seed)
    kind = case["kind"]
    if kind == "mlp":
        return dict(kind=kind, net=cg.MLP(i["net"]), X=i["X"], y=i["y"])
    if kind == "cylinder":
        return dict(kind=kind, boundary=case["boundary"], lmax=case["lmax"], **i)
    c = cg.Caps(i["R"], SEP, ldim=case["ldim"])
    if i["metal"]:
        c.set_drude(*i["metal"])
    if case.get("mixed"):
        c.set_precision(cg.PREC_MIXED)
    state = dict(kind=kind, caps=c, **{k: i[k] for k in ("xi", "m", "T") if k in i})
    if case.get("learned"):
        state["net"] = learned.train(epochs=1500)[0]
    return state


def run(state):
    kind = state["kind"]
    if kind == "mlp":
        loss, grad = state["net"].loss_grad(state["X"], state["y"])
        return dict(loss=np.float32(loss), grad=grad, predicted=state["net"].predict(state["X"]))
    if kind == "cylinder":
        return cg.capc_logdet(state["R"], state["d"], state["q"], state["boundary"], state["lmax"])
    c = state["caps"]
    if kind == "single":
        return np.float64(c.logdetD(state["xi"][0], state["m"][0]))
    if kind in ("batch", "spheres"):
        v, status = (c.logdetD_batch if kind == "batch" else c.logdetD2_batch)(state["xi"], state["m"])
        return dict(logdet=v, failed=status >= 16)
    E, info = c.free_energy_T0() if kind == "t0" else c.free_energy(state["T"], mlp=state.get("net"))
    E = np.float64(E)
    if kind == "t0":
        return dict(E=E)
    return dict(E=E, nxi=info["nxi"], xi=np.array(info["xi"]), terms=np.array(info["logdetD"]))


def work(case):
    """Operations of the sums and factorisations; the data of a call (its scalars or lists) is next to nothing."""
    kind = case["kind"]
    if kind == "mlp":
        return dict(bytes=case["n"] * 7 * 4, flops=case["n"] * 4 * 2 * (5 * 64 + 2 * 64 * 64 + 64))
    if kind == "cylinder":
        return dict(bytes=16 * case["nq"], flops=case["nq"] * 2 * (case["lmax"] ** 3 / 3 + 8 * case["lmax"] ** 2))
    ldim = case["ldim"]
    # terms of the sums: m runs to about 4.7 sqrt(R/L), the frequencies to 2 xi L/c = 14; an
    # adaptive T = 0 integral takes about 285 abscissae.  Six in ten matrices need their determinant
    perxi = 4.7 * math.sqrt(case["rl"])
    if kind == "energy":
        n, factored = 17 * 300 / case["T"] * perxi, 0.6
    elif kind == "t0":
        n, factored = 285 * perxi, 0.6
    else:
        n, factored = case.get("nxi", 1) * case.get("nm", 1), 1.0
    dim = 2 * ldim
    matrix = dim ** 3 / 3 + 60 * ldim ** 2 + (dim ** 3 if kind == "spheres" else 0)  # M^2 is symmetric
    return dict(bytes=16 * n, flops=n * (factored * matrix + 4 * ldim * 60 * 10))


# ---- values in 64 bits: the round trip as a Gram matrix over quadrature nodes ----
# M_{l1 l2} = int dx e^{-2 xi x} [r_TM v_l1 v_l2 + |r_TE| w_l1 w_l2], x = cosh t, with
# v_l = (A_l s P', B_l m P/s), w_l = (A_l m P/s, B_l s P'), s = sinh t, P = P_l^m(x) and A, B the
# normalisation times the square roots of the Mie coefficients.  The integrand decays at both
# ends of log s, so the trapezoidal rule converges beyond all orders.

def _mie(chi, lmax, eps):
    """log a_l, log b_l for l = 0..lmax (0 unused); eps = epsilon - 1 of the sphere or inf"""
    def tables(x):
        # rho_l = I_{l-1/2}/I_{l+1/2} downwards, K upwards, I from the Wronskian
        top = lmax + 60 + int(3 * x)
        r = (2 * top + 1) / x
        inv = np.zeros(lmax + 2)               # 1/rho_{l+1}
        for l in range(top - 1, -1, -1):
            if l <= lmax:
                inv[l] = 1 / r
            r = (2 * l + 1) / x + 1 / r
        logk, up = np.zeros(lmax + 1), np.zeros(lmax + 1)   # log K_{l+1/2}; K_{l+1/2}/K_{l-1/2}
        logk[0], up[0] = 0.5 * math.log(math.pi / (2 * x)) - x, 1.0
        for l in range(1, lmax + 1):
            up[l] = (2 * l - 1) / x + 1 / up[l - 1]
            logk[l] = logk[l - 1] + math.log(up[l])
        l = np.arange(lmax + 1)
        rho = (2 * l + 1) / x + inv[:lmax + 1]
        logi = -math.log(x) - logk - np.log(rho + 1 / up)   # I_{l+1/2}
        return rho, inv[:lmax + 1], logi, logk, up
    l = np.arange(lmax + 1)
    rho, inv, logi, logk, up = tables(chi)
    half_pi = math.log(math.pi / 2)
    if math.isinf(eps):
        with np.errstate(divide="ignore"):
            return half_pi + logi - logk + np.log(l + 1 + chi * inv) - np.log(l + chi / up), half_pi + logi - logk
    n = math.sqrt(1 + eps)
    rho_n, inv_n, _, _, _ = tables(n * chi)
    # everything over I_{l+1/2}(n chi) K_{l+1/2}(chi)
    gb = chi * (n * inv_n - inv)
    gd = chi * (1 / up + n * rho_n)
    gc = eps * (chi / up + l)
    ga = eps * (l + 1) + n * chi * (n * inv - inv_n)
    return half_pi + logi - logk + np.log(ga) - np.log(gc + gd), half_pi + logi - logk + np.log(gb) - np.log(gd)


def _gram(R, ldim, xi, m, metal, square=False):
    """log det(1 - M), or log det(1 - M^2), for lists xi (scaled by (L+R)/c) and m"""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    f64 = dict(dtype=torch.float64, device=dev)
    xi, m = np.asarray(xi, float), np.asarray(m, int)
    lmin = np.where(m == 0, 1, np.maximum(m, np.round(m / math.sqrt(2 * SEP / R)).astype(int) - ldim // 2))
    lmax = int(lmin.max()) + ldim
    h = 0.6 / math.sqrt(4 * lmax)
    out = np.empty(len(xi))
    mie = {}
    for x in sorted(set(xi)):
        eps = math.inf
        if metal:
            w = x * CL / (SEP + R)
            wp, ga = (v / 6.582119514e-16 for v in metal)
            eps = wp * wp / (w * (w + ga))
        mie[x] = (eps, *_mie(x * R / (R + SEP), lmax, eps))
    lo, hi = -20.0, math.log((2 * lmax + 100) / xi.min())
    nodes = int((hi - lo) / h) + 1
    step = max(1, int(1.5e9 / (nodes * 2 * ldim * 8)))
    for k in range(0, len(xi), step):
        X, M, lm = xi[k:k + step], m[k:k + step], lmin[k:k + step]
        n = len(X)
        mm = torch.tensor(np.maximum(M, 1), **f64)[:, None]
        md = torch.tensor(M, **f64)[:, None]
        s = torch.exp(lo + h * torch.arange(nodes, **f64))[None, :]
        x = torch.sqrt(1 + s * s)
        xt = torch.tensor(X, **f64)[:, None]
        eps = torch.tensor([mie[v][0] for v in X], **f64)[:, None]
        if metal:
            y = eps / (x * x)
            b = y / (torch.sqrt(1 + y) + 1)
            rte, rtm = b / (2 + b), (eps - b) / (eps + 2 + b)
        else:
            rte = rtm = torch.ones_like(x).expand(n, -1)
        # dx = s ds/dlog(s) ... = s * (s/x) dlog(s); log of the square root of weight and e^{-2 xi x}
        lw = 0.5 * (torch.log(h * s * s / x)) - xt * x
        V = torch.zeros((n, nodes, ldim, 2), **f64)
        W = torch.zeros((n, nodes, ldim, 2), **f64)
        logn = torch.zeros((n, ldim, 2), **f64)
        for i in range(n):
            l = np.arange(lm[i], lm[i] + ldim)
            lg = np.vectorize(math.lgamma)
            f = np.log(2.0 * l + 1) - np.log(l * (l + 1.0)) + lg(l - M[i] + 1.0) - lg(l + M[i] + 1.0)
            _, la, lb = mie[X[i]]
            logn[i] = torch.tensor(np.stack([0.5 * (f + la[l]), 0.5 * (f + lb[l])], axis=1), **f64)
        # P_l^{m'} by its ratio (stable upwards: P is the dominant solution for x > 1)
        mi = np.maximum(M, 1)
        logp = torch.tensor([math.lgamma(2 * v + 1) - math.lgamma(v + 1) - v * math.log(2) for v in mi], **f64)[:, None] + mm * torch.log(s)
        low = torch.zeros((n, nodes), **f64)       # P_{l-1}/P_l
        pos = torch.tensor(lm, device=dev)
        rows = torch.arange(n, device=dev)
        for j in range(int((lm + ldim - mi).max())):
            l = mm + j
            w = (l[:, 0].long() - pos)
            on = (w >= 0) & (w < ldim)
            if bool(on.any()):
                r, c = rows[on], w[on]
                e = torch.exp((logp + lw)[r][:, :, None] + logn[r, c][:, None, :])
                # m >= 1: s P' = P (l x - (l+m) P_{l-1}/P_l)/s; m = 0: s P' = P_l^1
                d = torch.where(md == 0, torch.ones_like(x), (l * x - (l + mm) * low) / s)[r]
                g = (md / s).expand(n, -1)[r]
                ta, tb = e[:, :, 0], e[:, :, 1]
                st, se = torch.sqrt(rtm.expand(n, -1))[r], torch.sqrt(rte.expand(n, -1))[r]
                V[r, :, c, 0], V[r, :, c, 1] = st * ta * d, st * tb * g
                W[r, :, c, 0], W[r, :, c, 1] = se * ta * g, se * tb * d
            ratio = ((2 * l + 1) * x - (l + mm) * low) / (l - mm + 1)
            logp = logp + torch.log(ratio)
            low = 1 / ratio
        V, W = V.reshape(n, nodes, 2 * ldim), W.reshape(n, nodes, 2 * ldim)
        A = V.transpose(1, 2) @ V + W.transpose(1, 2) @ W
        if square:
            A = A @ A
        tr = torch.diagonal(A, dim1=1, dim2=2).sum(1)
        C = torch.linalg.cholesky(torch.eye(2 * ldim, **f64) - A)
        ld = 2 * torch.log(torch.diagonal(C, dim1=1, dim2=2)).sum(1)
        out[k:k + n] = torch.where(tr < 1e-8, -tr, ld).cpu().numpy()
    return out


def _sum_m(R, ldim, xi, metal):
    """sum over m (m = 0 with weight 1/2) of log det(1 - M) at each xi, with the cutoff of the library"""
    terms = [[] for _ in xi]
    left, m0 = list(range(len(xi))), 0
    while left:
        v = _gram(R, ldim, np.repeat([xi[i] for i in left], 8), np.tile(np.arange(m0, m0 + 8), len(left)), metal).reshape(-1, 8)
        for i, row in zip(left, v):
            terms[i] += list(row)
        left = [i for i in left if not any(t / terms[i][0] < CUTOFF for t in terms[i])]
        m0 += 8
    got = []
    for t in terms:
        stop = next(k for k, v in enumerate(t) if v / t[0] < CUTOFF)
        got.append(math.fsum([t[0] / 2] + t[1:stop + 1]))
    return np.array(got)


def _drude_ht(R):
    x = SEP / R
    Z = (1 + x) * (1 - math.sqrt((x * x + 2 * x) / (x * x + 2 * x + 1)))
    l = np.arange(1, 20000)
    a = Z ** (2.0 * l)
    b = a * Z
    return 0.5 * (math.fsum((2 * l + 1) * np.log1p(-b)) + math.log1p(-(1 - Z * Z) * math.fsum(b * (1 - a) / (1 - b))))


def _bessel(x, n):
    """log K_k and log I_k, k = 0..n"""
    t = np.arange(0, 12, 0.01)
    w = np.where(t == 0, 0.5, 1.0) * 0.01
    k0, k1 = (float(np.sum(w * np.exp(-x * (np.cosh(t) - 1)) * np.cosh(v * t))) for v in (0, 1))
    if x < 1e-3:
        raise ValueError("argument below the range of the rule")
    logk, up = [math.log(k0) - x, math.log(k1) - x], [k1 / k0]       # up[k] = K_{k+1}/K_k
    for k in range(1, n + 1):
        up.append(2 * k / x + 1 / up[-1])
        logk.append(logk[-1] + math.log(up[-1]))
    top = n + 60 + int(3 * x)
    r = 0.0                                                          # I_{k+1}/I_k
    rat = np.zeros(n + 2)
    for k in range(top, -1, -1):
        r = 1 / (2 * (k + 1) / x + r)
        if k <= n + 1:
            rat[k] = r
    k = np.arange(n + 1)
    logk, up = np.array(logk), np.array(up)
    return logk[:n + 1], -math.log(x) - logk[:n + 1] - np.log(up[:n + 1] + rat[:n + 1])


def _cylinder(R, d, n, q, dn):
    x = R * q
    kr, ir = _bessel(x, n + 1)
    kq, _ = _bessel(2 * (R + d) * q, 2 * n + 1)
    if dn == "D":
        ratio = ir - kr
    else:
        ratio = np.empty(n + 1)
        ratio[0] = ir[1] - kr[1]
        ratio[1:] = np.logaddexp(ir[:n], ir[2:n + 2]) - np.logaddexp(kr[:n], kr[2:n + 2])
    m00 = math.exp(ratio[0] + kq[0])
    mu = np.arange(1, n + 1)
    t = 0.5 * (ratio[mu][:, None] + ratio[mu][None, :])
    U, V = np.exp(t + kq[mu[:, None] + mu[None, :]]), np.exp(t + kq[abs(mu[:, None] - mu[None, :])])
    w = np.exp(0.5 * (ratio[mu] + ratio[0]) + kq[mu])
    total = math.log1p(-m00)
    for M in (U - V, U + V + 2 / (1 - m00) * np.outer(w, w)):
        tr = float(np.trace(M))
        total += -tr if abs(tr) < 1e-8 else float(np.linalg.slogdet(np.eye(n) - M)[1])
    return total


def exact(case, seed):
    i = _inputs(case, seed)
    kind = case["kind"]
    if kind == "mlp":
        net = cg.MLP(i["net"])
        p = torch.tensor(net.params(), dtype=torch.float64, requires_grad=True)
        h, o = torch.tensor(i["X"], dtype=torch.float64), 0
        for a, b in ((64, 5), (64, 64), (64, 64), (1, 64)):
            h = h @ p[o:o + a * b].reshape(a, b).T + p[o + a * b:o + a * b + a]
            o += a * b + a
            h = torch.nn.functional.silu(h) if a > 1 else h
        loss = torch.mean((h[:, 0] - torch.tensor(i["y"], dtype=torch.float64)) ** 2)
        loss.backward()
        return dict(loss=loss.item(), grad=p.grad, predicted=h[:, 0].detach())
    if kind == "cylinder":
        if case["lmax"] > 400:
            return None
        return np.array([_cylinder(i["R"], i["d"], case["lmax"], q, case["boundary"]) for q in i["q"]])
    if case["ldim"] > 360:
        return None
    R, ldim, metal = i["R"], case["ldim"], i["metal"]
    if kind == "single":
        return np.float64(_gram(R, ldim, i["xi"], i["m"], metal)[0])
    if kind in ("batch", "spheres"):
        return dict(logdet=_gram(R, ldim, i["xi"], i["m"], metal, kind == "spheres"), failed=None)
    if ldim > 150:
        return None
    if kind == "t0":
        if case["metal"] == "drude":
            return None                    # F has the scale of gamma near zero, too narrow for the rule below
        # E (L+R)/(hbar c) = 1/(pi a) int dx F(x/a), a = 2 L/(L+R)
        x, w = np.polynomial.laguerre.laggauss(48)
        a = 2 * SEP / (SEP + R)
        F = _sum_m(R, ldim, x / a, metal)
        return dict(E=np.sum(w * np.exp(x) * F) / (a * math.pi))
    if case["metal"] != "drude":
        return None                        # the zero-frequency term has its own matrices there
    step = 2 * math.pi * KB * (R + SEP) * i["T"] / (HBAR * CL)
    terms = [_drude_ht(R)]
    while len(terms) == 1 or abs(terms[-1] / terms[0]) >= EPSREL:
        terms += list(_sum_m(R, ldim, np.array([len(terms) * step]), metal))
    terms = np.array(terms)
    E = step / math.pi * math.fsum([terms[0] / 2] + list(terms[1:]))
    return dict(E=np.float64(E), nxi=None, xi=step * np.arange(len(terms)), terms=terms)
