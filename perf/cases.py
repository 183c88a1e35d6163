"""Performance cases: what programs have this framework do, through its
public entry points (``oap_b200``), over the sizes they use.

listed() names the cases, draw() gives more of the same ranges, prepare()
makes what a program holds before the call (operators, images, handles, the
network) on the GPU from a seed, run() is one pass, work() what a pass cannot
do without, exact() the 64-bit result by plain torch / numpy.

Solves are asked for eigenvalues, the call without an eigenvector matrix, and
return them with whether every pair met the residual goal (the residuals
themselves are rounding-sized numbers below that goal).
"""

import ctypes as C

import numpy as np
import torch

import oap_b200 as B
from oap_b200 import warmstart as W

TOL = 1e-10
SHIFT = 4.0  # added to the planted diagonal entries of the dense operators


def listed():
    return [
        # the reference's CPU-sized solve: a few hundred rows, symmetric, a
        # decaying spectrum; one small operator after another (latency)
        dict(name="sym_256", kind="solve", spectrum="geometric", n=256, k=5, m=32, sort="LM", precision="mixed",
             fresh=True),
        # one member of a parameterised symmetric family, rightmost values at
        # the edge of a dense spectrum: many restarts, an operator that fits L2
        dict(name="sym_edge_2048", kind="solve", spectrum="edge", n=2048, k=8, m=24, sort="LR", precision="fp64",
             fresh=True),
        # an ordinary complex operator of odd size by the plain FP64 restart loop
        dict(name="complex_3001", kind="solve", spectrum="planted", cplx=True, n=3001, k=8, m=32, sort="LM",
             precision="fp64", fresh=True),
        # the benchmark's workload: large complex non-Hermitian operator, resident, top 16
        dict(name="complex_16384", kind="solve", spectrum="planted", cplx=True, n=16384, k=16, m=64, sort="LM",
             precision="mixed", fresh=False),
        # a large operator of odd size solved once: its preparation is part of the call
        dict(name="complex_fresh_9001", kind="solve", spectrum="planted", cplx=True, n=9001, k=8, m=40, sort="LM",
             precision="mixed", fresh=True),
        # a large real symmetric operator solved once
        dict(name="sym_fresh_12000", kind="solve", spectrum="planted", cplx=False, n=12000, k=8, m=40, sort="LM",
             precision="mixed", fresh=True),
        # thousands of uneven complex problems in one call
        dict(name="batch_2048", kind="batch", cplx=True, count=2048, nmin=32, nmax=512, k=4, hdim=24),
        # a few hundred small symmetric ones
        dict(name="batch_sym_300", kind="batch", cplx=False, count=300, nmin=24, nmax=160, k=3, hdim=16),
        # the image application: the Gram operator of 4096 images of 256 x 256 pixels, built ...
        dict(name="gram_build_4096", kind="gram_build", rows=4096, cols=65536),
        # ... or applied without building it, top 32
        dict(name="gram_solve_4096", kind="gram_solve", rows=4096, cols=65536, k=32, m=96),
        # the operator surface: a complex matrix product of ragged sizes
        dict(name="dot_1500", kind="dot", cplx=True, rows=1500, inner=1031, cols=1277),
        # one training step of the warm-start network (forward, backward, update)
        dict(name="train_256", kind="train", batch=256, hidden=256, out=2056),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["small", "edge", "plain", "plain", "mixed", "mixed", "batch", "batch", "gram_build",
                       "gram_solve", "dot", "train"])
    if kind == "small":
        m = rng.randint(20, 32)
        return dict(kind="solve", spectrum="geometric", n=_log_int(rng, 64, 640), k=rng.randint(2, 6), m=m, sort="LM",
                    precision=rng.choice(["mixed", "fp64"]), fresh=True)
    if kind == "edge":
        return dict(kind="solve", spectrum="edge", n=_log_int(rng, 500, 2500), k=rng.randint(4, 8),
                    m=rng.randint(24, 40), sort="LR", precision="fp64", fresh=True)
    if kind == "plain":
        return dict(kind="solve", spectrum="planted", cplx=rng.random() < 0.7, n=_log_int(rng, 700, 6000),
                    k=rng.randint(4, 12), m=rng.randint(28, 48), sort="LM", precision="fp64", fresh=True)
    if kind == "mixed":
        return dict(kind="solve", spectrum="planted", cplx=rng.random() < 0.7, n=_log_int(rng, 8192, 14000),
                    k=rng.randint(5, 16), m=rng.randint(40, 64), sort="LM", precision="mixed",
                    fresh=rng.random() < 0.5)
    if kind == "batch":
        nmax = _log_int(rng, 100, 512)
        return dict(kind="batch", cplx=rng.random() < 0.6, count=_log_int(rng, 100, 1500), nmin=rng.randint(24, 48),
                    nmax=nmax, k=rng.randint(2, 5), hdim=rng.randint(16, 28))
    if kind in ("gram_build", "gram_solve"):
        case = dict(kind=kind, rows=_log_int(rng, 300, 4000), cols=_log_int(rng, 2500, 60000))
        if kind == "gram_solve":
            case.update(k=rng.randint(6, 32), m=rng.randint(64, 96))
        return case
    if kind == "dot":
        return dict(kind="dot", cplx=rng.random() < 0.6, rows=_log_int(rng, 100, 1600), inner=_log_int(rng, 60, 1600),
                    cols=_log_int(rng, 30, 1600))
    return dict(kind="train", batch=_log_int(rng, 32, 512), hidden=rng.randint(100, 300), out=_log_int(rng, 250, 2100))


# ------------------------------------------------------------------ inputs --
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, *shape):
    return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g)


def _operator(case, seed):
    """(re, im or None) FP64 planes of a dense operator.
    geometric: symmetric, eigenvalues 1 .. 1e-3; edge: symmetric Gaussian
    (G + G^T) / (2 sqrt n); planted: Gaussian of unit spectral size plus 4 on
    k seeded diagonal positions."""
    n, g = case["n"], _generator(seed)
    if case["spectrum"] == "geometric":
        q, _ = torch.linalg.qr(_randn(g, n, n))
        lam = 10.0 ** (-3.0 * torch.arange(n, dtype=torch.float64, device="cuda") / (n - 1))
        a = (q * lam) @ q.T
        return ((a + a.T) * 0.5).contiguous(), None
    if case["spectrum"] == "edge" or not case["cplx"]:
        a = _randn(g, n, n)
        a = (a + a.T).div_(2.0 * n ** 0.5)
        b = None
    else:
        s = (1.0 / (2.0 * n)) ** 0.5
        a, b = _randn(g, n, n).mul_(s), _randn(g, n, n).mul_(s)
    if case["spectrum"] == "planted":
        pos = torch.randperm(n, generator=g, device="cuda")[:case["k"]]
        a[pos, pos] += SHIFT
    return a, b



def _batch(case, seed):
    """Independent operators of uneven sizes (Gaussian plus 4 on k diagonal
    positions; symmetric when real), one allocation for all."""
    rng = np.random.default_rng(seed)
    sizes = rng.integers(case["nmin"], case["nmax"] + 1, size=case["count"])
    at = np.concatenate([[0], np.cumsum((sizes * sizes + 31) // 32 * 32)])
    g = _generator(seed)
    total = int(at[-1])
    s = np.repeat((1.0 / (2.0 * sizes)) ** 0.5, np.diff(at)) if case["cplx"] else np.repeat(
        1.0 / (2.0 * sizes ** 0.5), np.diff(at))
    scale = torch.from_numpy(s).cuda()
    re = _randn(g, total).mul_(scale)
    im = _randn(g, total).mul_(scale) if case["cplx"] else None
    where = np.concatenate([o + rng.permutation(n)[:case["k"]] * (n + 1) for o, n in zip(at[:-1], sizes)])
    mats = []
    for o, n in zip(at[:-1], sizes):
        o, n = int(o), int(n)
        r = re[o:o + n * n].view(n, n)
        if case["cplx"]:
            mats.append((r, im[o:o + n * n].view(n, n)))
        else:
            r.copy_(r + r.T)
            mats.append((r, None))
    re[torch.from_numpy(where).cuda()] += SHIFT
    return mats


def _images(rows, cols, seed):
    """rows synthetic images of cols pixels as FP32 rows in [0, 1]: a smooth
    sum of 8 blobs along the pixels plus noise, quantised to 8 bits."""
    g = _generator(seed)
    x = torch.arange(cols, device="cuda", dtype=torch.float32)
    out = torch.empty(rows, cols, dtype=torch.float32, device="cuda")
    for r0 in range(0, rows, 512):
        cnt = min(512, rows - r0)
        img = torch.rand(cnt, cols, generator=g, device="cuda").mul_(16.0)
        p = torch.rand(3, cnt, 8, generator=g, device="cuda")
        for b in range(8):
            c, w = p[0, :, b, None] * cols, cols * (0.01 + 0.07 * p[1, :, b, None])
            img += (40.0 + 80.0 * p[2, :, b, None]) * torch.exp(-0.5 * ((x - c) / w) ** 2)
        out[r0:r0 + cnt] = img.clamp_(0, 255).floor_().div_(255.0)
    return out


def _train_inputs(case, seed):
    g = _generator(seed)
    x = torch.rand(case["batch"], 16, device="cuda", generator=g) * 2 - 1
    t = torch.randn(case["batch"], case["out"], device="cuda", generator=g)
    sizes = [16, case["hidden"], case["hidden"], case["out"]]
    parts = [(torch.rand(o * i, device="cuda", generator=g) * 2 - 1) / i ** 0.5 for i, o in zip(sizes, sizes[1:])]
    parts += [(torch.rand(o, device="cuda", generator=g) * 2 - 1) * 0.1 for o in sizes[1:]]
    return sizes, x, t, torch.cat(parts)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        planes = _operator(case, seed)
        s = B.Arnoldi(case["n"], case["m"], case["k"], is_complex=planes[1] is not None, sort=case["sort"],
                      precision=B.PREC_MIXED if case["precision"] == "mixed" else B.PREC_FP64, tolerance=TOL, seed=1)
        s.set_operator(*planes)
        return dict(case, solver=s, planes=planes)
    if kind == "batch":
        return dict(case, mats=_batch(case, seed))
    if kind == "gram_build":
        return dict(case, X=_images(case["rows"], case["cols"], seed))
    if kind == "gram_solve":
        X = _images(case["rows"], case["cols"], seed)
        s = B.Arnoldi(case["rows"], case["m"], case["k"], tolerance=TOL, seed=5)
        s.set_gram_operator(X)
        return dict(case, X=X, solver=s)
    if kind == "dot":
        g = _generator(seed)
        shapes = ((case["rows"], case["inner"]), (case["inner"], case["cols"]))
        ops = [(_randn(g, *sh), _randn(g, *sh) if case["cplx"] else None) for sh in shapes]
        shape = (case["rows"], case["cols"])
        out = [torch.empty(shape, dtype=torch.float64, device="cuda") if p is not None else None for p in ops[0]]
        return dict(case, ops=ops, out=out)
    sizes, x, t, p0 = _train_inputs(case, seed)
    net = W.Net(sizes, seed=seed % 1000 + 1)
    net.set_params(p0.cpu().numpy())
    return dict(case, net=net, x=x, t=t, params=torch.empty_like(p0), grads=torch.empty_like(p0))


def run(state):
    kind = state["kind"]
    if kind == "solve":
        s = state["solver"]
        if state["fresh"]:  # a program with a new operator for every solve
            s.set_operator(*state["planes"])
        ev, res, st = s.solve()
        return {"eigenvalues": np.array(ev), "converged": st == B.OK and max(res) <= TOL}
    if kind == "batch":
        ev, res, st, _, _ = B.solve_batched(state["mats"], state["k"], hdim=state["hdim"], tolerance=TOL)
        return {"eigenvalues": ev, "status": st}
    if kind == "gram_build":
        A, _ = B.gram_build(state["X"])
        return A
    if kind == "gram_solve":
        ev, res, st = state["solver"].solve()
        return {"eigenvalues": np.array(ev), "converged": st == B.OK and max(res) <= TOL}
    if kind == "dot":
        m = [B.mat(*p) for p in (state["out"], *state["ops"])]
        B.check(B.lib().oapb_dot_product(*[C.byref(x) for x in m],
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream)), "oapb_dot_product")
        return state["out"]
    net = state["net"]
    loss = net.backward(state["x"], state["t"])
    net.adam(1e-3)
    for which, dst in ((0, state["params"]), (1, state["grads"])):
        B.check(B.lib().oapb_mlp_copy(net.h, which, C.c_void_p(dst.data_ptr()), None), "oapb_mlp_copy")
    return {"loss": loss, "params": state["params"], "grads": state["grads"]}


def work(case):
    kind = case["kind"]
    if kind == "solve":
        planes = 2 if case.get("cplx") else 1
        n2 = float(case["n"]) ** 2
        # a factorization of m steps applies the operator m times
        return {"bytes": 8.0 * planes * n2, "flops": 2.0 * planes ** 2 * n2 * case["m"]}
    if kind == "batch":
        planes = 2 if case["cplx"] else 1
        n2 = case["count"] * (case["nmin"] ** 2 + case["nmin"] * case["nmax"] + case["nmax"] ** 2) / 3.0
        return {"bytes": 8.0 * planes * n2, "flops": 2.0 * planes ** 2 * n2 * case["hdim"]}
    if kind == "gram_build":
        r, c = float(case["rows"]), float(case["cols"])
        return {"bytes": 4.0 * (r * c + r * r), "flops": r * r * c}  # symmetric: one triangle
    if kind == "gram_solve":
        r, c = float(case["rows"]), float(case["cols"])
        return {"bytes": 4.0 * r * c, "flops": 4.0 * r * c * case["m"]}
    if kind == "dot":
        planes = 2 if case["cplx"] else 1
        m, k, n = float(case["rows"]), float(case["inner"]), float(case["cols"])
        return {"bytes": 8.0 * planes * (m * k + k * n + m * n), "flops": 2.0 * planes ** 2 * m * k * n}
    sizes = [16, case["hidden"], case["hidden"], case["out"]]
    params = float(sum(i * o + o for i, o in zip(sizes, sizes[1:])))
    # weights, gradients and the update's two moments read and written; both outputs written
    return {"bytes": 4.0 * (9 * params + case["batch"] * (sizes[0] + sizes[-1])), "flops": 6.0 * params * case["batch"]}


# ------------------------------------------------------------------- exact --
def _sorted(ev, sort, k):
    ev = np.asarray(ev).astype(complex)
    return ev[np.argsort(-(ev.real if sort == "LR" else np.abs(ev)), kind="stable")][:k]


def _dominant(A, k):
    """The k largest-magnitude eigenvalues of a batch of operators (..., n, n)
    that dominate the rest (ratio below about 0.5): subspace iteration on
    k + 4 vectors, Rayleigh-Ritz at the end."""
    b = min(k + 4, A.shape[-1])
    g = _generator(99)
    X = torch.randn(*A.shape[:-1], b, dtype=torch.float64, device="cuda", generator=g).to(A.dtype)
    eye = torch.eye(b, dtype=A.dtype, device="cuda")

    def orth(Y):
        for _ in range(2):
            L = torch.linalg.cholesky(Y.mH @ Y + 1e-300 * eye)
            Y = torch.linalg.solve_triangular(L.mH, Y, upper=True, left=False)
        return Y

    for _ in range(60):
        X = orth(A @ X)
    ev = np.linalg.eigvals((X.mH @ (A @ X)).cpu().numpy())
    return np.take_along_axis(ev, np.argsort(-np.abs(ev), axis=-1, kind="stable"), -1)[..., :k]


def _exact_batch(case, seed):
    mats = _batch(case, seed)
    if not case["cplx"]:
        return np.stack([_sorted(np.linalg.eigvalsh(re.cpu().numpy()), "LM", case["k"]) for re, _ in mats])
    out = np.zeros((case["count"], case["k"]), dtype=complex)
    order = np.argsort([re.shape[0] for re, _ in mats], kind="stable")
    for c0 in range(0, len(order), 256):  # of like size, padded with zeros to the largest
        idx = order[c0:c0 + 256]
        n = mats[idx[-1]][0].shape[0]
        A = torch.zeros(len(idx), n, n, dtype=torch.complex128, device="cuda")
        for j, i in enumerate(idx):
            re, im = mats[i]
            A[j, :re.shape[0], :re.shape[0]] = torch.complex(re, im)
        out[idx] = _dominant(A, case["k"])
    return out


def _exact_train(case, seed):
    sizes, x, t, p = _train_inputs(case, seed)
    x, t, p = x.double(), t.double(), p.double()
    Ws, bs, at = [], [], 0
    for i, o in zip(sizes, sizes[1:]):
        Ws.append(p[at:at + i * o].view(o, i))
        at += i * o
    for o in sizes[1:]:
        bs.append(p[at:at + o])
        at += o
    h1 = torch.tanh(x @ Ws[0].T + bs[0])
    h2 = torch.tanh(h1 @ Ws[1].T + bs[1])
    d = h2 @ Ws[2].T + bs[2] - t
    n = case["batch"]
    z3 = d / n
    z2 = (z3 @ Ws[2]) * (1 - h2 * h2)
    z1 = (z2 @ Ws[1]) * (1 - h1 * h1)
    grads = torch.cat([(z1.T @ x).reshape(-1), (z2.T @ h1).reshape(-1), (z3.T @ h2).reshape(-1), z1.sum(0), z2.sum(0),
                       z3.sum(0)])
    params = p - 1e-3 * grads / (grads.abs() + 1e-8)  # the first Adam step
    return {"loss": float(0.5 * (d * d).sum() / n), "params": params, "grads": grads}


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        re, im = _operator(case, seed)
        if case["spectrum"] == "planted":
            ev = _dominant(torch.complex(re, im) if im is not None else re, case["k"])
        else:
            ev = torch.linalg.eigvalsh(re).cpu().numpy()
        return {"eigenvalues": _sorted(ev, case["sort"], case["k"]), "converged": None}
    if kind == "batch":
        return {"eigenvalues": _exact_batch(case, seed), "status": None}
    if kind in ("gram_build", "gram_solve"):
        X = _images(case["rows"], case["cols"], seed).double()
        A = X @ X.T
        if kind == "gram_build":
            return A
        return {"eigenvalues": _sorted(torch.linalg.eigvalsh(A).cpu().numpy(), "LM", case["k"]), "converged": None}
    if kind == "dot":
        ops = prepare(case, seed)["ops"]
        a, b = (torch.complex(*p) if p[1] is not None else p[0] for p in ops)
        c = a @ b
        return [c.real.contiguous(), c.imag.contiguous()] if case["cplx"] else [c, None]
    return _exact_train(case, seed)
