"""Handles and host threads that use the same kernels with different dynamic
shared-memory sizes: what one sets does not refuse another's launch."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402

TOL = 1e-10


def operator(n, seed, k):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    A = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    A = (A + A.T) / (2 * n ** 0.5)
    i = torch.arange(k, device="cuda")
    A[i, i] += 4.0 + 0.05 * i.double()
    return A.contiguous()


def dense(m, k, cplx, per_step):
    n = 3 * m + 40
    A = operator(n, m, k)
    s = B.Arnoldi(n, m, k, is_complex=cplx, tolerance=TOL, seed=3, autotune=2 if per_step else True)
    s.set_operator(A, torch.zeros_like(A) if cplx else None)
    return s, A


def gram(m, k):
    g = torch.Generator(device="cuda")
    g.manual_seed(m)
    rows, cols = 3 * m + 12, 640
    U = torch.randn(rows, k, generator=g, device="cuda") * torch.linspace(9.0, 6.0, k, device="cuda")
    X = (U @ torch.randn(k, cols, generator=g, device="cuda") / cols ** 0.5
         + 0.02 * torch.randn(rows, cols, generator=g, device="cuda")).contiguous()
    s = B.Arnoldi(rows, m, k, tolerance=TOL, seed=3)
    s.set_gram_operator(X)
    Xd = X.double()
    return s, Xd @ Xd.T


# the larger handle first, then one of a smaller Krylov space: the basis
# products (m x vectors formed) and the small eigenproblem's workspace, on the
# one-launch cycles and the per-step kernels
@pytest.mark.parametrize("big,small,cplx,per_step", [((128, 60), (96, 32), False, False), ((128, 60), (96, 32), False, True),
                                                     ((64, 8), (20, 4), False, False), ((64, 40), (40, 8), True, True),
                                                     ((100, 50), (64, 46), True, False)])
def test_handle_after_a_smaller_one(big, small, cplx, per_step):
    pairs = [dense(*mk, cplx, per_step) for mk in (big, small)]
    for (s, A), (_, k) in zip(pairs, (big, small)):
        ev, res, st = s.solve()
        assert st == B.OK and max(res) <= TOL
        # eigenvalues of a symmetric operator: residuals <= 1e-10 leave rounding
        ref = torch.linalg.eigvalsh(A).cpu().numpy()
        ref = ref[np.argsort(-np.abs(ref))][:k]
        assert np.abs(np.sort(np.array(ev).real) - np.sort(ref)).max() <= A.shape[0] * 2.3e-16 * 4 * np.abs(ref).max()


def test_gram_handle_after_a_smaller_one():
    pairs = [gram(96, 32), gram(64, 45)]
    for (s, G), k in zip(pairs, (32, 45)):
        ev, res, st = s.solve()
        assert st == B.OK and max(res) <= TOL
        ref = torch.linalg.eigvalsh(G).flip(0)[:k].cpu().numpy()
        assert np.abs(np.array(ev).real - ref).max() <= (G.shape[0] + 640) * 2.3e-16 * 4 * ref[0]


def in_threads(work, count):
    """work(i) on `count` host threads at once; the first exception is raised here."""
    errors = []

    def run(i):
        try:
            work(i)
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(count)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def test_gram_operators_on_host_threads():
    # row counts that share an instance of the kernel with other rows per thread
    rows = (2000, 300, 1100, 2000)
    handles = []
    for i, r in enumerate(rows):
        g = torch.Generator(device="cuda")
        g.manual_seed(i)
        X = torch.randn(r, 640, device="cuda", generator=g)
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        s = B.Arnoldi(r, 24, 4, seed=3, max_restarts=6, stream=stream.cuda_stream)
        s.set_gram_operator(X)
        handles.append((s, stream, s.solve(allow_not_converged=True)))

    def work(i):
        s, _, ref = handles[i]
        for _ in range(60):
            assert s.solve(allow_not_converged=True) == ref  # the same launches: the same bits

    in_threads(work, len(rows))


def test_batched_solves_on_host_threads():
    shapes = [(40, 32, 512, 32), (60, 24, 40, 8), (40, 200, 300, 24), (60, 16, 24, 6)]  # problems, sizes, hdim
    sets = []
    for i, (count, lo, hi, hdim) in enumerate(shapes):
        rng = np.random.default_rng(i)
        sets.append(([(operator(int(n), 100 * i + j, 3), None) for j, n in enumerate(rng.integers(lo, hi + 1, count))], hdim))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in shapes]

    def solve(i):
        mats, hdim = sets[i]
        ev, res, st, _, _ = B.solve_batched(mats, 2, hdim=hdim, max_restarts=50, stream=streams[i].cuda_stream)
        return ev, res, st

    refs = [solve(i) for i in range(len(shapes))]

    def work(i):
        for _ in range(30):
            for a, b in zip(solve(i), refs[i]):
                assert np.array_equal(a, b)

    in_threads(work, len(shapes))


def test_block_passes_on_host_threads():
    # block widths of other stage counts and sizes on the tensor-core passes
    n = 1024
    widths = (4, 32, 12, 24)
    todo = []
    for i, b in enumerate(widths):
        A = operator(n, i, 3)
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        s = B.Arnoldi(n, 24, 4, precision=B.PREC_MIXED, stream=stream.cuda_stream)
        s.set_operator(A)
        X = torch.randn(b, n, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(b))
        ref = X @ A.T
        torch.cuda.synchronize()
        todo.append((s, ref, X, stream, n ** 0.5 * A.abs().max().item() * X.abs().max().item()))

    def work(i):
        s, ref, X, stream, scale = todo[i]
        for _ in range(60):
            # FP64-class slices: 2^-42 of each row's scale and FP32-class planes:
            # 2^-15 per product, the sums of n growing like sqrt(n)
            for precision, tol in ((B.PREC_FP64, 2.0 ** -42), (B.PREC_MIXED, 2.0 ** -15)):
                with torch.cuda.stream(stream):
                    W, _ = s.apply_block(X, precision=precision)
                    err = (W - ref).abs().max().item()
                assert err <= tol * scale

    in_threads(work, len(widths))


def test_qr_on_host_threads():
    sizes = (60, 70, 56, 65)
    mats = [operator(n, n, 2) for n in sizes]
    streams = [torch.cuda.Stream() for _ in sizes]
    torch.cuda.synchronize()

    def work(i):
        n, A = sizes[i], mats[i]
        with torch.cuda.stream(streams[i]):
            Q, R = torch.empty_like(A), torch.empty_like(A)
            for _ in range(200):
                a, q, r = B.mat(A), B.mat(Q), B.mat(R)
                B.check(B.lib().oapb_qr_givens(q, r, a, streams[i].cuda_stream), "oapb_qr_givens")
            assert (Q @ R - A).abs().max().item() <= 8 * n * 2.3e-16 * A.abs().max().item()

    in_threads(work, len(sizes))
