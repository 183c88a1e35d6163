"""The kept Ritz vectors of the symmetric path stay orthogonal over many restarts
and the values as accurate as the operator allows, on operators whose spectrum
is known exactly (H D H of a Hadamard matrix H, D of few bits, so that every
entry of the operator is exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402
from gpu_util import host, planes, zeros  # noqa: E402

TOL = 1e-10
EPS = 2.3e-16


def even_spectrum(n, cplx=False):
    """Eigenvalues 1, 1 - 1 / n, ..., 1 / n."""
    H = np.ones((1, 1))
    while H.shape[0] < n:
        H = np.block([[H, H], [H, -H]])
    d = 1 - np.arange(n) / n
    A = (H * d) @ H.T / n
    if cplx:  # phases 1, i, -1, -i: Hermitian, the same values
        p = 1j ** np.arange(n)
        A = p[:, None] * A * p.conj()
    return A, d


def check(A, d, k, ev, res, X):
    n = A.shape[0]
    # rounding of the products, growing like sqrt(n); the residuals' share of
    # an eigenvalue is their square over the spacing
    assert np.abs(np.sort(ev.real)[::-1] - d[:k]).max() <= 8 * np.sqrt(n) * EPS
    # vectors within residual / spacing of the eigenvectors are that far from
    # orthogonal; their lengths come from the basis, whose products are accurate
    # while it is orthogonal to sqrt(eps)
    spacing = 1.0 / n
    G = X.conj().T @ X
    assert np.abs(G - np.eye(k)).max() <= 1.5e-8 + 2 * res.max() / spacing


@pytest.mark.parametrize("per_step", [False, True])
@pytest.mark.parametrize("n,m,k,cplx", [(1024, 24, 6, False), (1024, 33, 8, False), (256, 40, 12, False),
                                        (1024, 24, 6, True), (512, 12, 4, False)])
def test_even_spectrum(n, m, k, cplx, per_step):
    A, d = even_spectrum(n, cplx)
    for seed in (2, 3):
        s = B.Arnoldi(n, m, k, is_complex=cplx, tolerance=TOL, seed=seed, max_restarts=2000,
                      autotune=2 if per_step else True)
        s.set_operator(*planes(A, cplx))
        v = zeros((n, k), cplx)
        ev, res, st = s.solve(vectors=v)
        assert st == B.OK
        check(A, d, k, np.array(ev), np.array(res), host(*v))


def test_even_spectrum_batched():
    k = 6
    probs = [even_spectrum(n, cplx) for n, cplx in ((1024, False), (512, True), (256, False), (1024, True))]
    vecs = [zeros((A.shape[0], k), True) for A, _ in probs]
    ev, res, st, _, rc = B.solve_batched([planes(A, np.iscomplexobj(A)) for A, _ in probs], k, hdim=24,
                                         max_restarts=2000, vectors=vecs)
    assert rc == B.OK
    for i, (A, d) in enumerate(probs):
        check(A, d, k, ev[i], res[i], host(*vecs[i]))
