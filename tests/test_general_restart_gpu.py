"""Restarts of non-Hermitian operators (Schur form and exact shifts of a general
Hessenberg matrix) over the Krylov dimensions where the rotation chain's columns
per lane, the rows per warp and the workspace's place change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402
from gpu_util import host, planes, zeros  # noqa: E402

TOL = 1e-10


def normal_matrix(n, seed, cplx):
    """A normal matrix with moduli exp(-3 j / n), phases at random (real: plane
    rotations, so conjugate pairs, and one positive value on top)."""
    rng = np.random.default_rng(seed)
    mod = np.exp(-3.0 * np.arange(n) / n)
    if cplx:
        Q, _ = np.linalg.qr(rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))
        lam = mod * np.exp(2j * np.pi * rng.random(n))
        return (Q * lam) @ Q.conj().T, lam
    Q, _ = np.linalg.qr(rng.normal(size=(n, n)))
    D = np.zeros((n, n))
    lam = []
    j = 0
    while j < n:
        if j < 4 or j + 1 == n:
            D[j, j] = mod[j] * (1 if j % 2 == 0 else -1)
            lam.append(D[j, j])
            j += 1
        else:
            t = np.pi * rng.random()
            c, s = mod[j] * np.cos(t), mod[j] * np.sin(t)
            D[j:j + 2, j:j + 2] = [[c, -s], [s, c]]
            lam += [c + 1j * s, c - 1j * s]
            j += 2
    return Q @ D @ Q.T, np.array(lam)


# 128 and 129: four columns per lane and eight; from about 75 the workspace is
# in global memory
@pytest.mark.parametrize("m", [5, 8, 31, 32, 33, 48, 64, 65, 97, 128, 129, 200, 256])
@pytest.mark.parametrize("cplx", [True, False])
def test_general_restarts(m, cplx):
    n, k = 2 * m + 30, 3
    A, lam = normal_matrix(n, m, cplx)
    s = B.Arnoldi(n, m, k, is_complex=cplx, tolerance=TOL, seed=7, max_restarts=2000)
    s.set_operator(*planes(A, cplx))
    ev, res, st = s.solve()
    assert st == B.OK and max(res) <= TOL
    # a normal matrix: each value lies within its residual norm of an eigenvalue
    # (which of them a restarted space of a few vectors finds is not settled)
    assert np.abs(np.array(ev)[:, None] - lam).min(axis=1).max() <= 2 * TOL * np.abs(lam).max()


@pytest.mark.parametrize("hdim", [4, 5, 17, 31, 32])
@pytest.mark.parametrize("cplx", [True, False])
def test_general_restarts_batched(hdim, cplx):
    k = 3
    probs = [normal_matrix(n, n + hdim, cplx) for n in (hdim, hdim + 1, 2 * hdim + 7, 90)]
    vecs = [zeros((A.shape[0], k), True) for A, _ in probs]
    ev, res, st, _, rc = B.solve_batched([planes(A, cplx) for A, _ in probs], k, hdim=hdim, max_restarts=3000,
                                         vectors=vecs)
    assert rc in (B.OK, B.NOT_CONVERGED)
    for i, (A, lam) in enumerate(probs):
        if st[i] == B.OK:
            assert res[i].max() <= TOL
        X = host(*vecs[i])
        r = np.linalg.norm(A @ X - X * ev[i], axis=0) / np.linalg.norm(X, axis=0)
        assert np.abs(r - res[i] * np.abs(ev[i]).max()).max() <= 4 * A.shape[0] * np.finfo(float).eps * np.abs(lam).max()
        near = np.abs(ev[i][:, None] - lam).min(axis=1)
        assert (near <= r + TOL * np.abs(lam).max()).all()
