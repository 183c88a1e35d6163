"""Symmetric and Hermitian operators in every sort order, the two by imaginary
parts (all zero) among them, and in the smallest Krylov spaces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402
from gpu_util import host, planes, zeros  # noqa: E402

TOL = 1e-10


def operator(n, seed, cplx):
    rng = np.random.default_rng(seed)
    G = rng.normal(size=(n, n)) + (1j * rng.normal(size=(n, n)) if cplx else 0)
    return (G + G.conj().T) / (2 * np.sqrt(n))


def check_pairs(A, ev, res, X):
    assert res.max() <= TOL
    # each value within its residual of an eigenvalue of the Hermitian matrix
    w = np.linalg.eigvalsh(A)
    assert np.abs(ev[:, None] - w).min(axis=1).max() <= 2 * TOL * np.abs(w).max()
    # distinct pairs: orthogonal vectors up to residual / gap
    G = X.conj().T @ X
    assert np.abs(G - np.diag(np.diag(G))).max() <= 1e-5 and np.abs(np.diag(G) - 1).max() <= 1e-6


@pytest.mark.parametrize("sort", ["LM", "LR", "SR", "LI", "SI"])
@pytest.mark.parametrize("n,m,k,cplx,per_step", [(300, 24, 4, False, False), (300, 24, 4, True, False), (200, 13, 3, False, True),
                                                 (400, 33, 6, True, True)])
def test_sorts(sort, n, m, k, cplx, per_step):
    A = operator(n, n + m, cplx)
    s = B.Arnoldi(n, m, k, is_complex=cplx, sort=sort, tolerance=TOL, seed=2, autotune=2 if per_step else True)
    s.set_operator(*planes(A, cplx))
    v = zeros((n, k), cplx)
    ev, res, st = s.solve(vectors=v)
    assert st == B.OK
    check_pairs(A, np.array(ev), np.array(res), host(*v))


@pytest.mark.parametrize("sort", ["LM", "LI", "SI"])
def test_sorts_batched(sort):
    k = 3
    A = [operator(n, n, n % 2 == 1) for n in (40, 81, 120, 201)]
    vecs = [zeros((a.shape[0], k), True) for a in A]
    ev, res, st, _, rc = B.solve_batched([planes(a, np.iscomplexobj(a)) for a in A], k, hdim=20, sort=sort, vectors=vecs)
    assert rc == B.OK
    for i, a in enumerate(A):
        check_pairs(a, ev[i], res[i], host(*vecs[i]))
