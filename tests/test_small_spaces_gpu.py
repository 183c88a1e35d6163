"""Restarts in Krylov spaces of a few vectors more than wanted: the vectors a
restart keeps leave it enough steps to converge within an ordinary budget."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402
from gpu_util import planes  # noqa: E402

TOL = 1e-10


# the restarts of all operators together, a third above what restarts that keep
# the wanted vectors alone need (4017, 4850 and 1892; with a guard vector 7266,
# 8853 and 1982)
@pytest.mark.parametrize("m,k,bound", [(3, 1, 5400), (5, 3, 6500), (4, 1, 2550)])
@pytest.mark.parametrize("batched", [False, True])
def test_symmetric(m, k, bound, batched):
    A = []
    for i in range(24):
        n = 80 + 3 * i
        G = np.random.default_rng(i).normal(size=(n, n))
        A.append((G + G.T) / (2 * n ** 0.5))
    if batched:
        ev, res, st, stats, rc = B.solve_batched([planes(a, False) for a in A], k, hdim=m, sort="LR", max_restarts=1500)
        assert rc == B.OK and res.max() <= TOL
        total = stats["restarts"]
    else:
        total = 0
        for a in A:
            s = B.Arnoldi(a.shape[0], m, k, sort="LR", tolerance=TOL, seed=2, max_restarts=1500)
            s.set_operator(*planes(a, False))
            ev, res, st = s.solve()
            assert st == B.OK and max(res) <= TOL
            total += s.stats()["restarts"]
    assert total <= bound


def normal_matrix(n, seed):
    rng = np.random.default_rng(seed)
    Q, _ = np.linalg.qr(rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))
    return (Q * (np.exp(-3.0 * np.arange(n) / n) * np.exp(2j * np.pi * rng.random(n)))) @ Q.conj().T


def test_batched_general_small_spaces():
    # five steps per restart: the batch needs about the restarts of the plain
    # loop on the same operators (other start vectors; 40 of them even that out)
    m, k = 11, 6
    A = [normal_matrix(100 + i, i) for i in range(40)]
    _, res, st, stats, rc = B.solve_batched([planes(a, True) for a in A], k, hdim=m, max_restarts=1000)
    assert rc == B.OK and res.max() <= TOL
    plain = 0
    for a in A:
        s = B.Arnoldi(a.shape[0], m, k, is_complex=True, tolerance=TOL, seed=1, max_restarts=1000)
        s.set_operator(*planes(a, True))
        s.solve()
        plain += s.stats()["restarts"]
    assert stats["restarts"] <= 1.4 * plain
