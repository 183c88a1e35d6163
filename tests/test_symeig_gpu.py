"""The symmetric path of the restart loop (Jacobi eigensolve, Ritz vectors kept
through a restart) on real symmetric and Hermitian operators."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402
from gpu_util import planes  # noqa: E402

TOL = 1e-10


def edge(n, seed, cplx=False):
    rng = np.random.default_rng(seed)
    G = rng.normal(size=(n, n)) + (1j * rng.normal(size=(n, n)) if cplx else 0)
    return (G + G.conj().T) / (2 * np.sqrt(n))


# odd and even m (the round robin's padding index), the thread counts' limits,
# k next to m, the one-launch cycles and the per-step kernels
@pytest.mark.parametrize("per_step", [False, True])
@pytest.mark.parametrize("n,m,k,cplx", [(40, 3, 1, False), (60, 16, 3, False), (200, 17, 16, False),
                                        (150, 24, 4, True), (300, 25, 6, False), (400, 40, 5, False),
                                        (500, 41, 8, True), (700, 97, 20, False), (900, 112, 10, False)])
def test_symmetric_restarts_against_lapack(n, m, k, cplx, per_step):
    # eigenvalues of a symmetric operator converge quadratically in the
    # residual (<= 1e-10): what is left is rounding, n eps |A| at most
    A = edge(n, n + m, cplx)
    s = B.Arnoldi(n, m, k, is_complex=cplx, sort="LR", tolerance=TOL, seed=2, max_restarts=2000,
                  autotune=2 if per_step else True)
    s.set_operator(*planes(A, cplx))
    ev, res, st = s.solve()
    assert st == B.OK and max(res) <= TOL and s.stats()["symtri"] > 0
    ref = np.linalg.eigvalsh(A)[::-1][:k]
    assert np.abs(np.array(ev).real - ref).max() <= n * 2.3e-16 * np.abs(ref).max() * 4
    assert np.abs(np.array(ev).imag).max() <= 1e-13


def test_batched_symmetric_restarts():
    sizes = [(20, 1), (33, 2), (70, 3), (129, 4)]
    A = [edge(n, s) for n, s in sizes]
    mats = [planes(a, False) for a in A]
    ev, res, st, stats, rc = B.solve_batched(mats, 3, hdim=13, sort="LR", max_restarts=2000)
    assert rc == B.OK and res.max() <= TOL
    for i, a in enumerate(A):
        ref = np.linalg.eigvalsh(a)[::-1][:3]
        assert np.abs(ev[i].real - ref).max() <= a.shape[0] * 2.3e-16 * np.abs(ref).max() * 4


def test_kept_vectors_survive_a_checkpoint(tmp_path):
    # the saved H holds the kept vectors' row below its diagonal block; a
    # resumed solve continues from it, also in a handle whose residual goal
    # makes the symmetry check fail (the loop then starts again from the
    # wanted Ritz vectors and takes the general path)
    n, m, k = 400, 16, 4
    A = edge(n, 7)
    a = planes(A, False)
    ref = np.linalg.eigvalsh(A)[::-1][:k]
    part = B.Arnoldi(n, m, k, sort="LR", max_restarts=3, seed=5)
    part.set_operator(*a)
    _, _, st = part.solve(allow_not_converged=True)
    assert st == B.NOT_CONVERGED
    p = tmp_path / "ck.bin"
    part.save(p)
    full = B.Arnoldi(n, m, k, sort="LR", seed=5)
    full.set_operator(*a)
    ev, _, _ = full.solve()
    back = B.Arnoldi(n, m, k, sort="LR", seed=9)
    back.set_operator(*a)
    back.load(p)
    ev2, res2, st2 = back.resume()
    assert st2 == B.OK and back.stats()["restarts"] == full.stats()["restarts"]
    assert np.allclose(np.array(ev2).real, np.array(ev).real, rtol=1e-12, atol=0)
    tight = B.Arnoldi(n, m, k, sort="LR", seed=9, tolerance=1e-17, max_restarts=400)
    tight.set_operator(*a)
    tight.load(p)
    ev3, res3, _ = tight.resume(allow_not_converged=True)
    assert tight.stats()["symtri"] == 0
    assert np.abs(np.array(ev3).real - ref).max() <= 1e-9
