"""The plain restart loop's one-launch cycles (dense operators) against the
per-step kernels on the same operator and start vector."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402
from gpu_util import planes, planted_complex  # noqa: E402

TOL = 1e-10


def operator(n, k, cplx):
    if cplx:
        return planted_complex(n, seed=n, nplant=k)
    rng = np.random.default_rng(n)
    A = rng.normal(size=(n, n))
    A = (A + A.T) / (2 * np.sqrt(n))
    A[np.arange(k), np.arange(k)] += 4.0
    return A


# one to 148 CTAs, a last CTA with fewer rows, odd n (8-byte operator loads),
# operator rows kept in shared memory or streamed, a basis wider than a warp,
# the largest m of the cycle and one above it
@pytest.mark.parametrize("n,m,k,cplx", [(2, 2, 1, False), (9, 6, 2, False), (63, 40, 4, True), (64, 33, 3, False),
                                        (1183, 48, 5, False), (1185, 36, 6, True), (1343, 45, 5, True),
                                        (2050, 64, 8, False), (2100, 128, 6, False), (1500, 130, 6, False),
                                        (3001, 34, 9, True)])
def test_cycle_matches_per_step_kernels(n, m, k, cplx):
    # both loops end at relative residuals <= 1e-10 and the operators'
    # outlying eigenvalues have condition numbers near 1, so the two sets of
    # eigenvalues agree within 4e-10 of the largest
    a = planes(operator(n, k, cplx), cplx)
    one = B.Arnoldi(n, m, k, is_complex=cplx, tolerance=TOL, seed=3)
    one.set_operator(*a)
    ev, res, st = one.solve()
    assert st == B.OK and max(res) <= TOL
    steps = B.Arnoldi(n, m, k, is_complex=cplx, tolerance=TOL, seed=3, autotune=2)  # a forced pass variant: per-step
    steps.set_operator(*a)
    ref, res2, st2 = steps.solve()
    assert st2 == B.OK
    assert np.abs(np.array(ev) - np.array(ref)).max() <= 4 * TOL * np.abs(ref).max()
    # the same launch on the same input gives the same bits (the sums over
    # CTAs run in a fixed order)
    for _ in range(20):
        again, res3, _ = one.solve()
        assert again == ev and res3 == res


def test_cycle_breakdown_and_zero_start():
    # an operator of rank 3: the Krylov space becomes invariant before m; the
    # cycle continues from random vectors as the per-step kernels do
    rng = np.random.default_rng(5)
    Q, _ = np.linalg.qr(rng.normal(size=(200, 3)))
    A = (Q * np.array([3.0, 2.0, 1.0])) @ Q.T
    s = B.Arnoldi(200, 12, 3, tolerance=TOL, seed=2)
    s.set_operator(*planes(A, False))
    ev, res, st = s.solve()
    assert st == B.OK
    assert np.allclose(np.array(ev).real, [3.0, 2.0, 1.0], rtol=1e-10)
    z = B.Arnoldi(200, 12, 3, init=B.INIT_USER)
    z.set_operator(*planes(A, False))
    z.set_start_vector(torch.zeros(200, dtype=torch.float64, device="cuda"))
    with pytest.raises(B.OapbError) as e:
        z.solve()
    assert e.value.status == B.ERR_BREAKDOWN
