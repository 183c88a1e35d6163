"""The mixed form's refinement on real non-symmetric operators whose wanted set
holds complex conjugate pairs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402


@pytest.mark.parametrize("n,k,pairs", [(8192, 4, 1), (8193, 6, 2), (8192, 8, 3)])
def test_conjugate_pairs(n, k, pairs):
    g = torch.Generator(device="cuda")
    g.manual_seed(n + k)
    A = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g) / n ** 0.5
    mod = 9.0 - 0.6 * np.arange(k)
    for p in range(pairs):  # planted 2 x 2 rotations, then real values of either sign
        c, s = mod[p] * np.cos(0.3 + p), mod[p] * np.sin(0.3 + p)
        i = 2 * p
        A[i, i] += c
        A[i + 1, i + 1] += c
        A[i, i + 1] += s
        A[i + 1, i] -= s
    for p in range(k - 2 * pairs):
        A[2 * pairs + p, 2 * pairs + p] += mod[pairs + p] * (1 if p % 2 == 0 else -1)
    # the same operator as a complex one by the plain restart loop, whose
    # residuals hold for complex vectors
    c = B.Arnoldi(n, 36, k, is_complex=True, tolerance=1e-12, seed=3)
    c.set_operator(A, torch.zeros_like(A))
    ref = np.array(c.solve()[0])
    del c
    s = B.Arnoldi(n, 32, k, precision=B.PREC_MIXED, tolerance=1e-10, seed=2)
    s.set_operator(A)
    ev, res, st = s.solve()
    assert st == B.OK and max(res) <= 1e-10
    assert s.trace()[-1][0] == 3 and s.stats()["fallbacks"] == 0  # the refinement delivered
    ev = np.array(ev)
    assert (np.abs(ev.imag) > 1).sum() == 2 * pairs
    # residuals of 1e-10 and 1e-12 of the largest value, eigenvalue condition
    # numbers near 1 (planted far outside the bulk): within 4e-10 of it
    d = np.abs(ev[:, None] - ref)
    tol = 4e-10 * np.abs(ref).max()
    assert d.min(axis=1).max() <= tol and d.min(axis=0).max() <= tol
