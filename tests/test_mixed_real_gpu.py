"""The mixed form's FP64-anchored refinement on real operators."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402

TOL = 1e-10


# one wanted vector, a count that fills no group of 8, the most with its four
# guard vectors; odd n; a non-symmetric operator with real outlying values
@pytest.mark.parametrize("n,k,sym", [(8192, 1, True), (8193, 5, True), (8200, 16, True), (8192, 28, True),
                                     (8192, 6, False)])
def test_real_operator_refinement(n, k, sym):
    g = torch.Generator(device="cuda")
    g.manual_seed(n + k)
    A = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    A = (A + A.T) / (2 * n ** 0.5) if sym else A / n ** 0.5
    for i in range(k):  # well apart, so that they stay real
        A[i, i] += 4.0 + 0.3 * i
    s = B.Arnoldi(n, max(k + 8, 32), k, precision=B.PREC_MIXED, tolerance=TOL, seed=2)
    s.set_operator(A)
    X = torch.zeros(n, k, dtype=torch.float64, device="cuda")
    ev, res, st = s.solve(vectors=(X, None))
    assert st == B.OK and max(res) <= TOL
    tr = s.trace()
    assert tr[-1][0] == 3 and s.stats()["fallbacks"] == 0  # the refinement delivered
    ev = np.array(ev)
    assert np.abs(ev.imag).max() <= 1e-9
    # residuals recomputed outside the library
    lam = torch.from_numpy(ev.real.copy()).cuda()
    R = A @ X - X * lam
    r = (R.norm(dim=0) / (X.norm(dim=0) * lam.abs().max())).max().item()
    assert r <= TOL * 1.01, r
