"""Symmetric restarts at the largest Krylov dimensions of the whole-CTA eigensolve
(its shared memory ends at m = 118) and of the one-launch cycles (128)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402
from gpu_util import planes  # noqa: E402


@pytest.mark.parametrize("per_step", [False, True])
@pytest.mark.parametrize("m,cplx", [(117, False), (118, False), (118, True), (119, False), (128, False), (129, True)])
def test_symmetric_restarts(m, cplx, per_step):
    n, k = 1200, 40
    rng = np.random.default_rng(m)
    G = rng.normal(size=(n, n)) + (1j * rng.normal(size=(n, n)) if cplx else 0)
    A = (G + G.conj().T) / (2 * np.sqrt(n))
    s = B.Arnoldi(n, m, k, is_complex=cplx, sort="LR", tolerance=1e-10, seed=2, max_restarts=500,
                  autotune=2 if per_step else True)
    s.set_operator(*planes(A, cplx))
    ev, res, st = s.solve()
    assert st == B.OK and max(res) <= 1e-10
    stats = s.stats()
    assert stats["restarts"] > 0 and stats["symtri"] == stats["restarts"] + 1
    ref = np.linalg.eigvalsh(A)[::-1][:k]
    # quadratic in the residual over the spacing: rounding is left
    assert np.abs(np.array(ev).real - ref).max() <= n * 2.3e-16 * np.abs(ref).max() * 4
