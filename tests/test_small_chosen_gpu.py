"""The chosen form of small dense operators runs in restart cycles whatever launch
variant of the operator pass is asked for, and while profiling."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402
from gpu_util import planes, planted_complex, planted_symmetric  # noqa: E402


@pytest.mark.parametrize("cplx", [False, True])
def test_forced_variants_and_profiling(cplx):
    n, m, k = 200, 24, 4
    A = planted_complex(n, 3, k) if cplx else planted_symmetric(n, 3)[0]

    def solve(**kw):
        s = B.Arnoldi(n, m, k, is_complex=cplx, precision=B.PREC_MIXED, tolerance=1e-10, seed=5, **kw)
        s.set_operator(*planes(A, cplx))
        out = s.solve()
        assert out[2] == B.OK and s.stats()["onchip"] == 1
        return out

    ref = solve()
    for autotune in (False, 2, 5, 7):
        assert solve(autotune=autotune) == ref
    assert solve(profile=True) == ref
    # the plain form keeps its per-step kernels for both
    s = B.Arnoldi(n, m, k, is_complex=cplx, tolerance=1e-10, seed=5, profile=True)
    s.set_operator(*planes(A, cplx))
    s.solve()
    st = s.stats()
    assert st["onchip"] == 0 and st["matvec_timed"] == st["matvecs"]
