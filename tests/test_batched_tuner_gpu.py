"""The batched solver's launch variant by the tuner against every forced one, on
large problems, which leave room for one CTA per SM or share an SM badly."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402


@pytest.mark.parametrize("count,lo,hi,cplx,hdim,k", [(200, 900, 1024, True, 24, 4), (160, 1400, 1600, False, 12, 2)])
def test_tuned_variant_is_among_the_fastest(count, lo, hi, cplx, hdim, k):
    rng = np.random.default_rng(1)
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    mats = []
    for n in rng.integers(lo, hi + 1, count):
        a, b = (torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
        s = 1 / (2 * n) ** 0.5
        a, b = (a * s, b * s) if cplx else ((a + a.T) * (s / 2 ** 0.5), None)
        i = torch.arange(k, device="cuda")
        a[i, i] += 4.0
        mats.append((a, b))

    def best(autotune):
        out = []
        for _ in range(4):
            torch.cuda.synchronize()
            t = time.perf_counter()
            rc = B.solve_batched(mats, k, hdim=hdim, max_restarts=40, autotune=autotune)[4]
            out.append(time.perf_counter() - t)
            assert rc == B.OK
        return min(out[1:])

    tuned = best(True)
    # every variant but the fastest takes 1.7 times its time and more here; half
    # of it covers the noise of a timed sample and of the host
    assert tuned <= 1.5 * min(best(2 + v) for v in range(5))
