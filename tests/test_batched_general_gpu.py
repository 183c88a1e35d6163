"""Batched restarts of non-Hermitian operators that a restarted space must find:
outlying values, every problem converged, within a bound on the restarts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402
from gpu_util import planes  # noqa: E402

TOL = 1e-10


def planted(n, k, seed, cplx):
    """Entries of variance 1 / n (spectral radius about 1) plus 4, 5, ... on k
    diagonal positions: so far apart that a real matrix's wanted values are real
    (a real solve's vectors are)."""
    rng = np.random.default_rng(seed)
    A = rng.normal(size=(n, n)) / np.sqrt(n)
    if cplx:
        A = (A + 1j * rng.normal(size=(n, n)) / np.sqrt(n)) / np.sqrt(2)
    A[np.arange(k), np.arange(k)] += 4.0 + np.arange(k)
    return A


@pytest.mark.parametrize("hdim,k", [(4, 2), (5, 3), (16, 3), (17, 5), (31, 4), (32, 6)])
@pytest.mark.parametrize("cplx", [True, False])
def test_outlying_values(hdim, k, cplx):
    sizes = [hdim + 12, 2 * hdim + 30, 97, 200, 301]
    probs = [planted(n, k, n + hdim, cplx) for n in sizes]
    for variant in (True, 2, 4):
        ev, res, st, stats, rc = B.solve_batched([planes(A, cplx) for A in probs], k, hdim=hdim, max_restarts=300,
                                                 autotune=variant)
        assert rc == B.OK and res.max() <= TOL
        # a restart applies the operator at least once and an application
        # contracts what is unwanted by about 4: 17 for 1e-10, five times that
        assert stats["restarts"] <= 85 * len(sizes)
        for i, A in enumerate(probs):
            ref = np.linalg.eigvals(A)
            ref = ref[np.argsort(-np.abs(ref))][:k]
            # residuals <= 1e-10 of the largest, condition numbers near 1
            d = np.abs(ev[i][:, None] - ref)
            assert max(d.min(axis=0).max(), d.min(axis=1).max()) <= 10 * TOL * np.abs(ref).max()
