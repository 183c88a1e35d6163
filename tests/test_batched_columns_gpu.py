"""The batched solver's column groups: residual checks of up to three pairs per
pass over the operator, and V Q and the Ritz vectors six columns at a time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402
from gpu_util import host, planes, zeros  # noqa: E402


@pytest.mark.parametrize("max_restarts", [1, 300])
@pytest.mark.parametrize("wanted", [1, 2, 3, 4, 6, 7, 13])
@pytest.mark.parametrize("kind", ["complex", "real", "symmetric"])
def test_reported_residuals_are_those_of_the_pairs(kind, wanted, max_restarts):
    rng = np.random.default_rng(11)
    As = []
    for n in (17, 24, 33, 127, 201):
        A = rng.normal(size=(n, n)) / np.sqrt(16 * n)  # the planted values stay real and apart
        if kind == "complex":
            A = A + 1j * rng.normal(size=(n, n)) / np.sqrt(16 * n)
        elif kind == "symmetric":
            A = A + A.T
        pos = rng.choice(n, 14, replace=False)
        A[pos, pos] += np.linspace(4.0, 8.0, 14)
        As.append(A)
    vecs = [zeros((A.shape[0], wanted), True) for A in As]
    ev, res, st, stats, rc = B.solve_batched(
        [planes(A) for A in As], wanted, hdim=24, max_restarts=max_restarts, vectors=vecs)
    if max_restarts == 300:
        assert rc == B.OK and (st == B.OK).all()
    for i, A in enumerate(As):
        X = host(*vecs[i])
        n = A.shape[0]
        assert np.isfinite(X).all() and np.isfinite(ev[i]).all()
        scale = np.abs(ev[i]).max()
        got = np.linalg.norm(A @ X - X * ev[i], axis=0) / np.linalg.norm(X, axis=0) / scale
        # two summations of n products of size |A||x|, each within n eps
        bound = 2 * n * np.finfo(float).eps * np.linalg.norm(np.abs(A), 2) / scale
        assert np.abs(got - res[i]).max() <= bound, (n, got, res[i])
        if max_restarts == 300:
            w = np.linalg.eigvals(A)
            w = np.sort(np.abs(w))[::-1][:wanted]
            assert np.abs(np.sort(np.abs(ev[i]))[::-1] - w).max() <= 1e-8 * w[0]
