"""The single-vector operator pass runs its tuned variant whenever a solve takes
it, also on handles whose solves otherwise run in restart cycles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402


def test_tuned_variant_after_the_operator_was_set():
    n = 6000
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    A = [torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g) / n ** 0.5 for _ in range(2)]
    kw = dict(is_complex=True, max_restarts=1, seed=3)
    want = B.Arnoldi(n, 20, 3, profile=True, **kw)  # the per-step kernels from the start
    want.set_operator(*A)
    want.solve(allow_not_converged=True)
    variant = want.stats()["matvec_variant"]
    assert variant != 0  # the default pass is a quarter slower at this size

    late = B.Arnoldi(n, 20, 3, **kw)
    late.set_operator(*A)
    ev, _, _ = late.solve(allow_not_converged=True)  # in cycles
    late.set_profile(True)
    late.solve(allow_not_converged=True)
    st = late.stats()
    assert st["matvec_variant"] == variant and st["matvec_timed"] > 0

    warm = B.Arnoldi(n, 20, 3, init=B.INIT_USER, **kw)
    warm.set_operator(*A)
    v = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    warm.set_start_vector(v, v)
    warm.set_start_shifts([0.5, -0.5])
    warm.solve(allow_not_converged=True)
    assert warm.stats()["matvec_variant"] == variant


def test_tuning_leaves_a_restored_factorization(tmp_path):
    # profiling switched on between load and resume: the pass is tuned at the
    # resume, the restored vectors stay as they were
    n, m, k = 900, 20, 4
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    A = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    A = (A + A.T) / (2 * n ** 0.5)
    part = B.Arnoldi(n, m, k, sort="LR", max_restarts=3, seed=5)
    part.set_operator(A)
    _, _, st = part.solve(allow_not_converged=True)
    assert st == B.NOT_CONVERGED
    part.save(tmp_path / "ck.bin")
    back = B.Arnoldi(n, m, k, sort="LR", seed=9)
    back.set_operator(A)
    back.load(tmp_path / "ck.bin")
    back.set_profile(True)
    ev, res, st = back.resume()
    assert st == B.OK and max(res) <= 1e-10
    ref = torch.linalg.eigvalsh(A).flip(0)[:k].cpu().numpy()
    assert np.abs(np.array(ev).real - ref).max() <= 4 * n * 2.3e-16 * np.abs(ref).max()
    full = B.Arnoldi(n, m, k, sort="LR", seed=5)
    full.set_operator(A)
    full.solve()
    # it went on from the saved space: as many restarts in all, within two
    assert abs(back.stats()["restarts"] - full.stats()["restarts"]) <= 2
