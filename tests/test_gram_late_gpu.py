"""The implicit Gram operator's exchange when one CTA of the cluster is late: its
peers' bounded waits run out, nobody leaves while sums can still arrive, and the
context stays usable.  Nothing here faults, traps or hangs the device."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402


# the first panel, one in the middle, the last (after it the late CTA has all sums
# and leaves by itself)
@pytest.mark.parametrize("late", [0, 7, 14, 15])
def test_late_cta(late):
    for _ in range(3):
        assert B.selftest_gram_wait(1000, late) == (B.ERR_TIMEOUT, 1)
        assert B.selftest_gram_wait(1000, -1) == (B.OK, 0)
    X = torch.randn(700, 1000, device="cuda")
    s = B.Arnoldi(700, 40, 3, tolerance=1e-10, seed=3)
    s.set_gram_operator(X)
    _, res, st = s.solve()
    assert st == B.OK and max(res) <= 1e-10


def test_arguments():
    for limit, late in ((0, 0), (200000, 0), (1000, 16), (1000, -2)):
        assert B.selftest_gram_wait(limit, late)[0] == B.ERR_ARG
