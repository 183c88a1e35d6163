"""The network's layer products at the edges of their tiles, chunks and K
splits, against the oracle's forward and gradients."""
import numpy as np
import pytest

from oracle import mlp as M

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oap_b200 import warmstart as W  # noqa: E402


# rows of odd length (padded BF16 rows), one sample, tiles filled and one
# beyond, K chunks split over clusters, the warm-start network's shape; a
# smaller batch after a larger one on the same handle
@pytest.mark.parametrize("sizes,batches", [([1, 1], [1]), ([5, 33, 129, 70], [1, 65, 300, 7]), ([16, 64, 64, 65], [64, 63]),
                                           ([31, 257, 40], [33]), ([16, 256, 256, 2056], [256, 100])])
@pytest.mark.parametrize("acts", [None, "sin"])
def test_layers_match_oracle(sizes, batches, acts):
    acts = None if acts is None else [M.SIN] * (len(sizes) - 1)
    net = W.Net(sizes, seed=3, acts=acts)
    rng = np.random.default_rng(sum(sizes))
    p = net.params()
    p[-sum(sizes[1:]):] = rng.uniform(-0.1, 0.1, sum(sizes[1:]))
    net.set_params(p)
    for b in batches:
        x = rng.uniform(-1, 1, size=(b, sizes[0])).astype(np.float32)
        t = rng.normal(size=(b, sizes[-1])).astype(np.float32)
        xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
        # both sides round weights and activations to BF16 and sum in FP32 or
        # better: what differs is a value that rounds to the other neighbour
        y = net.forward(xd).cpu().numpy()
        hf, _ = M.forward(p, sizes, x, acts)
        assert np.abs(y - hf[-1]).max() <= 1e-3 * max(1.0, np.abs(hf[-1]).max())
        loss = net.backward(xd, td)
        lo, go = M.loss_and_grads(p, sizes, x, t, acts)
        assert abs(loss - lo) <= 1e-4 * lo
        g = net.grads()
        assert np.linalg.norm(g - go) <= 1e-3 * np.linalg.norm(go)
    net.adam(1e-3)
    q = net.params()
    assert np.abs(q - p).max() <= 1.001e-3  # the first step moves a weight by at most lr
    # the BF16 copies follow the masters
    assert np.abs(net.forward(xd).cpu().numpy() - M.forward(q, sizes, x, acts)[0][-1]).max() <= 1e-3 * max(
        1.0, np.abs(y).max())
