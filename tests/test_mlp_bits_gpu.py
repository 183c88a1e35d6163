"""The network's layer products sum in k order in FP32: with linear layers every
output and gradient has the bits of that sum over the BF16 operands."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oap_b200 import warmstart as W  # noqa: E402
from oracle import mlp as M  # noqa: E402


def bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).bfloat16().float().numpy()


def product(A, B):
    """sum_k A[m, k] B[n, k] of BF16 values, in order of k: their products are
    exact in FP32, so an FP32 fused multiply-add is an FP32 addition of them."""
    acc = np.zeros((A.shape[0], B.shape[0]), np.float32)
    for k in range(A.shape[1]):
        acc += A[:, k, None] * B[None, :, k]
    return acc


def column_sums(Z):
    acc = np.zeros(Z.shape[1], np.float32)
    for row in Z:
        acc += row
    return acc


# sizes off and on the tiles of 16 and 32 and the chunks of 32, short and tall grids
@pytest.mark.parametrize("sizes,batch", [([1, 1], 1), ([5, 33, 70], 37), ([32, 64, 96], 64), ([31, 65, 129, 40], 100),
                                         ([16, 256, 2056], 96)])
def test_bits(sizes, batch):
    net = W.Net(sizes, seed=4, acts=[M.LINEAR] * (len(sizes) - 1))
    rng = np.random.default_rng(sum(sizes))
    p = net.params()
    p[-sum(sizes[1:]):] = rng.uniform(-0.1, 0.1, sum(sizes[1:]))
    net.set_params(p)
    x = rng.uniform(-1, 1, size=(batch, sizes[0])).astype(np.float32)
    t = rng.normal(size=(batch, sizes[-1])).astype(np.float32)

    Ws, bs, at = [], [], 0
    for i, o in zip(sizes, sizes[1:]):
        Ws.append(bf16(p[at:at + i * o].reshape(o, i)))
        at += i * o
    for o in sizes[1:]:
        bs.append(p[at:at + o])
        at += o
    hs = [bf16(x)]
    for Wl, bl in zip(Ws, bs):
        y = product(hs[-1], Wl) + bl
        hs.append(bf16(y))
    dZ = (y - t) / np.float32(batch)
    dWs, dbs = [], []
    for l in range(len(Ws) - 1, -1, -1):
        Zb = bf16(dZ)
        dWs.insert(0, product(Zb.T, hs[l].T).ravel())
        dbs.insert(0, column_sums(dZ))
        dZ = product(Zb, Ws[l].T)

    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    assert np.array_equal(net.forward(xd).cpu().numpy(), y)
    net.backward(xd, td)
    assert np.array_equal(net.grads(), np.concatenate(dWs + dbs))
