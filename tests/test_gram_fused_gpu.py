"""The implicit Gram operator's one-pass application at the edges of its row
and panel splits, and the two-pass path beyond a cluster's rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402


# panels of 64, 32 and 16 columns, one to eight CTAs per cluster, a last CTA
# and a last panel partly empty, rows that are not 16-byte aligned, fewer
# panels than clusters, the two-pass path above 8192 rows
@pytest.mark.parametrize("rows,cols", [(30, 7), (256, 640), (257, 1001), (512, 1000), (513, 333), (1024, 2048),
                                       (1025, 999), (2500, 3001), (4096, 1024), (7000, 250), (8192, 126), (8193, 128)])
@pytest.mark.parametrize("host", [False, True])
def test_gram_eigenvalues(rows, cols, host):
    # eigenvalues of the exact Gram of the FP32 values: the products are exact
    # in FP64 up to their sums' rounding, so what is left is (rows + cols) eps
    # of the largest
    g = torch.Generator(device="cuda")
    g.manual_seed(rows + cols)
    k = 4
    U = torch.randn(rows, k + 2, generator=g, device="cuda", dtype=torch.float64)
    V = torch.randn(k + 2, cols, generator=g, device="cuda", dtype=torch.float64)
    scale = torch.tensor([10.0, 8.0, 6.5, 5.0, 2.0, 1.0], device="cuda", dtype=torch.float64)
    X = ((U * scale) @ V / cols ** 0.5 + 0.02 * torch.randn(rows, cols, generator=g, device="cuda",
                                                             dtype=torch.float64)).float().contiguous()
    Xd = X.double()
    ref = torch.linalg.eigvalsh(Xd @ Xd.T if rows <= cols else Xd.T @ Xd).flip(0)[:k].cpu().numpy()
    s = B.Arnoldi(rows, min(20, rows), k, seed=3)
    if host:
        s.set_gram_operator_host(X.cpu().pin_memory(), max(1, cols // 3))
    else:
        s.set_gram_operator(X)
    ev, res, st = s.solve()
    assert st == B.OK and max(res) <= 1e-10
    assert np.abs(np.array(ev).real - ref).max() <= (rows + cols) * 2.3e-16 * 4 * ref[0]
    again, res2, _ = s.solve()  # fixed summation order: the same bits
    assert again == ev and res2 == res
