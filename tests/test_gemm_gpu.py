"""oapb_dot_product's matrix products at the edges of its tiles and K splits,
with every combination of planes."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402
import oracle as O  # noqa: E402

EPS = 2.3e-16


def product(a, b, out_planes, shape):
    """a, b: (re or None, im or None) numpy planes; the library's product."""
    up = lambda p: [torch.from_numpy(np.ascontiguousarray(x)).cuda() if x is not None else None for x in p]
    ta, tb = up(a), up(b)
    o = [torch.full(shape, 7.0, dtype=torch.float64, device="cuda") if w else None for w in out_planes]
    m = [B.mat(*x) for x in (o, ta, tb)]
    st = B.lib().oapb_dot_product(*[C.byref(x) for x in m], None)
    assert st == B.OK, B.status_string(st)
    torch.cuda.synchronize()
    return [x.cpu().numpy() if x is not None else None for x in o]


def check(a, b, out_planes, shape, k):
    full = lambda p: (p[0] if p[0] is not None else 0.0) + 1j * (p[1] if p[1] is not None else 0.0 * p[0])
    fa, fb = full(a) + 0j, full(b) + 0j
    ref = O.dot_product(fa, fb)
    # both sums have 2 k terms of rounding at most 2 k eps each
    bound = 4 * (k + 2) * EPS * (np.abs(fa) @ np.abs(fb)) * 2 ** 0.5 + 1e-300
    got = product(a, b, out_planes, shape)
    for g, r in zip(got, (ref.real, ref.imag)):
        if g is not None:
            assert (np.abs(g - r) <= bound).all()


# one element, tiles filled and one beyond, chunk remainders, deep products that
# split K over clusters (1 .. 8), more tiles than SMs
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (32, 16, 32), (33, 17, 31), (64, 15, 65), (65, 64, 129), (30, 1549, 30),
                                   (299, 1000, 30), (40, 130, 200), (3, 40, 700), (700, 33, 2), (900, 48, 1001)])
@pytest.mark.parametrize("cplx", [False, True])
def test_products_at_tile_edges(m, k, n, cplx):
    rng = np.random.default_rng(m + 10 * k + 100 * n)
    r = lambda *s: rng.normal(size=s)
    a, b = (r(m, k), r(m, k) if cplx else None), (r(k, n), r(k, n) if cplx else None)
    check(a, b, (True, cplx), (m, n), k)


@pytest.mark.parametrize("pa,pb,po", [((1, 1), (1, 0), (1, 1)), ((1, 0), (1, 1), (1, 1)), ((0, 1), (1, 1), (1, 1)),
                                      ((0, 1), (0, 1), (1, 1)), ((1, 0), (1, 0), (1, 1)), ((1, 1), (1, 1), (1, 0)),
                                      ((1, 1), (1, 1), (0, 1)), ((1, 0), (1, 0), (0, 1))])
def test_products_of_partial_planes(pa, pb, po):
    # an absent plane is zero, an absent output plane is not written
    rng = np.random.default_rng(3)
    m, k, n = 45, 70, 37
    a = tuple(rng.normal(size=(m, k)) if w else None for w in pa)
    b = tuple(rng.normal(size=(k, n)) if w else None for w in pb)
    if a[0] is None:
        a = (None, a[1])
    ra = (np.zeros((m, k)) if a[0] is None else a[0], a[1])
    rb = (np.zeros((k, n)) if b[0] is None else b[0], b[1])
    full = lambda p: p[0] + 1j * (p[1] if p[1] is not None else 0.0)
    ref = full(ra) @ full(rb)
    got = product(a, b, po, (m, n))
    bound = 4 * (k + 2) * EPS * (np.abs(full(ra)) @ np.abs(full(rb))) * 2 ** 0.5
    for g, r in zip(got, (ref.real, ref.imag)):
        if g is not None:
            assert (np.abs(g - r) <= bound).all()
