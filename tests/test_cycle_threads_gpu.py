"""Solves in restart cycles on several host threads and streams of one device."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import oap_b200 as B  # noqa: E402


def handle(n, m, k, seed, cplx=False, **kw):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    A = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    if not cplx:
        A = A + A.T
    A = A / (2 * n ** 0.5)
    i = torch.arange(k, device="cuda")
    A[i, i] += 4.0 + 0.1 * i.double()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    s = B.Arnoldi(n, m, k, is_complex=cplx, seed=seed, stream=stream.cuda_stream, **kw)
    s.set_operator(A, torch.zeros_like(A) if cplx else None)
    s.keep = stream
    return s


def test_cycles_of_threads_give_the_serial_results():
    # grids of 8 to 148 CTAs: some fit the device together, some only alone
    hs = [handle(n, m, k, n, cplx) for n, m, k, cplx in ((64, 16, 3, False), (256, 24, 4, False), (640, 32, 5, True),
                                                         (900, 24, 4, False), (1500, 20, 3, False), (1300, 24, 3, True))]
    refs = [s.solve() for s in hs]
    errors = []

    def run(i):
        try:
            for _ in range(25):
                assert hs[i].solve() == refs[i]
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(hs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_a_long_solve_does_not_hold_back_the_others():
    # a cyclic shift (all eigenvalues of modulus 1): no small Krylov space finds
    # the wanted ones, the solve uses its whole restart budget (seconds)
    n = 240
    stream = torch.cuda.Stream()
    A = torch.eye(n, dtype=torch.float64, device="cuda").roll(1, 0).contiguous()
    torch.cuda.synchronize()
    long = B.Arnoldi(n, 8, 3, seed=1, max_restarts=20000, stream=stream.cuda_stream)
    long.set_operator(A)
    short = handle(200, 24, 4, 2)
    ref = short.solve()
    done = []
    t = threading.Thread(target=lambda: done.append(long.solve(allow_not_converged=True)[2]))
    t.start()
    time.sleep(0.2)
    assert not done  # still running
    for _ in range(10):
        assert short.solve() == ref
    assert not done
    t.join()
    assert done == [B.NOT_CONVERGED]
