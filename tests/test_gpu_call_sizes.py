"""Entry points whose launches need shared memory by their call's sizes, called
side by side by two host threads with different sizes: a launch may not depend
on the size that another thread set in between."""
import threading

import pytest
import torch

from vtem_b200._abi import call, dptr, stream_ptr

pytestmark = pytest.mark.gpu
RUNS = 3000


def _coefficients(L, M):
    rf = torch.zeros((1, L, L), dtype=torch.float64, device="cuda")
    Ds = torch.empty((1, 2 * M + 1, 2 * M + 1), dtype=torch.complex128, device="cuda")
    return lambda: call("vtb_dirichlet_coeffs", dptr(rf), 1, L, L, L * L, M, M if 2 * M < 16 else 2, 1.0, dptr(Ds),
                        stream_ptr())


def _functions(P, M):
    Ds = torch.zeros((1, 2 * M + 1, 2 * M + 1), dtype=torch.complex128, device="cuda")
    out = torch.empty((1, P, P), dtype=torch.float64, device="cuda")
    return lambda: call("vtb_dirich_space", dptr(Ds), 1, M, M, P, P, P, P, dptr(out), stream_ptr())


def _basis(M):
    K = 2 * M + 1
    a = torch.zeros((K * K, 3), dtype=torch.complex128, device="cuda")
    smap = torch.arange(K * K, dtype=torch.int32, device="cuda")
    H = torch.empty((64 * 64, 3), dtype=torch.float64, device="cuda")
    return lambda: call("vtb_coeff_basis", dptr(a), dptr(smap), K * K, M, M, 1, 64, 64, 64, 64, dptr(H), 3, stream_ptr())


def _synthesis(P, M, Mt, f32):
    K = 2 * M + 1
    a = torch.zeros((K * K, 2 * Mt + 1), dtype=torch.complex128, device="cuda")
    smap = torch.arange(K * K, dtype=torch.int32, device="cuda")
    A = torch.empty((2 * K * K,), dtype=torch.complex128, device="cuda")
    u = torch.empty((2, P, P), dtype=torch.float32 if f32 else torch.float64, device="cuda")
    return lambda: call("vtb_coeff_synthesize", dptr(a), dptr(smap), K * K, M, M, Mt, 1.0, 0.0, 0.1, 2, P, P, P, P,
                        dptr(A), dptr(u), int(f32), stream_ptr())


@pytest.mark.parametrize("make,small,large", [
    (_coefficients, (64, 6), (256, 6)),                      # the tensor path
    (_coefficients, (300, 9), (400, 9)),                     # more than 16 bins one way
    (_functions, (128, 12), (180, 12)),
    (_basis, (8,), (14,)),
    (_synthesis, (64, 6, 1, False), (64, 6, 8, False)), (_synthesis, (64, 6, 1, True), (64, 6, 8, True)),
    (_synthesis, (72, 6, 1, False), (160, 6, 1, False)), (_synthesis, (72, 6, 1, True), (160, 6, 1, True)),
    (_synthesis, (72, 15, 1, False), (120, 15, 1, False)), (_synthesis, (72, 15, 1, True), (120, 15, 1, True)),
])
def test_two_threads(make, small, large):
    calls = [make(*small), make(*large)]
    torch.cuda.synchronize()
    errors, start = [], threading.Barrier(2)

    def work(f):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                for _ in range(RUNS):
                    f()
        except Exception as e:                               # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=work, args=(f,)) for f in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
