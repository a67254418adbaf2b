"""Float64 GEMM over its operand orders, copy widths, tile choices and edges."""
import numpy as np
import pytest
import torch

from vtem_b200._abi import call, dptr, stream_ptr

pytestmark = pytest.mark.gpu


def _operand(rng, rows, K, kind):
    """(device storage, element (0, 0), row stride, k stride, values (rows, K)) in one memory order."""
    v = rng.standard_normal((rows, K))
    if kind == "k":              # k contiguous
        t, r, k = torch.as_tensor(v, device="cuda"), K, 1
    elif kind == "k_odd":        # k contiguous, base 8 bytes off a 16-byte boundary
        buf = torch.zeros(rows * K + 1, dtype=torch.float64, device="cuda")
        buf[1:] = torch.as_tensor(v.reshape(-1), device="cuda")
        return buf, buf.data_ptr() + 8, K, 1, v
    elif kind == "r":            # rows contiguous
        t, r, k = torch.as_tensor(np.ascontiguousarray(v.T), device="cuda"), 1, rows
    else:                        # every second element of every third row
        t = torch.zeros((3 * rows, 2 * K), dtype=torch.float64, device="cuda")
        t[::3, ::2] = torch.as_tensor(v, device="cuda")
        r, k = 3 * 2 * K, 2
    return t, t.data_ptr(), r, k, v


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (64, 64, 16), (65, 33, 17), (63, 128, 64), (130, 31, 50), (2001, 129, 70),
                                   (700, 900, 33)])
@pytest.mark.parametrize("ka,kb", [("k", "k"), ("k", "r"), ("r", "k"), ("r", "r"), ("k_odd", "k"), ("x", "k"), ("r", "x")])
def test_gemm_f64_orders_and_edges(M, N, K, ka, kb):
    rng = np.random.default_rng(M + N + K)
    A, pa, am, ak, va = _operand(rng, M, K, ka)
    B, pb, bn, bk, vb = _operand(rng, N, K, kb)
    for cm, cn, beta in ((N, 1, 0.0), (1, M, 0.5)):
        c0 = rng.standard_normal((M, N))
        C = torch.as_tensor(c0 if cn == 1 else np.ascontiguousarray(c0.T), device="cuda")
        call("vtb_gemm_f64", M, N, K, pa, am, ak, pb, bn, bk, dptr(C), cm, cn, 1.25, beta, stream_ptr())
        got = C.cpu().numpy() if cn == 1 else C.cpu().numpy().T
        want = 1.25 * (va @ vb.T) + beta * c0
        # K rounded products and sums, then two operations, on each side
        tol = 2 * np.finfo(np.float64).eps * (K + 3) * (1.25 * (np.abs(va) @ np.abs(vb).T) + abs(beta) * np.abs(c0))
        assert np.all(np.abs(got - want) <= tol)
