"""Gradient flow on the coefficient system at every row and column split of
its kernels, against the same updates in float64 on the host
(vtem/neural_network.py:15-128)."""
import numpy as np
import pytest
import torch

from vtem_b200 import _abi
from vtem_b200._abi import call, dptr, stream_ptr

pytestmark = pytest.mark.gpu


def _run(Mr, ld, br, K, h, steps):
    nb = np.zeros(1, np.int64)
    call("vtb_rnn_coeff_workspace", K, nb.ctypes.data)
    work = torch.full((int(nb[0]),), 255, dtype=torch.uint8, device="cuda")
    x = torch.full((K,), 7.0, dtype=torch.float64, device="cuda")
    call("vtb_rnn_coeff_work", dptr(Mr), ld, dptr(br), dptr(x), K, h, steps, dptr(work), work.numel(), stream_ptr())
    return x.cpu().numpy(), int(work[:16].view(torch.int32)[2].item())


@pytest.mark.parametrize("K,pad", [(1, 0), (2, 3), (296, 0), (297, 1), (512, 0), (592, 0), (593, 0), (1024, 5), (1036, 0),
                                   (1037, 0), (1480, 0), (1481, 0), (1921, 0), (1924, 2), (1925, 0)])
@pytest.mark.parametrize("steps", [0, 1, 25, 402])
def test_gradient_flow_splits(K, pad, steps):
    rng = np.random.default_rng(K)
    A = rng.standard_normal((K, 8)) / np.sqrt(K)
    M = A @ A.T + np.diag(rng.uniform(0.1, 1.0, K))
    b = rng.standard_normal(K)
    h = 0.5
    buf = torch.full((K, K + pad), float("nan"), dtype=torch.float64, device="cuda")
    buf[:, :K] = torch.as_tensor(M, device="cuda")
    x, err = _run(buf, K + pad, torch.as_tensor(b, device="cuda"), K, h, steps)
    want = np.zeros(K)
    size = np.zeros(K)
    for _ in range(steps + 1):
        want = want + h * (b - M @ want)
        size = size + h * (np.abs(b) + np.abs(M) @ np.abs(want))
    assert err == 0
    # K rounded products an update, carried by updates that contract
    assert np.abs(x - want).max() <= 2 * np.finfo(np.float64).eps * (K + 4) * size.max()


def test_gradient_flow_wait_runs_out():
    """A limit of one poll: the status says so, and the next call is exact."""
    K = 700
    M = torch.eye(K, dtype=torch.float64, device="cuda") * 0.5
    b = torch.ones(K, dtype=torch.float64, device="cuda")
    with _abi.wait_limit(1):
        _, err = _run(M, K, b, K, 0.5, 200)
    assert err != 0
    x, err = _run(M, K, b, K, 1.0, 60)
    assert err == 0
    assert np.allclose(x, 2.0, rtol=0, atol=1e-12)


def _system(K):
    rng = np.random.default_rng(1000 + K)
    A = rng.standard_normal((K, 8)) / np.sqrt(K)
    M = A @ A.T + np.diag(rng.uniform(0.1, 1.0, K))
    return M, rng.standard_normal(K), np.linalg.eigvalsh(M)[-1]


@pytest.mark.parametrize("K", [1, 2, 3, 40, 300, 1925])
@pytest.mark.parametrize("steps", [100, 401, 402])
def test_steps_that_diverge(K, steps):
    """Above 2 / lambda_max the updates grow, and so would a squared map's
    rounding (all of these squared at least once): the iterate is that of the
    updates one by one, bit for bit."""
    M, b, top = _system(K)
    h = 2.4 / top
    Md, bd = torch.as_tensor(M, device="cuda"), torch.as_tensor(b, device="cuda")
    x, err = _run(Md, K, bd, K, h, steps)
    want, tmp = torch.empty_like(bd), torch.empty_like(bd)
    bar = torch.zeros(4, dtype=torch.int32, device="cuda")
    call("vtb_rnn_coeff", dptr(Md), K, dptr(bd), dptr(want), dptr(tmp), K, h, steps, dptr(bar), stream_ptr())
    assert err == 0 and int(bar[2].item()) == 0
    assert np.abs(x).max() > 100 * np.abs(b).max()
    assert np.array_equal(x, want.cpu().numpy())


@pytest.mark.parametrize("K", [1, 2, 3, 40, 300])
@pytest.mark.parametrize("steps", [25, 402])
def test_steps_near_the_largest_that_contracts(K, steps):
    M, b, top = _system(K)
    h = 1.9 / top
    x, err = _run(torch.as_tensor(M, device="cuda"), K, torch.as_tensor(b, device="cuda"), K, h, steps)
    want = np.zeros(K)
    size = np.zeros(K)
    for _ in range(steps + 1):
        want = want + h * (b - M @ want)
        size = size + h * (np.abs(b) + np.abs(M) @ np.abs(want))
    assert err == 0
    assert np.abs(x - want).max() <= 2 * np.finfo(np.float64).eps * (K + 4) * size.max()
