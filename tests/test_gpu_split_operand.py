"""The [hi | lo] operand of the split-bf16 products: float32 and float64
sources, wide and scalar loads (row lengths around 8, pitches and bases off
16 bytes), against the definition hi = bf16(x), lo = bf16(x - hi)."""
import numpy as np
import pytest
import torch

from vtem_b200 import tc, vrf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 0.75])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("rows,K,pitch,start", [(1, 1, 1, 0), (5, 7, 8, 0), (5, 8, 8, 0), (5, 8, 9, 0), (5, 9, 12, 0),
                                                (3, 64, 64, 1), (3, 64, 66, 2), (4, 65, 68, 4), (33, 100, 100, 0),
                                                (2, 2311, 2312, 0)])
def test_split(rows, K, pitch, start, dtype, scale):
    g = torch.Generator(device="cuda").manual_seed(rows * 1000 + K)
    base = torch.randn(start + rows * pitch, dtype=torch.float64, device="cuda", generator=g).to(dtype)
    X = base[start:].view(rows, pitch)[:, :K]
    if K > 2:
        X[0, 1], X[-1, K - 1] = float("inf"), float("nan")
    got = tc.split_bf16x2(X, scale=scale)
    Kp = tc.padded_k(K)
    x = X.double() * scale
    hi = x.float().to(torch.bfloat16)
    lo = (x - hi.double()).float().to(torch.bfloat16)
    want = torch.zeros((rows, 2 * Kp), dtype=torch.bfloat16, device="cuda")
    want[:, :K], want[:, Kp:Kp + K] = hi, lo
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.nan_to_num(got.float()), torch.nan_to_num(want.float()))


@pytest.mark.parametrize("layout", ["time", "neuron"])
@pytest.mark.parametrize("P", [9, 64, 100])
def test_projection_of_single_precision_video(P, layout):
    g = torch.Generator(device="cuda").manual_seed(P)
    V = torch.randn(37, P, device="cuda", generator=g)
    rf = torch.randn(21, P, dtype=torch.float64, device="cuda", generator=g)
    a, b, c = (vrf._project(v, rf, 0.5, P, layout, "bf16x3") for v in (V, V.double(), V.cpu().numpy()))
    assert a.dtype == torch.float64 and torch.equal(a, b) and torch.equal(a, c)
    assert np.isfinite(a.cpu().numpy()).all()
