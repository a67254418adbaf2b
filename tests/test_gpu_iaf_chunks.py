"""The integrate-and-fire scan works on chunks of 32 steps; clips and frame
blocks around that width, membranes that end a step exactly on the threshold
or a hair below it, steps of negative slope, quotients by 1 and not, and
inputs in both layouts, bit for bit against the reference-order C oracle
(vtem/ensemble_encode.py:466-545)."""
import numpy as np
import pytest
import torch

from oracle import vtem_oracle as O
from vtem_b200 import ensemble_encode

pytestmark = pytest.mark.gpu

DT = 2.0 ** -10


def _case(N, F, seed):
    rng = np.random.default_rng(seed)
    L = rng.standard_normal((F, N)) * 0.3
    kap = np.where(rng.random(N) < 0.5, 1.0, rng.uniform(0.7, 1.3, N))
    bia = rng.uniform(0.8, 1.6, N)
    dl = rng.uniform(2, 90, N) * DT
    v0 = rng.uniform(0, 1, N) * dl
    # constant drive 1: the membrane is a whole number of DT after each step,
    # on the threshold (k = 0) or below it by 1e-13 or 1e-9 (k = 1, 2)
    for k in range(min(3, N // 4)):
        L[:, k], kap[k], bia[k], v0[k] = 0.0, 1.0, 1.0, 0.0
        dl[k] = 40 * DT + (0.0, 1e-13, 1e-9)[k]
    if N > 6:
        L[F // 2:F // 2 + 5, 4] = -4.0              # falls through zero
        L[::3, 5] = -30.0                           # zigzag: steps of negative slope and falling membranes
    return L, kap, bia, dl, v0


@pytest.mark.parametrize("major", ["time", "neuron"])
@pytest.mark.parametrize("N,F,B", [(1, 2, 101), (9, 32, 101), (9, 33, 101), (9, 34, 33), (9, 65, 34), (9, 66, 32),
                                   (9, 97, 7), (9, 1000, 33), (9, 1001, 45), (133, 700, 101), (9, 640, 65),
                                   (9, 700, 2)])
def test_chunks(N, F, B, major):
    L, kap, bia, dl, v0 = _case(N, F, 7 * F + B)
    want = O.vtem_encode(L, DT, kap, bia, dl, v0, block_frames=B, max_spike_per_block=100000)
    e = ensemble_encode.IAF_encode(N, DT)
    e.load_parameters(h_kappa=kap, h_bias=bia, h_delta=dl, h_v0=v0)
    x = torch.as_tensor(np.ascontiguousarray(L if major == "time" else L.T), device="cuda")
    sp = e.encode_blocks(x, block_frames=B, layout=major)
    times, steps, cnt = sp.to_host_lists()
    got_t = [times[n][(steps[n] // (B - 1)) == b] for b in range(len(want.block_counts)) for n in range(N)]
    got_s = [steps[n][(steps[n] // (B - 1)) == b] for b in range(len(want.block_counts)) for n in range(N)]
    assert np.array_equal(np.concatenate(got_s), np.concatenate(want.block_steps))
    assert np.array_equal(np.concatenate(got_t), np.concatenate(want.block_spikes))
    assert np.array_equal(e.d_v0.cpu().numpy(), want.v0)
    assert sp.near_threshold == want.near_threshold


@pytest.mark.parametrize("F", [31, 64, 65, 300])
def test_random_thresholds_in_one_block(F):
    N = 12
    L, kap, bia, dl, v0 = _case(N, F, F)
    rng = np.random.default_rng(F)
    sig = dl * 0.05
    rn = rng.standard_normal((400, N))
    dv = dl.copy()
    ref = O.iaf_encode_block(L, DT, kap, bia, dl, v0.copy(), np.zeros(N), 400, randn=rn, sigma=sig, delta_value=dv)
    from vtem_b200._abi import call, dptr, stream_ptr
    d = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")
    x, dk, db, dd, dv0, dtc, drn, dsg, ddv = map(d, (L, kap, bia, dl, v0, np.zeros(N), rn, sig, dl))
    st = torch.zeros((N, 400), dtype=torch.float64, device="cuda")
    ss = torch.zeros((N, 400), dtype=torch.int32, device="cuda")
    cnt = torch.zeros(N, dtype=torch.int32, device="cuda")
    near = torch.zeros(1, dtype=torch.int64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    call("vtb_iaf_encode", dptr(x), N, 1, N, F, 1, DT, dptr(dk), dptr(db), dptr(dd), dptr(dv0), dptr(dtc), dptr(drn),
         0, N, 1, 400, dptr(dsg), dptr(ddv), dptr(st), dptr(ss), dptr(cnt), 400, dptr(near), 1e-12, dptr(status), 0.0,
         stream_ptr())
    got = cnt.cpu().numpy()
    assert np.array_equal(got, ref.spike_count)
    for n in range(N):
        assert np.array_equal(st[n, :got[n]].cpu().numpy(), ref.spikes[n])
        assert np.array_equal(ss[n, :got[n]].cpu().numpy(), ref.steps[n])
    assert np.array_equal(ddv.cpu().numpy(), dv)
    assert int(near) == ref.near_threshold
