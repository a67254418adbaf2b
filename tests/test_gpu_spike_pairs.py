"""Pairing of device spikes over neuron counts around its scan's width, empty
and single-spike neurons, against the oracle's consecutive pairs
(vtem/spike_store.py:279-351)."""
import numpy as np
import pytest
import torch

from vtem_b200 import ensemble_encode, spike_store

pytestmark = pytest.mark.gpu


def _spikes(N, cap, seed, T):
    rng = np.random.default_rng(seed)
    cnt = rng.integers(0, cap, N).astype(np.int32)
    cnt[rng.random(N) < 0.2] = 0
    B, dt = 11, 1e-3
    R = (B - 1) * dt
    time = np.full((N, cap), np.nan)
    step = np.full((N, cap), -1, np.int32)
    for n in range(N):
        t = np.sort(rng.uniform(1e-6, T - 1e-6, cnt[n]))
        step[n, :cnt[n]] = np.floor(t / dt)
        time[n, :cnt[n]] = t - (step[n, :cnt[n]] // (B - 1)) * R
    dev = [torch.as_tensor(x, device="cuda") for x in (time, step, cnt)]
    return ensemble_encode.DeviceSpikes(*dev, B, dt), time, step, cnt, R, B


@pytest.mark.parametrize("N,cap", [(1, 1), (1, 40), (31, 5), (33, 70), (1023, 6), (1024, 6), (1025, 33), (3000, 4)])
def test_pairs(N, cap):
    T = 0.5
    sp, time, step, cnt, R, B = _spikes(N, cap, N + cap, T)
    tk1, tk2, ind = (x.cpu().numpy() for x in spike_store.device_pairs(sp, T))
    want = [time[n, :cnt[n]] + (step[n, :cnt[n]] // (B - 1)).astype(np.float64) * R - 0.0 for n in range(N)]
    assert np.array_equal(tk1, np.concatenate([t[:-1] for t in want]))
    assert np.array_equal(tk2, np.concatenate([t[1:] for t in want]))
    assert np.array_equal(ind, np.repeat(np.arange(N), np.maximum(cnt - 1, 0)))


def test_spike_outside_is_refused():
    sp, *_ = _spikes(70, 9, 3, 0.5)
    with pytest.raises(ValueError):
        spike_store.device_pairs(sp, 0.25)
