"""Synthesis of the plain decoder at uniform times, against the oracle's
per-neuron regrouping of reconstruct_Kernel (vtem/dirichlet.py:354-420), at
the edges of its neuron chunks, pixel tiles and harmonic counts."""
import numpy as np
import pytest
import torch

from oracle import vtem_oracle as O
from vtem_b200 import dirichlet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,Py,Px,Mt,n,t0,Nt,order", [
    (1, 1, 1, 1, 1, 0.0, 1, "sorted"), (7, 5, 13, 2, 40, 0.1, 7, "any"), (33, 8, 8, 3, 100, 0.0, 8, "sorted"),
    (255, 4, 16, 4, 300, 0.0, 33, "any"), (257, 3, 43, 5, 900, 0.05, 101, "sorted"), (64, 9, 7, 6, 64, 0.0, 64, "sorted"),
    (40, 2, 32, 7, 200, 0.0, 321, "sorted"), (300, 16, 16, 8, 2000, 0.0, 700, "any"),
    (31, 6, 11, 9, 150, 0.3, 50, "sorted"), (96, 8, 9, 10, 500, 0.0, 65, "sorted"),
    (20, 5, 5, 11, 100, 0.1, 12, "sorted"),          # beyond 10 harmonics: the general path
])
def test_uniform_reconstruction(N, Py, Px, Mt, n, t0, Nt, order):
    rng = np.random.default_rng(N + Mt)
    Wt, T, dt = 2 * np.pi * 20, 0.4, 1e-3
    a = rng.uniform(0, T, n)
    b = a + rng.uniform(0.003, 0.05, n)
    ind = rng.integers(0, N, n).astype(np.int32)
    if order == "sorted":
        ind = np.sort(ind)
    c = rng.standard_normal(n)
    norm = rng.uniform(0.5, 1.0, N)
    phi = rng.standard_normal((N, Py, Px))
    one = np.ones(N)
    cp = dirichlet.dirichlet(N, a, b, ind, one, one, one, norm, Wt, Mt)
    cp.d_q = torch.as_tensor(c, device="cuda").reshape(-1, 1)
    frame = [t0, t0 + (Nt - 0.5) * dt]
    u = cp.reconstruct(phi, frame, dt).cpu().numpy()
    t = np.arange(frame[0], frame[1], dt)
    uo = O.reconstruct_factored(phi, a, b, c, t, ind, norm, Mt, Wt / Mt)
    assert u.shape == (Nt, Py, Px)
    # every term rounded with its argument (m W t), and two sums of N and n terms
    W, m = Wt / Mt, np.arange(1, Mt + 1)
    term = np.abs(c) * norm[ind] * ((b - a) + (4 / W) * (1 / m).sum())
    size = np.bincount(ind, weights=term, minlength=N) @ np.abs(phi).reshape(N, -1)
    tol = np.finfo(np.float64).eps * (8 + Mt * W * (t0 + T + Nt * dt) + N + n) * size.max()
    assert np.abs(u - uo).max() <= tol


@pytest.mark.parametrize("t0", [0.3, 5.0, -70.1])
def test_times_are_those_of_arange(t0):
    """np.arange steps by fl(t0 + dt) - t0; over many frames that is far from
    dt.  Against the general kernel on arange's own times."""
    N, Mt, n, Nt, dt = 9, 6, 60, 4000, 1e-4
    rng = np.random.default_rng(3)
    Wt = 2 * np.pi * 20
    a = t0 + rng.uniform(0, 0.4, n)
    b = a + rng.uniform(0.003, 0.05, n)
    ind = np.sort(rng.integers(0, N, n)).astype(np.int32)
    c, one, phi = rng.standard_normal(n), np.ones(N), rng.standard_normal((N, 6, 5))
    cp = dirichlet.dirichlet(N, a, b, ind, one, one, one, one, Wt, Mt)
    cp.d_q = torch.as_tensor(c, device="cuda").reshape(-1, 1)
    frame = [t0, t0 + (Nt - 0.5) * dt]
    u = cp.reconstruct(phi, frame, dt).cpu().numpy().reshape(Nt, -1)
    t = np.arange(frame[0], frame[1], dt)
    call = dirichlet.call
    d = [torch.as_tensor(x, device="cuda") for x in (phi, a, b, c, ind, one, t)]
    nb = np.zeros(1, np.int64)
    call("vtb_reconstruct_workspace", N, len(t), Mt, nb.ctypes.data)
    work = torch.empty(int(nb[0]), dtype=torch.uint8, device="cuda")
    want = torch.empty((len(t), 30), dtype=torch.float64, device="cuda")
    p = [x.data_ptr() for x in d]
    call("vtb_reconstruct", p[0], N, 30, p[1], p[2], p[3], p[4], p[5], n, p[6], len(t), Mt, Wt / Mt, want.data_ptr(),
         work.data_ptr(), work.numel(), dirichlet.stream_ptr())
    assert u.shape == (Nt, 30)
    # the rounding of the arguments m W t on both sides, and of two sums of N and n terms
    W, m = Wt / Mt, np.arange(1, Mt + 1)
    term = np.abs(c) * ((b - a) + (4 / W) * (1 / m).sum())
    size = np.bincount(ind, weights=term, minlength=N) @ np.abs(phi).reshape(N, -1)
    tol = 2 * np.finfo(np.float64).eps * (8 + Mt * W * (abs(t0) + 0.5) + N + n) * size.max()
    assert np.abs(u - want.cpu().numpy()).max() <= tol
