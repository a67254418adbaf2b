"""Receptive-field generation, Dirichlet coefficients and spatial functions at
the edges of their tiles, bin counts and copy widths, against the oracle."""
import numpy as np
import pytest
import torch

from oracle import vtem_oracle as O
from vtem_b200 import vrf
from vtem_b200._abi import call, dptr, stream_ptr

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("N,LPy,LPx,Mx,My,pad", [
    (1, 1, 1, 0, 0, 0), (3, 16, 16, 0, 3, 0), (5, 17, 23, 3, 2, 1), (4, 64, 64, 7, 7, 0), (2, 33, 50, 7, 3, 0),
    (3, 250, 66, 2, 7, 2), (2, 129, 256, 6, 6, 1), (700, 32, 32, 2, 2, 0),      # more RFs than blocks
    (3, 48, 40, 8, 3, 0), (2, 40, 48, 2, 9, 0)])                                # more than 16 bins one way
def test_dirichlet_coefficients(N, LPy, LPx, Mx, My, pad):
    rng = np.random.default_rng(N + LPx)
    rf = rng.standard_normal((N, LPy, LPx))
    buf = torch.full((N, LPy * LPx + pad), 1e300, dtype=torch.float64, device="cuda")
    buf[:, :LPy * LPx] = torch.as_tensor(rf.reshape(N, -1), device="cuda")
    Ds = torch.empty((N, 2 * My + 1, 2 * Mx + 1), dtype=torch.complex128, device="cuda")
    call("vtb_dirichlet_coeffs", dptr(buf), N, LPy, LPx, LPy * LPx + pad, Mx, My, 0.25, dptr(Ds), stream_ptr())
    want = O.compute_Ds(rf, Mx, My, 0.25)
    tol = 4 * EPS * (LPx + LPy) * 0.25 * np.abs(rf).sum(axis=(1, 2)).max()      # two sums of rounded products
    assert np.abs(Ds.cpu().numpy() - want).max() <= tol


@pytest.mark.parametrize("N,Mx,My,Px,Py,Px1,Py1", [
    (1, 0, 0, 1, 1, 1, 1), (3, 3, 2, 16, 14, 16, 16), (2, 6, 6, 13, 13, 13, 13), (4, 2, 7, 65, 5, 70, 15),
    (2, 4, 3, 33, 21, 12000, 40)])                                              # a period beyond the table
def test_spatial_functions(N, Mx, My, Px, Py, Px1, Py1):
    rng = np.random.default_rng(Px + Py)
    D = rng.standard_normal((N, 2 * My + 1, 2 * Mx + 1)) + 1j * rng.standard_normal((N, 2 * My + 1, 2 * Mx + 1))
    out = torch.empty((N, Py, Px), dtype=torch.float64, device="cuda")
    Dd = torch.as_tensor(D, device="cuda")
    call("vtb_dirich_space", dptr(Dd), N, Mx, My, Px, Py, Px1, Py1, dptr(out), stream_ptr())
    want = O.compute_dirich_space_fft(D, Mx, My, Px, Py, Px1, Py1)
    tol = 8 * EPS * (2 * Mx + 2 * My + 2) * np.abs(D).sum(axis=(1, 2)).max()
    assert np.abs(out.cpu().numpy() - want).max() <= tol


@pytest.mark.parametrize("Py,Px", [(1, 1), (16, 14), (31, 129), (33, 128), (65, 300)])
@pytest.mark.parametrize("gain", [False, True])
def test_receptive_fields(Py, Px, gain):
    rng = np.random.default_rng(Px)
    N, k = 9, 2.5
    al, th = rng.choice([0.05, 0.2, 1.0], N), rng.uniform(0, np.pi, N)
    x0, y0, ab = rng.uniform(-0.5, 0.5, N), rng.uniform(-0.5, 0.5, N), (np.arange(N) % 2).astype(np.int32)
    g = rng.uniform(0.5, 2, N) if gain else None
    b = vrf.vrf_gabor((Py, Px), dx=1.0 / Px, dy=1.0 / Py)
    b.load_parameters(num_neurons=N, h_alpha=al, h_l=th, h_x0=x0, h_y0=y0, h_ab=ab, KAPPA=k, h_gain=g)
    b.generate_visual_receptive_fields()
    want = O.gabor_rf(al, th, x0, y0, ab, Px, Py, 1.0, 1.0, -0.5, -0.5, k, g)
    # the modulation's and the envelope's arguments, up to k X and X^2 with e^{-X^2/2}: a few ulp of the largest
    reach = k * np.sqrt(2.0) * 1.5 / al.min()
    assert np.abs(b.gabors.cpu().numpy() - want).max() <= 8 * EPS * (4 + reach) * np.abs(want).max()
    c = vrf.vrf_cs((Py, Px), dx=1.0 / Px, dy=1.0 / Py)
    c.load_parameters(num_neurons=N, h_alpha=al, h_x0=x0, h_y0=y0, sigma_center=0.05, sigma_surround=0.15, h_gain=g)
    c.generate_visual_receptive_fields()
    want = O.cs_rf(al, x0, y0, Px, Py, 1.0, 1.0, -0.5, -0.5, 0.05, 0.15, g)
    centre = 1.0 / al.min() / 0.05 ** 2 / (2 * np.pi) * 2          # the two Gaussians cancel in part
    assert np.abs(c.filters.cpu().numpy() - want).max() <= 16 * EPS * centre
