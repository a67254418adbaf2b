"""Float64 Kronecker Gram at the edges of its pair, entry and neuron tiles,
against the definition."""
import numpy as np
import pytest
import torch

from vtem_b200._abi import call, dptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,Ks,Kt", [(1, 1, 1), (15, 5, 3), (16, 13, 7), (17, 5, 8), (33, 29, 9), (50, 49, 17), (300, 13, 21),
                                     (40, 113, 5)])
def test_kron_gram(N, Ks, Kt):
    rng = np.random.default_rng(N + Ks)
    d = rng.standard_normal((N, Ks)) + 1j * rng.standard_normal((N, Ks))
    V = rng.standard_normal((N, Kt, 2 * Kt)) + 1j * rng.standard_normal((N, Kt, 2 * Kt))
    W = V @ np.conj(V.transpose(0, 2, 1))                       # Hermitian, as a temporal Gram is
    W = 0.5 * (W + np.conj(W.transpose(0, 2, 1)))
    g = rng.standard_normal((N, Kt)) + 1j * rng.standard_normal((N, Kt))
    K = Ks * Kt
    ld = K + 3
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")
    M = torch.full((K, ld), 7.0 + 7.0j, dtype=torch.complex128, device="cuda")
    b = torch.empty(K, dtype=torch.complex128, device="cuda")
    dd, Wd, gd = t(d), t(W), t(g)
    call("vtb_coeff_gram", dptr(dd), N, Ks, dptr(Wd), dptr(gd), Kt, dptr(M), ld, dptr(b), stream_ptr())
    got = M.cpu().numpy()[:, :K].T                               # column-major
    want = np.einsum("ns,nt,nij->sitj", d, np.conj(d), W).reshape(K, K)
    size = np.einsum("ns,nt,nij->sitj", np.abs(d), np.abs(d), np.abs(W)).reshape(K, K)
    assert np.all(np.abs(got - want) <= 8 * np.finfo(np.float64).eps * (N + 4) * size)
    assert np.array_equal(got, np.conj(got.T))
    assert np.all(M.cpu().numpy()[:, K:] == 7.0 + 7.0j)


def test_more_pairs_than_a_grid_dimension():
    """2.2 million pairs of spatial indices (65,536 rows of 32 and more)."""
    Ks = 2100
    rng = np.random.default_rng(2)
    d = torch.as_tensor(rng.standard_normal(Ks) + 1j * rng.standard_normal(Ks), device="cuda")
    W = torch.full((1, 1, 1), 1.5, dtype=torch.complex128, device="cuda")
    g = torch.full((1, 1), 0.5 - 0.25j, dtype=torch.complex128, device="cuda")
    M = torch.zeros((Ks, Ks), dtype=torch.complex128, device="cuda")
    b = torch.empty(Ks, dtype=torch.complex128, device="cuda")
    call("vtb_coeff_gram", dptr(d), 1, Ks, dptr(W), dptr(g), 1, dptr(M), Ks, dptr(b), stream_ptr())
    want = 1.5 * torch.outer(d, d.conj())
    eps = np.finfo(np.float64).eps
    assert bool(((M.T - want).abs() <= 4 * eps * want.abs()).all())
    assert bool(((b - d * g[0, 0]).abs() <= 4 * eps * b.abs()).all())
