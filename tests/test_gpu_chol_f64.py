"""vtb_sym_chol_solve: the float64 tile Cholesky solve over sizes around its
tile, odd and even leading dimensions, against the normwise backward error of
a Cholesky solve; the pivot test; the solver that uses it."""
import numpy as np
import pytest
import torch

from oracle import vtem_oracle as O
from vtem_b200 import _abi, fast
from vtem_b200._abi import call, dptr, lib, stream_ptr

pytestmark = pytest.mark.gpu


def _solve(M, b, ld, rcond=1e-12):
    K = b.numel()
    A = torch.full((K, ld), 7.0, dtype=torch.float64, device="cuda")
    A[:, :K] = M                                          # column j at j*ld
    x = b.clone()
    w = torch.empty(int(lib().vtb_sym_chol_solve_bytes(K)), dtype=torch.uint8, device="cuda").random_()
    flag = torch.full((1,), 9, dtype=torch.int32, device="cuda")
    piv = torch.zeros(2, dtype=torch.float64, device="cuda")
    call("vtb_sym_chol_solve", dptr(A), ld, K, dptr(x), rcond, dptr(w), w.numel(), dptr(flag), dptr(piv), stream_ptr())
    return x, A, int(flag), piv.tolist()


def _spd(K, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    B = torch.randn(K, K + 8, dtype=torch.float64, device="cuda", generator=g)
    return B @ B.T / K + torch.eye(K, dtype=torch.float64, device="cuda"), torch.randn(K, dtype=torch.float64,
                                                                                         device="cuda", generator=g)


@pytest.mark.parametrize("pad", [0, 1, 6])
@pytest.mark.parametrize("K", [1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 161, 500, 979, 1921])
def test_solve(K, pad):
    M, b = _spd(K, K)
    x, A, flag, piv = _solve(M, b, K + pad)
    assert flag == 0
    eps = np.finfo(np.float64).eps
    r = (M @ x - b).norm() / (torch.linalg.matrix_norm(M) * x.norm())
    assert r.item() <= 4 * K * eps
    L = torch.tril(A[:, :K].T)
    assert ((L @ L.T - M).norm() / M.norm()).item() <= 4 * K * eps
    d = torch.diagonal(L) ** 2
    assert piv == pytest.approx([d.min().item(), d.max().item()], rel=8 * eps)
    assert torch.equal(A[:, :K].T.triu(1), M.triu(1))     # the upper triangle and the padding stay
    assert bool((A[:, K:] == 7.0).all())


@pytest.mark.parametrize("K", [40, 200])
def test_pivot_flags(K):
    M, b = _spd(K, 3)
    M[K - 1, K - 1] = -1.0
    assert _solve(M, b, K)[2] == 1
    D = torch.diag(torch.logspace(0, -8, K, dtype=torch.float64, device="cuda"))
    assert _solve(D, b, K, rcond=1e-7)[2] == 2
    assert _solve(D, b, K, rcond=1e-9)[2] == 0


@pytest.mark.parametrize("K", [65, 261, 979])
def test_tiles_of_the_call(K):
    """Two systems solved in turn in the same buffers: a tile read before its
    writer has published it would hold the other system's numbers."""
    systems = [_spd(K, s) for s in (1, 2)]
    ld = K + (K & 1)
    A = torch.empty((K, ld), dtype=torch.float64, device="cuda")
    x = torch.empty(K, dtype=torch.float64, device="cuda")
    w = torch.empty(int(lib().vtb_sym_chol_solve_bytes(K)), dtype=torch.uint8, device="cuda")
    flags = torch.zeros(100, dtype=torch.int32, device="cuda")
    first, same = [], torch.ones((), dtype=torch.bool, device="cuda")
    for i in range(100):
        M, b = systems[i & 1]
        A[:, :K] = M
        x.copy_(b)
        call("vtb_sym_chol_solve", dptr(A), ld, K, dptr(x), 1e-12, dptr(w), w.numel(), flags.data_ptr() + 4 * i, None,
             stream_ptr())
        if i < 2:
            first.append((A[:, :K].clone(), x.clone()))
        else:
            same &= (A[:, :K] == first[i & 1][0]).all() & (x == first[i & 1][1]).all()
    assert int(flags.abs().max()) == 0 and bool(same)


@pytest.mark.parametrize("K,extra", [(261, 20), (500, 40)])
def test_as_close_as_the_library(K, extra):
    """Against the solution refined in extended precision: as many roundings of
    the same sizes as a blocked factorisation in float64, so on average the
    library's error, a quarter left for the samples."""
    ratios = []
    for seed in range(8):
        g = torch.Generator(device="cuda").manual_seed(100 + seed)
        B = torch.randn(K, K + extra, dtype=torch.float64, device="cuda", generator=g)
        M = B @ B.T / K
        M = 0.5 * (M + M.T)
        b = M @ torch.randn(K, dtype=torch.float64, device="cuda", generator=g)
        x, _, flag, _ = _solve(M, b, K + (K & 1))
        nb = np.zeros(1, np.int64)
        call("vtb_sym_workspace", K, 1, nb.ctypes.data)
        work = torch.empty(int(nb[0]), dtype=torch.uint8, device="cuda")
        A, y = M.clone(), b.clone()
        st = torch.zeros(4, dtype=torch.float64, device="cuda")
        call("vtb_sym_factor", dptr(A), K, K, 1, 1e-12, dptr(work), work.numel(), dptr(st), st.data_ptr() + 8, stream_ptr())
        call("vtb_sym_potrs", dptr(A), K, dptr(y), K, 1, dptr(work), work.numel(), stream_ptr())
        assert flag == 0
        Ml, bl = M.cpu().numpy().astype(np.longdouble), b.cpu().numpy().astype(np.longdouble)
        inv = np.linalg.inv(M.cpu().numpy())
        exact = y.cpu().numpy().astype(np.longdouble)
        for _ in range(6):
            exact = exact + inv @ (bl - Ml @ exact).astype(np.float64)
        e = [np.sqrt(((v.cpu().numpy() - exact) ** 2).sum()) for v in (x, y)]
        ratios.append(float(e[0] / e[1]))
    assert np.exp(np.mean(np.log(ratios))) <= 1.25


def test_ill_conditioned_tiles_are_flagged():
    """A nearly dependent pair in every eighth row: the inverses of the
    diagonal tiles then cost digits (Skeel condition numbers of 40 and 10,000)."""
    for c, want in ((1e1, 0), (1e6, -1)):
        for K in (300, 31):
            g = torch.Generator(device="cuda").manual_seed(1)
            B = torch.randn(K, K + 40, dtype=torch.float64, device="cuda", generator=g)
            n = B[1::8].shape[0]
            B[1::8] = B[0::8][:n] + B[1::8] / c ** 0.5
            assert _solve(B @ B.T / K, B[:, 0].clone(), K + (K & 1), rcond=1e-16)[2] == want


def test_short_window_takes_the_library(monkeypatch):
    """A window of 0.6 temporal periods, the truncation switched off: the
    coefficients are the library's, bit for bit."""
    rng = np.random.default_rng(12)
    N, n, Mx, My, Mt = 60, 3000, 2, 2, 8
    Ds = rng.standard_normal((N, 2 * My + 1, 2 * Mx + 1)) + 1j * rng.standard_normal((N, 2 * My + 1, 2 * Mx + 1))
    Ds = 0.5 * (Ds + np.conj(Ds[:, ::-1, ::-1])) * O.ellipse_mask(Mx, My)[None]
    tk1 = rng.uniform(0, 0.6 * Mt / 20, n)
    t = [torch.as_tensor(x, device="cuda") for x in (tk1, tk1 + rng.uniform(0.004, 0.03, n),
                                                     np.sort(rng.integers(0, N, n)).astype(np.int32))]
    p = [rng.uniform(0.8, 1.2, N), rng.uniform(0.01, 0.05, N), rng.uniform(1, 3, N)]
    dec = fast.CoeffDecoder(torch.as_tensor(Ds, device="cuda"), rng.uniform(0.5, 1.0, N), Mx, My, 2 * np.pi * 20, Mt,
                            8, 8, 8, 8, solver="chol", rcond=1e-20)
    run = lambda: dec.coefficients(*t, *p, assume_sorted=True).clone()
    a = run()
    monkeypatch.setattr(fast, "CHOL_TILES_MAX", 0)
    assert torch.equal(a, run())


def test_wait_limit_runs_out_and_recovers():
    M, b = _spd(979, 5)
    with _abi.wait_limit(1):
        assert _solve(M, b, 980)[2] == 3
    assert _solve(M, b, 980)[2] == 0


def test_decoder_routes(monkeypatch):
    """One window by the tile solve, by the library and with the tile solve
    giving up: the same coefficients up to cond(M) rounding errors."""
    rng = np.random.default_rng(11)
    N, n, Mx, My, Mt = 40, 1500, 3, 2, 3
    Ds = rng.standard_normal((N, 2 * My + 1, 2 * Mx + 1)) + 1j * rng.standard_normal((N, 2 * My + 1, 2 * Mx + 1))
    Ds = 0.5 * (Ds + np.conj(Ds[:, ::-1, ::-1])) * O.ellipse_mask(Mx, My)[None]
    tk1 = rng.uniform(0, 0.3, n)
    t = [torch.as_tensor(x, device="cuda") for x in (tk1, tk1 + rng.uniform(0.004, 0.03, n),
                                                     np.sort(rng.integers(0, N, n)).astype(np.int32))]
    p = [rng.uniform(0.8, 1.2, N), rng.uniform(0.01, 0.05, N), rng.uniform(1, 3, N)]
    dec = fast.CoeffDecoder(torch.as_tensor(Ds, device="cuda"), rng.uniform(0.5, 1.0, N), Mx, My, 2 * np.pi * 20, Mt,
                            8, 8, 8, 8, solver="chol")
    run = lambda: dec.coefficients(*t, *p, assume_sorted=True).clone()
    tiles = run()
    assert dec._chol64 is not None and dec.last_solver == "chol"
    with _abi.wait_limit(1):
        gave_up = run()
    monkeypatch.setattr(fast, "CHOL_TILES_MAX", 0)
    library = run()
    assert torch.equal(gave_up, library)
    tol = 8 * dec.K * np.finfo(np.float64).eps * torch.linalg.cond(dec.M).item()
    assert tol < 1e-3 and (tiles - library).norm().item() <= tol * library.norm().item()
