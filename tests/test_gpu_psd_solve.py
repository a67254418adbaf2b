"""Pseudoinverse solve: the low-rank path, and the matrices it has to leave to
the eigendecomposition, against a float64 eigendecomposition on the host
(vtem/utils/linalg.py:591-631, the rule s > rcond * s_0)."""
import numpy as np
import pytest
import torch

from vtem_b200 import linalg
from vtem_b200._abi import call, dptr, stream_ptr

pytestmark = pytest.mark.gpu
RCOND = 1e-8


def _matrix(n, w, seed, groups=0):
    """Symmetric n x n with the eigenvalues w (and zeros); ``groups``: rows come in near-parallel groups."""
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((n, len(w)))
    if groups:
        A = A[np.arange(n) % groups] + 1e-2 * rng.standard_normal((n, len(w)))
    Q, _ = np.linalg.qr(A)
    G = (Q * w) @ Q.T
    return 0.5 * (G + G.T), Q


def _solve(G, q):
    Gd = torch.as_tensor(np.tril(G) + np.triu(np.full(G.shape, np.nan), 1), device="cuda")
    nb = np.zeros(1, np.int64)
    n = G.shape[0]
    call("vtb_solve_psd_workspace", n, nb.ctypes.data)
    work = torch.full((int(nb[0]),), 255, dtype=torch.uint8, device="cuda")
    qd = torch.as_tensor(q, device="cuda")
    c = torch.empty(n, dtype=torch.float64, device="cuda")
    kept = torch.zeros(1, dtype=torch.int32, device="cuda")
    ok = np.zeros(1, np.int32)
    call("vtb_solve_psd", dptr(Gd), n, dptr(qd), dptr(c), n, RCOND, dptr(work), work.numel(), dptr(kept), ok.ctypes.data,
         stream_ptr())
    assert torch.equal(torch.tril(Gd), torch.as_tensor(np.tril(G), device="cuda"))
    return bool(ok[0]), c.cpu().numpy(), int(kept.item())


@pytest.mark.parametrize("n,r,cond,groups", [(1, 0, 1, 0), (64, 3, 10, 0), (256, 1, 1, 0), (257, 31, 1e2, 0), (300, 32, 1e3, 0),
                                             (300, 33, 1e4, 7), (777, 100, 1e5, 0), (1000, 261, 1e3, 40),
                                             (600, 300, 1e3, 0)])
def test_low_rank_solve(n, r, cond, groups):
    w = np.geomspace(2.0, 2.0 / cond, r) if r else np.zeros(0)
    G, Q = _matrix(n, w, n + r, groups)
    x = Q @ np.random.default_rng(r).standard_normal(r)
    q = G @ x
    ok, c, kept = _solve(G, q)
    if r == 0:
        assert not ok                                            # nothing to factor
        return
    assert ok and kept == r
    # backward error of a few n eps |G|, amplified by the condition number, in G (on both sides) and q
    assert np.linalg.norm(c - x) <= 4 * np.finfo(np.float64).eps * np.sqrt(n) * 8 * cond * np.linalg.norm(x)


def _case(kind, n):
    rng = np.random.default_rng(5)
    if kind == "full":
        return _matrix(n, np.geomspace(1.0, 1e-3, n), 1)[0]
    if kind == "indefinite":
        return _matrix(n, np.concatenate([np.geomspace(1.0, 1e-2, 20), -np.geomspace(1.0, 1e-2, 20)]), 2)[0]
    if kind == "hidden":                                         # indefinite behind zero diagonal entries
        G = np.zeros((n, n))
        G[0, 0] = 1.0
        G[5, 9] = G[9, 5] = 0.5
        return G
    if kind == "truncates":                                      # eigenvalues on both sides of the rule
        return _matrix(n, np.concatenate([np.geomspace(1.0, 1e-3, 30), [1e-10, 1e-11]]), 3)[0]
    if kind == "zero":
        return np.zeros((n, n))
    return np.diag(rng.uniform(0.5, 1.0, n))                     # "diagonal"


@pytest.mark.parametrize("kind", ["full", "indefinite", "hidden", "truncates", "zero", "diagonal"])
def test_left_to_the_eigendecomposition(kind):
    n = 320
    G = _case(kind, n)
    q = np.random.default_rng(0).standard_normal(n)
    ok, _, _ = _solve(G, q)
    assert not ok
    c, kept = linalg.solve_eq_sym(torch.as_tensor(G, device="cuda"), torch.as_tensor(q, device="cuda").reshape(-1, 1),
                                  rcond=RCOND, return_kept=True)
    w, V = np.linalg.eigh(G)
    s = np.abs(w)
    keep = s > RCOND * s.max()
    # eigenvalues -s as the reference's singular values: U diag(1/s) U^T q on the kept ones
    want = V[:, keep] @ ((V[:, keep].T @ q) / s[keep])
    assert kept == keep.sum()
    size = max(np.linalg.norm(want), 1e-300)
    assert np.linalg.norm(c.cpu().numpy().ravel() - want) <= 1e-9 * size


@pytest.mark.parametrize("s,t", [(1, 1), (1, -1), (-1, 1), (-1, -1)])
def test_cycle_behind_zero_diagonal(s, t):
    """A four-cycle on rows of zero diagonal, the rest of low rank: no diagonal
    entry shows its eigenvalues +-2a, and a vector of +-1 with v5 v6 = s and
    v9 v10 = t lies in its null space."""
    n, r = 320, 20
    rng = np.random.default_rng(8)
    A = rng.standard_normal((n, r))
    A[[5, 6, 9, 10]] = 0.0
    Q, _ = np.linalg.qr(A)
    G = (Q * np.geomspace(1.0, 1e-2, r)) @ Q.T
    G = 0.5 * (G + G.T)
    for i, j, e in ((5, 9, 0.2), (5, 10, -0.2 * t), (6, 9, -0.2 * s), (6, 10, 0.2 * s * t)):
        G[i, j] = G[j, i] = e
    q = rng.standard_normal(n)
    assert not _solve(G, q)[0]
    c, kept = linalg.solve_eq_sym(torch.as_tensor(G, device="cuda"), torch.as_tensor(q, device="cuda").reshape(-1, 1),
                                  rcond=RCOND, return_kept=True)
    w, V = np.linalg.eigh(G)
    keep = np.abs(w) > RCOND * np.abs(w).max()
    want = V[:, keep] @ ((V[:, keep].T @ q) / np.abs(w[keep]))
    assert kept == keep.sum() == r + 2
    assert np.linalg.norm(c.cpu().numpy().ravel() - want) <= 1e-9 * np.linalg.norm(want)


@pytest.mark.parametrize("n,r", [(400, 60), (1900, 261)])
@pytest.mark.parametrize("cond", [1e2, 1e4, 1e6])
def test_as_close_as_the_eigendecomposition(n, r, cond):
    """Right-hand sides that weigh the spectrum differently, in G's range and
    out of it: the error against the known solution, which the rounding of G
    is part of on both sides, is that of the eigendecomposition."""
    w = np.geomspace(1.0, 1.0 / cond, r)
    G, Q = _matrix(n, w, n + r)
    rng = np.random.default_rng(4)
    for q in (Q @ (w * rng.standard_normal(r)), Q @ rng.standard_normal(r), rng.standard_normal(n)):
        want = Q @ ((Q.T @ q) / w)
        error = lambda c: np.linalg.norm(c - want) / np.linalg.norm(want)
        ok, c, kept = _solve(G, q)
        assert ok and kept == r
        nb = np.zeros(1, np.int64)
        call("vtb_solve_eq_sym_workspace", n, nb.ctypes.data)
        work = torch.empty(int(nb[0]), dtype=torch.uint8, device="cuda")
        Gd, qd = torch.as_tensor(G, device="cuda"), torch.as_tensor(q, device="cuda")
        ce = torch.empty_like(qd)
        call("vtb_solve_eq_sym", dptr(Gd), n, dptr(qd), dptr(ce), n, RCOND, dptr(work), work.numel(), None, stream_ptr())
        assert error(c) <= 2 * error(ce.cpu().numpy())
