"""Batched tile Cholesky: the host's plan of its CTAs, and its solves against
a float64 solve on the host."""
import numpy as np
import pytest
import torch

from vtem_b200 import _abi
from vtem_b200._abi import call, dptr, lib, stream_ptr
from vtem_b200.batch import INV_SYSTEM


def _plan(Ks):
    n = len(Ks)
    Ks = np.array(Ks, np.int32)
    host = np.zeros(int(lib().vtb_chol_batch_bytes(n)), np.uint8)
    grid = np.zeros(1, np.int32)
    one = np.full(n, 256, np.uint64)
    ld = Ks.astype(np.int64)
    ids = 4096 * (1 + np.arange(n)).astype(np.uint64)       # tells the systems apart in the plan's order
    p = lambda a: a.ctypes.data
    rc = np.ones(n)
    call("vtb_chol_batch_build", p(host), n, p(ids), p(ld), p(Ks), p(one), p(one), 256, p(one), p(one), p(rc), p(grid))
    size = (host.size - 296 * 16) // n
    order = [int(host[i * size:i * size + 8].view(np.uint64)[0]) // 4096 - 1 for i in range(n)]
    teams = host[n * size:].view(np.int32).reshape(-1, 4)[:int(grid[0])]
    return order, teams


@pytest.mark.parametrize("Ks", [[1], [64], [65], [129], [1921], [63, 65, 129, 700], [261] * 12, list(range(1, 400, 2)),
                                [1921] * 49, [1921] * 50, [1] * 300 + [1921]])
def test_plan_covers_every_system_once(Ks):
    order, teams = _plan(Ks)
    assert sorted(order) == list(range(len(Ks)))
    assert 1 <= len(teams) <= 296
    seen = []
    b = 0
    while b < len(teams):
        first, count, rank, size = teams[b]
        assert rank == 0 and count >= 1
        assert all(tuple(teams[b + r]) == (first, count, r, size) for r in range(size))
        for i in range(first, first + count):
            T = -(-Ks[order[i]] // 64)
            assert size >= min(T, 3)                         # a worker for T = 2, both pools from T = 3
        seen += list(range(first, first + count))
        b += size
    assert sorted(seen) == list(range(len(Ks)))


class _Batch(object):
    def __init__(self, mats, rcond=1e-6):
        n = len(mats)
        self.n = n
        self.K = np.array([m.shape[0] for m in mats], np.int32)
        self.ld = np.array([(k + 3) // 4 * 4 for k in self.K], np.int64)
        self.A = [torch.zeros((int(k), int(l)), dtype=torch.float32, device="cuda") for k, l in zip(self.K, self.ld)]
        for a, m in zip(self.A, mats):
            a[:, :m.shape[0]] = torch.as_tensor(m, device="cuda")
        f = lambda name, dt: [torch.zeros(int(getattr(lib(), name)(int(k))), dtype=dt, device="cuda") for k in self.K]
        self.dinv, self.linv = f("vtb_chol_dinv_floats", torch.float32), f("vtb_chol_inverse_floats", torch.float32)
        self.sw = f("vtb_chol_solve_inverse_bytes", torch.uint8)
        self.status = torch.zeros(n, dtype=torch.int32, device="cuda")
        self.piv = torch.zeros(2 * n, dtype=torch.float64, device="cuda")
        nb = np.zeros(1, np.int64)
        call("vtb_chol_batch_work_bytes", n, self.K.ctypes.data, nb.ctypes.data)
        self.work = torch.empty(int(nb[0]), dtype=torch.uint8, device="cuda")
        host = np.zeros(int(lib().vtb_chol_batch_bytes(n)), np.uint8)
        grid = np.zeros(1, np.int32)
        u = lambda ts: np.array([t.data_ptr() for t in ts], np.uint64)
        args = [u(self.A), self.ld, self.K, u(self.dinv), u(self.linv),
                np.array([self.status.data_ptr() + 4 * i for i in range(n)], np.uint64),
                np.array([self.piv.data_ptr() + 16 * i for i in range(n)], np.uint64), np.full(n, rcond)]
        a = [x.ctypes.data for x in args]
        call("vtb_chol_batch_build", host.ctypes.data, n, a[0], a[1], a[2], a[3], a[4], self.work.data_ptr(), a[5], a[6],
             a[7], grid.ctypes.data)
        self.grid = int(grid[0])
        self.desc = torch.as_tensor(host).cuda()
        rng = np.random.default_rng(n)
        self.b = [rng.standard_normal(int(k)) for k in self.K]
        self.x = [[torch.as_tensor(b, device="cuda").clone() for b in self.b] for _ in range(2)]
        tiles = (self.K.astype(np.int64) + 63) // 64
        tiles = tiles * (tiles + 1) // 2
        self.tiles = int(tiles.sum())
        d = np.zeros(n, INV_SYSTEM)
        for i in range(n):
            d[i] = (self.linv[i].data_ptr(), self.sw[i].data_ptr(), (self.x[0][i].data_ptr(), self.x[1][i].data_ptr()),
                    0, self.K[i], tiles[:i].sum())
        self.systems = torch.as_tensor(np.frombuffer(d.tobytes(), np.uint8).copy()).cuda()

    def factor(self):
        self.status.zero_()
        call("vtb_chol_batch_factor", dptr(self.desc), self.n, self.grid, dptr(self.work), self.work.numel(), stream_ptr())
        torch.cuda.synchronize()
        return self.status.cpu().numpy()

    def solve(self, which):
        call("vtb_chol_batch_solve", dptr(self.systems), self.n, self.tiles, which, stream_ptr())
        return [x.cpu().numpy() for x in self.x[which]]


def _spd(K, cond, seed):
    rng = np.random.default_rng(seed)
    Q, _ = np.linalg.qr(rng.standard_normal((K, K)))
    return (Q * np.geomspace(1.0, 1.0 / cond, K)) @ Q.T


@pytest.mark.gpu
@pytest.mark.parametrize("Ks", [[1, 63, 64, 65, 127, 128, 129, 193], [300, 1, 517, 64], [130] * 60 + [65] * 20 + [3] * 30])
def test_batch_solves(Ks):
    cond = 30.0
    mats = [_spd(k, cond, i) for i, k in enumerate(Ks)]
    bt = _Batch(mats)
    assert np.all(bt.factor() == 0)
    for which in (1, 0):
        for m, b, x in zip(mats, bt.b, bt.solve(which)):
            want = np.linalg.solve(m, b)
            # a float32 factor and its inverse: K roundings amplified by the condition number
            assert np.linalg.norm(x - want) <= 8 * 6e-8 * (len(b) + 8) ** 0.5 * cond * np.linalg.norm(want)


@pytest.mark.gpu
def test_batch_refusals_stay_with_their_system():
    mats = [_spd(k, 30.0, k) for k in (100, 200, 260, 64)]
    mats[1] = mats[1] - 2.0 * np.eye(200)                        # not positive definite
    mats[2] = np.diag(np.concatenate([np.ones(130), np.full(130, 1e-5)]))   # pivots 1e5 apart
    bt = _Batch(mats, rcond=1e-4)
    assert list(bt.factor()) == [0, 1, 2, 0]
    x = bt.solve(0)
    for i in (0, 3):
        want = np.linalg.solve(mats[i], bt.b[i])
        assert np.linalg.norm(x[i] - want) <= 1e-3 * np.linalg.norm(want)


@pytest.mark.gpu
def test_batch_wait_limit_runs_out():
    mats = [_spd(k, 30.0, k) for k in (700, 500, 300)]
    bt = _Batch(mats)
    with _abi.wait_limit(1):
        st = bt.factor()
    assert np.any(st == 3)
    for a, m in zip(bt.A, mats):
        a[:, :m.shape[0]] = torch.as_tensor(m, device="cuda")
    assert np.all(bt.factor() == 0)
    for m, b, x in zip(mats, bt.b, bt.solve(0)):
        want = np.linalg.solve(m, b)
        assert np.linalg.norm(x - want) <= 1e-3 * np.linalg.norm(want)
