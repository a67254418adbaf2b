"""Spike Gram kernel at the edges of its tiles, harmonic passes and strips,
against the oracle's cosine form (vtem/dirichlet.py:272-350)."""
import numpy as np
import pytest

from oracle import vtem_oracle as O
from vtem_b200 import dirichlet
from vtem_b200._abi import call, dptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,Mt,lower,lamb,shift", [
    (1, 1, False, 0.0, 0.0), (2, 3, True, 0.5, 0.0), (63, 8, False, 0.25, 0.0), (64, 10, False, 0.0, 3.0),
    (65, 11, True, 0.25, 0.0), (129, 20, False, 0.25, 0.0), (193, 21, False, 0.0, 0.0), (321, 31, True, 0.0, 0.0),
    (2750, 8, False, 0.5, 0.0),       # more tiles than one a block: strips of four
])
def test_gram_tiles_match_oracle(n, Mt, lower, lamb, shift):
    rng = np.random.default_rng(n + Mt)
    N, Wt, T = 37, 2 * np.pi * 20, 0.4
    a = rng.uniform(0, T, n) + shift
    b = a + rng.uniform(0.003, 0.05, n)
    ind = rng.integers(0, N, n).astype(np.int32)                 # any order
    D = rng.standard_normal((N, N))                              # any matrix, not a symmetric one
    one = np.ones(N)
    cp = dirichlet.dirichlet(N, a, b, ind, one, one, one, one, Wt, Mt)
    cp.compute_G(D, lamb, lower_only=lower)
    G = cp.d_G.cpu().numpy()
    cp.d_G.fill_(7.0)                                            # and without the table of harmonics
    Dd = dirichlet._dev(D)
    call("vtb_compute_G", dptr(cp.d_tk1), dptr(cp.d_tk2), dptr(cp.d_neuron_ind), n, Wt, Mt, dptr(Dd), N, lamb, int(lower),
         dptr(cp.d_G), n, stream_ptr())
    G1 = cp.d_G.cpu().numpy()
    Go = O.compute_G(a, b, ind, D, Wt, Mt, lamb=lamb)
    # four cosines a harmonic, each off by its own rounding and its argument's, in both forms
    W, m, eps = Wt / Mt, np.arange(1, Mt + 1), np.finfo(np.float64).eps
    tol = 8 * eps * (2 / W ** 2) * ((1 + m * W * (T + shift)) / m ** 2).sum() * np.abs(D).max() + 4 * eps * lamb
    keep = np.tril(np.ones((n, n), bool)) if lower else np.ones((n, n), bool)
    assert np.abs(G - Go)[keep].max() <= tol
    assert np.abs(G1 - Go)[keep].max() <= tol
    assert np.all(G1[~keep] == 7.0)


@pytest.mark.parametrize("T,Mt,shift", [(0.3, 4, 0.0), (1.0, 8, 0.0), (3.0, 8, 100.0), (2.0, 12, 0.0)])
@pytest.mark.parametrize("table", [True, False])
def test_error_does_not_grow_with_time(T, Mt, shift, table):
    """Against the entries in extended precision: the interval's harmonics are
    powers and products of at most eight correctly rounded factors (two units of
    rounding each on average, squared entries: four in all), whatever phase m W t
    they stand for.  Cosines of rounded arguments are off by m W t units."""
    rng = np.random.default_rng(Mt)
    n, Wt, L = 300, 2 * np.pi * 20, np.longdouble
    a = rng.uniform(0, T, n) + shift
    b = a + rng.uniform(0.02, 0.06, n)
    W, one = Wt / Mt, np.ones(1)
    al, bl = a.astype(L) - L(a[0]), b.astype(L) - L(a[0])
    rows = [bl - al]
    for m in range(1, Mt + 1):
        k = m * L(W)
        rows += [np.sqrt(L(2)) * (np.sin(k * bl) - np.sin(k * al)) / k, np.sqrt(L(2)) * (np.cos(k * al) - np.cos(k * bl)) / k]
    R = np.stack(rows, 1)
    want = R @ R.T
    cp = dirichlet.dirichlet(1, a, b, np.zeros(n, np.int32), one, one, one, one, Wt, Mt)
    cp.compute_G(np.ones((1, 1)))
    if not table:
        Dd = dirichlet._dev(np.ones((1, 1)))
        call("vtb_compute_G", dptr(cp.d_tk1), dptr(cp.d_tk2), dptr(cp.d_neuron_ind), n, Wt, Mt, dptr(Dd), 1, 0.0, 0,
             dptr(cp.d_G), n, stream_ptr())
    G = cp.d_G.cpu().numpy()
    assert np.sqrt(((G - want) ** 2).sum() / (want ** 2).sum()) <= 4 * np.finfo(np.float64).eps
