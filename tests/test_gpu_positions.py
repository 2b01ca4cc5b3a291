"""The flagged cells' list and the 2D neighbouring pairs against the mask itself,
at sizes around the 16-cell loads, the 512-cell warps and the 4096-cell chunks,
from few flagged cells to nearly all, for a search from psi and on a given
theta, and for repeated searches (the counters start at zero each time)."""
import numpy as np
import pytest

from gpu_util import params

pytestmark = pytest.mark.gpu


def pairs(mask):
    """s_run.cpp:101-109 over ascending offsets: consecutive entries one apart in a row, or one row apart in a column."""
    N = mask.shape[1]
    off = np.flatnonzero(mask.reshape(-1)).astype(np.int64)
    dx, dy = np.diff(off % N), np.diff(off // N)
    return int((((dy == 0) & (dx == 1)) | ((dy == 1) & (dx == 0))).sum())


@pytest.mark.parametrize("thr", [1, 60, 97])   # the share of flagged cells grows with the threshold percent
@pytest.mark.parametrize("nd,N,precision", [(2, 4, 64), (2, 6, 32), (2, 22, 32), (2, 30, 64), (2, 62, 64), (2, 64, 32),
                                            (2, 66, 32), (2, 130, 64), (2, 514, 32), (3, 4, 64), (3, 6, 32), (3, 10, 32),
                                            (3, 16, 64), (3, 18, 32), (3, 34, 64), (3, 66, 32)])
def test_positions_and_pairs_follow_the_mask(axs, nd, N, precision, thr):
    rng = np.random.default_rng(N + thr)
    p = params(axs, nd=nd, N=N, precision=precision, thr=thr)
    with axs.Lattice(p) as L:
        for theta in (None, rng.uniform(-np.pi, np.pi, L.shape), None):
            L.upload(*[rng.standard_normal(L.shape) for _ in range(4)])
            n, cores, mask = L.find_strings(theta=theta, want_mask=True)
            assert n == int(mask.sum())
            assert cores == (n - pairs(mask) if nd == 2 else n)
            got = L.string_positions()
            want = np.argwhere(mask)
            assert np.array_equal(got, want[:, ::-1] if nd == 2 else want)
            assert np.array_equal(L.string_positions(), got)
            n2, cores2, mask2 = L.find_strings(theta=theta, want_mask=True)
            assert (n2, cores2) == (n, cores) and np.array_equal(mask2, mask)


def test_sparse_columns(axs):
    """Flagged cells a row apart with other cells between them, next to the row's and the lattice's ends."""
    N = 64
    p = params(axs, nd=2, N=N)
    rng = np.random.default_rng(1)
    with axs.Lattice(p) as L:
        for _ in range(20):
            theta = np.zeros((N, N))
            for _ in range(12):   # a vortex flags the cells around it
                j, i = rng.integers(0, N, 2)
                theta[j, i], theta[(j + 1) % N, i] = 2.2, -2.2
                theta[(j + 2) % N, i] = rng.choice([0.0, 2.2])
            n, cores, mask = L.find_strings(theta=theta, want_mask=True)
            assert cores == n - pairs(mask)


@pytest.mark.parametrize("share", [2e-5, 1e-3, 0.03, 0.3])   # of the sites off a uniform angle
@pytest.mark.parametrize("N", [4, 16, 34, 256, 512, 1022, 1540])
def test_pairs_over_empty_stretches(axs, N, share):
    """Next entries in the same lane, another lane, a later warp's cells or none: few entries, far apart, also one row
    apart with nothing between."""
    rng = np.random.default_rng(N)
    with axs.Lattice(params(axs, nd=2, N=N, precision=32)) as L:
        off = rng.random(L.shape) < max(share, 1.0 / N ** 2)
        off[N // 2, N // 3] = off[N // 2 + 1, N // 3] = True   # stacked: entries N apart
        th = np.where(off, rng.uniform(-np.pi, np.pi, L.shape), 0.3)
        for theta in (None, th):
            L.upload(np.sin(th), np.cos(th), np.zeros(L.shape), np.zeros(L.shape))
            n, cores, mask = L.find_strings(theta=theta, want_mask=True)
            assert n == int(mask.sum()) and cores == n - pairs(mask)


def test_dense_search_takes_no_longer_than_its_cells(axs):
    """A 2D search reads each cell a few times whatever the share of flagged ones: noise within three times a uniform
    field's time at 8192^2 (noise takes 0.66 ms; 8.6 when each candidate pair looked at the N cells between)."""
    import time
    N = 8192
    rng = np.random.default_rng(1)
    best = []
    with axs.Lattice(params(axs, nd=2, N=N, precision=32)) as L:
        for a in (np.ones(L.shape, np.float32), rng.standard_normal(L.shape, np.float32)):
            L.upload(a, a[::-1], dtype=np.float32)
            t = []
            for _ in range(6):
                t0 = time.perf_counter()
                L.find_strings()
                t.append(time.perf_counter() - t0)
            best.append(min(t))
    assert best[1] <= 3 * best[0], best
