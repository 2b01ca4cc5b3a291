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
