"""The spectrum binner's row groups (up to four rows of the half spectrum with
the same |n|^2 at every ix, binned together): slices of one mode and ragged
ones, groups of one, two and four rows, rows staged four and (many bins) two at
a time, slices on both sides of 16 modes. Against the oracle, counts equal, with the bounds of the other spectrum tests: FP64 1e-11
(axion 1e-10), FP32 1e-5 (axion 1e-4) relative."""
import numpy as np
import pytest

from gpu_util import orc, params, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("nd,N,nbins", [(3, 4, 12), (3, 6, 12), (3, 10, 12), (3, 34, 12), (3, 66, 12), (3, 126, 12),
                                        (3, 34, 1300), (2, 6, 12), (2, 250, 12), (2, 958, 12), (2, 962, 12)])
def test_groups_of_rows(axs, oracle, nd, N, nbins, precision):
    p = params(axs, nd, N, precision, T_initial=0.0)
    op = orc(params(axs, nd, N, 64, T_initial=0.0))
    with axs.Lattice(p) as L:
        L.init_flat(5, 1.0)
        L.evolve(2)
        tau, _ = L.time
        g = L.download()
        first = L.powerspec(1), L.axion_spectrum(nbins)
        again = L.powerspec(1), L.axion_spectrum(nbins)
    for a, b in zip(first, again):   # a later call of the same binning: the same bits
        for x, y in zip(a, b):
            assert np.array_equal(x, y, equal_nan=True)
    tol = 1e-11 if precision == 64 else 1e-5
    pk, ks, cnt = first[0]
    pko, kso, cnto = oracle.powerspec(op, g[1])
    ok = cnto > 0
    assert np.array_equal(cnt, cnto)
    assert rel(pk[ok], pko[ok]) <= tol and rel(ks[ok], kso[ok]) <= 1e-11
    k, apk, acnt = first[1]
    ko, apko, acnto = oracle.axion_spectrum(op, *g, tau, nbins)
    ok = acnto > 0
    assert np.array_equal(acnt, acnto)
    assert rel(apk[ok], apko[ok]) <= (1e-10 if precision == 64 else 1e-4) and rel(k[ok], ko[ok]) <= 1e-11


@pytest.mark.parametrize("nd,N,precision,nbins", [(2, 2600, 64, 700), (2, 2712, 64, 12), (2, 250, 32, 3000), (3, 34, 64, 2100),
                                                  (3, 66, 32, 4000)])
def test_bins_in_passes(axs, oracle, nd, N, precision, nbins):
    """More bins than one pass holds (the reference's at 2600^2 and, with rows in segments, 2712^2; logarithmic ones from
    about 2000): each pass takes only the slices that hold its modes."""
    test_groups_of_rows(axs, oracle, nd, N, nbins, precision)
