"""2D steps, several per launch: the steps of one call in one or a few launches
give the bits of one launch per step, for every stencil radius and precision,
at sizes around the tiles' edges (regions of 32 and 64 sites, tiles from 8
sites, halos that wrap a lattice smaller than the region more than once), and
match the oracle within 1e-12 after 10 steps."""
import numpy as np
import pytest

from gpu_util import orc, params, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("stencil,N", [(0, 4), (0, 6), (0, 26), (0, 30), (0, 62), (0, 64), (0, 66), (0, 128), (0, 502),
                                       (1, 6), (1, 60), (1, 130), (1, 276), (2, 8), (2, 54), (2, 180), (3, 10), (3, 58),
                                       (3, 108), (3, 110), (3, 200)])
def test_steps_per_launch_bit_identical(axs, oracle, precision, stencil, N):
    p = params(axs, nd=2, N=N, precision=precision, stencil_setting=stencil)
    f = oracle.init_thermal(orc(p), 3)
    outs = []
    for calls in ([10, 3], [1] * 13, [2, 11], [12, 1]):
        with axs.Lattice(p) as L:
            L.upload(*f)
            for i, n in enumerate(calls):
                L.evolve(n)
                if i == 0 and n == 10 and precision == 64:
                    want = oracle.evolve(orc(p), *f, 10)
                    for a, b in zip(L.download(), want):
                        assert rel(a, b) <= 1e-12
            outs.append((L.time, L.download()))
    for t, o in outs[1:]:
        assert t == outs[0][0]
        for a, b in zip(o, outs[0][1]):
            assert np.array_equal(a, b)


def test_ensemble_of_uneven_2d_lattices(axs, oracle):
    """Members whose launches would take different numbers of steps advance together and keep the bits of a lattice alone."""
    sizes = (6, 64, 130, 400)
    plist = [params(axs, nd=2, N=n, precision=32) for n in sizes]
    fields = [oracle.init_thermal(orc(p), 5 + i) for i, p in enumerate(plist)]
    E = axs.Ensemble(plist)
    for m, f in zip(E.members, fields):
        m.upload(*f)
    E.evolve(9)
    E.evolve(20)
    got = [m.download() for m in E.members]
    E.close()
    for p, f, g in zip(plist, fields, got):
        with axs.Lattice(p) as L:
            L.upload(*f)
            L.evolve(29)
            for a, b in zip(g, L.download()):
                assert np.array_equal(a, b)


def test_table_follows_a_reset_clock(axs, oracle):
    """The coefficients formed ahead serve only the clock they were formed for."""
    p = params(axs, nd=2, N=64)
    f = oracle.init_thermal(orc(p), 3)
    outs = []
    for reset in (False, True):
        with axs.Lattice(p) as L:
            L.upload(*f)
            if reset:   # leaves tables for other clocks behind
                L.evolve(7)
                L.set_time(2.5, 0)
                L.evolve(5)
                L.set_time(1.0, 0)
                L.upload(*f)
            L.evolve(11)
            outs.append(L.download())
    for a, b in zip(*outs):
        assert np.array_equal(a, b)
