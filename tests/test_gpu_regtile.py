"""Several 3D steps per pass with the tile in registers give the bits of the
generic kernel: sizes around the tiles' edges (regions of 64 columns and 32, 40
or 48 rows; halos that wrap small lattices more than once), z-chunks down to two
planes, intervals of every length modulo the steps per pass, both forms of the
equation, and as one table over an uneven ensemble."""
import os

import numpy as np
import pytest

from gpu_util import orc, params

pytestmark = pytest.mark.gpu
VARIANTS = (58, 59, 60, 61)


def forced(force, fn):
    prev = os.environ.get("AXS_FORCE_CONFIG")
    os.environ["AXS_FORCE_CONFIG"] = force
    try:
        return fn()
    finally:
        if prev is None:
            del os.environ["AXS_FORCE_CONFIG"]
        else:
            os.environ["AXS_FORCE_CONFIG"] = prev


@pytest.mark.parametrize("N,zchunk,form", [(16, 2, 0), (18, 32, 0), (34, 4, 0), (54, 16, 1), (56, 8, 0), (58, 32, 0), (60, 64, 0),
                                           (66, 8, 0), (112, 32, 0), (130, 64, 0)])
def test_register_tiles_bit_identical(axs, oracle, N, zchunk, form):
    p = params(axs, nd=3, N=N, precision=32, form=form)
    f = oracle.init_thermal(orc(p), 3)

    def run():
        with axs.Lattice(p) as L:
            L.upload(*f)
            for n in (2, 1, 3, 4, 5, 6, 7):
                L.evolve(n)
            return L.describe(), L.time, L.download()

    d0, t0, want = forced("0,0,0", run)
    assert "generic" in d0
    for v in VARIANTS:
        d, t, got = forced("1,%d,%d" % (v, zchunk), run)
        assert "register-tile z-march variant %d" % v in d, d
        assert t == t0
        for a, b in zip(got, want):
            assert np.array_equal(a, b), v


@pytest.mark.parametrize("variant", VARIANTS)
def test_ensemble_on_register_tiles(axs, oracle, variant):
    plist = [params(axs, nd=3, N=n, precision=32, lambda_=lam) for n, lam in ((64, 1.0), (18, 0.5), (50, 2.0), (96, 4.0))]
    fields = [oracle.init_thermal(orc(p), 9 + i) for i, p in enumerate(plist)]

    def ensemble():
        E = axs.Ensemble(plist)
        for m, f in zip(E.members, fields):
            m.upload(*f)
        E.evolve(6)
        E.evolve(5)
        d, out = E.describe(), [m.download() for m in E.members]
        E.close()
        return d, out

    def alone(p, f):
        with axs.Lattice(p) as L:
            L.upload(*f)
            L.evolve(11)
            return L.download()

    d, got = forced("1,%d,32" % variant, ensemble)
    assert "register-tile" in d
    for p, f, g in zip(plist, fields, got):
        for a, b in zip(g, forced("0,0,0", lambda: alone(p, f))):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("N", [112, 250, 320, 384])
def test_tuned_intervals_of_every_length(axs, N):
    """A tuned lattice takes an interval in passes of its register tiles and, where they are faster, of a shared-memory
    kernel for one or two steps: intervals of 1 to 8, 20, 25 and 26 steps give the bits of the generic kernel."""
    p = params(axs, 3, N, 32)
    f = [np.random.default_rng(i).standard_normal((N, N, N)).astype(np.float32) for i in range(4)]
    n = (1, 2, 1, 3, 4, 5, 2, 6, 7, 8, 20, 25, 26) if N < 300 else (1, 2, 4, 7, 20)
    out = []
    for force in (None, "0,0,64"):
        if force:
            os.environ["AXS_FORCE_CONFIG"] = force
        try:
            with axs.Lattice(p) as L:
                L.upload(*f, dtype=np.float32)
                for k in n:
                    L.evolve(k)
                out.append((L.download(dtype=np.float32), L.time, L.describe()))
        finally:
            os.environ.pop("AXS_FORCE_CONFIG", None)
    assert out[0][1] == out[1][1]
    for a, b in zip(out[0][0], out[1][0]):
        assert np.array_equal(a, b), out[0][2]


def test_tuned_ensemble_intervals(axs):
    """The same for an ensemble of mixed sizes, against the members alone."""
    ps = [params(axs, 3, N, 32) for N in (96, 200, 128, 64)]
    with axs.Ensemble(ps) as E:
        for i, m in enumerate(E.members):
            m.init_flat(i, 1.0)
        for k in (1, 2, 1, 4, 3, 5, 20):
            E.evolve(k)
        d, out = E.describe(), [m.download(dtype=np.float32) for m in E.members]
    for i, p in enumerate(ps):
        with axs.Lattice(p) as L:
            L.init_flat(i, 1.0)
            L.evolve(36)
            for a, b in zip(L.download(dtype=np.float32), out[i]):
                assert np.array_equal(a, b), d


def test_short_intervals_keep_the_two_step_kernels_times(axs):
    """Intervals of one and two steps at 512^3: 0.67 and 0.75 ms by the shared-memory kernels, 0.80 and 1.01 on register
    tiles alone. A third step costs less than half a step more."""
    with axs.Lattice(params(axs, 3, 512, 32)) as L:
        L.init_flat(1, 1.0)
        L.autotune()   # also where the environment turns it off for the first step
        L.evolve(3)
        t = {}
        for k in (1, 2, 3):
            for _ in range(3):
                L.evolve_timed(k)
            t[k] = min(L.evolve_timed(k) for _ in range(10))
    assert t[2] <= 1.25 * t[1] and t[1] <= 0.72 * t[3], t
