"""3D lattices whose size no tile divides: the z-march kernels on overlapping
tiles (the last one of a row or column starts at N - tx or N - ty, the
momentum out of place) give the bits of the generic per-site kernel, at sizes
just above and below the tiles', with an odd last step, calls in between and
as members of an ensemble."""
import os

import numpy as np
import pytest

from gpu_util import orc, params

pytestmark = pytest.mark.gpu


def evolved(axs, p, f, force, calls=(6, 5, 1)):
    prev = os.environ.get("AXS_FORCE_CONFIG")
    os.environ["AXS_FORCE_CONFIG"] = force
    try:
        with axs.Lattice(p) as L:
            L.upload(*f)
            for n in calls:
                L.evolve(n)
                L.background()
            return L.describe(), L.download()
    finally:
        if prev is None:
            del os.environ["AXS_FORCE_CONFIG"]
        else:
            os.environ["AXS_FORCE_CONFIG"] = prev


# variants of axs_step.cu's table: one-step (0, 5, 16, 27, 38), two-step (17, 30, 31, 39), radius 2 (21, 41, 50),
# radius 3 (22, 23, 51) and 4 (26, 44); 23 does not fit shared memory in FP64
@pytest.mark.parametrize("precision,stencil,N,variants", [
    (32, 0, 18, (27, 31, 38, 39)), (32, 0, 30, (16, 30, 39)), (32, 0, 50, (5, 16, 17, 30, 31, 39)),
    (32, 0, 66, (0, 16, 30, 39)), (32, 0, 70, (30, 31, 39)), (64, 0, 10, (16, 27)), (64, 0, 42, (0, 16, 27, 38)),
    (32, 1, 18, (21, 41)), (32, 1, 70, (21, 41, 50)), (64, 1, 22, (21,)), (32, 2, 28, (23, 51)), (64, 2, 20, (22,)),
    (32, 3, 36, (26, 44)), (64, 3, 20, (26,))])
def test_overlapping_tiles_bit_identical(axs, oracle, precision, stencil, N, variants):
    p = params(axs, nd=3, N=N, precision=precision, stencil_setting=stencil)
    f = oracle.init_thermal(orc(p), 3)
    d0, want = evolved(axs, p, f, "0,0,0")
    assert "generic" in d0
    for v in variants:
        d, got = evolved(axs, p, f, "1,%d,32" % v)
        assert "z-march variant %d" % v in d, d
        for a, b in zip(got, want):
            assert np.array_equal(a, b), v


def test_ensemble_with_untiled_members(axs, oracle):
    """Exact and overlapping members in one table, for an in-place one-step variant and a two-step one."""
    plist = [params(axs, nd=3, N=n, precision=32) for n in (64, 34, 50)]
    fields = [oracle.init_thermal(orc(p), 9 + i) for i, p in enumerate(plist)]
    for force in ("1,27,32", "1,39,32"):
        os.environ["AXS_FORCE_CONFIG"] = force
        try:
            E = axs.Ensemble(plist)
            for m, f in zip(E.members, fields):
                m.upload(*f)
            E.evolve(6)
            E.evolve(5)
            got = [m.download() for m in E.members]
            E.close()
        finally:
            del os.environ["AXS_FORCE_CONFIG"]
        for p, f, g in zip(plist, fields, got):
            _, want = evolved(axs, p, f, "0,0,0", calls=(11,))
            for a, b in zip(g, want):
                assert np.array_equal(a, b), force
