"""The generic 3D step (a column march in z-chunks) against the oracle at sizes
around its choices: chunks of one, two and four planes, blocks of 32 x 8 columns
and of 256 columns in a plane's order, both with a remainder."""
import os

import numpy as np
import pytest

from gpu_util import orc, params, rel

pytestmark = pytest.mark.gpu


@pytest.fixture
def generic():
    os.environ["AXS_FORCE_CONFIG"] = "0,0,64"
    yield
    del os.environ["AXS_FORCE_CONFIG"]


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("N,stencils", [(4, (0,)), (6, (0, 1)), (10, (0, 3)), (16, (0, 2)), (32, (1,)), (34, (0, 3)), (44, (2,)),
                                        (54, (0,)), (58, (3,)), (60, (0,)), (62, (1,)), (64, (0, 3)), (66, (2,)), (96, (0,)),
                                        (162, (2,)), (170, (0,))])
def test_sizes_against_oracle(axs, oracle, generic, N, stencils, precision):
    for st in stencils:
        p = params(axs, 3, N, precision, stencil_setting=st)
        f = [np.random.default_rng(N + i).standard_normal((N, N, N)) for i in range(4)]
        if precision == 32:
            f = [a.astype(np.float32).astype(np.float64) for a in f]
        with axs.Lattice(p) as L:
            L.upload(*f)
            L.evolve(3)
            g = L.download()
            assert "generic" in L.describe()
        o = oracle.evolve(orc(p), *f, 3)
        for q in range(4):
            # the bounds of the step's other tests against the oracle
            assert rel(g[q], o[q]) <= (1e-12 if precision == 64 else 1e-5), (N, st, q)


def test_small_steps_are_short(axs, generic):
    """22^3 FP64 of radius 4: 5.7 us per step with chunks of one plane; 16 with four planes, each a trip to L2 after the
    other."""
    with axs.Lattice(params(axs, 3, 22, 64, stencil_setting=3)) as L:
        L.init_flat(1, 1.0)
        L.evolve(3)
        best = min(L.evolve_timed(20) for _ in range(8)) * 50
    assert best <= 11, best


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("N,stencils", [(6, (0, 1)), (10, (0, 3)), (22, (1, 3)), (30, (0,)), (34, (2,)), (38, (0, 3)), (42, (1,)),
                                        (54, (0, 3)), (66, (0,)), (72, (2,))])
def test_staged_marches_on_small_lattices(axs, oracle, N, stencils, precision):
    """The staged column marches (pi_n, energies, axion field) with chunks of two, four and eight planes and a remainder."""
    for st in stencils:
        p = params(axs, 3, N, precision, stencil_setting=st)
        with axs.Lattice(p) as L:
            L.init_flat(3, 1.0)
            L.evolve(4)
            g = L.download()
            en = L.energies()
            k, pk, cnt = L.axion_spectrum(8)
            tau = L.time[0]
            pin = [axs.PinnedBuffer(L.shape, np.float64 if precision == 64 else np.float32) for _ in range(4)]
            fn = axs._lib.axs_download if precision == 64 else axs._lib.axs_download_f32
            axs._check(fn(L._h, *[b.array.ctypes.data for b in pin]))
            for a, b in zip(g, pin):
                assert np.array_equal(a, b.array.astype(np.float64))
                b.free()
        op = orc(p)
        eo = oracle.energies(op, *g, tau)
        ko, pko, cnto = oracle.axion_spectrum(op, g[0], g[1], g[2], g[3], tau, 8)
        tol = 1e-12 if precision == 64 else 2e-6   # the bounds of the other energy and spectrum tests
        for q in range(3):
            assert abs(en[q] - eo[q]) <= 10 * tol * max(1e-3, abs(eo[q])), (N, st, q)
        assert np.array_equal(cnt, cnto)
        ok = cnto > 0
        assert rel(pk[ok], pko[ok]) <= (1e-10 if precision == 64 else 1e-4), (N, st)
