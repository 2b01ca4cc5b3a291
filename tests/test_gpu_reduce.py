"""Background means (s_run.cpp:135-150), energies and the finite check."""
import numpy as np
import pytest

from gpu_util import orc, params, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 2e-6)])
@pytest.mark.parametrize("nd,N,stencil,steps,prs,lap", [
    (2, 64, 0, 15, 1, 0), (3, 32, 0, 15, 1, 0),
    (3, 20, 0, 15, 1, 0),    # columns past the edge of the 32 x 8 blocks
    (3, 36, 0, 9, 0, 0),
    (3, 32, 0, 0, 1, 0),     # a fresh state: pih holds pi_0
    (3, 24, 1, 15, 1, 0),    # radius 2..4: the z-column march of that radius
    (3, 24, 2, 15, 1, 0),
    (3, 20, 3, 9, 0, 0),     # radius 4, columns past the edge of the blocks
    (3, 24, 3, 0, 1, 0),     # radius 4, fresh
    (3, 16, 0, 6, 1, 1),     # spectral Laplacian
    (2, 48, 3, 12, 1, 0),    # radius 4 in 2D
])
def test_background_and_energies(axs, oracle, precision, tol, nd, N, stencil, steps, prs, lap):
    """The device's background means take the mean of pi_n without the
    Laplacian part of the half kick (it sums to zero over the periodic
    lattice); the oracle averages the per-site pi_n that download() forms with
    the full stencil, so these cases also check that cancellation for every
    stencil and the spectral operator."""
    p = params(axs, nd, N, precision, T_initial=0.0, stencil_setting=stencil, prs=prs, laplacian=lap)
    op = orc(p)
    with axs.Lattice(p) as L:
        L.init_flat(6, 1.0)
        if steps:
            L.evolve(steps)
        g = L.download()
        tau, _ = L.time
        bg = L.background()
        en = L.energies()
    bo = oracle.background(op, *g)
    eo = oracle.energies(op, *g, tau)
    for q in range(6):
        assert abs(bg[q] - bo[q]) <= tol * max(1.0, abs(bo[q])), (q, bg[q], bo[q])
    for q in range(3):
        assert abs(en[q] - eo[q]) <= tol * max(1e-3, abs(eo[q])) * 10, (q, en[q], eo[q])


def test_finite_check_flags_seeded_nan(axs):
    p = params(axs, 3, 32, 64)
    with axs.Lattice(p) as L:
        L.init_flat(1, 1.0)
        assert L.check_finite()
        f = list(L.download())
        f[2][3, 4, 5] = np.nan
        L.upload(*f)
        assert not L.check_finite()


def test_background_angle_and_modulus_edge_cases(axs):
    """FP64 means of |theta| = |atan2(phi1, phi2)| and |phi| over sites that
    the table rotation serves and sites it hands to the library (zeros, values
    outside float range, the branch cut at theta = +-pi), against numpy, on a
    fresh state (pi_n is the uploaded pi)."""
    N = 4
    p = params(axs, 3, N, 64)
    rng = np.random.default_rng(5)
    p1 = rng.standard_normal(N ** 3)
    p2 = rng.standard_normal(N ** 3)
    special = [(0.0, 0.0), (0.0, -1.0), (-0.0, -1.0), (1e-13, -1.0), (-1e-13, -1.0), (1.0, 0.0), (-1.0, 0.0),
               (1e100, 3e100), (-2e-200, 1e-200), (3e-40, -5e-40), (1e-300, -2.0), (2.5, -1e-17)]
    for i, (a, b) in enumerate(special):
        p1[i], p2[i] = a, b
    z = np.zeros(N ** 3)
    with axs.Lattice(p) as L:
        L.upload(p1.reshape(N, N, N), p2.reshape(N, N, N), z.reshape(N, N, N), z.reshape(N, N, N))
        bg = L.background()
    th = np.mean(np.abs(np.arctan2(p1, p2)))
    ph = np.mean(np.sqrt(p1 * p1 + p2 * p2))
    assert abs(bg[4] - th) <= 1e-15 * th, (bg[4], th)
    assert abs(bg[5] - ph) <= 1e-15 * ph, (bg[5], ph)


@pytest.mark.parametrize("b", [1.0 + 2.0 ** -23 * (1 - 2.0 ** -20), 1.5, 3.0 - 2.0 ** -22 * (1 - 2.0 ** -20), 1.9999999])
@pytest.mark.parametrize("t", [3.0e-3, -1.0e-3, 7.0e-5, 1.0e-9])
def test_background_small_angle_to_double_precision(axs, t, b):
    """FP64 sites next to the positive phi2 axis: |theta| is the quotient's series alone, no table entry is added that
    would cover a short reciprocal. Every site is the same, 64 of them, so the mean is the site's value: three roundings of
    2^-53 for |theta|, one and a small part of one for |phi|."""
    a = t * b
    z = np.zeros((4, 4, 4))
    with axs.Lattice(params(axs, 3, 4, 64)) as L:
        L.upload(z + a, z + b, z, z)
        bg = L.background()
    la, lb = np.longdouble(a), np.longdouble(b)
    th, ph = abs(np.arctan2(la, lb)), np.sqrt(la * la + lb * lb)
    assert abs(bg[4] - th) <= 3.1 * 2.0 ** -53 * th, float((bg[4] - th) / th)
    assert abs(bg[5] - ph) <= 1.1 * 2.0 ** -53 * ph, float((bg[5] - ph) / ph)


def test_first_fp64_background_of_a_process(axs):
    """The call that brings the angle table to the device uses it on another stream at once: a new process's first call,
    and one from a second thread started with it, give what later calls give."""
    import subprocess
    import sys
    code = """
import sys, threading
sys.path[:0] = %r
import numpy as np, axs
rng = np.random.default_rng(0)
N = 8
f = [rng.standard_normal((N, N, N)) for _ in range(4)]
lats = [axs.Lattice(axs.default_params(NDIMS=3, N=N, precision=axs.F64)) for _ in range(2)]
for L in lats:
    L.upload(*f)
first = [None, None]
def go(i):
    first[i] = lats[i].background()
ts = [threading.Thread(target=go, args=(i,)) for i in range(2)]
[t.start() for t in ts]
[t.join() for t in ts]
again = lats[0].background()
assert np.array_equal(first[0], again) and np.array_equal(first[1], again), (first, again)
th = np.mean(np.abs(np.arctan2(f[0], f[1])))
assert abs(again[4] - th) <= 1e-14, (again[4], th)
""" % ([p for p in sys.path if p],)
    for _ in range(3):
        r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stderr


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("nd,N", [(2, 4), (2, 6), (3, 4), (3, 10)])
def test_finite_check_at_every_place(axs, nd, N, precision):
    """One NaN or infinity anywhere (first, last and other components of psi and of pih) is seen; the largest and smallest
    finite values are not."""
    dt = np.float32 if precision == 32 else np.float64
    info = np.finfo(dt)
    rng = np.random.default_rng(N)
    ok = [rng.choice([info.max, -info.max, info.tiny, -info.smallest_subnormal, 0.0, -0.0, 1.0], (N,) * nd).astype(dt) for _ in range(4)]
    with axs.Lattice(params(axs, nd, N, precision)) as L:
        L.upload(*ok, dtype=dt)
        assert L.check_finite()
        places = [0, 1, 2, 3, N ** nd - 2, N ** nd - 1, *rng.integers(0, N ** nd, 6)]
        for f in range(4):
            for at, bad in zip(places, [np.nan, np.inf, -np.inf] * 4):
                g = [a.copy() for a in ok]
                g[f].reshape(-1)[at] = bad
                L.upload(*g, dtype=dt)
                assert not L.check_finite(), (f, at, bad)
        L.upload(*ok, dtype=dt)
        assert L.check_finite()
