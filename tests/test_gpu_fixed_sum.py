"""The FP64 neighbour sums, formed on the integer pipe (sum_fixed), through
axs_laplacian at dx = 1, against exact sums (rational arithmetic).

With M the largest neighbour's magnitude a term loses at most 2^-59 M and the
sum S is rounded once (half an ulp: 2^-53 |S|); the Laplacian S - 2 d c adds
one more rounding (2^-53 |L|). Terms all tiny or huge take FP64 additions
instead, each within 2^-53 of a partial sum no larger than the terms'
magnitudes together (and within half the smallest subnormal).
"""
from fractions import Fraction

import numpy as np
import pytest

from gpu_util import params

pytestmark = pytest.mark.gpu


def field(kind, shape, rng):
    r = rng.uniform(-1.0, 1.0, shape)
    if kind == "random":
        return r
    if kind == "smooth":   # nearly equal terms: every partial sum rounds
        return 1.0 + 1e-7 * r
    if kind == "wide":     # neighbours up to 2^80 apart
        return np.ldexp(r, rng.integers(-40, 41, shape))
    if kind == "integers":
        return rng.integers(-1000, 1001, shape).astype(np.float64)
    if kind == "sparse":   # zeros of either sign among a few values
        return np.where(rng.random(shape) < 0.1, r, np.copysign(0.0, r))
    if kind == "cancel":   # pairs that cancel but for their last places
        return np.where(np.indices(shape).sum(0) % 2 == 0, 1.0, -1.0) * (0.3 + 2.0 ** -50 * rng.integers(0, 4, shape))
    if kind == "edge_low":   # around the exponent below which the FP64 additions take over
        return np.ldexp(r, -1023 + rng.integers(60, 69, shape))
    if kind == "tiny":
        return r * 1e-309
    if kind == "edge_high":
        return np.ldexp(r, rng.integers(1004, 1012, shape))
    raise KeyError(kind)


@pytest.mark.parametrize("nd,N", [(2, 10), (3, 6)])
@pytest.mark.parametrize("kind", ["random", "smooth", "wide", "integers", "sparse", "cancel", "edge_low", "tiny",
                                  "edge_high"])
def test_fixed_point_sum(axs, kind, nd, N):
    rng = np.random.default_rng(5)
    f = field(kind, (N,) * nd, rng)
    with axs.Lattice(params(axs, nd=nd, N=N, precision=64, space_step=1.0)) as L:
        L.upload(f, np.zeros_like(f))
        got = L.laplacian(axs.PHI1)
    nb = np.stack([np.roll(f, s, d) for d in range(nd) for s in (1, -1)], -1)
    for at in np.ndindex(f.shape):
        v = [float(x) for x in nb[at]]
        exact = sum(map(Fraction, v))
        S, want = float(exact), exact - 2 * nd * Fraction(float(f[at]))
        big, total = max(abs(x) for x in v), sum(abs(x) for x in v)
        # exponent field below 64 or above 0x7ef: the FP64 additions
        fp64 = not 2.0 ** (64 - 1023) <= big < 2.0 ** (0x7f0 - 1023)
        err = 5 * 2.0 ** -53 * total + 5 * 2.0 ** -1075 if fp64 else len(v) * 2.0 ** -59 * big + 2.0 ** -53 * abs(S)
        assert abs(Fraction(float(got[at])) - want) <= (err + 2.0 ** -53 * abs(float(want))) * (1 + 2.0 ** -40) + 2.0 ** -1074, (at, v)
    if kind == "integers":
        assert np.array_equal(got, nb.sum(-1) - 2 * nd * f)   # exact sums stay exact


@pytest.mark.parametrize("nd,N", [(2, 12), (3, 8)])
@pytest.mark.parametrize("depth", [8, 13, 28, 60, 200])   # the small terms' exponents below the cancelling ones'
def test_fixed_point_sum_of_cancelling_terms(axs, depth, nd, N):
    """Every second site is 0 and its neighbours are +-0.7 or far smaller, so the large ones often cancel exactly. The sum
    keeps its own relative accuracy: below 2^-14 of the largest term's power of two by rounding alone (or 2^-100 of that
    term), above it within the alignment's loss."""
    rng = np.random.default_rng(depth)
    odd = np.indices((N,) * nd).sum(0) % 2 == 1
    big = 0.7 * rng.choice([-1.0, 1.0], (N,) * nd)
    f = np.where(odd, np.where(rng.random((N,) * nd) < 0.5, big, np.ldexp(rng.uniform(-1.0, 1.0, (N,) * nd), -depth)), 0.0)
    with axs.Lattice(params(axs, nd=nd, N=N, precision=64, space_step=1.0)) as L:
        L.upload(f, np.zeros_like(f))
        got = L.laplacian(axs.PHI1)
    nb = np.stack([np.roll(f, s, d) for d in range(nd) for s in (1, -1)], -1)
    cancelled = 0
    for at in np.argwhere(~odd):
        at = tuple(at)
        v = [float(x) for x in nb[at]]
        exact, top = sum(map(Fraction, v)), max(abs(x) for x in v)
        cancelled += top == 0.7 and abs(exact) < 2.0 ** -16
        loss = 2.0 ** -100 * top if abs(exact) < 2.0 ** -16 * top else len(v) * 2.0 ** -59 * top
        assert abs(Fraction(float(got[at])) - exact) <= 2.0 ** -53 * abs(exact) * (1 + 2.0 ** -40) + loss, (at, v)
    assert cancelled > 3 or depth < 28
