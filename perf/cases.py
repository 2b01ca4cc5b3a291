"""What a user of this framework has it do, as timed cases.

The work is the run loop of a lattice simulation: intervals of leapfrog steps,
then at each output the string search, the background means and energies, a
spectrum, and the fields themselves. A case is one of

  evolve    one interval of `steps` steps, then the synchronised state (both
            fields and both derivatives) into the program's own arrays
  interval  a whole output of the run loop: steps, string count, means, the
            axion spectrum, and the two fields as host arrays
  ensemble  one interval of independent lattices of uneven sizes, their string
            counts and their states
  strings   the string search and the list of flagged cells
  spectrum  the axion kinetic spectrum and the power spectrum of a field
  means     the background means and the energies

in 2D and 3D, FP32 and FP64, with stencil radius 1 to 4. The program's arrays
are torch tensors on the GPU (the C ABI takes any address that the device
reaches), except where a case says host arrays. Lattices keep evolving from
pass to pass, as in a run; the analysis cases look at one evolved state.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "axion-strings_gb300"))
import axs  # noqa: E402

#: dx, dt: the 2D/3D runs of the benchmark, and the parameter file's default.
GRID = {"run": (0.5, 0.1), "default": (1.0, 0.3)}
ENSEMBLE_SIZES = (64, 96, 128, 160, 192)
LEAD = 4   # steps that the analysis cases' state has taken


def listed():
    return [
        # the parameter file's default lattice at its sampling cadence: the smallest call, all latency
        dict(name="interval_2d_128_f64", kind="interval", nd=2, N=128, bits=64, stencil=0, steps=10, T=4.0, grid="default", host=True),
        # the 2D reference run: a string count every 100 steps
        dict(name="evolve_2d_512_f64", kind="evolve", nd=2, N=512, bits=64, stencil=0, steps=100, T=0.0, grid="run"),
        # a 2D FP32 lattice of no round size
        dict(name="evolve_2d_1500_f32", kind="evolve", nd=2, N=1500, bits=32, stencil=0, steps=50, T=0.0, grid="run"),
        # the 3D FP64 run at its string cadence of 20 steps, a whole output with host fields
        dict(name="interval_3d_256_f64", kind="interval", nd=3, N=256, bits=64, stencil=0, steps=20, T=0.0, grid="run", host=True),
        # a small 3D FP64 lattice, thermal mass on
        dict(name="evolve_3d_128_f64", kind="evolve", nd=3, N=128, bits=64, stencil=0, steps=20, T=4.0, grid="run"),
        # a 3D size that no tile divides
        dict(name="evolve_3d_250_f32", kind="evolve", nd=3, N=250, bits=32, stencil=0, steps=20, T=0.0, grid="run"),
        # the precision form at its full size: the largest
        dict(name="evolve_3d_1024_f32", kind="evolve", nd=3, N=1024, bits=32, stencil=0, steps=20, T=0.0, grid="run"),
        # a higher-order Laplacian
        dict(name="evolve_3d_384_f32_r2", kind="evolve", nd=3, N=384, bits=32, stencil=1, steps=10, T=0.0, grid="run"),
        # the batched ensemble, 50-step interval
        dict(name="ensemble_24_f32", kind="ensemble", nd=3, N=24, bits=32, stencil=0, steps=50, T=0.0, grid="run"),
        # the production run's analysis: strings every 10 steps, spectra and means
        dict(name="strings_3d_512_f32", kind="strings", nd=3, N=512, bits=32, stencil=0, steps=0, T=0.0, grid="run"),
        dict(name="spectrum_3d_512_f32", kind="spectrum", nd=3, N=512, bits=32, stencil=0, steps=0, T=0.0, grid="run"),
        dict(name="means_3d_512_f32", kind="means", nd=3, N=512, bits=32, stencil=0, steps=0, T=0.0, grid="run"),
    ]


def _log_even(rng, lo, hi):
    return 2 * int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2))


def draw(rng):
    kind = rng.choice(["evolve", "evolve", "evolve", "interval", "ensemble", "strings", "spectrum", "means"])
    nd = 3 if kind == "ensemble" else rng.choice([2, 3])
    bits = 32 if kind == "ensemble" else rng.choice([32, 64])
    if kind == "ensemble":
        N = rng.randint(6, 32)   # members
    elif nd == 2:
        N = _log_even(rng, 64, 4096)
    else:
        N = _log_even(rng, 24, 640 if bits == 32 and kind != "interval" else 300)
    sites = sum(n ** 3 for n in _members(N)) if kind == "ensemble" else N ** nd
    stencil = rng.choice([0, 0, 0, 1, 2, 3]) if kind == "evolve" else 0
    T, grid = rng.choice([(0.0, "run"), (0.0, "run"), (4.0, "run")]) if nd == 3 else rng.choice([(0.0, "run"), (4.0, "default")])
    steps = 0
    if kind in ("evolve", "interval", "ensemble"):
        most = 100 if sites < 2_000_000 else 50 if sites < 20_000_000 else 20   # the cadences in use; long intervals on small lattices
        steps = rng.randint(5, most)
    return dict(kind=kind, nd=nd, N=N, bits=bits, stencil=stencil, steps=steps, T=T, grid=grid, host=kind == "interval")


def _members(n):
    """The sizes of an ensemble of n lattices: a fixed uneven mix."""
    return [ENSEMBLE_SIZES[(3 * i * i + 2 * i + 1) % 5] for i in range(n)]


def _params(case, N, lam=1.0):
    dx, dt = GRID[case["grid"]]
    return axs.default_params(NDIMS=case["nd"], N=N, lambda_=lam, T_initial=case["T"], space_step=dx, time_step=dt, stencil_setting=case["stencil"],
                              precision=axs.F32 if case["bits"] == 32 else axs.F64, prs=1, thr=1)


def _fields(nd, N, dx, seed, dtype, kcut):
    """Both components of a Gaussian random field with power for 0 < |k| < kcut, <|phi|^2> = 1."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    L = N * dx
    k2 = torch.zeros([1] * nd, device="cuda", dtype=torch.float64)
    for d in range(nd):
        k = 2 * math.pi / L * torch.fft.fftfreq(N, 1.0 / N, device="cuda", dtype=torch.float64)
        k2 = k2 + k.reshape([N if i == d else 1 for i in range(nd)]) ** 2
    spec = torch.complex(torch.randn([N] * nd, device="cuda", dtype=dtype, generator=g), torch.randn([N] * nd, device="cuda", dtype=dtype, generator=g))
    spec *= (k2 > 0) & (k2 < max(kcut * kcut, (2.5 * 2 * math.pi / L) ** 2))   # small boxes: the lowest modes
    f = torch.fft.ifftn(spec)
    del spec
    f *= 1.0 / torch.view_as_real(f).double().square().sum().div(N ** nd).sqrt().item() if N ** nd < 1 << 28 else 1.0 / (torch.linalg.vector_norm(f).item() / math.sqrt(N ** nd))
    return f.real.contiguous(), f.imag.contiguous()


def _upload(lattice, fields):
    torch.cuda.synchronize()   # the lattice has a stream of its own
    fn = axs._lib.axs_upload_f32 if fields[0].dtype == torch.float32 else axs._lib.axs_upload
    axs._check(fn(lattice._h, *[f.data_ptr() for f in fields]))


def _state_into(lattice, out):
    fn = axs._lib.axs_download_f32 if out[0].dtype == torch.float32 else axs._lib.axs_download
    axs._check(fn(lattice._h, *[o.data_ptr() for o in out]))


def _dtype(case):
    return torch.float32 if case["bits"] == 32 else torch.float64


def _seeded(case, seed, N, i=0):
    # a run starts with kcut = 1; the analysis looks at a network further on, whose strings are further apart
    kcut = 0.25 if case["kind"] in ("strings", "spectrum", "means") else 1.0
    f1, f2 = _fields(case["nd"], N, GRID[case["grid"]][0], 1_000_003 * seed + i, _dtype(case), kcut)
    return f1, f2, torch.zeros_like(f1)


def _lambda(i):
    return float(np.float32(0.5 * 8.0 ** ((7 * i % 24) / 24.0)))   # log-spaced in [0.5, 4)


def prepare(case, seed):
    if case["kind"] == "ensemble":
        sizes = _members(case["N"])
        ens = axs.Ensemble([_params(case, n, _lambda(i)) for i, n in enumerate(sizes)])
        for i, (n, m) in enumerate(zip(sizes, ens.members)):
            f1, f2, z = _seeded(case, seed, n, i)
            _upload(m, (f1, f2, z, z))
        out = [torch.empty(sum(n ** 3 for n in sizes), device="cuda", dtype=torch.float32) for _ in range(4)]
        at = np.cumsum([0] + [n ** 3 for n in sizes])
        ens.evolve(0)   # tuned, as by a run's first interval
        return {"case": case, "ens": ens, "out": out, "views": [[o[at[i]:at[i + 1]] for o in out] for i in range(len(sizes))]}
    lat = axs.Lattice(_params(case, case["N"]))
    f1, f2, z = _seeded(case, seed, case["N"])
    _upload(lat, (f1, f2, z, z))
    del f1, f2, z
    state = {"case": case, "lat": lat}
    lat.autotune()
    if case["kind"] in ("evolve",):
        state["out"] = [torch.empty(lat.shape, device="cuda", dtype=_dtype(case)) for _ in range(4)]
    if case["kind"] in ("strings", "spectrum", "means"):
        lat.evolve(LEAD)
        torch.cuda.synchronize()
    if case["kind"] == "strings":   # room for the list, as a program that follows the network keeps
        state["list"] = np.full((lat.length // 8 + 64, case["nd"]), -1, dtype=np.int32)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        ens = state["ens"]
        ens.evolve(case["steps"])
        n, _ = ens.find_strings()
        for m, v in zip(ens.members, state["views"]):
            _state_into(m, v)
        return state["out"], n
    lat = state["lat"]
    if kind == "evolve":
        lat.evolve(case["steps"])
        _state_into(lat, state["out"])
        return state["out"]
    if kind == "interval":
        lat.evolve(case["steps"])
        n, cores, _ = lat.find_strings()
        means = lat.background()
        k, pk, count = lat.axion_spectrum(128)
        f = lat.download(dtype=np.float64 if case["bits"] == 64 else np.float32, fields=(True, True, False, False))
        return f[0], f[1], means, k, pk, count, n, cores
    if kind == "strings":
        n, cores, _ = lat.find_strings()
        pos, total = state["list"], ctypes.c_int64()
        axs._check(axs._lib.axs_string_positions(lat._h, pos.ctypes.data, len(pos), ctypes.byref(total)))
        return pos, total.value, n, cores
    if kind == "spectrum":
        return lat.axion_spectrum(128) + lat.powerspec(axs.PHI2)
    return lat.background(), lat.energies()


# ---------------------------------------------------------------- the same in 64 bits

def _coefs(setting, nd):
    """The Laplacian's weights, which the framework holds in single precision."""
    f = np.float32
    w = [[f(-2.0) * f(nd), f(1)], [f(-5) / f(2) * f(nd), f(4) / f(3), f(-1) / f(12)],
         [f(-49) / f(18) * f(nd), f(3) / f(2), f(-3) / f(20), f(1) / f(90)],
         [f(-205) / f(72) * f(nd), f(8) / f(5), f(-1) / f(5), f(8) / f(315), f(-1) / f(560)]][setting]
    return [float(x) for x in w]


def _lap(a, w, dx):
    s = w[0] * a
    for r, c in enumerate(w[1:], 1):
        t = torch.zeros_like(a)
        for d in range(a.dim()):
            t += torch.roll(a, r, d)
            t += torch.roll(a, -r, d)
        s += c * t
    return s.div_(dx * dx)


def _evolve64(case, f1, f2, steps, lam):
    """Leapfrog steps of psi'' = lap psi - lam/tau^2 psi (|psi|^2 - tau^2 + T^2/3), the first a pure drift."""
    dx, dt = (float(np.float32(v)) for v in GRID[case["grid"]])
    w, T3 = _coefs(case["stencil"], case["nd"]), float(np.float32(case["T"])) ** 2 / 3.0
    psi, tau = [f1.double(), f2.double()], 1.0
    pi = [torch.zeros_like(p) for p in psi]
    for s in range(steps):
        for p, q in zip(psi, pi):   # pi at the half step
            p.add_(q, alpha=dt)
        tau += dt
        g = psi[0] * psi[0]
        g += psi[1] * psi[1]
        g += T3 - tau * tau
        g *= -lam / (tau * tau)
        kick = [_lap(p, w, dx).addcmul_(g, p) for p in psi]
        for q, k in zip(pi, kick):
            q.add_(k, alpha=dt if s < steps - 1 else 0.5 * dt)
    return psi, pi, tau


def _means64(psi, pi):
    r = torch.hypot(psi[0], psi[1])
    return np.array([float(v) for v in (psi[0].mean(), psi[1].mean(), pi[0].mean(), pi[1].mean(), torch.atan2(psi[0], psi[1]).abs().mean(), r.mean())])


def _energies64(case, psi, pi, tau, lam):
    dx = float(np.float32(GRID[case["grid"]][0]))
    kin = sum((0.5 * ((q - p / tau) / tau).square()).mean() for p, q in zip(psi, pi))
    grad = sum((0.5 * ((torch.roll(p, -1, d) - p) / tau / dx).square()).mean() for p in psi for d in range(p.dim()))
    pot = 0.25 * lam * ((psi[0].square() + psi[1].square()) / (tau * tau) - 1).square().mean()
    return np.array([float(kin), float(grad), float(pot)])


def _modes(f):
    """|F|^2, |n|^2 and the weight of each mode of the half spectrum."""
    N, nd = f.shape[0], f.dim()
    F = torch.fft.rfftn(f)
    p = torch.view_as_real(F).square().sum(-1)
    n2 = torch.zeros([1] * nd, device=f.device, dtype=torch.int64)
    for d in range(nd):
        n = torch.fft.fftfreq(N, 1.0 / N, device=f.device, dtype=torch.float64)[: N if d < nd - 1 else N // 2 + 1].round().long()
        n2 = n2 + (n * n).reshape([-1 if i == d else 1 for i in range(nd)])
    wt = torch.full((N // 2 + 1,), 2.0, device=f.device, dtype=torch.float64)
    wt[0] = wt[-1] = 1.0
    return p.reshape(-1), n2.reshape(-1), wt.expand(p.shape).reshape(-1)


def _binned(p, n2, wt, bin_of, nbins):
    ok = (bin_of >= 0) & (bin_of < nbins)
    b, w = bin_of[ok], wt[ok]
    return [torch.bincount(b, weights=x, minlength=nbins).cpu().numpy() for x in (p[ok] * w, n2[ok].double().sqrt() * w, w)]


def _axion64(case, psi, pi, tau, nbins=128):
    N, nd = case["N"], case["nd"]
    L = N * float(np.float32(GRID[case["grid"]][0]))
    f = (psi[1] * pi[0] - psi[0] * pi[1]) / (tau * torch.hypot(psi[0], psi[1]))
    p, n2, wt = _modes(f)
    ratio = math.sqrt(nd) * N / 2.0
    first = torch.tensor([0] + [math.ceil(math.exp(math.log(ratio) * b / nbins) ** 2) for b in range(1, nbins)], device=p.device)
    at = torch.searchsorted(first, n2, right=True) - 1
    at[n2 == 0] = -1
    ps, ns, c = _binned(p, n2, wt, at, nbins)
    d = np.maximum(c, 1)
    return 2 * math.pi * ns / d / L, L ** nd / float(N ** nd) ** 2 * ps / d, None


def _power64(case, f):
    N, nd = case["N"], case["nd"]
    L = N * float(np.float32(GRID[case["grid"]][0]))
    p, n2, wt = _modes(f)
    at = n2.double().sqrt().floor().long() - 1
    at[(n2 == 0) | (4 * n2 >= N * N)] = -1
    ps, ns, c = _binned(p, n2, wt, at, N // 2)
    with np.errstate(all="ignore"):
        k = ns / c
        return ps / (2 * math.pi * k if nd == 2 else 4 * math.pi * k * k), k * (2 * math.pi / L), None


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        parts = []
        for i, n in enumerate(_members(case["N"])):
            f1, f2, _ = _seeded(case, seed, n, i)
            psi, pi, _ = _evolve64(case, f1, f2, case["steps"], _lambda(i))
            parts.append([a.reshape(-1) for a in psi + pi])
        return [torch.cat([p[j] for p in parts]) for j in range(4)], None
    if kind == "strings":
        return None   # whole numbers
    f1, f2, _ = _seeded(case, seed, case["N"])
    psi, pi, tau = _evolve64(case, f1, f2, case["steps"] or LEAD, 1.0)
    del f1, f2
    if kind == "evolve":
        return psi + pi
    if kind == "interval":
        return (psi[0], psi[1], _means64(psi, pi)) + _axion64(case, psi, pi, tau) + (None, None)
    if kind == "spectrum":
        return _axion64(case, psi, pi, tau) + _power64(case, psi[1])
    return _means64(psi, pi), _energies64(case, psi, pi, tau, 1.0)


def work(case):
    """The state read once and written once, the outputs written once; the arithmetic of the steps and of what is looked at."""
    kind, es = case["kind"], case["bits"] // 8
    sites = float(sum(n ** 3 for n in _members(case["N"])) if kind == "ensemble" else case["N"] ** case["nd"])
    R, nd = case["stencil"] + 1, case["nd"]
    step = 2 * (2 * nd * R + R) + 13   # neighbour sums and weights of both components, the kick and the drift
    fft = 2.5 * math.log2(sites)
    if kind in ("evolve", "ensemble"):
        return {"bytes": 12 * es * sites, "flops": case["steps"] * step * sites}
    if kind == "interval":
        return {"bytes": 10 * es * sites, "flops": (case["steps"] * step + 20 + 30 + step + 6 + fft + 3) * sites}
    if kind == "strings":
        return {"bytes": 2 * es * sites, "flops": 40 * sites}
    if kind == "spectrum":
        return {"bytes": 4 * es * sites, "flops": (step + 6 + 2 * (fft + 3)) * sites}
    return {"bytes": 4 * es * sites, "flops": (30 + step + 30) * sites}
