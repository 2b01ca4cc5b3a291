"""The whole state in one pass (axs_download into arrays the device reaches)
gives the bits of the copy through host staging, for 2D and 3D, every stencil
radius, both precisions, fresh and stepped states, at sizes around the march's
32 x 8 columns and its shortest z-chunks."""
import numpy as np
import pytest

from gpu_util import params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("nd,N,stencil", [(2, 4, 0), (2, 30, 0), (2, 34, 1), (2, 70, 2), (2, 66, 3),
                                          (3, 4, 0), (3, 6, 1), (3, 8, 2), (3, 10, 3), (3, 18, 0), (3, 34, 0),
                                          (3, 64, 0), (3, 66, 1), (3, 40, 2), (3, 36, 3), (3, 130, 0)])
def test_direct_snapshot_equals_staged(axs, precision, nd, N, stencil):
    p = params(axs, nd=nd, N=N, precision=precision, stencil_setting=stencil)
    dt = np.float64 if precision == 64 else np.float32
    with axs.Lattice(p) as L:
        rng = np.random.default_rng(2)
        L.upload(*[rng.standard_normal(L.shape) for _ in range(4)])
        for steps in (0, 3):
            L.evolve(steps)
            want = L.download(dtype=dt)
            out = [axs.PinnedBuffer(L.shape, dt) for _ in range(4)]
            fn = axs._lib.axs_download if precision == 64 else axs._lib.axs_download_f32
            axs._check(fn(L._h, *[o.array.ctypes.data for o in out]))
            for a, b in zip(out, want):
                assert np.array_equal(a.array, b), steps
            for o in out:
                o.free()


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("N", [4, 6, 18, 64])
def test_axion_spectrum_of_small_lattices(axs, oracle, precision, N):
    """The march's planes wrap more than once on the smallest lattices (its ring runs A = 5 planes ahead)."""
    from gpu_util import orc
    p = params(axs, nd=3, N=N, precision=precision)
    f = oracle.init_thermal(orc(p), 4)
    with axs.Lattice(p) as L:
        L.upload(*f)
        L.evolve(4)
        k, pk, c = L.axion_spectrum(8)
        g = L.download()
        tau = L.time[0]
    ref = (g[1] * g[2] - g[0] * g[3]) / (tau * np.hypot(g[0], g[1]))
    F = np.abs(np.fft.fftn(ref)) ** 2
    n = np.fft.fftfreq(N, 1.0 / N)
    n2 = (n[:, None, None] ** 2 + n[None, :, None] ** 2 + n[None, None, :] ** 2).round().astype(int)
    ratio = np.sqrt(3.0) * N / 2
    edges = [0] + [int(np.ceil(np.exp(np.log(ratio) * b / 8) ** 2)) for b in range(1, 8)]
    at = np.searchsorted(edges, n2, side="right") - 1
    at[n2 == 0] = -1
    norm = (N * 0.5) ** 3 / float(N ** 3) ** 2
    for b in range(8):
        assert c[b] == (at == b).sum()
        if c[b]:
            # the tests of both precisions against the oracle: 1e-10 and 1e-4
            assert abs(pk[b] - norm * F[at == b].mean()) <= (1e-10 if precision == 64 else 1e-4) * pk[b]


@pytest.mark.parametrize("fields", [(0, 1), (0, 1, 2, 3), (1,), (2,)])
def test_large_pageable_downloads(axs, fields):
    """Destinations large enough to be touched ahead of the copies (several chunks, not page-aligned) get the values of
    the pinned ones, and nothing outside them is written."""
    p = params(axs, nd=3, N=202, precision=64)
    with axs.Lattice(p) as L:
        L.init_flat(7, 1.0)
        L.evolve(3)
        pins = [axs.PinnedBuffer(L.shape, np.float64) for _ in range(4)]
        axs._check(axs._lib.axs_download(L._h, *[o.array.ctypes.data for o in pins]))
        raw = [np.full(L.length + 24, -7.0) for _ in fields]
        got = {f: r[13:13 + L.length] for f, r in zip(fields, raw)}
        axs._check(axs._lib.axs_download(L._h, *[got[f].ctypes.data if f in got else None for f in range(4)]))
        for f in fields:
            assert np.array_equal(got[f].reshape(L.shape), pins[f].array)
        for r in raw:
            assert (r[:13] == -7.0).all() and (r[13 + L.length:] == -7.0).all()
        c = L.checkpoint()
        with axs.Lattice(p) as M:
            M.restore(c)
            for a, b in zip(M.download(), pins):
                assert np.array_equal(a, b.array)
        for o in pins:
            o.free()


@pytest.mark.parametrize("where", ["pinned", "device"])
@pytest.mark.parametrize("first", [True, False])
def test_pair_of_two_kinds_of_memory(axs, where, first):
    """One array of a pair page-locked or on the device, the other pageable and large enough to be touched by host
    threads: both get the values, and the host writes to the pageable one only."""
    p = params(axs, nd=3, N=128, precision=64)
    with axs.Lattice(p) as L:
        L.init_flat(7, 1.0)
        L.evolve(3)
        want = L.download()
        host = np.empty(L.shape)
        assert host.nbytes >= 8 << 20
        if where == "pinned":
            other = axs.PinnedBuffer(L.shape, np.float64)
            ptr, get = other.array.ctypes.data, lambda: other.array
        else:
            torch = pytest.importorskip("torch")
            dev = torch.full(L.shape, -7.0, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            ptr, get = dev.data_ptr(), lambda: dev.cpu().numpy()
        pair = (ptr, host.ctypes.data) if first else (host.ctypes.data, ptr)
        axs._check(axs._lib.axs_download(L._h, None, None, *pair))
        a, b = (get(), host) if first else (host, get())
        assert np.array_equal(a, want[2]) and np.array_equal(b, want[3])
        if where == "pinned":
            other.free()
