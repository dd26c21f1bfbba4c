"""finaliseGrid, initialiseDegrid and finaliseWeights against their formulas in
64 bits, at image sides that are not powers of two (even and odd halves,
rectangular, padded), for one and several grids and planes, host and device."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ARCSEC = math.pi / (180 * 3600)
CELL = 30.0 * ARCSEC


def correction(n):
    """Low-passed inverse spheroidal of one axis (SphFuncVisGridder::correctConvolution) in 64 bits."""
    from oracle.spheroidal import SpheroidalFunction
    half = n // 2
    f = SpheroidalFunction(3 * math.pi, 1.0)(np.abs(np.arange(n) - half) / float(half)).astype(np.float32)
    f[0] = np.float32(3.0) * (f[1] - f[2]) + f[3]
    b = np.fft.fftshift(np.fft.fft(np.fft.ifftshift(f.astype(np.float64))))
    b[:half - 3] = 0
    b[half + 4:] = 0
    b = np.fft.fftshift(np.fft.ifft(np.fft.ifftshift(b)))
    return 1.0 / (b * (float(f[half]) / b[half])).real


def centred(a, forward):
    f = np.fft.fft2 if forward else (lambda x, axes: np.fft.ifft2(x, axes=axes, norm="forward"))
    return np.fft.fftshift(f(np.fft.ifftshift(a, axes=(0, 1)), axes=(0, 1)), axes=(0, 1))


def setup(kind, nx, ny, npol, nchan, padding):
    from yandasoft_b200 import gridder as G
    ps = {"gridder": kind, "gridder.padding": padding}
    if kind == "WStack":
        ps.update({"gridder.WStack.wmax": 2000.0, "gridder.WStack.nwplanes": 3})
    return G, G.VisGridderFactory.make(ps), G.Axes(CELL, CELL, freq=(1.0e9, 1.01e9) if nchan > 1 else None)


def screens(kind, pnx, pny):
    if kind != "WStack":
        return [None]
    import oracle.cf as cf
    uvc = (1.0 / (CELL * pnx), 1.0 / (CELL * pny))
    return [cf.wstack_screen(pnx, pny, uvc[0], uvc[1], w)(np.ones((pnx, pny), dtype=np.complex64)).astype(np.complex128)
            for w in (-2000.0, 0.0, 2000.0)]


SIZES = [("SphFunc", 64, 64, 1, 1, 1.0), ("SphFunc", 90, 150, 2, 3, 1.0), ("SphFunc", 100, 60, 1, 1, 1.5),
         ("WStack", 90, 66, 4, 1, 1.0), ("WStack", 130, 130, 1, 1, 1.2), ("SphFunc", 1000, 258, 1, 1, 1.0)]


@pytest.mark.parametrize("kind,nx,ny,npol,nchan,padding", SIZES)
def test_finalise(kind, nx, ny, npol, nchan, padding):
    """Image from the grids in 64 bits.  Compared with the correction divided
    out: a single-precision FFT of N = nx ny <= 2^18 points is within
    eps sqrt(log2 N) ~ 3e-7 of its norm, the rounded sums over grids add as
    much: 1e-6."""
    import torch
    G, g, axes = setup(kind, nx, ny, npol, nchan, padding)
    rng = np.random.default_rng(5)
    nrow, fr = 300, np.array([1.0e9, 1.005e9, 1.01e9])
    uvw = rng.uniform(-400, 400, (nrow, 3))
    vis = np.asfortranarray(rng.standard_normal((nrow, 3, npol)) + 1j * rng.standard_normal((nrow, 3, npol)),
                            dtype=np.complex64)
    g.initialiseGrid(axes, (nx, ny, npol, nchan))
    g.grid(G.Accessor(uvw, fr, vis))
    grids = g.grids()
    host = g.finaliseGrid()
    dev = torch.full((nchan, npol, ny, nx), 7.0, device="cuda")
    g.finaliseGrid(dev)
    assert np.array_equal(dev.cpu().numpy().transpose(3, 2, 1, 0), host)
    for a, b in zip(grids, g.grids()):
        assert np.array_equal(a, b)
    pnx, pny = grids[0].shape[:2]
    ref = 0.0
    for a, s in zip(grids, screens(kind, pnx, pny)):
        t = centred(a.astype(np.complex128), False)
        ref = ref + (t if s is None else t * s[:, :, None, None]).real
    x0, y0 = (pnx - nx) // 2, (pny - ny) // 2
    ref = ref[x0:x0 + nx, y0:y0 + ny]
    corr = (correction(pnx)[:, None] * correction(pny)[None, :])[x0:x0 + nx, y0:y0 + ny, None, None]
    assert np.linalg.norm(ref) > 0
    assert np.linalg.norm(host / corr - ref) <= 1e-6 * np.linalg.norm(ref)
    wh = g.finaliseWeights()
    wd = torch.full((nchan, npol, ny, nx), 7.0, device="cuda")
    g.finaliseWeights(wd)
    sums = g.sum_weights().sum(0).astype(np.float32)
    assert np.array_equal(wh, np.broadcast_to(sums, (nx, ny, npol, nchan)))
    assert np.array_equal(wd.cpu().numpy().transpose(3, 2, 1, 0), wh)


@pytest.mark.parametrize("kind,nx,ny,npol,nchan,padding", SIZES)
@pytest.mark.parametrize("on_device", [False, True])
def test_initialise_degrid(kind, nx, ny, npol, nchan, padding, on_device):
    """Grids of a model image in 64 bits: rounding of the corrected pixels and
    a single-precision FFT, 1e-6 of the norm as above."""
    import torch
    G, g, axes = setup(kind, nx, ny, npol, nchan, padding)
    rng = np.random.default_rng(6)
    img = np.asfortranarray(rng.standard_normal((nx, ny, npol, nchan)), dtype=np.float32)
    give = torch.from_numpy(np.ascontiguousarray(img.transpose(3, 2, 1, 0))).cuda().permute(3, 2, 1, 0) \
        if on_device else img
    g.initialiseDegrid(axes, give)
    assert not g.isModelEmpty()
    grids = g.grids()
    pnx, pny = grids[0].shape[:2]
    x0, y0 = (pnx - nx) // 2, (pny - ny) // 2
    pad = np.zeros((pnx, pny, npol, nchan))
    pad[x0:x0 + nx, y0:y0 + ny] = img
    pad *= (correction(pnx)[:, None] * correction(pny)[None, :])[:, :, None, None]
    for a, s in zip(grids, screens(kind, pnx, pny)):
        ref = centred(pad if s is None else np.conj(pad * s[:, :, None, None]), True)
        assert np.linalg.norm(a - ref) <= 1e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("on_device", [False, True])
@pytest.mark.parametrize("where", [None, 0, -1])
def test_model_empty(on_device, where):
    """A model is empty when no pixel, first and last included, differs from zero."""
    import torch
    G, g, axes = setup("SphFunc", 90, 66, 1, 1, 1.0)
    img = np.zeros((90, 66, 1, 1), dtype=np.float32, order="F")
    if where is not None:
        img[where, where, 0, 0] = -1e-30
    give = torch.from_numpy(np.ascontiguousarray(img.transpose(3, 2, 1, 0))).cuda().permute(3, 2, 1, 0) \
        if on_device else img
    g.initialiseDegrid(axes, give)
    assert g.isModelEmpty() == (where is None)
    if where is None:
        assert not np.any(g.grids()[0])


def test_corrections_follow_the_shape():
    """One handle through several shapes, host and device models in turn: the
    first pass after each change takes the new shape's correction factors (the
    grids and images of a handle that never had another shape)."""
    import torch
    G, g, axes = setup("SphFunc", 64, 64, 1, 1, 1.0)
    rng = np.random.default_rng(7)
    uvw = rng.uniform(-400, 400, (200, 3))
    vis = np.asfortranarray(rng.standard_normal((200, 1, 1)), dtype=np.complex64)
    acc = G.Accessor(uvw, np.array([1.0e9]), vis)
    for k, (nx, ny) in enumerate([(90, 66), (128, 64), (66, 90), (256, 256), (64, 128), (90, 66)]):
        img = np.asfortranarray(rng.standard_normal((nx, ny, 1, 1)), dtype=np.float32)
        give = torch.from_numpy(np.ascontiguousarray(img.transpose(3, 2, 1, 0))).cuda().permute(3, 2, 1, 0) \
            if k % 2 else img
        fresh = setup("SphFunc", nx, ny, 1, 1, 1.0)[1]
        for h in (g, fresh):
            h.initialiseDegrid(axes, give)
        assert np.array_equal(g.grids()[0], fresh.grids()[0])
        for h in (g, fresh):
            h.initialiseGrid(axes, (nx, ny, 1, 1))
            h.grid(acc)
        assert np.array_equal(g.finaliseGrid(), fresh.finaliseGrid())


@pytest.mark.parametrize("on_device", [False, True])
def test_empty_model_is_not_transformed(on_device):
    """An empty model costs a look at it and cleared grids, not the screens and
    transforms of its 17 grids: less than half of what another model takes (the
    transforms alone are several times the rest)."""
    import time
    import torch
    from yandasoft_b200 import gridder as G
    n = 2048
    g = G.VisGridderFactory.make({"gridder": "WStack", "gridder.WStack.wmax": 2000.0, "gridder.WStack.nwplanes": 17})
    axes = G.Axes(CELL, CELL)
    best = {}
    for value in (1.0, 0.0):
        img = np.zeros((n, n, 1, 1), dtype=np.float32, order="F")
        img[n // 2 + 3, n // 2 - 7, 0, 0] = value
        give = torch.from_numpy(np.ascontiguousarray(img.transpose(3, 2, 1, 0))).cuda().permute(3, 2, 1, 0) \
            if on_device else torch.from_numpy(np.ascontiguousarray(img.transpose(3, 2, 1, 0))).pin_memory().numpy() \
            .transpose(3, 2, 1, 0)
        times = []
        for _ in range(6):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            g.initialiseDegrid(axes, give)
            times.append(time.perf_counter() - t0)
        assert g.isModelEmpty() == (value == 0.0)
        best[value] = min(times[1:])
    print("initialiseDegrid %s: %.3f ms, empty %.3f ms" % (on_device, 1e3 * best[1.0], 1e3 * best[0.0]))
    upload = 0.0 if on_device else 1e-3 * n * n * 4 / 40e6      # 17 MB at 40 GB/s and above
    assert best[0.0] - upload < 0.5 * (best[1.0] - upload)


@pytest.mark.parametrize("on_device", [False, True])
def test_model_beyond_a_smaller_grid(on_device):
    """With padding below 1 the grid is smaller than the image: an empty model
    is taken as such, any other refused, also one whose only pixel lies outside
    the grid."""
    import torch
    G, _, axes = setup("SphFunc", 64, 64, 1, 1, 0.5)
    for at in (None, (0, 0), (32, 32)):
        g = setup("SphFunc", 64, 64, 1, 1, 0.5)[1]
        img = np.zeros((64, 64, 1, 1), dtype=np.float32, order="F")
        if at:
            img[at[0], at[1], 0, 0] = 1.0
        give = torch.from_numpy(np.ascontiguousarray(img.transpose(3, 2, 1, 0))).cuda().permute(3, 2, 1, 0) \
            if on_device else img
        if at is None:
            g.initialiseDegrid(axes, give)
            assert g.isModelEmpty()
        else:
            with pytest.raises(G.AskapError):
                g.initialiseDegrid(axes, give)


# sides that are powers of two fold the centring into the passes beside the FFT:
# with screens, several planes and channels, extraction from a padded grid,
# rectangular both ways
ROLLED = [("WStack", 64, 64, 4, 1, 1.0), ("WStack", 128, 32, 2, 3, 1.0), ("SphFunc", 32, 128, 2, 3, 1.0),
          ("SphFunc", 64, 32, 1, 1, 2.0), ("WStack", 32, 64, 3, 1, 2.0), ("SphFunc", 256, 512, 4, 1, 1.0)]


@pytest.mark.parametrize("kind,nx,ny,npol,nchan,padding", ROLLED)
def test_finalise_rolled(kind, nx, ny, npol, nchan, padding):
    test_finalise(kind, nx, ny, npol, nchan, padding)


@pytest.mark.parametrize("kind,nx,ny,npol,nchan,padding", ROLLED)
@pytest.mark.parametrize("on_device", [False, True])
def test_initialise_degrid_rolled(kind, nx, ny, npol, nchan, padding, on_device):
    test_initialise_degrid(kind, nx, ny, npol, nchan, padding, on_device)
