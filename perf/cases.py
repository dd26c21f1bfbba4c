"""Performance cases of the gridder: imaging, prediction and major cycles through
the public Python interface (yandasoft_b200.gridder), from one integration on a
small grid to tens of millions of samples on stacked 4096^2 grids.

A case is a dict of plain values:

  op        "predict"  initialiseDegrid of a model, degrid of a zeroed cube
            "chunk"    degrid of one more accessor chunk with the model in place
            "image"    initialiseGrid, grid, finaliseGrid, finaliseWeights
            "psf"      the same for the point spread function (dopsf)
            "cold"     "image" on a gridder made by the call: convolution functions included
            "major"    one major cycle over a plan made once: new model, degrid_plan,
                       subtract, grid_plan, finaliseGrid
            "cycle"    the same for several uneven instances as one CUDA graph (MajorCycle)
  gridder   SphFunc, WProject, WStack, WStackWProject, AWProject, with nwplanes,
            nwstacks, oversample, maxsupport, (AWProject) dish
  nx, cell  image side and cell (arcsec); npol, nchan_img: its polarisations and channels
  ntime     integrations of `dt` seconds of a 36-antenna, 630-baseline array, the first of a
            track of `track` seconds centred on transit (its largest |w| sets wmax)
  nchan     channels over f0..f1 (Hz)
  flags     a few percent of the samples flagged; weights: noise other than one
  delay     per-row phase rotation delays; mfs: first Taylor term weights
  host      the cubes are the caller's pinned host memory instead of device memory

`exact` evaluates the same outputs in 64 bits with torch alone: convolution
functions, index arithmetic, tap sums and transforms.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from yandasoft_b200 import gridder as G
from yandasoft_b200 import simulate

ARCSEC = math.pi / (180 * 3600)
C_LIGHT = 299792458.0

_DEFAULTS = dict(npol=1, nchan_img=1, dt=10.0, track=3600.0, f0=940e6, f1=948e6, nwplanes=33, nwstacks=17, oversample=4,
                 maxsupport=1024, dish=12.0, instances=1, flags=False, weights=False, delay=False, mfs=False,
                 host=False)


def listed():
    return [
        # one integration of a calibrator-sized field: the call that a streaming ingest makes per
        # timestamp, all launches and latency
        dict(name="chunk_sph_one_integration", op="chunk", gridder="SphFunc", nx=512, cell=16.0, ntime=1, nchan=4,
             npol=2, oversample=128, flags=True),
        # a quick-look image of a minute of data, both hands, real flags and weights
        dict(name="image_wproject_minute", op="image", gridder="WProject", nx=1024, cell=8.0, ntime=6, nchan=8,
             npol=2, oversample=8, maxsupport=512, flags=True, weights=True),
        # an hour of narrow-band W-projection on 2048^2 (1.8e6 samples): ordinary imaging and its prediction
        dict(name="image_wproject_hour", op="image", gridder="WProject", nx=2048, cell=8.0, ntime=360, nchan=8,
             nwplanes=65, weights=True),
        dict(name="predict_wproject_hour", op="predict", gridder="WProject", nx=2048, cell=8.0, ntime=360, nchan=8,
             nwplanes=65, delay=True, flags=True),
        # the PSF of a continuum field, no w-term: small kernels, oversample 128
        dict(name="psf_sph_continuum", op="psf", gridder="SphFunc", nx=3000, cell=6.0, ntime=120, nchan=37, npol=2,
             oversample=128, f0=700e6, f1=1000e6, weights=True, flags=True),
        # w-stacked image, Taylor-term weights, data on a ragged size
        dict(name="image_wstack_taylor", op="image", gridder="WStack", nx=1536, cell=10.0, ntime=101, nchan=23,
             npol=2, nwplanes=21, f0=700e6, f1=1000e6, mfs=True, delay=True),
        # full-polarisation continuum, W-stacking with W-projection, an hour of the full track (4.4e7
        # samples x 4 polarisations): the large image and one major cycle over a kept plan; half of
        # the hour imaged from cubes that the caller holds on the host
        dict(name="image_wstackwproject_continuum", op="image", gridder="WStackWProject", nx=4096, cell=4.0, ntime=720,
             dt=5.0, nchan=96, npol=4, oversample=8, maxsupport=512, f0=700e6, f1=1000e6, track=28800.0),
        dict(name="major_wstackwproject_continuum", op="major", gridder="WStackWProject", nx=4096, cell=4.0,
             ntime=720, dt=5.0, nchan=96, npol=4, oversample=8, maxsupport=512, f0=700e6, f1=1000e6, track=28800.0),
        dict(name="image_host_continuum", op="image", gridder="WStackWProject", nx=2048, cell=8.0, ntime=360,
             dt=5.0, nchan=96, npol=4, nwstacks=9, oversample=8, maxsupport=512, f0=700e6, f1=1000e6, track=28800.0,
             host=True),
        # wide-field W-projection: supports of tens of cells, uneven instances in one graph
        dict(name="cycle_wproject_widefield", op="cycle", gridder="WProject", nx=4096, cell=4.0, ntime=90, nchan=9,
             track=14400.0, instances=4),
        # one beam of a phased-array feed per instance, convolution functions per channel
        dict(name="cycle_awproject_beams", op="cycle", gridder="AWProject", nx=2048, cell=4.0, ntime=20, dt=5.0,
             nchan=24, npol=2, f0=700e6, f1=1000e6, maxsupport=256, instances=3),
        # a new pointing: the first image of a gridder, its convolution functions made by the call
        dict(name="cold_awproject_pointing", op="cold", gridder="AWProject", nx=2048, cell=4.0, ntime=20, dt=5.0,
             nchan=12, npol=2, f0=700e6, f1=1000e6, maxsupport=256, weights=True),
    ]


def draw(rng):
    """One more case of the same ranges; none costs more than the largest listed one."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["chunk", "predict", "image", "image", "psf", "cold", "major", "cycle"])
    kind = rng.choice(["SphFunc", "WProject", "WProject", "WStack", "WStackWProject", "AWProject"])
    c = dict(op=op, gridder=kind, npol=rng.choice([1, 1, 2, 4]), flags=rng.random() < 0.5, weights=rng.random() < 0.5,
             delay=rng.random() < 0.3, mfs=op != "cycle" and rng.random() < 0.2, dt=rng.choice([5.0, 10.0]))
    c["nx"] = 2 * log_int(256, 2048)
    c["cell"] = round(min(10.0, max(4.0, rng.uniform(0.8, 1.2) * 14000.0 / c["nx"])), 2)
    c["nchan"] = log_int(1, 64)
    c["ntime"] = max(1, min(720, log_int(2e3, 8e6) // (630 * c["nchan"])))
    c["track"] = rng.choice([3600.0, 3600.0, 14400.0])
    if rng.random() < 0.5:
        c.update(f0=700e6, f1=1000e6)
    c["oversample"] = 128 if kind in ("SphFunc", "WStack") else 8 if c["nx"] * c["cell"] < 9000 else 4
    if kind == "WStack":
        c["nwplanes"] = rng.choice([5, 9, 15, 21])
    if kind == "WStackWProject":
        c.update(nwstacks=rng.choice([5, 9, 17]), nwplanes=rng.choice([9, 17, 33]), maxsupport=512)
    if kind == "AWProject":
        c.update(nwplanes=rng.choice([9, 17, 33]), maxsupport=256, nx=2048, cell=4.0, oversample=4,
                 nchan=min(24, max(6, c["nchan"])), ntime=min(c["ntime"], 40), f0=700e6, f1=1000e6)
    if kind in ("WStack", "WStackWProject"):
        c["nx"] = min(c["nx"], 2560)
    if op == "cycle":
        c["instances"] = rng.choice([2, 3, 4])
    if op in ("chunk", "predict", "image") and kind != "AWProject" and rng.random() < 0.25:
        c["host"] = True
    if op in ("image", "predict") and kind in ("SphFunc", "WProject") and c["nx"] <= 1400 and c["nchan"] >= 4:
        c["nchan_img"] = rng.choice([1, 2, 4])
    while c["ntime"] > 1 and work(c)["flops"] > 1e11:
        c["ntime"] //= 2
    return c


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _full(case):
    return {**_DEFAULTS, **case}


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _instances(c):
    """The case of each instance: sides and track lengths fall from one to the next."""
    out = []
    for i in range(c["instances"]):
        d = dict(c)
        if i and c["gridder"] != "AWProject":
            d["nx"] = max(512, c["nx"] >> (i % 3) & ~1)
            d["cell"] = c["cell"] * min(2.0, c["nx"] / d["nx"])
        d["ntime"] = max(1, c["ntime"] * (c["instances"] - i) // c["instances"])
        out.append(d)
    return out


def _track(c, seed):
    """uvw (nrow, 3) in metres, the shortest baseline first in each integration; channel frequencies; wmax."""
    arr = simulate.random_disk_array(36, 6000.0, -26.7, seed)
    uvw, ntime, nbl = simulate.uvw_track(arr, -45.0 * simulate.DEG, max(c["track"], c["ntime"] * c["dt"]), c["dt"])
    freq = c["f0"] + (np.arange(c["nchan"]) + 0.5) * (c["f1"] - c["f0"]) / c["nchan"]
    wmax = math.ceil(float(np.abs(uvw[:, 2]).max()) * float(freq.max()) / C_LIGHT * 1.02 / 100.0) * 100.0
    uvw = uvw.reshape(ntime, nbl, 3)[:c["ntime"]]
    k = int(np.argmin(np.linalg.norm(uvw[0], axis=1)))
    uvw[:, [0, k]] = uvw[:, [k, 0]]
    return np.ascontiguousarray(uvw.reshape(-1, 3)), freq, wmax


def _data(c, seed):
    """Point sources and noise over the track, and a model image of other sources, on the device.
    Cubes are [pol][chan][row], the memory of a column-major (row, chan, pol) cube."""
    dev = _device()
    uvw, freq, wmax = _track(c, seed)
    nrow, nchan, npol = len(uvw), c["nchan"], c["npol"]
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    rng = np.random.default_rng(seed + 1)
    half = 0.25 * c["nx"] * c["cell"] * ARCSEC
    src = np.stack([rng.uniform(-half, half, 3), rng.uniform(-half, half, 3), rng.uniform(0.1, 1.0, 3)], 1)
    U = torch.from_numpy(uvw).to(dev)
    vis = torch.view_as_complex(torch.randn((npol, nchan, nrow, 2), generator=gen, device=dev) * 0.01)
    for l, m, s in src:
        cyc = (l * U[:, 0] + m * U[:, 1] + (math.sqrt(1 - l * l - m * m) - 1) * U[:, 2]) / C_LIGHT
        for ch in range(nchan):
            ph = cyc * float(freq[ch])
            ph = (ph - torch.floor(ph)).float() * (2 * math.pi)
            v = torch.polar(torch.full_like(ph, float(s)), ph)
            vis[0, ch] += v
            if npol > 1:
                vis[npol - 1, ch] += v
    d = dict(uvw=U, freq=torch.from_numpy(freq).to(dev), vis=vis, noise=None, flag=None, delay=None, uvw_np=uvw,
             freq_np=freq, nrow=nrow, wmax=wmax)
    if c["weights"]:
        nz = torch.rand((npol, nchan, nrow), generator=gen, device=dev) * 0.75 + 0.75
        d["noise"] = torch.complex(nz, torch.zeros_like(nz))
    if c["flags"]:
        bad = torch.rand((nchan, nrow), generator=gen, device=dev) < 0.03
        bad[:, 0] = False
        d["flag"] = bad.to(torch.uint8)[None].expand(npol, -1, -1).contiguous()
    if c["delay"]:
        d["delay"] = torch.randn((nrow,), generator=gen, device=dev, dtype=torch.float64) * 0.05
    nx = c["nx"]
    img = torch.zeros((c["nchan_img"], npol, nx, nx), device=dev)       # memory of (nx, ny, npol, nchan) column-major
    k = rng.integers(nx // 4, nx - nx // 4, size=(100, 2))
    flux = torch.from_numpy(np.exp(rng.uniform(math.log(0.01), 0.0, 100)).astype(np.float32)).to(dev)
    for p in sorted({0, npol - 1}):
        img[:, p, torch.from_numpy(k[:, 1]).to(dev), torch.from_numpy(k[:, 0]).to(dev)] = flux
    d["model"] = img
    return d


def _parset(c, wmax):
    g = c["gridder"]
    p = {"gridder": g}
    if g == "SphFunc":
        p["gridder.SphFunc.oversample"] = c["oversample"]
    else:
        p.update({"gridder.%s.wmax" % g: wmax, "gridder.%s.nwplanes" % g: c["nwplanes"]})
        if g != "WStack":
            p.update({"gridder.%s.oversample" % g: c["oversample"], "gridder.%s.cutoff" % g: 1e-3,
                      "gridder.%s.maxsupport" % g: c["maxsupport"]})
        if g == "WStackWProject":
            p["gridder.%s.nwstacks" % g] = c["nwstacks"]
        if g == "AWProject":
            p.update({"gridder.%s.maxfeeds" % g: 1, "gridder.%s.diameter" % g: "%gm" % c["dish"],
                      "gridder.%s.blockage" % g: "1m"})
    if c["mfs"]:
        p.update({"visweights": "MFS", "visweights.MFS.reffreq": 0.5 * (c["f0"] + c["f1"]) * 1.1})
    return p


def _axes(c):
    fr = None
    if c["nchan_img"] > 1:
        step = (c["f1"] - c["f0"]) / c["nchan_img"]
        fr = (c["f0"] + 0.5 * step, c["f1"] - 0.5 * step)
    return G.Axes(c["cell"] * ARCSEC, c["cell"] * ARCSEC, freq=fr)


def _make(c, parset):
    g = G.VisGridderFactory.make(parset)
    if c["mfs"]:
        g.customiseForContext("image.i.field.taylor.1")
    return g


def _accessor(c, d, vis):
    shape = (d["nrow"], c["nchan"], c["npol"])
    if c["host"]:
        # column-major views of pinned cubes
        cube = vis.numpy().transpose(2, 1, 0)
        return G.Accessor(d["uvw_np"], d["freq_np"], cube, shape=shape, **{
            k: None if d[k] is None else d[k].cpu().numpy() if k == "delay" else d[k].cpu().numpy().transpose(2, 1, 0)
            for k in ("noise", "flag", "delay")})
    return G.Accessor(d["uvw"], d["freq"], vis, noise=d["noise"], flag=d["flag"], delay=d["delay"], shape=shape)


def _shape(c):
    return (c["nx"], c["nx"], c["npol"], c["nchan_img"])


class _State:
    pass


def _prepare_one(c, seed, op):
    s = _State()
    s.c, s.op = c, op
    d = _data(c, seed)
    s.axes, s.shape = _axes(c), _shape(c)
    s.parset = _parset(c, d["wmax"])
    s.image = torch.empty((c["nchan_img"], c["npol"], c["nx"], c["nx"]), device=_device())
    s.weights = torch.empty_like(s.image)
    # the gridder reads device images by their column-major shape
    s.model = d.pop("model").permute(3, 2, 1, 0)
    s.obs = _accessor(c, d, d["vis"].cpu().pin_memory() if c["host"] else d["vis"])
    s.keep = d
    if op in ("predict", "chunk", "major"):
        s.cube = torch.zeros_like(d["vis"])
        if c["host"]:
            s.cube = s.cube.cpu().pin_memory()
        s.acc = _accessor(c, d, s.cube)
        s.dg = _make(c, s.parset)
        s.dg.initialiseDegrid(s.axes, s.model)
        if c["gridder"] != "AWProject":
            s.dg.build_cf()
        s.stream = torch.cuda.ExternalStream(s.dg.stream_handle())
    if op in ("image", "psf", "major"):
        s.gg = _make(c, s.parset)
        s.gg.initialiseGrid(s.axes, s.shape, dopsf=op == "psf")
        if c["gridder"] != "AWProject":
            s.gg.build_cf()
    if c["gridder"] == "AWProject" and op in ("predict", "chunk"):
        s.dg.degrid(s.acc)          # convolution functions come with the first chunk
    if c["gridder"] == "AWProject" and op in ("image", "psf"):
        s.gg.grid(s.obs)
    if op == "major":
        s.resid = torch.empty_like(d["vis"])
        s.racc = _accessor(c, d, s.resid)
        if c["host"]:
            raise ValueError("plans need device-resident cubes")
        s.plan = s.gg.plan(s.obs)
    return s


def prepare(case, seed):
    c = _full(case)
    if c["op"] != "cycle":
        return _prepare_one(c, seed, c["op"])
    s = _State()
    s.c, s.op, s.inst = c, "cycle", []
    for i, d in enumerate(_instances(c)):
        t = _prepare_one(d, seed + 1000 * i, "")
        t.dg, t.gg = _make(d, t.parset), _make(d, t.parset)
        t.dg.initialiseDegrid(t.axes, t.model)
        t.gg.initialiseGrid(t.axes, t.shape)
        s.inst.append(t)
    s.cyc = G.MajorCycle([t.dg for t in s.inst], [t.gg for t in s.inst], [t.obs for t in s.inst])
    return s


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def _clear(s):
    if s.c["host"]:
        s.cube.zero_()
    else:
        with torch.cuda.stream(s.stream):
            s.cube.zero_()


def run(s):
    if s.op == "chunk":
        _clear(s)
        s.dg.degrid(s.acc)
        return {"vis": s.cube}
    if s.op == "predict":
        s.dg.initialiseDegrid(s.axes, s.model)
        _clear(s)
        s.dg.degrid(s.acc)
        s.dg.finaliseDegrid()
        return {"vis": s.cube}
    if s.op in ("image", "psf", "cold"):
        g = _make(s.c, s.parset) if s.op == "cold" else s.gg
        g.initialiseGrid(s.axes, s.shape, dopsf=s.op == "psf")
        g.grid(s.obs)
        g.finaliseGrid(s.image)
        g.finaliseWeights(s.weights)
        return {"image": s.image, "weights": s.weights}
    if s.op == "major":
        s.dg.initialiseDegrid(s.axes, s.model)
        _clear(s)
        s.dg.degrid_plan(s.plan, s.acc)
        with torch.cuda.stream(s.stream):
            torch.sub(s.keep["vis"], s.cube, out=s.resid)
        s.dg.synchronize()
        s.gg.initialiseGrid(s.axes, s.shape)
        s.gg.grid_plan(s.plan, s.racc)
        s.gg.finaliseGrid(s.image)
        return {"vis": s.cube, "image": s.image}
    for t in s.inst:
        t.dg.initialiseDegrid(t.axes, t.model)
        t.gg.initialiseGrid(t.axes, t.shape)
    s.cyc.run(1)
    for t in s.inst:
        t.gg.finaliseGrid(t.image)
    return {"images": [t.image for t in s.inst]}


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def _ngrids(c):
    return {"WStack": c["nwplanes"], "WStackWProject": c["nwstacks"]}.get(c["gridder"], 1)


def work(case):
    c = _full(case)
    total = {"bytes": 0.0, "flops": 0.0}
    for i, d in enumerate(_instances(c)):
        uvw, freq, wmax = _track(d, 1 + 1000 * i)
        n = len(uvw) * d["nchan"]
        width = 2 * _cf(d, wmax, freq, "cpu", support_only=True) + 1
        passes = 2 if d["op"] in ("major", "cycle") else 1
        cells = d["nx"] ** 2 * d["npol"] * d["nchan_img"]
        cube = 8.0 * n * d["npol"]
        b = uvw.nbytes + cube * (2 if passes == 2 else 1)
        if d["op"] != "psf":
            b += 4.0 * cells * passes
        if d["weights"]:
            b += cube
        if d["flags"]:
            b += n * d["npol"]
        if d["op"] in ("image", "psf", "cold"):
            b += 4.0 * cells * (2 if d["op"] == "psf" else 1)
        f = 8.0 * width ** 2 * n * d["npol"] * passes
        if d["op"] != "chunk":
            f += passes * _ngrids(d) * cells * 5.0 * 2 * math.log2(d["nx"])
        if d["op"] == "cold":
            f += d["nwplanes"] * d["nchan"] * d["maxsupport"] ** 2 * 5.0 * 2 * math.log2(d["maxsupport"])
        total["bytes"] += b
        total["flops"] += f
    return total


# --------------------------------------------------------------------------
# the same outputs in 64 bits
# --------------------------------------------------------------------------
def _grdsf(c, nu):
    """Prolate spheroidal function psi_{1,0}(c, nu) over (1 - nu^2)^(1/2), 1 at 0: eigenvector of the
    spheroidal equation in orthonormal associated Legendre functions of order 1."""
    nt, m, c2 = 24, 1, c * c
    b = np.zeros((nt, nt))
    for r in range(nt):
        l = 2 * r + m
        b[r, r] = l * (l + 1) + c2 * (2 * l * (l + 1) - 2 * m * m - 1) / ((2 * l - 1) * (2 * l + 3))
        if r + 1 < nt:
            b[r, r + 1] = b[r + 1, r] = c2 / (2 * l + 3) * math.sqrt(
                (l + m + 1) * (l + m + 2) * (l - m + 1) * (l - m + 2) / ((2 * l + 1) * (2 * l + 5)))
    w, v = np.linalg.eigh(b)
    a = v[:, 0]

    def series(x):
        s = np.sqrt(np.maximum(0.0, 1.0 - x * x))
        p0, p1 = -math.sqrt(0.75) * s, None
        acc, prev, cur = a[0] * p0, p0, x * math.sqrt(5.0) * p0
        for l in range(3, 2 * nt):
            nxt = math.sqrt((4.0 * l * l - 1) / (l * l - 1.0)) * (
                x * cur - math.sqrt(((l - 1.0) ** 2 - 1) / (4.0 * (l - 1.0) ** 2 - 1)) * prev)
            prev, cur = cur, nxt
            if l % 2 == 1:
                acc = acc + a[(l - 1) // 2] * cur
        return acc

    nu = np.asarray(nu, dtype=np.float64)
    inside = np.abs(nu) < 1.0
    x = np.where(inside, nu, 0.0)
    return np.where(inside, series(x) / series(np.zeros(1))[0] / np.sqrt(1.0 - x * x), 0.0)


def _edge(f):
    f = f.copy()
    f[0] = 3.0 * (f[1] - f[2]) + f[3]
    if len(f) % 2:
        f[-1] = f[0]
    return f


def _cfft(a, forward=True):
    s = torch.fft.ifftshift(a, dim=(-2, -1))
    s = torch.fft.fft2(s) if forward else torch.fft.ifft2(s, norm="forward")
    return torch.fft.fftshift(s, dim=(-2, -1))


def _wterms(n, wmax):
    half = (n - 1) // 2
    return (np.arange(n) - half) * (wmax / half if n > 1 else 1.0)


def _support(plane, os_):
    """Support of one transformed plane: furthest cell of the peak's row and column above the cutoff."""
    a = plane.abs()
    k = int(torch.argmax(a))
    py, px = divmod(k, a.shape[1])
    cut = 1e-3 * float(a[py, px])
    row = torch.nonzero(a[py] > cut).flatten()
    col = torch.nonzero(a[:, px] > cut).flatten()
    h = a.shape[0] // 2
    size = 2 * max(abs(int(q) - h) for q in (row[0], row[-1], col[0], col[-1]))
    return max(3, size // (2 * os_))


def _cf(c, wmax, freq, dev, support_only=False):
    """CF matrices [plane][fv][fu][y][x] in complex128 (planes of a channel follow each other), or the support."""
    os_, kind = c["oversample"], c["gridder"]
    if kind in ("SphFunc", "WStack"):
        os_ = 128 if kind == "WStack" else os_
        if support_only:
            return 3
        i = np.arange(7)
        nu = np.abs(os_ * (i[None, :] - 3) + np.arange(os_)[:, None]) / (3.0 * os_)
        b = torch.from_numpy(_grdsf(3 * math.pi, nu) * (1 - nu * nu)).to(dev)
        cf = b[:, None, :, None] * b[None, :, None, :]
        cf = cf / cf.abs().sum((-1, -2), keepdim=True)
        return cf[None].to(torch.complex128)
    n, q = c["maxsupport"], c["maxsupport"] // os_
    if kind == "WStackWProject":
        wmax = 0.5 * wmax / ((c["nwstacks"] - 1) // 2)
    cell = c["cell"] * ARCSEC
    uvcell = 1.0 / (cell * c["nx"])
    aw = kind == "AWProject"
    ccell = 1.0 / (q * uvcell)
    terms = _wterms(c["nwplanes"], wmax)
    x = (torch.arange(n if aw else q, device=dev, dtype=torch.float64) - (n if aw else q) // 2) * ccell
    r2 = x[None, :] ** 2 + x[:, None] ** 2
    inside = r2 < 1.0
    bend = 1.0 - torch.sqrt(torch.where(inside, 1.0 - r2, torch.ones_like(r2)))
    amps = []
    if aw:
        o = torch.arange(n, device=dev, dtype=torch.float64) - n / 2.0
        rr = o[None, :] ** 2 + o[:, None] ** 2
        for f in freq[:1] if support_only else freq:
            cm = uvcell / os_ * (C_LIGHT / f)
            rmax2, rmin2 = (c["dish"] / (2 * cm)) ** 2, (1.0 / (2 * cm)) ** 2
            if rmin2 + 1 >= rmax2:
                rmin2 -= 1
            disk = ((rr >= rmin2) & (rr <= rmax2)).to(torch.float64)
            pat = _cfft(torch.complex(disk, torch.zeros_like(disk)) / float(disk.sum()), False)
            amps.append((pat.abs() ** 2).cpu() if support_only else pat.abs() ** 2)
    else:
        t = torch.from_numpy(_edge(_grdsf(3 * math.pi, np.abs(np.arange(q) - q // 2) / float(q // 2)))).to(dev)
        amps.append(t[None, :] * t[:, None])

    def plane(amp, w):
        s = torch.where(inside, torch.polar(amp, -2 * math.pi * w * bend), torch.zeros((), dtype=torch.complex128,
                                                                                       device=dev))
        if not aw:
            buf = torch.zeros((n, n), dtype=torch.complex128, device=dev)
            lo = n // 2 - q // 2
            buf[lo:lo + q, lo:lo + q] = s
            s = buf
        s = _cfft(s)
        return s / float(n * n) if aw else s

    S = _support(plane(amps[0], terms[0]), os_)
    if support_only:
        return S
    k = (torch.arange(-S, S + 1, device=dev)[None, :] * os_ + torch.arange(os_, device=dev)[:, None] + n // 2)
    out = torch.empty((len(amps) * len(terms), os_, os_, 2 * S + 1, 2 * S + 1), dtype=torch.complex128, device=dev)
    for a, amp in enumerate(amps):
        for i, w in enumerate(terms):
            cut = plane(amp, float(w))[k[:, None, :, None], k[None, :, None, :]]
            out[a * len(terms) + i] = cut * float(os_ * os_) if aw else cut / cut.real.sum((-1, -2), keepdim=True)
    return out


def _nint(x):
    return torch.where(x > 0, torch.trunc(x + 0.5), torch.trunc(x - 0.5))


def _indices(c, d, cf, dev):
    """Per sample [chan][row]: cell u, v, matrix index, grid plane, image channel, whether it is on the grid and used."""
    os_ = cf.shape[1]
    f = d["freq"][:, None]
    U = d["uvw"]
    uvcell = 1.0 / (c["cell"] * ARCSEC * float(c["nx"]))

    def axis(x):
        s = f * x[None] / (C_LIGHT * uvcell)
        i = _nint(s)
        fr = _nint(os_ * (i - s))
        i, fr = torch.where(fr < 0, i + 1, torch.where(fr >= os_, i - 1, i)), torch.where(
            fr < 0, fr + os_, torch.where(fr >= os_, fr - os_, fr))
        return i.long() + c["nx"] // 2, fr.long()

    iu, fu = axis(U[:, 0])
    iv, fv = axis(U[:, 1])
    w = U[None, :, 2] / C_LIGHT * f
    wmax = d["wmax"]
    gp, cp = torch.zeros_like(iu), torch.zeros_like(iu)

    def plane_of(ww, n, top):
        half = (n - 1) // 2
        return half + _nint(ww / (top / half)).long()

    kind = c["gridder"]
    if kind == "WStack":
        gp = plane_of(w, c["nwplanes"], wmax)
    elif kind == "WStackWProject":
        gp = plane_of(w, c["nwstacks"], wmax)
        half = (c["nwstacks"] - 1) // 2
        cp = plane_of(w - (gp - half).double() * (wmax / half), c["nwplanes"], 0.5 * (wmax / half))
    elif kind in ("WProject", "AWProject"):
        cp = plane_of(w, c["nwplanes"], wmax)
        if kind == "AWProject":
            cp = cp + c["nwplanes"] * torch.arange(c["nchan"], device=dev)[:, None]
    S = (cf.shape[-1] - 1) // 2
    used = torch.ones_like(iu, dtype=torch.bool) if d["flag"] is None else d["flag"][0] == 0
    ic = torch.zeros(c["nchan"], dtype=torch.long, device=dev)
    if c["nchan_img"] > 1:
        step = (c["f1"] - c["f0"]) / c["nchan_img"]
        ic = _nint((d["freq"] - (c["f0"] + 0.5 * step)) / step).long()
    on = used & (iu - S > 0) & (iv - S > 0) & (iu + S < c["nx"]) & (iv + S < c["nx"])
    return iu, iv, fu + os_ * (fv + os_ * cp), gp, ic[:, None].expand_as(iu), on, used


def _corrections(nx):
    h = nx // 2
    b = _edge(_grdsf(3 * math.pi, np.abs(np.arange(nx) - h) / float(h)))
    b = np.fft.fftshift(np.fft.fft(np.fft.ifftshift(b)))
    b[:h - 3] = 0
    b[h + 4:] = 0
    b = np.fft.fftshift(np.fft.ifft(np.fft.ifftshift(b))).real
    b = b / b[h]
    return np.where(np.abs(b) > 1e-10, 1.0 / b, 0.0)


def _image_factors(c, d, dev):
    """Grid correction [y][x] and the w-stack screens."""
    nx = c["nx"]
    corr = torch.ones((nx, nx), dtype=torch.float64, device=dev)
    if c["gridder"] != "AWProject":
        f = torch.from_numpy(_corrections(nx)).to(dev)
        corr = f[:, None] * f[None, :]
    if _ngrids(c) == 1:
        return corr, [None]
    x = (torch.arange(nx, device=dev, dtype=torch.float64) - nx // 2) * (c["cell"] * ARCSEC)
    r2 = x[None, :] ** 2 + x[:, None] ** 2
    bend = torch.where(r2 < 1.0, 1.0 - torch.sqrt(torch.clamp(1.0 - r2, min=0.0)), torch.zeros_like(r2))
    one = torch.ones_like(bend)
    return corr, [torch.polar(one, -2 * math.pi * float(w) * bend)
                  for w in _wterms(_ngrids(c), d["wmax"])]


def _mfs(c, d):
    if not c["mfs"]:
        return None
    ref = 0.5 * (c["f0"] + c["f1"]) * 1.1
    return ((d["freq"] - ref) / ref)[:, None]


def _phasor(d):
    if d["delay"] is None:
        return None
    ph = 2 * math.pi * d["freq"][:, None] * d["delay"][None] / C_LIGHT
    return torch.polar(torch.ones_like(ph), ph)


def _blocks(n, width):
    step = max(1, int(3e7) // width ** 2)
    for a in range(0, n, step):
        yield slice(a, min(n, a + step))


def _cells(nx, iu, iv, S, dev):
    o = torch.arange(-S, S + 1, device=dev)
    return ((iv[:, None, None] + o[None, :, None]) * nx + iu[:, None, None] + o[None, None, :]).reshape(len(iu), -1)


def _exact_predict(c, d, model, cf, dev):
    nx, S = c["nx"], (cf.shape[-1] - 1) // 2
    iu, iv, ci, gp, ic, on, used = _indices(c, d, cf, dev)
    corr, screens = _image_factors(c, d, dev)
    flat = cf.reshape(-1, cf.shape[-1] ** 2)
    out = torch.zeros(d["vis"].shape, dtype=torch.complex128, device=dev)
    val = torch.zeros_like(out)
    for p in range(c["npol"]):
        for ch in range(c["nchan_img"]):
            m = (model[ch, p].double() * corr).to(torch.complex128)
            for g, scr in enumerate(screens):
                grid = _cfft(m if scr is None else torch.conj(m * scr)).reshape(-1)
                sel = torch.nonzero((on & (gp == g) & (ic == ch)).reshape(-1)).flatten()
                for b in _blocks(len(sel), cf.shape[-1]):
                    k = sel[b]
                    cells = _cells(nx, iu.reshape(-1)[k], iv.reshape(-1)[k], S, dev)
                    val[p].view(-1)[k] = (flat[ci.reshape(-1)[k]] * torch.conj(grid[cells])).sum(1)
        mf, ph = _mfs(c, d), _phasor(d)
        if mf is not None:
            val[p] *= mf
        if ph is not None:
            val[p] *= ph
        # a used sample off the grid takes the value of the last one on it (rows outer, channels inner)
        t = val[p].t().reshape(-1)
        o = on.t().reshape(-1)
        last = torch.cummax(torch.where(o, torch.arange(len(o), device=dev), torch.full((), -1, device=dev)), 0).values
        t = torch.where(last >= 0, t[last.clamp(min=0)], torch.zeros_like(t)).reshape(d["nrow"], c["nchan"]).t()
        out[p] = torch.where(used, t, torch.zeros_like(t))
    return out


def _exact_image(c, d, vis, cf, dev, psf=False, weights=True):
    nx, S = c["nx"], (cf.shape[-1] - 1) // 2
    iu, iv, ci, gp, ic, on, _ = _indices(c, d, cf, dev)
    corr, screens = _image_factors(c, d, dev)
    flat = cf.reshape(-1, cf.shape[-1] ** 2)
    image = torch.zeros((c["nchan_img"], c["npol"], nx, nx), dtype=torch.float64, device=dev)
    wimg = None if c["gridder"] == "AWProject" else torch.zeros_like(image)
    mf, ph = _mfs(c, d), _phasor(d)
    for p in range(c["npol"]):
        wt = torch.ones_like(d["vis"][p].real, dtype=torch.float64)
        if d["noise"] is not None:
            wt = 1.0 / d["noise"][p].real.double() ** 2
        v = wt.to(torch.complex128) if psf else torch.conj(vis[p].to(torch.complex128)) * wt
        if ph is not None and not psf:
            v = v * ph
        if mf is not None:
            v = v * mf
        for ch in range(c["nchan_img"]):
            if wimg is not None:
                wimg[ch, p] = torch.where(on & (ic == ch), wt, torch.zeros_like(wt)).sum()
            for g, scr in enumerate(screens):
                grid = torch.zeros(nx * nx, dtype=torch.complex128, device=dev)
                sel = torch.nonzero((on & (gp == g) & (ic == ch)).reshape(-1)).flatten()
                for b in _blocks(len(sel), cf.shape[-1]):
                    k = sel[b]
                    cells = _cells(nx, iu.reshape(-1)[k], iv.reshape(-1)[k], S, dev)
                    t = (flat[ci.reshape(-1)[k]] * v.reshape(-1)[k][:, None]).reshape(-1)
                    parts = torch.view_as_real(grid)
                    parts[:, 0].index_add_(0, cells.reshape(-1), t.real)
                    parts[:, 1].index_add_(0, cells.reshape(-1), t.imag)
                back = _cfft(grid.reshape(nx, nx), False)
                image[ch, p] += (back if scr is None else back * scr).real
            image[ch, p] *= corr
    return {"image": image, "weights": wimg} if weights else image


def exact(case, seed):
    c = _full(case)
    cost = sum(i["ntime"] * 630.0 * i["nchan"] * i["npol"] for i in _instances(c)) * (
        2 if c["op"] in ("major", "cycle") else 1)
    if c["gridder"] == "WProject":
        cost *= 8.0 if c["nx"] * c["cell"] > 12000 else 2.0
    if cost > 3e7:
        return None          # minutes in 64 bits
    dev = _device()
    if c["op"] != "cycle":
        d = _data(c, seed)
        cf = _cf(c, d["wmax"], d["freq_np"], dev)
        if c["op"] in ("predict", "chunk"):
            return {"vis": _exact_predict(c, d, d["model"], cf, dev)}
        if c["op"] == "major":
            vis = _exact_predict(c, d, d["model"], cf, dev)
            return {"vis": vis, "image": _exact_image(c, d, d["vis"].to(torch.complex128) - vis, cf, dev,
                                                      weights=False)}
        return _exact_image(c, d, d["vis"], cf, dev, psf=c["op"] == "psf")
    images = []
    for i, e in enumerate(_instances(c)):
        d = _data(e, seed + 1000 * i)
        cf = _cf(e, d["wmax"], d["freq_np"], dev)
        vis = _exact_predict(e, d, d["model"], cf, dev)
        images.append(_exact_image(e, d, d["vis"].to(torch.complex128) - vis, cf, dev, weights=False))
    return {"images": images}
