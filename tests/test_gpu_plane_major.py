"""k_grid_pl (plane-major gridding) and k_grid_cf (CF-major) against the oracle at the edges of its
layouts: CF widths around multiples of a warp's 32 residues, one and several
parts and groups, staged and unstaged tables, one to four polarisations, tiles
and work items of odd sizes, and scratch in several batches."""
import math

import numpy as np
import pytest

from parity_helpers import make_pair, rel_l2

pytestmark = pytest.mark.gpu

ARCSEC = math.pi / (180 * 3600)
CELL = 40.0 * ARCSEC
NX = 512
# grids relative L2 of the repository's parity tests: FP32 sums in another order
TOL = 1e-5


def _inputs(npol, diameter, seed):
    from yandasoft_b200 import simulate
    ds = simulate.make_dataset(duration_s=80.0, nchan=3, npol=npol, seed=seed, diameter_m=diameter)
    rng = np.random.default_rng(seed + 1)
    flag = np.zeros(ds.vis.shape, dtype=bool, order="F")
    flag[rng.random(ds.vis.shape[:2]) < 0.05, :] = True
    noise = np.asfortranarray(rng.uniform(0.5, 2.0, ds.vis.shape).astype(np.float32).astype(np.complex64))
    return ds, flag, noise, rng.standard_normal(ds.nrow) * 0.05


def _pair(support, os_):
    """WProject gridders whose CFs (support about 35 uncut) are cut to `support`, on the GPU's own CFs."""
    params = {"wmax": 6000.0, "nwplanes": 5, "oversample": os_, "maxsupport": 1024, "limitsupport": support}
    return make_pair("WProject", params)


def _adopt_cf(og, gg):
    og.cache.cfs = [None if c is None else np.asfortranarray(c) for c in gg.convolution_functions()]
    og._flat = og.cache.flatten()


@pytest.mark.parametrize("support,os_,npol,tile,item,diameter,mode", [
    (3, 4, 1, 0, 0, 600.0, ""), (3, 8, 2, 24, 300, 600.0, ""), (3, 8, 4, 8, 64, 60.0, "psf"),
    (4, 8, 4, 40, 5000, 60.0, ""), (6, 8, 4, 32, 700, 600.0, ""), (6, 8, 3, 32, 257, 600.0, "pcf"),
    (6, 8, 1, 33, 2048, 60.0, ""), (7, 8, 4, 16, 129, 600.0, ""), (8, 4, 2, 56, 100, 600.0, "pcf"),
    (9, 8, 4, 40, 3000, 60.0, ""), (12, 4, 2, 24, 511, 600.0, ""), (13, 4, 4, 64, 1000, 60.0, ""),
    (15, 4, 1, 32, 90, 600.0, "psf"), (19, 4, 4, 32, 400, 600.0, ""), (24, 4, 1, 56, 1300, 600.0, ""),
    (27, 4, 1, 48, 800, 60.0, "pcf"), (30, 4, 2, 32, 2000, 600.0, ""), (33, 4, 1, 88, 350, 600.0, "")])
def test_against_oracle(support, os_, npol, tile, item, diameter, mode):
    import oracle
    from yandasoft_b200.gridder import Accessor, Axes
    ds, flag, noise, delay = _inputs(npol, diameter, 100 + support)
    og, gg = _pair(support, os_)
    if tile:
        gg.set_tile(tile)
    if item:
        gg.set_item_size(item)
    kw = {"psf": {"dopsf": True}, "pcf": {"dopcf": True}}.get(mode, {})
    axes = Axes(CELL, CELL)
    acc = Accessor(ds.uvw, ds.freq, ds.vis, noise=noise, flag=flag, delay=delay).to_device()
    chunk = oracle.Chunk(uvw=ds.uvw, freq=ds.freq, vis=ds.vis, noise=noise, flag=flag, delay=delay)
    gg.set_grid_variant(64)
    gg.initialiseGrid(axes, (NX, NX, npol, 1), **kw)
    gg.grid(acc)
    assert gg.support()[0] == support
    direct = np.stack(gg.grids())
    sw = gg.sum_weights()
    og.initialise_grid(NX, NX, npol, 1, CELL, CELL, **kw)
    og.init_cf(chunk)
    _adopt_cf(og, gg)
    og.grid(chunk)
    ref = np.stack(og.grids)
    assert np.abs(ref).max() > 0
    assert rel_l2(direct, ref) < TOL
    assert np.array_equal(sw, og.sumw)
    # a plan of both record orders, run to run the same bits
    plan = gg.plan(acc)
    for k in range(2):
        gg.initialiseGrid(axes, (NX, NX, npol, 1), **kw)
        gg.grid_plan(plan, acc)
        again = np.stack(gg.grids())
        assert rel_l2(again, ref) < TOL
        assert k == 0 or np.array_equal(again, first)
        first = again
    # the CF-major kernel over the same plan
    gg.set_grid_variant(1)
    gg.initialiseGrid(axes, (NX, NX, npol, 1), **kw)
    gg.grid_plan(plan, acc)
    assert rel_l2(np.stack(gg.grids()), ref) < TOL


def test_scratch_batches():
    """More work items than the scratch holds at a time: the same sums as the
    CF-major kernel's, whose scratch holds them all."""
    from yandasoft_b200 import simulate
    from yandasoft_b200.gridder import Accessor, Axes
    ds = simulate.make_dataset(duration_s=600.0, nchan=16, npol=4, seed=5, diameter_m=600.0)
    acc = Accessor(ds.uvw, ds.freq, ds.vis).to_device()
    out = []
    for variant in (64, 1):
        _, gg = _pair(6, 8)
        gg.set_tile(64)
        gg.set_item_size(64)
        gg.set_grid_variant(variant)
        gg.initialiseGrid(Axes(CELL, CELL), (NX, NX, 4, 1))
        plan = gg.plan(acc)
        # four slots of (64 + 12)^2 cells x 4 polarisations per item
        assert plan.info()["nitems"] * 4 * 76 * 76 * 4 * 8 > 5 << 30
        gg.grid_plan(plan, acc)
        out.append((np.stack(gg.grids()), gg.sum_weights()))
    assert rel_l2(out[0][0], out[1][0]) < TOL
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("support,os_,npol,tile,item,diameter,mode", [
    (3, 4, 1, 0, 0, 600.0, ""), (3, 8, 2, 24, 300, 60.0, "psf"), (4, 8, 4, 40, 5000, 60.0, ""),
    (6, 8, 4, 32, 700, 600.0, ""), (6, 8, 3, 32, 257, 600.0, "pcf"), (7, 8, 4, 24, 129, 600.0, ""),
    (8, 4, 2, 56, 100, 600.0, "pcf"), (9, 8, 4, 40, 3000, 60.0, ""), (12, 4, 2, 24, 511, 600.0, ""),
    (15, 4, 1, 32, 90, 600.0, "psf"), (19, 4, 4, 32, 400, 600.0, ""), (24, 4, 1, 56, 1300, 600.0, ""),
    (27, 4, 1, 48, 800, 60.0, "pcf"), (30, 4, 2, 32, 2000, 600.0, "")])
def test_cf_major_same_sums(support, os_, npol, tile, item, diameter, mode):
    """The default CF-major kernel adds a cell's samples in the order of the
    padded layout (variant 2: half its threads, the same order), bit for bit;
    against the oracle within the order of its sums."""
    import oracle
    from yandasoft_b200.gridder import Accessor, Axes
    ds, flag, noise, delay = _inputs(npol, diameter, 200 + support)
    og, gg = _pair(support, os_)
    if tile:
        gg.set_tile(tile)
    if item:
        gg.set_item_size(item)
    kw = {"psf": {"dopsf": True}, "pcf": {"dopcf": True}}.get(mode, {})
    acc = Accessor(ds.uvw, ds.freq, ds.vis, noise=noise, flag=flag, delay=delay).to_device()
    out = []
    for variant in (0, 2):
        gg.set_grid_variant(variant)
        gg.initialiseGrid(Axes(CELL, CELL), (NX, NX, npol, 1), **kw)
        gg.grid(acc)
        out.append(np.stack(gg.grids()))
    assert gg.support()[0] == support
    assert np.array_equal(out[0], out[1])
    chunk = oracle.Chunk(uvw=ds.uvw, freq=ds.freq, vis=ds.vis, noise=noise, flag=flag, delay=delay)
    og.initialise_grid(NX, NX, npol, 1, CELL, CELL, **kw)
    og.init_cf(chunk)
    _adopt_cf(og, gg)
    og.grid(chunk)
    assert rel_l2(out[0], np.stack(og.grids)) < TOL


@pytest.mark.parametrize("support,os_,npol,tile", [(37, 4, 1, 56), (23, 4, 1, 108), (22, 4, 1, 28)])
def test_cf_major_full_ring(support, os_, npol, tile):
    """Widths and tiles at which k_grid_cf's ring fills its shared-memory
    budget to the byte, the kernel's static shared memory included."""
    from yandasoft_b200.gridder import Accessor, Axes
    ds, flag, noise, delay = _inputs(npol, 600.0, 200 + support)
    acc = Accessor(ds.uvw, ds.freq, ds.vis, noise=noise, flag=flag, delay=delay).to_device()
    out = []
    params = {"wmax": 9000.0, "nwplanes": 5, "oversample": os_, "maxsupport": 1024, "limitsupport": support}
    for variant in (0, 64):
        _, gg = make_pair("WProject", params)
        gg.set_tile(tile)
        gg.set_grid_variant(variant)
        gg.initialiseGrid(Axes(CELL, CELL), (NX, NX, npol, 1))
        gg.grid(acc)
        assert gg.support()[0] == support
        out.append((np.stack(gg.grids()), gg.sum_weights()))
    assert np.abs(out[1][0]).max() > 0
    assert rel_l2(out[0][0], out[1][0]) < TOL
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("support,npol,tile,item", [(6, 3, 8, 0), (24, 4, 16, 0), (6, 3, 64, 300), (24, 4, 56, 100)])
def test_halo_sums_of_passes(support, npol, tile, item):
    """Several passes of polarisations with nearly all tiles empty (one halo sum
    over all of them: 4096 and 1024 tiles, under 64 items) and with many items
    to a tile (a sum per pass): the padded layout's sums, bit for bit."""
    from yandasoft_b200 import simulate
    from yandasoft_b200.gridder import Accessor, Axes
    ds = simulate.make_dataset(duration_s=80.0 if item else 10.0, nchan=3 if item else 1, npol=npol, seed=7,
                               diameter_m=600.0 if item else 60.0)
    acc = Accessor(ds.uvw, ds.freq, ds.vis).to_device()
    out = []
    for variant in (1, 2):
        _, gg = _pair(support, 4)
        gg.set_tile(tile)
        if item:
            gg.set_item_size(item)
        gg.set_grid_variant(variant)
        gg.initialiseGrid(Axes(CELL, CELL), (NX, NX, npol, 1))
        plan = gg.plan(acc)
        assert (plan.info()["nitems"] * 16 < (NX // tile) ** 2) == (item == 0)
        gg.grid_plan(plan, acc)
        out.append(np.stack(gg.grids()))
    assert np.abs(out[0]).max() > 0 and np.array_equal(out[0], out[1])
