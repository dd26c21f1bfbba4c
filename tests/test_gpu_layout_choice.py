"""Which record order and grid kernel a pass takes: the handle's own choice
(set_grid_variant, the autotuner, or the automatic choice of its gridder kind),
never what a plan or another handle happens to bring along."""
import math

import numpy as np
import pytest

from parity_helpers import make_pair

pytestmark = pytest.mark.gpu

ARCSEC = math.pi / (180 * 3600)
CELL = 40.0 * ARCSEC
NX = 512


def _data(npol, seed, diameter=600.0):
    from yandasoft_b200 import simulate
    return simulate.make_dataset(duration_s=80.0, nchan=3, npol=npol, seed=seed, diameter_m=diameter)


def _wproject(support, os_=8, **more):
    params = {"wmax": 6000.0, "nwplanes": 5, "oversample": os_, "maxsupport": 1024, "limitsupport": support, **more}
    return make_pair("WProject", params)[1]


def _grid(g, npol, run):
    from yandasoft_b200.gridder import Axes
    g.initialiseGrid(Axes(CELL, CELL), (NX, NX, npol, 1))
    run(g)
    return np.stack(g.grids())


@pytest.mark.parametrize("support,npol", [(3, 2), (6, 4), (19, 1)])
def test_plan_does_not_choose_the_order(support, npol):
    """A WProject plan made under variant 64 holds both record orders; under
    the automatic choice it grids CF-major, the same bits as a plan made
    without, through this handle and through another of the same parset."""
    from yandasoft_b200.gridder import Accessor, Axes
    ds = _data(npol, 300 + support)
    acc = Accessor(ds.uvw, ds.freq, ds.vis).to_device()
    want = _grid(_wproject(support), npol, lambda g: g.grid(acc))
    assert np.abs(want).max() > 0
    g = _wproject(support)
    g.set_grid_variant(64)
    g.initialiseGrid(Axes(CELL, CELL), (NX, NX, npol, 1))
    plan = g.plan(acc)
    planes = _grid(g, npol, lambda g: g.grid_plan(plan, acc))
    assert not np.array_equal(planes, want)              # the other order rounds differently
    for variant in (0, 1):
        g.set_grid_variant(variant)
        assert np.array_equal(_grid(g, npol, lambda g: g.grid_plan(plan, acc)), want)
    assert np.array_equal(_grid(_wproject(support), npol, lambda g: g.grid_plan(plan, acc)), want)


@pytest.mark.parametrize("kind,os_", [("AWProject", 4), ("AWProject", 8), ("WProject", 4), ("SphFunc", 8)])
def test_tuning_serves_its_own_class(kind, os_):
    """What the autotuner keeps for one gridder kind and oversampling says
    nothing of another's kernels: a fresh WProject handle of the same padded CF
    width and polarisations grids its untuned bits after either was tuned."""
    from yandasoft_b200 import gridder as G
    npol = 4
    ds = _data(npol, 330)
    acc = G.Accessor(ds.uvw, ds.freq, ds.vis).to_device()
    axes = G.Axes(CELL, CELL)
    G.autotune_reset()
    try:
        fresh = _wproject(6)
        want = _grid(fresh, npol, lambda g: g.grid(acc))
        info = fresh.plan(acc).info()
        more = {"diameter": "12m", "blockage": "1m", "cutoff": 1e-3} if kind == "AWProject" else {}
        params = {"wmax": 2500.0, "nwplanes": 5, "oversample": os_, "maxsupport": 512, "limitsupport": 6, **more}
        tuner = make_pair(kind, params if kind != "SphFunc" else {})[1]
        tuner.initialiseGrid(axes, (NX, NX, npol, 1))
        rep = tuner.autotune(acc, max_trials=12)
        assert (rep["cf_width"], rep["npol"]) == (16, npol)
        g = _wproject(6)
        assert np.array_equal(_grid(g, npol, lambda g: g.grid(acc)), want)
        assert g.plan(acc).info() == info
    finally:
        G.autotune_reset()


@pytest.mark.parametrize("npol", [1, 4])
@pytest.mark.parametrize("variant", [64, 65, 66, 67, 80, 194])
def test_plane_major_bits_beside(npol, variant):
    """Bit 64 stands alone: the bits up to 128 beside it change nothing, and a
    table that the plane-major kernel does not take (CFs of several sizes, up
    to 16 wide) is gridded as with variant 1, bit for bit."""
    from yandasoft_b200.gridder import Accessor
    ds = _data(npol, 340)
    acc = Accessor(ds.uvw, ds.freq, ds.vis).to_device()
    for more, same in (({}, 64), ({"variablesupport": True}, 1)):
        out = []
        for v in (variant, same):
            g = _wproject(6, **more)
            g.set_grid_variant(v)
            out.append(_grid(g, npol, lambda g: g.grid(acc)))
        sizes = {c.shape for c in g.convolution_functions() if c is not None}
        assert (len(sizes) > 1) == bool(more)
        assert np.abs(out[1]).max() > 0
        assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("kind,support", [("AWProject", 6), ("WProject", 6)])
def test_tuner_times_the_automatic_choice(kind, support):
    """default_ms is the time of what an untuned handle runs (plane-major for
    AWProject, CF-major for the others): with one trial it is that trial's, and
    the choice kept grids the untuned bits."""
    from yandasoft_b200 import gridder as G
    ds = _data(2, 350)
    acc = G.Accessor(ds.uvw, ds.freq, ds.vis).to_device()
    more = {"diameter": "12m", "blockage": "1m", "cutoff": 1e-3} if kind == "AWProject" else {}
    params = {"wmax": 2500.0, "nwplanes": 5, "oversample": 4, "maxsupport": 512, "limitsupport": support, **more}
    G.autotune_reset()
    try:
        want = _grid(make_pair(kind, params)[1], 2, lambda g: g.grid(acc))
        tuner = make_pair(kind, params)[1]
        tuner.initialiseGrid(G.Axes(CELL, CELL), (NX, NX, 2, 1))
        rep = tuner.autotune(acc, max_trials=1)
        assert rep["trials"] == 1 and rep["variant"] == (64 if kind == "AWProject" else 1)
        assert rep["default_ms"] == rep["best_ms"] > 0
        assert np.array_equal(_grid(tuner, 2, lambda g: g.grid(acc)), want)
    finally:
        G.autotune_reset()


@pytest.mark.parametrize("more,variant", [({"variablesupport": True}, 0), ({}, 2), ({}, 17)])
def test_inverse_is_made_with_the_plan(more, variant):
    """Layouts and tables whose kernel reads the inverse permutation get it with
    the plan, before any pass: the first pass over a plan launches what every
    later one does."""
    from yandasoft_b200 import gridder as G
    ds = _data(2, 360)
    acc = G.Accessor(ds.uvw, ds.freq, ds.vis).to_device()
    g = _wproject(6, **more)
    g.set_grid_variant(variant)
    g.initialiseGrid(G.Axes(CELL, CELL), (NX, NX, 2, 1))
    plan = g.plan(acc)
    n, out = [], []
    for _ in range(2):
        before = G.kernel_launch_count()
        out.append(_grid(g, 2, lambda g: g.grid_plan(plan, acc)))
        n.append(G.kernel_launch_count() - before)
    assert n[0] == n[1]
    assert np.abs(out[0]).max() > 0 and np.array_equal(out[0], out[1])


def test_inverse_for_another_layout():
    """A plan made under the automatic choice has no inverse permutation; the
    first pass that needs it makes it, and the next one, of another handle on
    another stream, finds it complete."""
    from yandasoft_b200.gridder import Accessor, Axes
    ds = _data(4, 370)
    acc = Accessor(ds.uvw, ds.freq, ds.vis).to_device()
    a, b = _wproject(6), _wproject(6)
    a.initialiseGrid(Axes(CELL, CELL), (NX, NX, 4, 1))
    want = _grid(a, 4, lambda g: g.grid(acc))
    for variant in (16, 17):
        ref = _wproject(6)
        ref.set_grid_variant(variant)
        want = _grid(ref, 4, lambda g: g.grid(acc))
        plan = a.plan(acc)
        for g in (a, b, a):
            g.set_grid_variant(variant)
            assert np.array_equal(_grid(g, 4, lambda g: g.grid_plan(plan, acc)), want)
        a.set_grid_variant(0)


@pytest.mark.parametrize("kind,variant", [("AWProject", 0), ("WProject", 64)])
def test_slot_beyond_32_bits(kind, variant):
    """A tile whose slot the plane-major kernel cannot index (4 polarisations,
    (23200 + 12)^2 cells: above 2^31 elements) is refused, as by variant 1."""
    from yandasoft_b200 import gridder as G
    ds = _data(4, 380)
    acc = G.Accessor(ds.uvw, ds.freq, ds.vis).to_device()
    more = {"diameter": "12m", "blockage": "1m", "cutoff": 1e-3} if kind == "AWProject" else {}
    params = {"wmax": 2500.0, "nwplanes": 5, "oversample": 4, "maxsupport": 512, "limitsupport": 6, **more}
    for v in (variant, 1):
        g = make_pair(kind, params)[1]
        g.set_tile(23200)
        g.set_item_size(1 << 20)
        g.set_grid_variant(v)
        g.initialiseGrid(G.Axes(CELL, CELL), (NX, NX, 4, 1))
        with pytest.raises(G.AskapError) as e:
            g.grid(acc)
        assert e.value.code == 9


def _kernels(run):
    """Names of the grid kernels that run() launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    names = " ".join(e.key for e in prof.key_averages())
    if "k_" not in names:
        pytest.skip("the profiler traced no kernels")
    return {k for k in ("k_grid<", "k_grid_cf<", "k_grid_pl<") if k in names}


@pytest.mark.parametrize("support,npol,kernel", [
    (19, 4, "k_grid_cf<"), (20, 1, "k_grid_cf<"), (21, 1, "k_grid<"), (21, 2, "k_grid_cf<"), (22, 3, "k_grid<"),
    (22, 4, "k_grid_cf<"), (23, 1, "k_grid<"), (23, 2, "k_grid<"), (23, 4, "k_grid<"), (24, 1, "k_grid_cf<"),
    (24, 4, "k_grid_cf<")])
def test_cf_major_kernel_by_width(support, npol, kernel):
    """CF-major passes take the faster of their two kernels (widths around 47,
    where k_grid's padding is thin); the sums are the same bit for bit."""
    import bench
    from yandasoft_b200.gridder import Accessor
    ds = _data(npol, 390 + support)
    acc = Accessor(ds.uvw, ds.freq, ds.vis).to_device()
    out = []
    for variant in (0, 2):
        g = _wproject(support, 4, wmax=12000.0)
        g.set_tile(48 if support < 24 else 56)
        g.set_grid_variant(variant)
        out.append(_grid(g, npol, lambda g: g.grid(acc)))
        assert g.support()[0] == support
        if variant == 0:
            assert _kernels(lambda: g.grid(acc)) == {kernel}
            assert bench.grid_kernel(variant, support, npol) + "<" == kernel    # the name that the bench prints
    assert np.abs(out[0]).max() > 0 and np.array_equal(out[0], out[1])


@pytest.mark.parametrize("support,npol,nchan,dt,kernel", [
    (3, 1, 16, 1200.0, "k_grid_pl<"), (6, 1, 16, 1200.0, "k_grid_cf<"), (6, 1, 16, 0.5, "k_grid_pl<"),
    (6, 1, 8, 1200.0, "k_grid_pl<"), (6, 2, 16, 1200.0, "k_grid_pl<"), (12, 4, 16, 1200.0, "k_grid_pl<"),
    (14, 2, 16, 1200.0, "k_grid_cf<"), (14, 2, 16, 0.5, "k_grid_pl<"), (19, 1, 16, 1200.0, "k_grid_cf<"),
    (19, 1, 16, 0.5, "k_grid_pl<"), (23, 2, 16, 1200.0, "k_grid<"), (23, 2, 16, 0.5, "k_grid_pl<"),
    (23, 4, 16, 1200.0, "k_grid_pl<")])
def test_awproject_order_by_samples(support, npol, nchan, dt, kernel):
    """AWProject's automatic choice: plane-major, but CF-major where the samples
    of a CF plane hardly share footprints (integrations 20 minutes apart; eight
    of half a second do) and the CFs are wide or the polarisation single, unless
    the CF-major kernel needs several passes or the chunk is small.  Through a
    plan and through grid(), whose plans serve gridding only; either order's grid agrees with the
    other's."""
    from yandasoft_b200 import simulate
    from yandasoft_b200.gridder import Accessor
    ds = simulate.make_dataset(duration_s=8 * dt, dt_s=dt, nchan=nchan, npol=npol, seed=400, diameter_m=600.0)
    acc = Accessor(ds.uvw, ds.freq, ds.vis).to_device()
    params = {"wmax": 5500.0, "nwplanes": 17, "oversample": 4, "maxsupport": 512, "limitsupport": support,
              "diameter": "12m", "blockage": "1m", "cutoff": 1e-3}
    out = []
    for variant in (0, 1, 64):
        g = make_pair("AWProject", params)[1]
        g.set_grid_variant(variant)
        g.set_tile(48)
        out.append(_grid(g, npol, lambda g: g.grid(acc)))
        assert g.support()[0] == support
        if variant == 0:
            assert _kernels(lambda: g.grid(acc)) == {kernel}
            plan = g.plan(acc)
            assert _kernels(lambda: g.grid_plan(plan, acc)) == {kernel}
            iu, iv, cfi, st = plan.samples(g, acc)
            on = st == 3
            cells = np.unique(np.stack([cfi[on] // 16, iu[on], iv[on]]), axis=1).shape[1]
            print("%.2f samples per CF plane and cell" % (on.sum() / cells))
    assert np.array_equal(out[0], out[2] if kernel == "k_grid_pl<" else out[1])
    assert np.linalg.norm(out[1] - out[2]) <= 1e-5 * np.linalg.norm(out[1])
