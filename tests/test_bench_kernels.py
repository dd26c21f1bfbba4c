"""The bench line names the kernels that run and charges them what they move (CPU)."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


@pytest.mark.parametrize("variant,support,npol,name", [
    (0, 6, 4, "k_grid_cf"), (1, 19, 4, "k_grid_cf"), (256, 6, 1, "k_grid_cf"), (0, 23, 1, "k_grid"),
    (1, 23, 2, "k_grid"), (0, 22, 2, "k_grid_cf"), (0, 22, 1, "k_grid"), (0, 24, 1, "k_grid_cf"), (2, 6, 4, "k_grid"),
    (17, 6, 4, "k_grid"), (64, 6, 4, "k_grid_pl"), (193 | 512, 23, 1, "k_grid_pl")])
def test_grid_kernel(variant, support, npol, name):
    import bench
    assert bench.grid_kernel(variant, support, npol) == name
    assert bench.kgrid_traffic({"tile": 32, "nvalid": 1000, "nitems": 10}, support, npol, name) > 0


def test_shared_memory_fraction():
    """The measured config-1 passes (1.39e9 visibilities, 169 taps, 1965 MHz)
    stay below the shared-memory pipe's own rate: 30.0 ms per 1.76e8
    visibilities for k_grid_cf, 93.5 ms for all in k_grid_pl."""
    import bench
    w = {"gridder": "WStackWProject", "nwstacks": 17, "nx": 4096}
    for name, nvis, ms in (("k_grid_cf", 4 * 4.4e7, 30.0), ("k_grid_pl", 1.39e9, 93.5)):
        d = {"nrow": int(nvis / 4 / 96), "nchan": 96}
        r = bench.roofline(w, d, {"tile": 32, "nvalid": int(nvis / 4), "nitems": 5000}, 6, 4, nvis, ms, 129.1, 6545.6,
                           "measured", 1.965e9, 22e6, (name, "k_degrid_r"))
        assert r["kernel"] == name
        assert 0 < r[name]["smem"]["frac"] < 1 and 0 < r["k_degrid_r"]["smem"]["frac"] < 1
