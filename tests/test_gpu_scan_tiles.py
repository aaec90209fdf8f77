"""The scan of the bin histogram on either side of its two- and three-launch forms.

Up to 2,048 tiles of 4,096 bins every block of the scan adds up the tiles
before its own; that grows with the square of the tiles, so larger grids scan
the tiles' sums in a launch between.  Bin bounds must be the histogram's prefix
sums in both, at the edge and well beyond it.
"""
from __future__ import annotations

import numpy as np
import pytest

from pbf_b200 import Particles
from pbf_b200.scenes import Scene

pytestmark = pytest.mark.gpu

S = 1.2


def _grid(dims):
    """A scene whose grid has these bins (ceil(extent / s) + 2 an axis)."""
    return Scene("grid", (8, 8, 8), tuple((d - 2.5) * S for d in dims))


@pytest.mark.parametrize("dims,tiles", [((16, 16, 15), 1), ((16, 16, 16), 2), ((127, 256, 256), 2033),
                                        ((255, 181, 181), 2040), ((2047, 16, 256), 2048), ((128, 256, 256), 2049),
                                        ((300, 200, 181), 2652), ((400, 400, 400), 15626)])
def test_bin_bounds_at_the_scans_edge(dims, tiles):
    sc = _grid(dims)
    rng = np.random.default_rng(tiles)
    n = 5000
    box = np.array(sc.box_max, np.float32)
    x = (rng.uniform(0.0, 1.0, (n, 3)) * box).astype(np.float32)
    x[:40] = box * np.float32(0.5)  # a crowd
    x[40:80] = box                  # the last bins
    with Particles(sc.params(), n) as g:
        bins = g._lib.pbf_num_bins(g.ctx)
        assert bins == np.prod(dims) and (bins + 1 + 4095) // 4096 == tiles
        g.upload(x)
        g.find_neighbors()
        got = g.bins()
        count = np.bincount(got["sorted_keys"], minlength=bins)
        end = np.cumsum(count)
        assert np.array_equal(got["bin_end"], end) and np.array_equal(got["bin_begin"], end - count)
        cell = np.floor((x + np.float32(S)) / np.float32(S)).astype(np.int64)
        key = (cell[:, 2] * dims[1] + cell[:, 1]) * dims[0] + cell[:, 0]
        order = np.argsort(key, kind="stable")
        assert np.array_equal(got["sorted_ids"], order) and np.array_equal(got["sorted_keys"], key[order])
        assert g.stats()["error_flags"] == 0


def test_a_large_grid_scans_its_tiles_in_a_launch():
    launches = []
    for dims in ((2047, 16, 256), (128, 256, 256)):
        with Particles(_grid(dims).params(), 512) as g:
            launches.append(g.launches_per_step())
            g.upload(_grid((8, 8, 8)).positions())
            g.set_timing(True)
            g.step(1)
            assert sum(k["launches"] for k in g.kernel_times().values()) == launches[-1]
    assert launches[1] == launches[0] + 1
