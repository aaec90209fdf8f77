"""PBF_FLAG_KEY_RANGE of the list fill: raised by the visits a list makes, not by those after it is full.

A particle in the grid's last bin along x has visits outside the grid.  In the
reference's order (x offset outer) they come last, so a list that its lower
bins fill makes none of them; a list that stays short makes them all, and at
the low edge they come first.  A few such particles of a warp are walked by
the whole warp, more by their own lanes: the flag is the same.
"""
from __future__ import annotations

import numpy as np
import pytest

from pbf_b200 import Particles, _abi, make_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exact", [0, 1])
@pytest.mark.parametrize("edge", [1, 4, 12])
@pytest.mark.parametrize("below,high", [(80, True), (60, True), (59, True), (20, True), (80, False)])
def test_flags_of_edge_particles(exact, edge, below, high):
    sc = make_scene("dam_2k", exact_math=exact, neighbor_cap=60)
    p = sc.params()
    s = np.float32(p.neighbor_bin_spacing)
    rng = np.random.default_rng(below + edge)
    dimx = int(np.ceil((sc.box_max[0] - 0.0) / float(s))) + 2
    face = (dimx - 2) * s if high else np.float32(0.0)  # the last bin begins here; the first one ends
    sign = 1 if high else -1
    near = np.float32([face, 3.5 * s, 3.5 * s])
    inner = near + rng.uniform(0.02, 0.1, (below, 3)) * [-sign, 1, 1]
    outer = near + rng.uniform(0.02, 0.1, (edge, 3)) * [sign, 1, 1]
    x = np.concatenate([inner, outer]).astype(np.float32)
    with Particles(p, len(x)) as g:
        g.upload(np.clip(x, 0.0, np.float32(sc.box_max)).astype(np.float32))
        g.set_array(_abi.ARRAY_POSITION_STARS, x)
        g.find_neighbors()
        count = g.neighbors(60)[1]
        assert np.all(count[below:] == min(60, below + edge - 1))
        full = high and below + edge - 1 >= 60  # before the visits outside come
        assert g.stats()["error_flags"] == (0 if full else _abi.PBF_FLAG_KEY_RANGE)
