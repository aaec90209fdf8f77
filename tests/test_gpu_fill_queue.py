"""The queue of particles the mask fill leaves: one entry a warp, never more.

Random lanes of every warp sit on bin faces, so that the float re-hash sends
them around the row tests and the warp reaches the queue in two parts: as many
entries as there are warps, the queue exactly full, each naming its warp's
lanes.  A warp that queued its parts one by one would take an entry past the
last.  All lists must be the exact ones, bit for bit.
"""
from __future__ import annotations

import numpy as np
import pytest

from pbf_b200 import Particles, make_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65536, 65537, 65567, 70000])
@pytest.mark.parametrize("share", [0.05, 0.5])
def test_a_warp_is_queued_once(n, share):
    sc = make_scene("dam_65k", gamma=0.0)
    p = sc.params()
    rng = np.random.default_rng(n)
    s = np.float32(p.neighbor_bin_spacing)
    i = np.arange(n)
    x = (np.stack([i % 41, i // 41 % 41, i // 1681], 1) * 0.5 + 1.0 + rng.uniform(-0.1, 0.1, (n, 3))).astype(np.float32)
    face = np.nextafter((np.round(x / s) * s).astype(np.float32), np.float32(-99))
    x = np.where((rng.random(n) < share)[:, None], face, x).astype(np.float32)
    got = []
    for exact in (0, 1):
        p.exact_math = exact
        with Particles(p, n) as g:  # as many slots as particles: the queue has no entry to spare
            g.upload(x)
            g.find_neighbors()
            got.append(g.neighbors(p.neighbor_cap))
            assert g.stats()["error_flags"] == 0
    assert np.array_equal(got[0][1], got[1][1])
    assert np.array_equal(got[0][0], got[1][0])
