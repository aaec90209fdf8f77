"""Density/lambda and delta-p with both lanes' sums in one thread.

From 196,608 (delta-p) and 262,144 particles on, the two-lane shapes run one
thread a particle; a batch's scenes, and the persistent step of the same batch,
whose passes keep two lanes, show that the bits are the same.
"""
from __future__ import annotations

import numpy as np
import pytest

from pbf_b200 import Particles, _abi, make_batch, make_scene

pytestmark = pytest.mark.gpu

SHAPES = {"density": (2, 128), "delta_p": (2, 128), "viscosity": (2, 128), "vorticity": (4, 128),
          "apply_vorticity": (2, 128)}


@pytest.mark.parametrize("squeeze", [1.0, 0.9])
@pytest.mark.parametrize("scenes,n_max", [(5, 60000), (9, 65536)])  # past the first, past both sizes
def test_batch_equals_its_scenes_and_the_persistent_step(scenes, n_max, squeeze):
    b = make_batch(scenes, seed=21, n_min=30000, n_max=n_max)
    x = (b.positions() * np.float32(squeeze)).astype(np.float32)
    assert b.n >= 196608 and (scenes == 5 or b.n >= 262144)
    got = []
    for persistent in (False, True):
        with Particles.batch(b) as g:
            g.set_tuning(SHAPES)
            if persistent:
                g.set_persistent(True)
            g.upload(x)
            g.step(3)
            assert g.stats()["error_flags"] == 0
            got.append({w: g.get_array(w) for w in (_abi.ARRAY_POSITIONS, _abi.ARRAY_VELOCITIES, _abi.ARRAY_LAMBDAS)})
    for w, a in got[0].items():
        assert np.array_equal(a, got[1][w]), w
    sc, end = b.scenes[1], b.offsets[1:3]
    with Particles(sc.params(), sc.n) as g:
        g.set_tuning(SHAPES)
        g.upload(x[end[0]:end[1]])
        g.step(3)
        for w, a in got[0].items():
            assert np.array_equal(g.get_array(w), a[end[0]:end[1]]), w


@pytest.mark.parametrize("options", [{}, {"scorr": (0.1, 4.0, 0.2)}])
def test_lanes_agree(options):
    """Four lanes (another order of the sums) against the one-thread form of two."""
    sc = make_scene("dam_65k", lattice=(64, 65, 67), box_max=(80.0, 81.0, 83.0), **options)
    x = (sc.positions() * np.float32(0.95)).astype(np.float32)
    res = []
    for lanes in (2, 4):
        with Particles(sc.params(), sc.n) as g:
            g.set_tuning({"density": (lanes, 128), "delta_p": (lanes, 128)})
            g.upload(x)
            g.step(1)
            res.append((g.positions(), g.densities()))
    assert np.abs(res[0][0] - res[1][0]).max() <= 1e-5 * max(sc.box_max)
    np.testing.assert_allclose(res[0][1], res[1][1], rtol=1e-5)
