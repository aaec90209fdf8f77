"""Scenes that share a 16-slot group of the walk bytes, in the persistent step.

A scene whose particles move far marks its lists to be walked whole while its
neighbours in memory may be passes ahead, between the viscosity pass that
writes the weights of the walked entries and the one that reads them: a mark
must stay within its own scene's slots.  Many small scenes of odd sizes, pressed
together so that most steps mark, must give the bits of a launch per pass.
"""
from __future__ import annotations

import numpy as np
import pytest

from pbf_b200 import Particles, _abi
from pbf_b200.scenes import Batch, Scene

pytestmark = pytest.mark.gpu
SHAPES = {"density": (2, 128, 0), "delta_p": (2, 128, 0), "viscosity": (2, 128, 0), "vorticity": (4, 128, 0),
          "apply_vorticity": (2, 128, 0)}


@pytest.mark.parametrize("squeeze", [0.99, 0.85])
@pytest.mark.parametrize("sizes", [[(3, 3, 3), (11, 13, 17), (5, 7, 3), (3, 5, 3)] * 6,
                                   [(3, 3, 3), (23, 19, 21), (7, 5, 5)] * 3])
def test_marks_stay_within_their_scene(sizes, squeeze):
    rng = np.random.default_rng(len(sizes))
    b = Batch("odd", tuple(Scene("s", k, (13.0, 13.0, 13.0), solve_steps=4) for k in sizes))
    x = (b.positions() * np.float32(squeeze)).astype(np.float32)
    v = rng.uniform(-6.0, 6.0, x.shape).astype(np.float32)
    assert any(o % 16 for o in b.offsets[1:-1])
    got = []
    for persistent in (False, True):
        with Particles.batch(b) as g:
            g.set_tuning(SHAPES)
            g.set_persistent(persistent)
            g.upload(x, v)
            out = []
            for _ in range(12):
                g.step(1)
                out += [g.get_array(_abi.ARRAY_POSITIONS), g.get_array(_abi.ARRAY_VELOCITIES)]
            got.append(out)
            assert g.stats()["error_flags"] == 0
    for a, c in zip(*got):
        assert np.isfinite(a).all() and np.array_equal(a, c)
