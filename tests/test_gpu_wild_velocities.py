"""An exact step from infinite velocities: x* is clamped into the box, but a nudge moves a particle by its velocity.

Two such particles are clamped into the same corner and nudged off one another,
to infinity; the bits that follow must be the oracle's, which walks whole lists.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import ARRAY_POSITIONS, ARRAY_VELOCITIES, OracleSim
from pbf_b200 import Particles, make_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.inf, -np.inf])
@pytest.mark.parametrize("n", [1203, 70000])
@pytest.mark.parametrize("gamma", [0.0, 1.0])
def test_two_infinite_velocities(bad, n, gamma):
    sc = make_scene("dam_2k" if n == 1203 else "dam_65k", gamma=gamma, exact_math=1)
    p = sc.params()
    box = np.float32(sc.box_max)
    rng = np.random.default_rng(6)
    i = np.arange(n)
    k = 11 if n == 1203 else 41
    x = (np.stack([i % k, i // k % k, i // (k * k)], 1) * 0.48 + rng.uniform(-0.02, 0.02, (n, 3))).astype(np.float32)
    x = np.clip(x if bad < 0 else box - x, 0.0, box).astype(np.float32)
    v = rng.uniform(-2.0, 2.0, (n, 3)).astype(np.float32)
    v[[n // 3, n // 2]] = bad
    o = OracleSim(p, n)
    o.set_state(x, v)
    o.step(1)
    with Particles(p, n) as g:
        g.upload(x, v)
        g.step(1)
        assert not np.isfinite(g.positions()).all()
        assert np.array_equal(g.positions(), o.get(ARRAY_POSITIONS), equal_nan=True)
        assert np.array_equal(g.velocities(), o.get(ARRAY_VELOCITIES), equal_nan=True)
