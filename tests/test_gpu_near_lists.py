"""The gathers walk a list's near entries only, and whole lists where particles moved.

A list holds its entries within h plus a margin first; a gather walks the
others too once a particle around has moved half the margin since the fill.
Steps whose position corrections pass the margin many times over must still
agree with the reference-ordered oracle within the fast path's tolerance (1e-5
of the box scale after one step); with the marks left out the far entries'
contributions would be missing.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import ARRAY_POSITIONS, OracleSim
from pbf_b200 import Particles, make_batch, make_scene

pytestmark = pytest.mark.gpu


def _oracle_step(p, x):
    q = type(p).from_buffer_copy(p)
    q.exact_math = 1
    o = OracleSim(q, len(x))
    o.set_state(x)
    o.step(1)
    return o.get(ARRAY_POSITIONS)


@pytest.mark.parametrize("squeeze", [0.97, 0.9, 0.8])
@pytest.mark.parametrize("K", [1, 3, 8])
@pytest.mark.parametrize("cap", [60, 64])
def test_large_corrections_match_the_oracle(squeeze, K, cap):
    sc = make_scene("dam_2k", lambda_epsilon=20.0, solve_steps=K, neighbor_cap=cap)
    p = sc.params()
    x = (sc.positions() * np.float32(squeeze) + np.float32(3.0)).astype(np.float32)
    ref = _oracle_step(p, x)
    fell = np.abs(ref - x)[:, [0, 2]].max()  # the corrections alone: nothing moves in x and z before them
    if squeeze < 0.95 and K > 1:
        assert fell > 0.05 * sc.h  # past the margin
    with Particles(p, sc.n) as g:
        g.upload(x)
        g.step(1)
        got = g.positions()
        assert g.stats()["error_flags"] == 0
    assert np.abs(got - ref).max() <= 1e-5 * max(sc.box_max)


@pytest.mark.parametrize("radius", [0.9, 1.0, 1.15, 1.2, 1.3])
def test_smoothing_radius_at_and_past_the_bin_spacing(radius):
    """h + margin at, around and past s: near entries are then all of the list."""
    sc = make_scene("dam_2k", lambda_epsilon=20.0)
    p = sc.params()
    p.smoothing_radius = radius  # s stays 1.2
    x = (sc.positions() * np.float32(0.9) + np.float32(3.0)).astype(np.float32)
    ref = _oracle_step(p, x)
    with Particles(p, sc.n) as g:
        g.upload(x)
        g.step(1)
        assert np.abs(g.positions() - ref).max() <= 1e-5 * max(sc.box_max)


def test_marks_across_scenes_change_no_bit():
    """A batch's scenes that move past the margin equal contexts of their own, bit for bit."""
    b = make_batch(4, seed=11, n_min=900, n_max=4000, lambda_epsilon=20.0)
    x = (b.positions() * np.float32(0.9) + np.float32(0.4)).astype(np.float32)
    with Particles.batch(b) as g:
        g.upload(x)
        g.step(3)
        got = g.split(g.positions())
    for sc, part, xs in zip(b.scenes, got, np.split(x, b.offsets[1:-1])):
        with Particles(sc.params(), sc.n) as g:
            g.upload(xs)
            g.step(3)
            assert np.array_equal(g.positions(), part)
