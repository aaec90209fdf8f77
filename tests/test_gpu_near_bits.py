"""Exact math walks a list's near entries only, in their places, and stays bit for bit the reference's.

The entries left out are past h, where every kernel is exactly zero.  Where
particles move past half the margin, or are nudged apart, whole lists are
walked; where a zero is not sure (no relaxation, no iteration, a falling power
in s_corr) the near entries are all.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import ARRAY_POSITIONS, OracleSim
from pbf_b200 import Particles, make_scene

pytestmark = pytest.mark.gpu


def _same_bits(p, x, steps):
    o = OracleSim(p, len(x))
    o.set_state(x)
    with Particles(p, len(x)) as g:
        g.upload(x)
        for k in range(steps):
            g.step(1)
            o.step(1)
            assert np.array_equal(g.positions(), o.get(ARRAY_POSITIONS), equal_nan=True), k


def _scene(n, squeeze, **kw):
    sc = make_scene(n, **kw)
    p = sc.params()
    p.exact_math = 1
    return p, (sc.positions() * np.float32(squeeze) + np.float32(3.0)).astype(np.float32)


@pytest.mark.parametrize("squeeze", [1.0, 0.9, 0.8])
@pytest.mark.parametrize("K", [1, 4])
@pytest.mark.parametrize("cap", [7, 33, 60, 64])
def test_large_corrections_keep_the_bits(squeeze, K, cap):
    p, x = _scene("dam_2k", squeeze, lambda_epsilon=20.0, solve_steps=K, neighbor_cap=cap)
    _same_bits(p, x, 3)


@pytest.mark.parametrize("radius", [0.9, 1.0, 1.15, 1.2, 1.3])
def test_smoothing_radius_at_and_past_the_bin_spacing(radius):
    p, x = _scene("dam_2k", 0.9)
    p.smoothing_radius = radius
    _same_bits(p, x, 3)


@pytest.mark.parametrize("change", [{"solve_steps": 0}, {"lambda_epsilon": 0.0}])
def test_zeros_that_are_none(change):
    p, x = _scene("dam_2k", 0.9)
    for k, v in change.items():
        setattr(p, k, v)
    _same_bits(p, x, 1)  # what a NaN velocity does next is refused by the oracle


@pytest.mark.parametrize("scorr", [(0.1, 4.0, 0.2), (0.1, -2.0, 0.2), (0.1, 0.0, 0.2)])
def test_scorr_equals_the_stages(scorr):
    """Against the stage calls, which walk whole lists: CUDA's powf is not the oracle's."""
    p, x = _scene("dam_2k", 0.9, scorr=scorr)
    with Particles(p, len(x)) as g, Particles(p, len(x)) as e:
        g.upload(x)
        e.upload(x)
        g.step(1)
        e.apply_external_forces()
        e.predict_positions()
        e.find_neighbors()
        for sub in range(p.solve_steps):
            e.compute_densities()
            e.compute_pressure_lambdas()
            e.compute_pressure_dps(substep=sub)
            e.update_position_stars()
        for stage in ("update_velocities", "apply_surface_tension", "apply_viscosity", "compute_vorticity",
                      "apply_vorticity", "apply_viscosity", "update_positions"):
            getattr(e, stage)()
        for array in ("positions", "velocities", "densities", "lambdas"):
            assert np.array_equal(getattr(g, array)(), getattr(e, array)(), equal_nan=True), array


def test_coincident_particles():
    """Pairs at one place are nudged apart: their lists, and all around them, in full."""
    p, x = _scene("dam_2k", 0.95)
    x[1::7] = x[0::7][: len(x[1::7])]
    _same_bits(p, x, 4)
