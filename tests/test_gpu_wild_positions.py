"""Stage calls after an x* has become NaN: it reaches as far in fast math as in exact math.

Without relaxation a particle alone has a lambda of -0 / 0, and the push of the
mover sphere is 0 / 0 at its very centre.  The surface stage, a force of zeros
without surface tension, and every stage after it must then leave the same
particles without a finite result as the exact stages, which walk whole lists.
"""
from __future__ import annotations

import numpy as np
import pytest

from pbf_b200 import Particles, _abi, make_scene

pytestmark = pytest.mark.gpu

TAIL = ("update_velocities", "apply_surface_tension", "apply_viscosity", "compute_vorticity", "apply_vorticity",
        "apply_viscosity", "update_positions")


def _lattice(n, seed):
    """A bar, longer than the stages carry a value."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    x = np.stack([i % 6, i // 6 % 6, i // 36], 1) * 0.5 + 1.3 + rng.uniform(-0.02, 0.02, (n, 3))
    return x.astype(np.float32), rng.uniform(-2.0, 2.0, (n, 3)).astype(np.float32)


def _finite(g, out):
    out += [np.isfinite(g.velocities()), np.isfinite(g.scratch()), np.isfinite(g.position_stars())]


def _compare(runs):
    exact, fast = runs
    assert any(not a.all() for a in exact) and all(a.any() for a in exact)
    for k, (a, b) in enumerate(zip(exact, fast)):
        assert np.array_equal(a, b), k


@pytest.mark.parametrize("gamma", [0.0, 1.0])
def test_at_the_centre_of_the_mover(gamma):
    x, v = _lattice(2400, 1)
    runs = []
    for exact in (1, 0):
        p = make_scene("dam_65k", exact_math=exact, gamma=gamma).params()
        d = np.float32(0.25)
        centre = x[500] + d
        p.mover_radius = 0.3
        for a in range(3):
            p.mover_center[a] = centre[a]
        with Particles(p, len(x)) as g:
            g.upload(x, v)
            g.find_neighbors()
            g.compute_densities()
            scratch = np.zeros_like(x)
            scratch[500] = centre - x[500]  # exact: the sum has the centre's bits
            assert np.array_equal(x[500] + scratch[500], centre)
            g.set_array(_abi.ARRAY_SCRATCH, scratch)
            g.update_position_stars()
            out = []
            for stage in TAIL:
                getattr(g, stage)()
                _finite(g, out)
            runs.append(out)
    _compare(runs)


@pytest.mark.parametrize("gamma", [0.0, 1.0])
def test_without_relaxation(gamma):
    x, v = _lattice(2400, 2)
    # two particles beyond h of all others, in the lists of some
    x = np.concatenate([x, [[1.3 + 2.5 + 1.1, 2.8, 2.0], [0.21, 2.8, 2.0]]]).astype(np.float32)
    v = np.concatenate([v, np.zeros((2, 3))]).astype(np.float32)
    runs = []
    for exact in (1, 0):
        p = make_scene("dam_65k", exact_math=exact, gamma=gamma, lambda_epsilon=0.0).params()
        with Particles(p, len(x)) as g:
            g.upload(x, v)
            g.find_neighbors()
            out = []
            g.compute_densities()
            g.compute_pressure_lambdas()
            out.append(np.isfinite(g.lambdas()))
            g.compute_pressure_dps()
            g.update_position_stars()
            for stage in TAIL:
                getattr(g, stage)()
                _finite(g, out)
            runs.append(out)
    assert not runs[0][0].all()
    _compare(runs)
