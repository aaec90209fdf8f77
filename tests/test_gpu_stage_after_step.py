"""Stage calls that follow a fused step walk the step's lists.

A stage call is accepted after pbf_step or pbf_group_step without a search of
its own.  The fast stage kernels read the slots past a list's end at slot n,
the record that adds nothing, so that record has to be there whichever calls
came before.  Each stage after a step is compared, bit for bit, with the same
stage of a context that was searched from the same positions (the same lists)
and given the step's state array by array.
"""
from __future__ import annotations

import numpy as np
import pytest

from pbf_b200 import Particles, SceneGroup, _abi, make_scene

pytestmark = pytest.mark.gpu

STAGES = ("compute_densities", "compute_pressure_lambdas", "compute_pressure_dps", "apply_surface_tension",
          "apply_viscosity", "compute_vorticity", "apply_vorticity")
ARRAYS = (_abi.ARRAY_POSITIONS, _abi.ARRAY_POSITION_STARS, _abi.ARRAY_VELOCITIES, _abi.ARRAY_SCRATCH,
          _abi.ARRAY_DENSITIES, _abi.ARRAY_LAMBDAS)


def _state(n, seed):
    rng = np.random.default_rng(seed)
    k = int(np.ceil(n ** (1 / 3)))
    i = np.arange(n)
    x = np.stack([i % k, i // k % k, i // (k * k)], 1) * 0.48 + 1.3 + rng.uniform(-0.02, 0.02, (n, 3))
    return x.astype(np.float32), rng.uniform(-2.0, 2.0, (n, 3)).astype(np.float32)


def _searched(g, sc, x, v):
    """A context whose lists are a search's, with g's state in its arrays."""
    h = Particles(sc.params(), len(x))
    h.upload(x, v)
    h.apply_external_forces()
    h.predict_positions()
    h.find_neighbors()
    for a, b in zip(g.neighbors(sc.neighbor_cap), h.neighbors(sc.neighbor_cap)):
        assert np.array_equal(a, b)
    for which in ARRAYS:
        h.set_array(which, g.get_array(which))
    return h


def _same_stages(g, h):
    for stage in STAGES:
        getattr(g, stage)()
        getattr(h, stage)()
        for which in ARRAYS:
            a = g.get_array(which)
            assert np.isfinite(a).all(), (stage, which)
            assert np.array_equal(a, h.get_array(which)), (stage, which)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 300, 1000])
@pytest.mark.parametrize("before", ["nothing", "spare slots", "more particles", "fewer, then added"])
@pytest.mark.parametrize("options", [{}, {"gamma": 1.0, "scorr": (0.1, 4.0, 0.2)}])
def test_stages_after_a_step(n, before, options):
    sc = make_scene("dam_2k", **options)
    x, v = _state(n, n)
    with Particles(sc.params(), n if before == "nothing" else n + 400) as g:
        if before == "more particles":
            g.upload(*_state(n + 37, 5))
            g.step(2)
        if before == "fewer, then added":
            first = n // 2
            g.upload(x[:first], v[:first])
            g.add_particles(x[first:], v[first:])
        else:
            g.upload(x, v)
        g.step(1)
        with _searched(g, sc, x, v) as h:
            _same_stages(g, h)


@pytest.mark.parametrize("n", [9, 1000])
def test_stages_after_a_group_step(n):
    sc = make_scene("dam_2k")
    states = [_state(n, 1), _state(n + 5, 2)]
    sims = [Particles(sc.params(), n + 100) for _ in states]
    for g, (x, v) in zip(sims, states):
        g.upload(x, v)
    with SceneGroup(sims) as group:
        group.step(1)
        group.sync()
        for g, (x, v) in zip(sims, states):
            with _searched(g, sc, x, v) as h:
                _same_stages(g, h)
    for g in sims:
        g.close()


def test_stages_after_a_saved_state(tmp_path):
    sc = make_scene("dam_2k")
    n = 1000
    x, v = _state(n, 3)
    with Particles(sc.params(), n + 8) as g:
        g.upload(x, v)
        g.step(3)
        g.save_state(tmp_path / "s")
        x, v = g.positions(), g.velocities()
    with Particles(sc.params(), n + 50) as g:
        g.load_state(tmp_path / "s")
        g.step(1)
        with _searched(g, sc, x, v) as h:
            _same_stages(g, h)
