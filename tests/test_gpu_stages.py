"""The fast per-stage kernels against the exact ones, stage by stage.

Both contexts run the reference's loop through the stage calls on the same
state.  The fast sums run over two lanes with fused multiply-adds: a sum of at
most 64 terms is within 64 * 2^-24 = 4e-6 of its terms' scale, so densities
agree to 1e-5 of the largest and lambdas to 1e-4 (they carry the difference
density - rest density); positions to 1e-5 of the box scale, the fast path's
parity bar; a position's last bit is 1e-6 in the 13-unit box, 6e-5 in a velocity
over dt = 0.016, so velocities agree to 4e-4 plus 1e-4 of the largest.
"""
from __future__ import annotations

import numpy as np
import pytest

from pbf_b200 import Particles, _abi, make_scene

pytestmark = pytest.mark.gpu


def _state(n, seed):
    rng = np.random.default_rng(seed)
    k = int(np.ceil(n ** (1 / 3)))
    i = np.arange(n)
    x = np.stack([i % k, i // k % k, i // (k * k)], 1) * 0.48 + 1.3 + rng.uniform(-0.02, 0.02, (n, 3))
    return x.astype(np.float32), rng.uniform(-2.0, 2.0, (n, 3)).astype(np.float32)


def _close(a, b, rel, floor):
    assert np.abs(a - b).max() <= rel * np.abs(b).max() + floor


def _compare(f, e):
    _close(f.position_stars(), e.position_stars(), 0.0, 1.3e-4)
    _close(f.densities(), e.densities(), 1e-5, 0.0)
    _close(f.lambdas(), e.lambdas(), 1e-4, 1e-12)
    _close(f.velocities(), e.velocities(), 1e-4, 4e-4)


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 63, 64, 65, 129, 1000])
@pytest.mark.parametrize("options", [{}, {"gamma": 1.0}, {"scorr": (0.1, 4.0, 0.2)}])
def test_stages_follow_the_exact_ones(n, options):
    sc = make_scene("dam_2k", **options)
    x, v = _state(n, n)
    with Particles(sc.params(), n) as f, Particles(sc.with_(exact_math=1).params(), n) as e:
        both = (f, e)
        for g in both:
            g.upload(x, v)
            g.apply_external_forces()
            g.predict_positions()
            g.find_neighbors()
        for sub in range(3):
            for g in both:
                g.compute_densities()
                g.compute_pressure_lambdas()
                g.compute_pressure_dps(substep=sub)
                g.update_position_stars()
            _compare(f, e)
        for stage in ("update_velocities", "apply_surface_tension", "apply_viscosity", "compute_vorticity",
                      "apply_vorticity", "apply_viscosity", "update_positions"):
            for g in both:
                getattr(g, stage)()
            _compare(f, e)
        _close(f.scratch(), e.scratch(), 1e-3, 1e-3)
        assert f.stats()["error_flags"] == 0


@pytest.mark.parametrize("resident", [1, 16, 500, 777])
def test_a_span_leaves_the_others_alone(resident):
    sc = make_scene("dam_2k")
    n = 1000
    x, v = _state(n, 7)
    with Particles(sc.params(), n) as f:
        f.upload(x, v)
        f.find_neighbors()
        span = (0, resident)
        for stage, arrays in (("compute_densities", (4, 1)), ("compute_pressure_lambdas", (5,)),
                              ("compute_pressure_dps", (3,)), ("update_position_stars", (1,)),
                              ("apply_viscosity", (2,)), ("compute_vorticity", (3,)), ("apply_vorticity", (2,))):
            before = [f.get_array(w) for w in arrays]
            getattr(f, stage)(span)
            for w, old in zip(arrays, before):
                assert np.array_equal(f.get_array(w)[resident:], old[resident:]), (stage, w)


def test_positions_set_between_stages_are_seen():
    """x* set by the caller after the search: the lists are walked whole again."""
    sc = make_scene("dam_2k")
    n = 1000
    x, v = _state(n, 3)
    moved = (x * np.float32(0.93)).astype(np.float32)  # entries from beyond the near radius come within h
    with Particles(sc.params(), n) as f, Particles(sc.with_(exact_math=1).params(), n) as e:
        for g in (f, e):
            g.upload(x, v)
            g.find_neighbors()
            g.set_array(_abi.ARRAY_POSITION_STARS, moved)
            g.compute_densities()
            g.compute_pressure_lambdas()
        _close(f.densities(), e.densities(), 1e-5, 0.0)
        _close(f.lambdas(), e.lambdas(), 1e-4, 1e-12)


@pytest.mark.parametrize("densities", ["computed", "missing", "zeroed"])
def test_no_surface_tension_changes_no_velocity(densities):
    """gamma = 0 adds exactly zero, except where a density is still 0: NaN there, as in exact math."""
    sc = make_scene("dam_2k")
    n = 1000
    x, v = _state(n, 5)
    got = []
    for exact in (0, 1):
        with Particles(sc.with_(exact_math=exact).params(), n) as g:
            g.upload(x, v)
            g.find_neighbors()
            if densities != "missing":
                g.compute_densities()
            if densities == "zeroed":
                rho = g.densities()
                rho[:200] = 0.0
                g.set_array(_abi.ARRAY_DENSITIES, rho)
            g.apply_surface_tension()
            got.append(g.velocities())
    assert np.array_equal(np.isnan(got[0]), np.isnan(got[1]))
    fine = ~np.isnan(got[1])
    assert np.array_equal(got[0][fine], v[fine])
    assert fine.all() == (densities == "computed") and not (densities == "missing" and fine.any())
