"""Infinities, NaN and zero densities reach as far through near lists as through whole ones.

Zero times such a value is NaN, so the reference spreads it to every particle
whose list holds it, also past h where the weight is zero.  The exact stage
calls walk whole lists; the fast ones, and the fused steps of both kinds, must
leave the same particles without a finite result.
"""
from __future__ import annotations

import numpy as np
import pytest

from pbf_b200 import Particles, _abi, make_scene

pytestmark = pytest.mark.gpu

N = 1203


def _state(seed):
    rng = np.random.default_rng(seed)
    i = np.arange(N)
    x = np.stack([i % 11, i // 11 % 11, i // 121], 1) * 0.48 + 1.3 + rng.uniform(-0.02, 0.02, (N, 3))
    return x.astype(np.float32), rng.uniform(-2.0, 2.0, (N, 3)).astype(np.float32)


def _both(run):
    """run(context) in exact and in fast math: what it returns must be finite at the same places."""
    got = []
    for exact in (1, 0):
        with Particles(make_scene("dam_2k", exact_math=exact).params(), N) as g:
            got.append([np.isfinite(a) for a in run(g)])
    assert any(not a.all() for a in got[0])  # the value does spread
    for a, b in zip(*got):
        assert np.array_equal(a, b)


def _after(g):
    """The stages that carry a velocity on, each from the one before."""
    out = []
    g.apply_viscosity()
    out.append(g.velocities())
    g.compute_vorticity()
    out.append(g.scratch())
    g.apply_vorticity()
    out.append(g.velocities())
    g.apply_viscosity()
    out.append(g.velocities())
    return out


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("where", ["uploaded", "set"])
def test_a_velocity(bad, where):
    x, v = _state(1)

    def run(g):
        w = v.copy()
        w[600, 1] = bad
        g.upload(x, w if where == "uploaded" else v)
        g.find_neighbors()
        g.compute_densities()
        if where == "set":
            g.set_array(_abi.ARRAY_VELOCITIES, w)
        return _after(g)

    _both(run)


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_a_scratch_vector_and_a_lambda(bad):
    x, v = _state(2)

    def run(g):
        g.upload(x, v)
        g.find_neighbors()
        g.compute_densities()
        g.compute_pressure_lambdas()
        lam = g.lambdas()
        lam[700] = bad
        g.set_array(_abi.ARRAY_LAMBDAS, lam)
        g.compute_pressure_dps()
        out = [g.scratch()]
        w = np.zeros((N, 3), np.float32)
        w[300, 2] = bad
        g.set_array(_abi.ARRAY_SCRATCH, w)
        g.apply_vorticity()
        return out + [g.velocities()]

    _both(run)


@pytest.mark.parametrize("case", ["none computed", "one set to zero", "part computed"])
def test_densities_that_are_zero(case):
    x, v = _state(3)

    def run(g):
        g.upload(x, v)
        g.find_neighbors()
        if case != "none computed":
            g.compute_densities((0, N if case == "one set to zero" else N - 40))
        if case == "one set to zero":
            rho = g.densities()
            rho[500] = 0.0
            g.set_array(_abi.ARRAY_DENSITIES, rho)
        return _after(g)

    _both(run)


def test_a_position_and_the_velocity_it_gives():
    x, v = _state(4)

    def run(g):
        g.upload(x, v)
        g.find_neighbors()
        g.compute_densities()
        far = x.copy()
        far[400] = np.inf
        g.set_array(_abi.ARRAY_POSITIONS, far)
        g.update_velocities()
        return _after(g)

    _both(run)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, 1e30])
@pytest.mark.parametrize("n", [N, 70000])
def test_a_fused_step_from_a_position_out_of_all_bounds(bad, n):
    """The step clamps x* into the box, but the velocity it gives is infinite."""
    sc = make_scene("dam_2k") if n == N else make_scene("dam_65k")
    box = np.float32(sc.box_max)
    rng = np.random.default_rng(5)
    i = np.arange(n)
    k = 11 if n == N else 41
    x = (np.stack([i % k, i // k % k, i // (k * k)], 1) * 0.48 + rng.uniform(-0.02, 0.02, (n, 3))).astype(np.float32)
    corner = box if bad > 0 else np.float32([0, 0, 0])
    x = np.clip(x if bad < 0 else box - x, 0.0, box).astype(np.float32)  # around the corner it is clamped to
    x[n // 2] = bad
    got = {}
    for exact in (1, 0):
        p = sc.params()
        p.exact_math = exact
        with Particles(p, n) as g:
            g.upload(x)
            g.step(1)
            got["step", exact] = g.velocities(), g.positions()
            if exact:
                g.upload(x)
                g.apply_external_forces()
                g.predict_positions()
                g.find_neighbors()
                for sub in range(p.solve_steps):
                    g.compute_densities()
                    g.compute_pressure_lambdas()
                    g.compute_pressure_dps(substep=sub)
                    g.update_position_stars()
                for stage in ("update_velocities", "apply_surface_tension", "apply_viscosity", "compute_vorticity",
                              "apply_vorticity", "apply_viscosity", "update_positions"):
                    getattr(g, stage)()
                got["stages", 1] = g.velocities(), g.positions()
    assert np.isfinite(corner).all() and not np.isfinite(got["stages", 1][0]).all()
    for a, b, c in zip(got["stages", 1], got["step", 1], got["step", 0]):
        assert np.array_equal(a, b, equal_nan=True)
        assert np.array_equal(np.isfinite(a), np.isfinite(c))


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_a_density(bad):
    x, v = _state(6)

    def run(g):
        g.upload(x, v)
        g.find_neighbors()
        g.compute_densities()
        rho = g.densities()
        rho[300] = bad
        g.set_array(_abi.ARRAY_DENSITIES, rho)
        g.compute_pressure_lambdas()
        out = [g.lambdas()]
        g.compute_pressure_dps()
        return out + [g.scratch()]

    _both(run)
