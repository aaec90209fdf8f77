"""Downloads that overlap the step before them return the state after it.

From 131,072 particles on, a download right after a step copies the positions
out while the step's last passes run.  It must return what the per-array
access returns once everything is done, after steps, repeated steps, and steps
followed by other calls.
"""
from __future__ import annotations

import numpy as np
import pytest

from pbf_b200 import Particles, _abi, learn, make_batch, make_scene

pytestmark = pytest.mark.gpu


def _check(g):
    d = g.download()
    assert np.array_equal(d["x"], g.positions(), equal_nan=True)
    assert np.array_equal(d["v"], g.velocities(), equal_nan=True)  # (no iteration: densities of 0, NaN)
    assert np.array_equal(d["rho"], g.densities())
    assert np.array_equal(d["lambda"], g.lambdas())
    return d["x"]


@pytest.mark.parametrize("lattice", [(32, 32, 31), (32, 32, 64), (64, 32, 63), (64, 32, 64), (64, 32, 65)])
@pytest.mark.parametrize("options", [{}, {"exact_math": 1}, {"gamma": 1.0}, {"solve_steps": 0}])
def test_download_after_a_step(lattice, options):
    sc = make_scene("dam_65k", lattice=lattice, **options)
    x = sc.positions()
    with Particles(sc.params(), sc.n) as g:
        g.upload(x)
        for steps in (1, 2, 1):
            before = g.positions()
            g.step(steps)
            assert not np.array_equal(_check(g), before)
        g.step(1)
        g.apply_external_forces()
        g.set_array(_abi.ARRAY_POSITIONS, x)  # the state is no longer the step's
        assert np.array_equal(_check(g), x)
        g.step(1)
        g.upload(x)
        assert np.array_equal(g.download()["x"], x)


def test_download_after_a_learned_step_and_a_batch():
    params, norm, _ = learn.load_model()
    sc = make_scene("dam_65k", lattice=(64, 32, 66), lambda_epsilon=1.0, solver=1, max_iterations=4)
    with Particles(sc.params(), sc.n) as g:
        g.mlp_set(params, norm)
        g.upload(sc.positions())
        for _ in range(3):
            g.step(1)
            _check(g)
    b = make_batch(12, seed=2, n_min=8192, n_max=32768)
    with Particles.batch(b) as g:
        g.upload(b.positions())
        g.step(2)
        _check(g)
        g.set_persistent(True)
        g.step(2)
        _check(g)
