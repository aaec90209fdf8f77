"""update_position_stars without lists of the present particles marks nothing.

The stage needs no search, so it may follow calls that replace the particles a
search has keyed: a larger or smaller upload, added particles, an autotune.
The moves (scratch set by the caller, the clamp into the box) must then touch
no list; positions, and everything a later search and step give, are those of
a context that was never searched before.
"""
from __future__ import annotations

import numpy as np
import pytest

from pbf_b200 import Particles, _abi, make_scene

pytestmark = pytest.mark.gpu

CAPACITY = 1500


def _state(n, seed):
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    x = np.stack([i % 10, i // 10 % 10, i // 100], 1) * 0.5 + 1.0 + rng.uniform(-0.02, 0.02, (n, 3))
    return x.astype(np.float32), rng.uniform(-2.0, 2.0, (n, 3)).astype(np.float32)


def _replace(g, how):
    if how == "more":
        g.upload(*_state(CAPACITY, 2))
    elif how == "as many":
        g.upload(*_state(600, 2))
    elif how == "fewer":
        g.upload(*_state(17, 2))
    elif how == "none, then added":
        g.upload(np.zeros((0, 3), np.float32))
        g.find_neighbors()
        g.add_particles(*_state(CAPACITY, 2))
    elif how == "autotuned":
        g.upload(*_state(600, 2))
        g.find_neighbors()
        g.autotune(1)
        g.set_tuning({f: (2, 128) for f in _abi.TUNE_FAMILIES})
    elif how == "added":
        g.upload(*_state(600, 2))
        g.find_neighbors()
        x, v = _state(900, 3)
        g.add_particles(x + np.float32(40.0), v)  # outside the 13-unit box: the clamp moves them far


def _follow(g, how):
    _replace(g, how)
    n = g.local_count()
    g.set_array(_abi.ARRAY_SCRATCH, np.random.default_rng(n).uniform(-0.3, 0.3, (n, 3)).astype(np.float32))
    g.update_position_stars()
    out = [g.position_stars()]
    g.predict_positions()
    g.find_neighbors()
    for _ in range(2):
        g.compute_densities()
        g.compute_pressure_lambdas()
        g.compute_pressure_dps()
        g.update_position_stars()
    out += [g.position_stars(), g.densities(), g.lambdas()]
    g.step(1)
    out += list(g.download().values())
    assert g.stats()["error_flags"] == 0
    return out


@pytest.mark.parametrize("how", ["more", "as many", "fewer", "none, then added", "autotuned", "added"])
def test_moves_of_particles_no_search_has_keyed(how):
    sc = make_scene("dam_2k")
    got = []
    for searched in (False, True):
        with Particles(sc.params(), CAPACITY) as g:
            g.set_tuning({f: (2, 128) for f in _abi.TUNE_FAMILIES})
            if searched:
                g.upload(*_state(600, 1))
                g.find_neighbors()
                got.append(_follow(g, how))
            else:  # the same particles in a new context
                with Particles(sc.params(), CAPACITY) as h:
                    _replace(h, how)
                    x, v = h.positions(), h.velocities()
                g.upload(x, v)
                n = g.local_count()
                g.set_array(_abi.ARRAY_SCRATCH,
                            np.random.default_rng(n).uniform(-0.3, 0.3, (n, 3)).astype(np.float32))
                g.update_position_stars()
                first = g.position_stars()
                assert np.isfinite(first).all()
                want = first
    assert np.array_equal(got[0][0], want)


@pytest.mark.parametrize("how", ["more", "as many", "fewer", "added"])
def test_what_follows_is_a_new_contexts(how):
    sc = make_scene("dam_2k")
    got = []
    for searched in (False, True):
        with Particles(sc.params(), CAPACITY) as g:
            if searched:
                g.upload(*_state(600, 1))
                g.find_neighbors()
                g.compute_densities()
                g.update_position_stars()
            got.append(_follow(g, how))
    for a, b in zip(*got):
        assert np.array_equal(a, b)
