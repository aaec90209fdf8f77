"""Stage calls in fast math on particles far closer than their spacing.

The reference divides the spiky gradient by r + FLT_EPSILON; compute_densities
nudges particles that sit on one another apart by v dt / 50, so r is often of
that size.  The stages that use the gradient must follow the exact ones there.
Bounds: a sum of at most 64 terms, each with a handful of operations and two
fast intrinsics (2 ulp each), is within 64 * 2^-20 of its terms' largest, which
is (h - r)^2 r / (r + eps) <= h^2 times the constants and factors; lambda's
denominator holds a positive sum (64 * 2^-20 of itself) and a squared one of
the same terms (at most 64 times the first, so 2 * 64 * 64 * 2^-20 of it).
"""
from __future__ import annotations

import numpy as np
import pytest

from pbf_b200 import Particles, _abi, make_scene

pytestmark = pytest.mark.gpu

N = 900
TERM = 64 * 2.0 ** -20


def _pairs(gap, seed=0):
    """A lattice in pairs `gap` apart, in random directions, within the first bins (fine coordinates)."""
    rng = np.random.default_rng(seed)
    i = np.arange(N // 2)
    x = np.stack([i % 8, i // 8 % 8, i // 64], 1) * 0.45 + 0.4 + rng.uniform(-0.02, 0.02, (N // 2, 3))
    x[:6] = rng.uniform(1e-5, 2e-5, (6, 3))  # at the origin even the smallest gaps are representable
    d = rng.normal(size=(N // 2, 3))
    d *= gap / np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([x, np.maximum(x.astype(np.float32) + d, 0)]).astype(np.float32), \
        rng.uniform(-2, 2, (N, 3)).astype(np.float32)


def _run(exact, gap, scorr=0.0):
    sc = make_scene("dam_2k", exact_math=exact, lambda_epsilon=20.0, scorr=(scorr, 4.0, 0.2))
    x, v = _pairs(gap)
    rng = np.random.default_rng(1)
    with Particles(sc.params(), N) as g:
        g.upload(x, v)
        g.find_neighbors()
        g.set_array(_abi.ARRAY_DENSITIES, rng.uniform(1.5, 2.0, N).astype(np.float32))
        g.compute_pressure_lambdas()
        out = {"lambda": g.lambdas()}
        g.set_array(_abi.ARRAY_LAMBDAS, rng.uniform(-0.01, 0.0, N).astype(np.float32))
        g.compute_pressure_dps()
        out["dp"] = g.scratch()
        g.compute_vorticity()
        out["omega"] = g.scratch()
        p = g.params()
        p.gamma = 0.0
        g.set_params(p)
        g.set_array(_abi.ARRAY_VELOCITIES, v)
        g.apply_surface_tension()
        out["color"] = g.scratch()
        return out, p


@pytest.mark.parametrize("gap", [1e-8, 3e-8, 1e-7, 1e-6, 1e-5, 1e-4, 1e-3])
def test_gradient_stages_of_close_pairs(gap):
    (e, p), (f, _) = _run(1, gap), _run(0, gap)
    h = p.smoothing_radius
    spiky = 45.0 / (np.pi * h ** 6) * h * h
    assert np.abs(f["lambda"] - e["lambda"]).max() <= 2 * 64 * TERM * np.abs(e["lambda"]).max()
    assert np.abs(f["dp"] - e["dp"]).max() <= TERM * 0.02 * spiky / p.rest_density
    assert np.abs(f["omega"] - e["omega"]).max() <= 2 * TERM * 4.0 * spiky
    assert np.abs(f["color"] - e["color"]).max() <= TERM * h * spiky / 1.5


@pytest.mark.parametrize("gap", [1e-7, 1e-4])
def test_artificial_pressure_of_close_pairs(gap):
    """(W / W(dq))^4 of a close pair is the largest: k times it on top of the lambdas."""
    (e, p), (f, _) = _run(1, gap, 0.1), _run(0, gap, 0.1)
    spiky = 45.0 / (np.pi * p.smoothing_radius ** 6) * p.smoothing_radius ** 2
    most = 0.02 + 0.1 * (1.0 - 0.2 ** 2) ** -12
    assert np.abs(f["dp"] - e["dp"]).max() <= TERM * most * spiky / p.rest_density
