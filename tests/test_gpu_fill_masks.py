"""The list fill from mask words against the oracle's lists.

The fill tests a row of three bins into 32-bit mask words, at most 96
candidates a row; other particles (longer rows, positions whose float re-hash
leaves the integer neighbour bins) are walked in the reference's order.  Fast
math writes its lists in slot order and drops the candidates past the cap by
the reference's order, exact math writes the reference's order, and both take
more or fewer warps a tile of 32 particles by the particle count; all must
export the same lists, bit for bit.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import OracleSim
from pbf_b200 import Particles, make_batch, make_scene

pytestmark = pytest.mark.gpu


def _lists(p, n, x, exact):
    p.exact_math = exact
    with Particles(p, n) as g:
        g.upload(x)
        g.find_neighbors()
        idx, cnt = g.neighbors(p.neighbor_cap)
        st = g.stats()
        assert st["error_flags"] == 0
        return idx, cnt


def _row_of(count, s, rng):
    """`count` particles spread over the three bins of one row, beside a loose lattice."""
    x = rng.uniform([3 * s, 3 * s, 3 * s], [6 * s, 4 * s, 4 * s], (count, 3))
    g = np.stack(np.meshgrid(*[np.arange(0.7, 12.0, 1.1)] * 3, indexing="ij"), -1).reshape(-1, 3)
    return np.concatenate([x, g[(g[:, 0] > 7 * s)]]).astype(np.float32)


@pytest.mark.parametrize("count", [1, 31, 32, 33, 63, 64, 65, 95, 96, 97, 128, 200])
@pytest.mark.parametrize("cap", [1, 8, 33, 60, 64])
def test_rows_at_the_mask_words_edges(count, cap):
    sc = make_scene("dam_2k", neighbor_cap=cap)
    p = sc.params()
    x = _row_of(count, p.neighbor_bin_spacing, np.random.default_rng(1000 * cap + count))
    fast, exact = _lists(p, len(x), x, 0), _lists(p, len(x), x, 1)
    assert np.array_equal(fast[1], exact[1]) and np.array_equal(fast[0], exact[0])
    o = OracleSim(p, len(x))
    o.set_state(x)
    o.stage(2)
    oi, oc = o.neighbors()
    assert np.array_equal(fast[1], oc) and np.array_equal(fast[0], oi)


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_positions_on_bin_faces(seed):
    """Coordinates on and one ulp beside bin faces, and on the walls: the float re-hash decides the bins."""
    sc = make_scene("dam_2k")
    p = sc.params()
    rng = np.random.default_rng(seed)
    s = np.float32(p.neighbor_bin_spacing)
    x = rng.uniform(0.0, 13.0, (4001, 3)).astype(np.float32)
    face = (np.round(x / s) * s).astype(np.float32)
    face = np.where(rng.random(x.shape) < 0.3, np.nextafter(face, np.float32(99)), face)
    face = np.where(rng.random(x.shape) < 0.3, np.nextafter(face, np.float32(-99)), face)
    x = np.clip(np.where(rng.random(x.shape) < 0.4, face, x), 0.0, 13.0).astype(np.float32)
    fast, exact = _lists(p, len(x), x, 0), _lists(p, len(x), x, 1)
    assert np.array_equal(fast[1], exact[1]) and np.array_equal(fast[0], exact[0])


@pytest.mark.parametrize("squeeze", [1.0, 0.85, 0.7])
def test_batch_lists(squeeze):
    """Scenes of their own boxes and bin keys: two small grids share a warp."""
    b = make_batch(5, seed=3, n_min=600, n_max=3000)
    x = (b.positions() * np.float32(squeeze)).astype(np.float32)
    got = []
    for exact in (0, 1):
        with Particles.batch(b.with_(exact_math=exact)) as g:
            g.upload(x)
            g.find_neighbors()
            got.append(g.neighbors(60))
            assert g.stats()["error_flags"] == 0
    assert np.array_equal(got[0][1], got[1][1]) and np.array_equal(got[0][0], got[1][0])


@pytest.mark.parametrize("n", [1, 31, 32, 33, 40960, 40961, 61440, 61441, 70003])
@pytest.mark.parametrize("squeeze,cap", [(1.0, 60), (0.8, 60), (0.8, 33)])
def test_particle_counts_at_the_dispatch_edges(n, squeeze, cap):
    sc = make_scene("dam_65k", neighbor_cap=cap)
    p = sc.params()
    i = np.arange(n)
    rng = np.random.default_rng(n)
    x = np.stack([i % 41, i // 41 % 41, i // 1681], 1) * 0.5 * squeeze + 1.0 + rng.uniform(-0.1, 0.1, (n, 3))
    x = x.astype(np.float32)
    o = OracleSim(p, n)
    o.set_state(x)
    o.stage(2)
    want = o.neighbors()
    for exact in (0, 1):
        got = _lists(p, n, x, exact)
        assert np.array_equal(got[1], want[1]) and np.array_equal(got[0], want[0])
