"""Exact math, particles nudged off one another: near lists are walked again in full, whole lists once.

Piles of coincident particles, in bins small enough for near lists and in bins
so crowded that their lists are whole, must both keep the oracle's bits.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import ARRAY_POSITIONS, OracleSim
from pbf_b200 import Particles, make_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pile", [2, 30, 90, 97, 300])
@pytest.mark.parametrize("cap", [16, 60, 64])
def test_piles_keep_the_bits(pile, cap):
    sc = make_scene("dam_2k", neighbor_cap=cap, exact_math=1)
    p = sc.params()
    x = sc.positions()
    rng = np.random.default_rng(pile)
    x[rng.permutation(len(x))[:pile]] = np.float32([3.1, 3.2, 2.9])
    o = OracleSim(p, len(x))
    o.set_state(x)
    with Particles(p, len(x)) as g:
        g.upload(x)
        for k in range(3):
            g.step(1)
            o.step(1)
            assert np.array_equal(g.positions(), o.get(ARRAY_POSITIONS), equal_nan=True), k
