"""Crowded bins among many particles: sorted in shared memory, or by the bitmap.

Above 1,048,576 particles bins of 1,025 to 8,192 are sorted by a block in
shared memory, larger ones (and all of them below) go by the bitmap of the
reference indices; either gives the stable sort by bin (numpy's here), also
when an earlier search has already permuted the slots.
"""
from __future__ import annotations

import numpy as np
import pytest

from pbf_b200 import Particles, make_scene

pytestmark = pytest.mark.gpu

SIZES = (1024, 1025, 2047, 2048, 2049, 4095, 4097, 8191, 8192, 8193, 20000)


@pytest.mark.parametrize("n", [1048576, 1048577, 1048703, 1300001])
def test_every_size_is_the_stable_sort(n):
    sc = make_scene("dam_1m")
    p = sc.params()
    s = np.float32(p.neighbor_bin_spacing)
    rng = np.random.default_rng(n)
    x = rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32) * np.float32([150.0, 150.0, 60.0])
    take = rng.permutation(n)
    at = 0
    for i, m in enumerate(SIZES):
        x[take[at:at + m]] = np.float32([10 + 3 * i, 70, 62]) * s + s * rng.uniform(0.05, 0.95, (m, 3))
        at += m
    with Particles(p, n) as g:
        g.upload(x)
        for xs in (x, x[::-1]):
            g.set_array(1, np.ascontiguousarray(xs))  # x*
            g.find_neighbors()
            bins = g.bins()
            by_id = np.empty(n, np.int64)
            by_id[bins["sorted_ids"]] = bins["sorted_keys"]
            order = np.argsort(by_id, kind="stable")
            assert np.array_equal(bins["sorted_ids"], order)
            assert np.array_equal(bins["sorted_keys"], by_id[order])
            count = np.bincount(by_id)
            assert set(SIZES) <= set(count.tolist())
            assert g.stats()["error_flags"] == 0
