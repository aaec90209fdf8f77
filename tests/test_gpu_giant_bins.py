"""Bins that hold a sixteenth of all particles or more: ordered by all blocks of the sort.

Around the population where such a bin begins (twice the words of the indices'
bitmap and 4, at least 1,025), with one and with as many as there can be, at
starts of every alignment, the sort must be numpy's stable one, also when an
earlier search has permuted the slots, and in the search on device arrays.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import pbf_b200
from oracle.oracle import OracleSim
from pbf_b200 import Particles, make_scene

pytestmark = pytest.mark.gpu


def _least(n):
    return max(2 * ((n + 127) // 128 * 4) + 4, 1025)


def _piles(n, sizes, s, rng):
    x = rng.uniform(0.0, 9.0, (n, 3))
    x[:, 2] += 20.0
    take, at = rng.permutation(n), 0
    for i, m in enumerate(sizes):
        x[take[at:at + m]] = (np.array([1 + 2 * (i % 6), 1 + 2 * (i // 6), 3]) + rng.uniform(0.1, 0.9, (m, 3))) * s
        at += m
    return x.astype(np.float32)


def _stable(g):
    bins = g.bins()
    by_id = np.empty(len(bins["sorted_ids"]), np.int64)
    by_id[bins["sorted_ids"]] = bins["sorted_keys"]
    order = np.argsort(by_id, kind="stable")
    assert np.array_equal(bins["sorted_ids"], order) and np.array_equal(bins["sorted_keys"], by_id[order])
    assert g.stats()["error_flags"] == 0
    return np.bincount(by_id)


@pytest.mark.parametrize("n", [1100, 2048, 16384, 16511, 65536, 262147])
@pytest.mark.parametrize("many", [1, 2, 15])
def test_around_the_least_giant(n, many):
    least = _least(n)
    sc = make_scene("dam_65k")
    p = sc.params()
    rng = np.random.default_rng(n + many)
    for off in (-1, 0, 1, 2, 3):
        sizes = [least + off] * many
        while sum(sizes) > n:
            sizes.pop()
        x = _piles(n, sizes, p.neighbor_bin_spacing, rng)
        with Particles(p, n) as g:
            g.upload(x)
            for xs in (x, x[::-1]):
                g.set_array(1, np.ascontiguousarray(xs))  # x*
                g.find_neighbors()
                assert np.count_nonzero(_stable(g) == least + off) >= len(sizes)


@pytest.mark.parametrize("n,m", [(1030, 1030), (65536, 65536), (65536, 60001), (300000, 299993)])
def test_almost_everything_in_one_bin(n, m):
    sc = make_scene("dam_65k")
    p = sc.params()
    x = _piles(n, [m], p.neighbor_bin_spacing, np.random.default_rng(m))
    with Particles(p, n) as g:
        g.upload(x)
        for _ in range(2):
            g.find_neighbors()
            assert _stable(g).max() == m
        g.step(2)
        _stable(g)


@pytest.mark.parametrize("n,m", [(3000, 2000), (20000, 1300), (65536, 5000)])
def test_search_on_device_arrays(n, m):
    torch = pytest.importorskip("torch")
    sc = make_scene("dam_65k")
    p = sc.params()
    x = _piles(n, [m] * min(4, n // m), p.neighbor_bin_spacing, np.random.default_rng(n))
    o = OracleSim(p, n)
    o.set_state(x)
    o.stage(2)
    idx, cnt = o.neighbors()
    d = torch.from_numpy(x).cuda()
    out = torch.empty((n, p.neighbor_cap), dtype=torch.int32, device="cuda")
    count = torch.empty(n, dtype=torch.int32, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    assert pbf_b200.lib().pbf_find_neighbors_noalloc(C.byref(p), ptr(d), n, ptr(out), ptr(count), None,
                                                     C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    assert np.array_equal(count.cpu().numpy(), cnt) and np.array_equal(out.cpu().numpy(), idx)
