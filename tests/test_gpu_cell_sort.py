"""The cell sort: every bin in ascending reference index, whatever its size.

Bins up to 1,024 particles are ordered by counting, larger ones from a bitmap
of the indices; both must give the stable sort by bin id (numpy's here), on
states whose slots are already permuted by an earlier step, and for the search
on device arrays, which shares the kernels.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import pbf_b200
from pbf_b200 import Particles, make_batch, make_scene

pytestmark = pytest.mark.gpu


def _crowds(sizes, n, s, seed):
    """`sizes[i]` particles in bin (2 + 2i, 2, 2), mixed by index with loose particles; n in all."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.0, 12.9, (n, 3))
    take = rng.permutation(n)
    at = 0
    for i, m in enumerate(sizes):
        lo = np.array([(1 + 2 * i) * s, s, s])
        x[take[at:at + m]] = lo + s * rng.uniform(0.05, 0.95, (m, 3))
        at += m
    return x.astype(np.float32)


def _check_bins(g, n):
    bins = g.bins()
    ids, keys = bins["sorted_ids"].astype(np.int64), bins["sorted_keys"].astype(np.int64)
    by_id = np.empty(n, np.int64)
    by_id[ids] = keys
    order = np.argsort(by_id, kind="stable")
    assert np.array_equal(ids, order)
    assert np.array_equal(keys, by_id[order])
    count = np.bincount(by_id, minlength=len(bins["bin_begin"]))
    assert np.array_equal(bins["bin_end"] - bins["bin_begin"], count)
    assert g.stats()["error_flags"] == 0


@pytest.mark.parametrize("sizes", [(1, 2), (1023, 1024, 1025), (2047, 1, 1500), (4096, 4097, 33), (6000,)])
@pytest.mark.parametrize("extra", [0, 1, 31, 777])
def test_bins_are_the_stable_sort(sizes, extra):
    sc = make_scene("dam_2k")
    p = sc.params()
    n = sum(sizes) + 900 + extra
    x = _crowds(sizes, n, p.neighbor_bin_spacing, extra)
    with Particles(p, n) as g:
        g.upload(x)
        g.find_neighbors()
        _check_bins(g, n)
        assert np.bincount(g.bins()["sorted_keys"]).max() >= max(sizes)
        g.set_array(1, x[::-1].copy())  # x*: the slots keep the first search's order
        g.find_neighbors()
        _check_bins(g, n)


def test_everything_in_one_bin_and_a_batch():
    sc = make_scene("dam_2k")
    p = sc.params()
    n = 5003
    x = (3 * p.neighbor_bin_spacing + np.random.default_rng(3).uniform(0.1, 1.0, (n, 3))).astype(np.float32)
    with Particles(p, n) as g:
        g.upload(x)
        g.find_neighbors()
        _check_bins(g, n)
    b = make_batch(3, seed=5, n_min=1500, n_max=4000)
    x = b.positions()
    x[:1400] = (1.3 + np.random.default_rng(4).uniform(0.0, 1.0, (1400, 3))).astype(np.float32)
    with Particles.batch(b) as g:
        g.upload(x)
        g.find_neighbors()
        _check_bins(g, b.n)


@pytest.mark.parametrize("sizes", [(1024, 1025), (3000, 40), (5000,)])
def test_search_on_device_arrays(sizes):
    torch = pytest.importorskip("torch")
    sc = make_scene("dam_2k")
    p = sc.params()
    n = sum(sizes) + 701
    x = _crowds(sizes, n, p.neighbor_bin_spacing, 9)
    d = torch.from_numpy(x).cuda()
    idx = torch.empty((n, 60), dtype=torch.int32, device="cuda")
    cnt = torch.empty(n, dtype=torch.int32, device="cuda")
    flags = torch.empty(1, dtype=torch.int32, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    rc = pbf_b200.lib().pbf_find_neighbors_noalloc(C.byref(p), ptr(d), n, ptr(idx), ptr(cnt), ptr(flags),
                                                   C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    assert int(flags[0]) == 0
    p.exact_math = 1
    with Particles(p, n) as g:
        g.upload(x)
        g.find_neighbors()
        want, count = g.neighbors(60)
    assert np.array_equal(cnt.cpu().numpy(), count)
    assert np.array_equal(idx.cpu().numpy(), want)
