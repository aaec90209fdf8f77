"""Crowded bins, walked run by run or 32 candidates at a time.

A bin of more than 512 particles is walked by its runs of bit-identical
positions when four looks say that they are long, else candidate by candidate.
Either walk must give the oracle's lists, around the bin size where the look
begins and from all distinct to all identical points, in fast and exact math
and in the search on device arrays.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import pbf_b200
from oracle.oracle import OracleSim
from pbf_b200 import Particles, make_scene

pytestmark = pytest.mark.gpu


def _scene(size, kind, s, rng):
    """`size` particles in one bin, loose ones around it; indices mixed."""
    pile = np.array([3.4, 3.4, 3.4]) * s
    x = 3 * s + s * rng.uniform(0.05, 0.95, (size, 3))
    if kind == "one point":
        x[:] = pile
    elif kind == "mostly":
        x[rng.random(size) < 0.9] = pile
    elif kind == "half":
        x[: size // 2] = pile
    elif kind == "short runs":
        x = np.repeat(x[: (size + 19) // 20], 20, axis=0)[:size]
    loose = rng.uniform(0.0, 12.9, (900, 3))
    loose = loose[np.any((loose < 3 * s) | (loose >= 4 * s), axis=1)]
    x = np.concatenate([x, loose]).astype(np.float32)
    return x if kind == "short runs" else x[rng.permutation(len(x))]


@pytest.mark.parametrize("size", [511, 512, 513, 640, 1025, 2979, 4096, 4097, 6000])
@pytest.mark.parametrize("kind", ["distinct", "short runs", "half", "mostly", "one point"])
def test_lists_of_a_crowded_bin(size, kind):
    torch = pytest.importorskip("torch")
    sc = make_scene("dam_2k")
    p = sc.params()
    x = _scene(size, kind, np.float32(p.neighbor_bin_spacing), np.random.default_rng(size))
    n = len(x)
    o = OracleSim(p, n)
    o.set_state(x)
    o.stage(2)
    idx, cnt = o.neighbors()
    for exact in (0, 1):
        p.exact_math = exact
        with Particles(p, n) as g:
            g.upload(x)
            g.find_neighbors()
            got = g.neighbors(p.neighbor_cap)
            assert np.array_equal(got[1], cnt) and np.array_equal(got[0], idx)
            assert g.stats()["error_flags"] == 0
    d = torch.from_numpy(x).cuda()
    out = torch.empty((n, p.neighbor_cap), dtype=torch.int32, device="cuda")
    count = torch.empty(n, dtype=torch.int32, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    assert pbf_b200.lib().pbf_find_neighbors_noalloc(C.byref(p), ptr(d), n, ptr(out), ptr(count), None,
                                                     C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    assert np.array_equal(count.cpu().numpy(), cnt) and np.array_equal(out.cpu().numpy(), idx)
