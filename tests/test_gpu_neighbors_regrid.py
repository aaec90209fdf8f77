"""The lists a call returned stay the ones returned while they are valid.

New parameters keep the lists when the number of bins, the bin spacing and the
cap stay: a box with its edges exchanged, another time step.  The fast path
puts its lists back into the reference's order by the bins they were built in,
which need not be the bins of the parameters at the time of the call.
"""
from __future__ import annotations

import numpy as np
import pytest

from pbf_b200 import Particles, make_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [(17.0, 13.0, 20.0), (20.0, 17.0, 13.0), (20.0, 13.0, 17.0), (13.0, 17.0, 20.0)])
@pytest.mark.parametrize("exact", [0, 1])
@pytest.mark.parametrize("how", ["search", "step"])
def test_lists_outlive_new_box_edges(box, exact, how):
    sc = make_scene("dam_2k", box_max=(13.0, 17.0, 20.0), exact_math=exact)
    x = sc.positions()
    with Particles(sc.params(), sc.n) as g:
        g.upload(x)
        if how == "search":
            g.find_neighbors()
        else:
            g.step(2)
        want = g.neighbors(sc.neighbor_cap)
        g.set_params(sc.with_(box_max=box, time_step=0.008).params())
        got = g.neighbors(sc.neighbor_cap)
        assert np.array_equal(got[1], want[1]) and np.array_equal(got[0], want[0])
        g.step(1)  # the new box's lists
        with Particles(sc.with_(box_max=box, time_step=0.008).params(), sc.n) as h:
            if how == "search":
                h.upload(x)
                h.step(1)
                for a, b in zip(g.neighbors(sc.neighbor_cap), h.neighbors(sc.neighbor_cap)):
                    assert np.array_equal(a, b)
