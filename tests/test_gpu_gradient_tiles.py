"""The gradient kernel at the edges of its 128-sample tiles and its grid.

One sample, the last and first row of a tile, one tile and a row, one row past
a tile for every SM (a CTA's second tile), and several tiles a CTA, against the
float64 restatement: cosine and norm of every parameter block as bfloat16
operands (2^-9 an operand) leave them.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp_oracle as mo
from pbf_b200 import Particles, make_scene

pytestmark = pytest.mark.gpu

BLOCKS = ((mo.OFF_W1, mo.OFF_B1), (mo.OFF_B1, mo.OFF_W2), (mo.OFF_W2, mo.OFF_B2), (mo.OFF_B2, mo.OFF_W3),
          (mo.OFF_W3, mo.OFF_B3), (mo.OFF_B3, mo.N_PARAMS))


@pytest.mark.parametrize("n", [1, 127, 128, 129, 128 * 148 + 1, 128 * 148 * 2 + 77])
def test_gradient_at_tile_edges(n):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 12)).astype(np.float32)
    t = np.tanh(x[:, 0] - x[:, 3]).astype(np.float32)
    sc = make_scene("dam_2k")
    with Particles(sc.params(), max(512, n * 13 // 6 + 1)) as g:
        g.mlp_init(5)
        params, _ = g.mlp_get()
        grad, loss = g.mlp_gradients(x, t)
        again, _ = g.mlp_gradients(x, t)
    want_loss, want = mo.loss_and_grad(params, x, t)
    assert abs(loss - want_loss) <= 0.02 * want_loss
    np.testing.assert_allclose(again, grad, rtol=1e-3, atol=1e-5 * np.abs(grad).max())  # only the atomics' order
    for a, b in BLOCKS:
        u, v = grad[a:b].astype(np.float64), want[a:b]
        assert np.linalg.norm(u - v) <= 0.05 * np.linalg.norm(v), (a, b)
