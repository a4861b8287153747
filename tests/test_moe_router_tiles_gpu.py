"""Router logits of many rows by tiles (16 rows x 16 experts, columns in a ring of bulk copies) and the routing of rows from registers (32, 64, 128 or 256
experts a warp): logits and choices are those of the CPU path to the bit, the layer within 1e-3 relative L2 (sums of f32 in another order), as
for the other expert-bank tests."""
import numpy as np
import pytest

import fixtures as fx
import infr_b200
from fixtures import Q4K
from infr_b200 import synth
from test_moe_gpu import _run

pytestmark = pytest.mark.gpu


def _layer(n_expert, ne, nff):
    bank = lambda out, k, seed: np.concatenate([synth.weight(Q4K, out, k, seed + e % 3) for e in range(n_expert)])
    return bank(nff, ne, 40), bank(nff, ne, 50), bank(ne, nff, 60), synth.normal(7, (n_expert, ne), 1.0 / np.sqrt(ne))


@pytest.mark.parametrize("rows,ne,n_expert,n_used", [
    (65, 256, 17, 2),    # half a chunk of columns, tiles with one row and one expert
    (70, 512, 33, 4),    # one chunk
    (66, 768, 5, 5),     # one and a half
    (81, 2304, 65, 3),   # more chunks than the ring holds
    (9, 256, 128, 32),   # the largest of 128 experts' registers, every choice of a lane
    (7, 256, 129, 6),    # the smallest of 256
    (5, 256, 256, 8),
    (6, 256, 257, 8),    # more than a warp's registers
])
def test_tiles_and_rows(backend, oracle, rows, ne, n_expert, n_used):
    gate, up, down, router = _layer(n_expert, ne, 256)
    x = synth.normal(8, (rows, ne))
    x[0, :8] = 0.0
    x[1] = x[0]  # ties
    dims = dict(rows=rows, ne=ne, n_expert=n_expert, n_used=n_used, n_ff_exp=256, wdt=Q4K, down_dt=Q4K)
    got, ids, w, lg = _run(backend, x, router, gate, up, down, rows, ne, n_expert, n_used, 256)
    want, o_ids, o_w, o_lg = oracle.moe_ffn(x, router, gate, up, down, **dims)
    np.testing.assert_array_equal(lg.view(np.uint32), o_lg.reshape(lg.shape).view(np.uint32))
    np.testing.assert_array_equal(ids, o_ids.reshape(ids.shape))
    assert fx.rel_l2(got, want) < 1e-3

