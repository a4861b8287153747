"""Expert banks as 8-row items at the edges of their launch: few items (many CTAs each), more items than the device holds at once,
one K block, rows so long that a CTA holds one group of warps only; and the rows per expert at which slabs of the tensor-memory GEMM
take over.

The integer products are exact, so a result differs from the CPU path's by the order of f32 additions alone: 1e-3 relative L2, as for
the other expert-bank tests."""
import numpy as np
import pytest

import fixtures as fx
import infr_b200
from fixtures import Q4K
from infr_b200 import synth
from test_moe_gpu import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,ne,n_expert,n_used,nff,down_dt", [
    (2, 1024, 4, 1, 2048, Q4K),              # at most two items: a tile or two a CTA
    (2, 256, 2, 2, 256, infr_b200.Q6K),      # one K block, one tile for some groups of warps and none for others
    (9, 512, 8, 8, 1280, infr_b200.Q6K),     # every row on every expert: items of eight rows and of one
    (40, 256, 200, 6, 256, Q4K),             # more items than SMs
    (27, 512, 4, 2, 512, Q4K),               # 13.5 pairs an expert: items of every size
    (28, 512, 4, 2, 512, Q4K),               # 14: slabs of 32 rows
    (55, 512, 4, 2, 512, Q4K),               # 27.5: the last of them
    (56, 512, 4, 2, 512, Q4K),               # 28: slabs of 64 rows
    (150, 256, 3, 2, 1280, Q4K),             # 100: two of them
    (2, 14336, 2, 1, 256, Q4K),              # 56 blocks a row: no room for two groups' rings
])
def test_items_at_the_edges(backend, oracle, rows, ne, n_expert, n_used, nff, down_dt):
    gate = np.concatenate([synth.weight(Q4K, nff, ne, 900 + 3 * e) for e in range(n_expert)])
    up = np.concatenate([synth.weight(Q4K, nff, ne, 901 + 3 * e) for e in range(n_expert)])
    down = np.concatenate([synth.weight(down_dt, ne, nff, 902 + 3 * e) for e in range(n_expert)])
    router = synth.normal(7, (n_expert, ne), 1.0 / np.sqrt(ne))
    x = synth.normal(8, (rows, ne))
    got, ids, _, _ = _run(backend, x, router, gate, up, down, rows, ne, n_expert, n_used, nff, wdt=Q4K, down_dt=down_dt)
    want, o_ids, _, _ = oracle.moe_ffn(x, router, gate, up, down, rows=rows, ne=ne, n_expert=n_expert, n_used=n_used, n_ff_exp=nff,
                                       wdt=Q4K, down_dt=down_dt)
    np.testing.assert_array_equal(ids, o_ids)
    assert fx.rel_l2(got, want) < 1e-3
    assert np.abs(want).max() > 1e-4
