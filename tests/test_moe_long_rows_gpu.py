"""Expert banks whose rows are too long for the 8-row items (eight staged rows of more than 69 blocks do not fit a CTA): slabs of the tensor-memory GEMM take
them at every number of rows per expert.

The integer products are exact, so a result differs from the CPU path's by the order of f32 additions alone: 1e-3 relative L2, as for
the other expert-bank tests."""
import numpy as np
import pytest

import fixtures as fx
from fixtures import Q4K
from infr_b200 import synth
from test_moe_gpu import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,ne,n_expert,n_used,nff", [
    (24, 256, 4, 2, 24576),   # 12 pairs an expert, long rows in down
    (9, 24576, 2, 2, 256),    # 9, long rows in gate and up
    (3, 256, 4, 2, 17920),    # 1.5, one block above what items take
    (24, 256, 4, 2, 17664),   # the longest that items take
])
def test_long_expert_rows(backend, oracle, rows, ne, n_expert, n_used, nff):
    gate, up = (np.concatenate([synth.weight(Q4K, nff, ne, 10 * k + e) for e in range(n_expert)]) for k in (1, 2))
    down = np.concatenate([synth.weight(Q4K, ne, nff, 30 + e) for e in range(n_expert)])
    router, x = synth.normal(7, (n_expert, ne), 1.0 / np.sqrt(ne)), synth.normal(8, (rows, ne))
    got, ids, _, _ = _run(backend, x, router, gate, up, down, rows, ne, n_expert, n_used, nff, wdt=Q4K, down_dt=Q4K)
    want, o_ids, _, _ = oracle.moe_ffn(x, router, gate, up, down, rows=rows, ne=ne, n_expert=n_expert, n_used=n_used, n_ff_exp=nff, wdt=Q4K, down_dt=Q4K)
    np.testing.assert_array_equal(ids, o_ids)
    assert fx.rel_l2(got, want) < 1e-3
