"""Expert banks in Q6_K on the matrix unit (gemv_q6_mma_grouped_kernel) vs the CPU restatement, at the edges of its tiles: one block a
row, odd numbers of blocks (rows that start two bytes off a word), items of one to eight rows, tiles per warp, rows too long for it.

Tolerance: block sums are the CPU's integers; between the banks values are coded in 8 bits, where the order of f32 additions can move a
code by one: the layer's bar of 1e-3."""
import numpy as np
import pytest

import fixtures as fx
import infr_b200
from infr_b200 import Q6K, synth
from test_moe_gpu import _run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    b = infr_b200.CudaBackend(device=0)
    yield b
    b.close()


@pytest.mark.parametrize("rows,ne,n_expert,n_used,nff", [
    (2, 256, 2, 1, 256),     # one block a row
    (17, 768, 3, 1, 1280),   # 3 and 5 blocks; items of 8 rows and a rest
    (40, 2304, 4, 2, 2048),  # 9 and 8 blocks: two warps a CTA, one CTA an SM
    (9, 3584, 3, 1, 1792),   # 14 blocks: the longest rows that two warps have room for; 7: the longest with room for two CTAs
    (9, 3840, 3, 1, 256),    # 15 blocks: the byte-dot kernel
    (9, 4608, 3, 1, 256),    # 18 blocks
])
def test_moe_q6_banks_match_cpu(be, oracle, rows, ne, n_expert, n_used, nff):
    bank = lambda o, i, s: np.concatenate([synth.weight(Q6K, o, i, s + 3 * e) for e in range(n_expert)])
    gate, up, down = bank(nff, ne, 1), bank(nff, ne, 2), bank(ne, nff, 3)
    router = synth.normal(7, (n_expert, ne), 1.0 / np.sqrt(ne))
    x = synth.normal(8, (rows, ne))
    got, ids, _, _ = _run(be, x, router, gate, up, down, rows, ne, n_expert, n_used, nff, wdt=Q6K, down_dt=Q6K)
    want, o_ids, _, _ = oracle.moe_ffn(x, router, gate, up, down, rows=rows, ne=ne, n_expert=n_expert, n_used=n_used, n_ff_exp=nff, wdt=Q6K, down_dt=Q6K)
    np.testing.assert_array_equal(ids, o_ids)
    assert fx.rel_l2(got, want) < 1e-3
    assert max(fx.rel_l2(got[r], want[r]) for r in range(rows)) < 3e-3
