"""Slots of the grouped expert GEMM that no pair has: nobody lays them out, so what an earlier op left in the context's scratch is multiplied there.  The layer has
the same bits over a scratch of 0xFF (NaN as f16 and as f32) as over one of zeroes."""
import numpy as np
import pytest

import infr_b200
from infr_b200 import Q4K, Q6K, synth

pytestmark = pytest.mark.gpu


def _fill_scratch(be, nbytes, code):
    """The first nbytes of the scratch: the int8 codes of a Q6_K batch that is quantised once and walked (9 blocks a row: no tiled copy)."""
    in_f = 2304
    m = nbytes // in_f + 1
    x = np.full((m, in_f), code / 127, np.float32)
    x[:, ::256] = float(code != 0)  # the block's largest value: code 127
    be.run_linear(Q6K, synth.weight(Q6K, 8, in_f, seed=3), x, m, in_f, 8)


@pytest.mark.parametrize("rows,n_expert,n_used", [
    (64, 16, 4),    # 16 pairs an expert: slabs of 32 slots, half empty
    (150, 20, 4),   # 30: slabs of 64
    (40, 8, 3),     # 15
])
def test_what_empty_slots_hold_is_not_seen(rows, n_expert, n_used):
    ne, nff = 512, 256
    dims = dict(rows=rows, ne=ne, n_expert=n_expert, n_used=n_used, n_ff_exp=nff, wdt=Q4K, down_dt=Q4K)
    bank = lambda out, k, seed: np.concatenate([synth.weight(Q4K, out, k, seed + e) for e in range(n_expert)])
    router, x = synth.normal(1, (n_expert, ne), ne ** -0.5), synth.normal(2, (rows, ne))
    banks = bank(nff, ne, 10), bank(nff, ne, 40), bank(ne, nff, 70)
    pairs = rows * n_used
    nbytes = 2 * (pairs * (8 * nff + 4 * ne) + 3 * (pairs + 64 * (n_expert + 1)) * (ne + nff)) + (1 << 20)  # more than the layer takes
    got = []
    for code in (0, -1):
        be = infr_b200.CudaBackend(device=0)  # a context of its own: the fill makes the scratch, and the layer finds it as it was left
        bufs = [be.from_numpy(a) for a in (x, router, *banks)]
        out = be.alloc(x.nbytes)
        _fill_scratch(be, nbytes, code)
        be.moe_ffn(bufs[0], bufs[0], *bufs[1:], out, **dims)
        got.append(be.download(out, np.float32))
        be.close()
    assert np.isfinite(got[0]).all() and np.abs(got[0]).max() > 0
    assert got[0].tobytes() == got[1].tobytes()
