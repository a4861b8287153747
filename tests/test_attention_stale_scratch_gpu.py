"""Key tiles past a row's causal end: nobody writes their partial sums, so the merge must not read what an earlier op left in
the context's scratch.  The scratch is filled with the int8 codes of a Linear whose rows code as -1 (0xFF: NaN as f32)."""
import numpy as np
import pytest

import fixtures as fx
import infr_b200
from infr_b200 import Q6K, synth

pytestmark = pytest.mark.gpu
HD = 128


def _fill_scratch(be, nbytes):
    """A Q6_K batch that is quantised once and walked (9 blocks a row: no tiled copy); its codes start the scratch, and it
    needs no more scratch than nbytes."""
    in_f = 2304
    m = int(nbytes / (in_f * (1 + 4 / 256 + 4 / 32 + 4 / 16))) - 8
    x = np.full((m, in_f), -1 / 127, np.float32)
    x[:, ::256] = 1.0  # the block's largest value: code 127, all others -1
    be.run_linear(Q6K, synth.weight(Q6K, 8, in_f, seed=3), x, m, in_f, 8)


@pytest.mark.parametrize("n_seq,rows,positions", [
    (1, 20, [120]),            # one CTA per row: rows 0..7 end in the first tile
    (1, 96, [100]),            # rows share a tile; whole blocks of them end in the first
    (1, 113, [500]),
    (4, 1, [700, 20, 300, 127]),   # a decode batch of unequal lengths
    (6, 20, [300, 0, 120, 128, 255, 31]),
])
@pytest.mark.parametrize("q8", [False, True])
def test_rows_that_end_before_the_last_tile(oracle, n_seq, rows, positions, q8):
    n_head, n_kv, pos = 32, 8, max(positions)
    ctx, kvd, k = pos + rows, n_kv * HD, n_head * HD
    kc = synth.normal(1, (n_seq, ctx, kvd)).astype(np.float16)
    vc = synth.normal(2, (n_seq, ctx, kvd)).astype(np.float16)
    q = synth.normal(3, (n_seq, rows, k))
    be = infr_b200.CudaBackend(device=0)  # a context of its own: the scratch is as large as the attention makes it
    kb, vb, qb, sp = be.from_numpy(kc.view(np.uint16)), be.from_numpy(vc.view(np.uint16)), be.from_numpy(q), be.from_numpy(np.array(positions, np.int32))
    kw = dict(rows=rows, pos=pos, n_head=n_head, n_kv=n_kv, head_dim=HD, scale=HD ** -0.5, n_seq=n_seq, seq_stride=ctx * kvd, seq_pos=sp)
    n = n_seq * rows
    ob, qs, d, sums = be.alloc(n * k * 4), be.alloc(n * k), be.alloc(n * k // 256 * 4), be.alloc(n * k // 32 * 4)

    def run():
        if q8:
            be.attention_q8(qb, kb, vb, qs, d, sums, **kw)
            return be.download(qs, np.int8).reshape(n, -1, 256) * be.download(d, np.float32).reshape(n, -1, 1)
        be.attention(qb, kb, vb, ob, **kw)
        return be.download(ob, np.float32)
    run()
    _fill_scratch(be, n * n_head * ((pos + rows + 127) // 128) * (HD + 2) * 4)
    got = run().reshape(n_seq, rows, k)
    for s in range(n_seq):
        want = oracle.attention(q[s], kc[s].view(np.uint16), vc[s].view(np.uint16), rows, n_head, n_kv, HD, HD ** -0.5, positions[s])
        # f32 sums: 1e-5; 8-bit codes: half a step of 1 / 127 of the largest of 256 values, ~3 standard deviations
        assert fx.rel_l2(got[s], want) < (1.5e-2 if q8 else 1e-5), s
    be.close()
