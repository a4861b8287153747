"""The merge of an attention row's key tiles at its edges: one tile, eight and nine, sixteen and seventeen (three kernels), rows that end
in any of them, f32 and int8 results.

The bound is that of the other attention tests: f32 sums of at most 2300 keys in another order than the oracle's."""
import numpy as np
import pytest

import fixtures as fx
from infr_b200 import synth
from test_decode_ops_gpu import TIGHT, _f16_cache, _q8_bufs, _q8_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_head,n_kv,hd", [(8, 2, 128), (4, 4, 64), (2, 1, 128)])
@pytest.mark.parametrize("tiles", [1, 8, 9, 16, 17])
def test_merge_of_key_tiles(backend, oracle, n_head, n_kv, hd, tiles):
    pos = np.array([128 * tiles - 1, 0, 127, 128, 64 * tiles, 128 * tiles - 129, 128 * tiles - 2][: 7 if tiles > 1 else 3], np.int32)
    n_seq, ctx = len(pos), 128 * tiles
    kc, vc = _f16_cache(21, n_seq * ctx, n_kv * hd), _f16_cache(22, n_seq * ctx, n_kv * hd)
    q = 2.0 * synth.normal(23, (n_seq, n_head * hd))
    scale = 1.0 / np.sqrt(hd)
    qb, kb, vb, db, pb = backend.from_numpy(q), backend.from_numpy(kc), backend.from_numpy(vc), backend.alloc(q.nbytes), backend.from_numpy(pos)
    kw = dict(rows=1, pos=int(pos.max()), n_head=n_head, n_kv=n_kv, head_dim=hd, scale=scale, n_seq=n_seq, seq_stride=ctx * n_kv * hd, seq_pos=pb)
    backend.attention(qb, kb, vb, db, **kw)
    got = backend.download(db, np.float32).reshape(q.shape)
    for s in range(n_seq):
        want = oracle.attention(q[s], kc[s * ctx:(s + 1) * ctx], vc[s * ctx:(s + 1) * ctx], 1, n_head, n_kv, hd, scale, int(pos[s]))
        assert fx.rel_l2(got[s], want) < TIGHT, s
    a, b = _q8_bufs(backend, n_seq, n_head * hd), _q8_bufs(backend, n_seq, n_head * hd)
    backend.quantize_q8(256, db, n_seq, n_head * hd, *a)
    backend.attention_q8(qb, kb, vb, *b, **kw)
    _q8_equal(backend, b, a)
