"""Attention whose tiles are fetched by tensor copies: a whole tile, or those boxes of 16 rows that have keys.  What lies behind a sequence's last key, in its
box or in the next sequence, is NaN here.  A sequence's result depends on that sequence alone, so the bits are those of a call with it alone, which has too
few tiles for tensor copies and is held against references by the other attention tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = [1, 15, 16, 17, 31, 33, 112, 113, 127, 128, 129, 143, 144, 145, 255, 256]


@pytest.mark.parametrize("n_head,n_kv,hd,n_seq,rows,gap", [
    (32, 8, 128, 64, 1, 0), (16, 16, 64, 40, 1, 8), (8, 4, 64, 128, 1, 24),  # a tile for a row; sequences apart by no whole number of rows
    (16, 2, 128, 240, 1, 8), (8, 8, 128, 64, 1, 8),
    (32, 8, 128, 6, 16, 8), (8, 8, 128, 40, 33, 0), (16, 2, 128, 48, 5, 8),  # shared tiles
])
@pytest.mark.parametrize("paged", [False, True])
def test_boxes_have_the_bits_of_single_sequences(backend, n_head, n_kv, hd, n_seq, rows, gap, paged):
    rng = np.random.default_rng(hd + n_seq)
    keys = np.array([KEYS[i % len(KEYS)] for i in range(n_seq)])  # of a sequence's first row
    pos, row, pages = int(keys.max()) - 1, n_kv * hd, (int(keys.max()) + rows + 126) // 128
    ctx, stride = pos + rows, (pos + rows) * row + gap
    q = rng.standard_normal((n_seq, rows, n_head * hd)).astype(np.float32)
    kv = np.full((2, n_seq, pages * 128, row), np.nan, np.float16)
    for s, n in enumerate(keys):
        kv[:, s, : n + rows - 1] = rng.standard_normal((2, n + rows - 1, row))
    kw = dict(rows=rows, n_head=n_head, n_kv=n_kv, head_dim=hd, scale=hd**-0.5)
    qb, sp, out = backend.from_numpy(q), backend.from_numpy((keys - 1).astype(np.int32)), backend.alloc(q.nbytes)
    if paged:
        table = rng.permutation(n_seq * pages).reshape(n_seq, pages).astype(np.int32)
        pool = np.empty((2, n_seq * pages, 128, row), np.float16)
        pool[:, table.ravel()] = kv.reshape(2, -1, 128, row)
        kb, vb = (backend.from_numpy(a.view(np.uint16)) for a in pool)
        backend.attention_paged(qb, kb, vb, backend.from_numpy(table), pages, n_seq * pages, pos=pos, n_seq=n_seq, seq_pos=sp, dst=out, **kw)
    else:
        flat = np.full((2, n_seq * stride), np.nan, np.float16)
        for s in range(n_seq):
            flat[:, s * stride : s * stride + ctx * row] = kv[:, s, :ctx].reshape(2, -1)
        kb, vb = (backend.from_numpy(a.view(np.uint16)) for a in flat)
        backend.attention(qb, kb, vb, out, pos=pos, n_seq=n_seq, seq_stride=stride, seq_pos=sp, **kw)
    got = backend.download(out, np.float32).reshape(q.shape)
    for s in range(min(n_seq, len(KEYS))):
        n = int(keys[s])
        one = backend.alloc(q[s].nbytes)
        backend.attention(*(backend.from_numpy(a) for a in (q[s], kv[0, s, : n + rows - 1].view(np.uint16), kv[1, s, : n + rows - 1].view(np.uint16))), one, pos=n - 1, **kw)
        assert np.isfinite(got[s]).all() and got[s].tobytes() == backend.download(one, np.float32).tobytes(), (s, n)
