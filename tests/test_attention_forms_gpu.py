"""Attention by tensor copies, every form of it: a tile for a row and tiles that rows share, by the number of query heads a KV head has.  The form that ran is
read from the launch.  What lies behind a sequence's last key is NaN; the bits are those of a call with that sequence alone, which has too few tiles for
tensor copies and is held against references by the other attention tests."""
import numpy as np
import pytest

from kernel_trace import launched

pytestmark = pytest.mark.gpu

KEYS = [1, 15, 16, 17, 31, 33, 112, 113, 127, 128, 129, 143, 144, 145, 255, 256]


def _form(backend, call):
    return [f"{name}<{args}>" for name, args, _ in launched(backend, call, ("attn_chunk_kernel", "attn_split_kernel"))]


@pytest.mark.parametrize("n_head,n_kv,hd,n_seq,rows,gap,form", [
    (8, 8, 128, 40, 33, 8, "attn_chunk_kernel<1, true>"),
    (16, 8, 128, 20, 19, 0, "attn_chunk_kernel<2, true>"),
    (32, 8, 128, 24, 16, 8, "attn_chunk_kernel<4, true>"),
    (16, 2, 128, 96, 7, 24, "attn_chunk_kernel<8, true>"),
    (32, 8, 128, 64, 1, 8, "attn_split_kernel<128, 4, true>"),
    (32, 4, 64, 128, 1, 0, "attn_split_kernel<64, 8, true>"),
])
@pytest.mark.parametrize("paged", [False, True])
def test_forms_have_the_bits_of_single_sequences(backend, n_head, n_kv, hd, n_seq, rows, gap, form, paged):
    rng = np.random.default_rng(n_head + n_seq)
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
        kb, vb, tb = *(backend.from_numpy(a.view(np.uint16)) for a in pool), backend.from_numpy(table)
        call = lambda: backend.attention_paged(qb, kb, vb, tb, pages, n_seq * pages, pos=pos, n_seq=n_seq, seq_pos=sp, dst=out, **kw)
    else:
        flat = np.full((2, n_seq * stride), np.nan, np.float16)
        for s in range(n_seq):
            flat[:, s * stride : s * stride + ctx * row] = kv[:, s, :ctx].reshape(2, -1)
        kb, vb = (backend.from_numpy(a.view(np.uint16)) for a in flat)
        call = lambda: backend.attention(qb, kb, vb, out, pos=pos, n_seq=n_seq, seq_stride=stride, seq_pos=sp, **kw)
    assert _form(backend, call) == [form]
    got = backend.download(out, np.float32).reshape(q.shape)
    for s in range(len(KEYS)):
        n = int(keys[s])
        one = backend.alloc(q[s].nbytes)
        bufs = [backend.from_numpy(a) for a in (q[s], kv[0, s, : n + rows - 1].view(np.uint16), kv[1, s, : n + rows - 1].view(np.uint16))]
        assert [f.split(", ")[-1] for f in _form(backend, lambda: backend.attention(*bufs, one, pos=n - 1, **kw))] == ["false>"]
        assert np.isfinite(got[s]).all() and got[s].tobytes() == backend.download(one, np.float32).tobytes(), (s, n)
