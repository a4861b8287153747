"""Attention of a prompt chunk: query rows share a key / value tile.  Every row must have the bits of the row on its own (a call
with one row), whatever rows share its tile, also where a later token's values are not finite."""
import numpy as np
import pytest

from infr_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_head,n_kv", [(8, 8), (16, 8), (32, 8), (32, 4)])  # 1, 2, 4, 8 heads per KV head
@pytest.mark.parametrize("rows,pos", [(113, 0), (130, 126), (97, 500), (256, 700)])
def test_chunk_rows_equal_single_rows(backend, n_head, n_kv, rows, pos):
    be, hd, kvd = backend, 128, n_kv * 128
    kc = synth.normal(1, (pos + rows, kvd)).astype(np.float16)
    vc = synth.normal(2, (pos + rows, kvd)).astype(np.float16)
    vc[pos + rows - 1, :] = np.inf  # the last token's values: no earlier row may see them
    q = synth.normal(3, (rows, n_head * hd))
    kb, vb = be.from_numpy(kc.view(np.uint16)), be.from_numpy(vc.view(np.uint16))
    qb, ob = be.from_numpy(q), be.alloc(q.nbytes)
    be.attention(qb, kb, vb, ob, rows=rows, pos=pos, n_head=n_head, n_kv=n_kv, head_dim=hd, scale=hd ** -0.5)
    got = be.download(ob, np.float32).reshape(rows, -1)
    assert np.isfinite(got[:-1]).all() and not np.isfinite(got[-1]).any()
    for r in sorted({0, 1, 2, 3, rows // 2, rows - 3, rows - 2}):
        q1, o1 = be.from_numpy(q[r:r + 1]), be.alloc(n_head * hd * 4)
        be.attention(q1, kb, vb, o1, rows=1, pos=pos + r, n_head=n_head, n_kv=n_kv, head_dim=hd, scale=hd ** -0.5)
        np.testing.assert_array_equal(got[r], be.download(o1, np.float32))


@pytest.mark.parametrize("n_head,n_kv", [(8, 8), (16, 8), (32, 8), (32, 4)])
@pytest.mark.parametrize("rows,positions", [(40, [300, 300, 300]), (35, [300, 0, 127]), (40, [90, 511, 256])])
def test_chunks_of_several_sequences(backend, n_head, n_kv, rows, positions):
    """Sequences of equal and of their own positions, contiguous and paged caches, f32 and 8-bit results: each sequence has the
    bits of a call of its own."""
    be, hd, kvd, k, b, pos = backend, 128, n_kv * 128, n_head * 128, len(positions), max(positions)
    pages = (pos + rows + 127) // 128
    ctx = pages * 128
    kc = synth.normal(1, (b, ctx, kvd)).astype(np.float16).view(np.uint16)
    vc = synth.normal(2, (b, ctx, kvd)).astype(np.float16).view(np.uint16)
    q = synth.normal(3, (b, rows, k))
    kw = dict(rows=rows, n_head=n_head, n_kv=n_kv, head_dim=hd, scale=hd ** -0.5)
    want = np.empty((b, rows, k), np.float32)
    for s, p in enumerate(positions):
        o = be.alloc(rows * k * 4)
        be.attention(be.from_numpy(q[s]), be.from_numpy(kc[s]), be.from_numpy(vc[s]), o, pos=p, **kw)
        want[s] = be.download(o, np.float32).reshape(rows, k)
    kb, vb, qb, out = be.from_numpy(kc), be.from_numpy(vc), be.from_numpy(q), be.alloc(q.nbytes)
    sp = be.from_numpy(np.array(positions, np.int32))
    kw.update(pos=pos, n_seq=b)

    def check():
        np.testing.assert_array_equal(be.download(out, np.float32).reshape(want.shape), want)
    be.attention(qb, kb, vb, out, seq_stride=ctx * kvd, seq_pos=sp, **kw)
    check()
    if len(set(positions)) == 1:
        be.attention(qb, kb, vb, out, seq_stride=ctx * kvd, **kw)
        check()
    # pages in another order, one spare
    table = np.random.default_rng(4).permutation(b * pages + 1)[:b * pages].astype(np.int32).reshape(b, pages)
    pool = [np.zeros((b * pages + 1, 128, kvd), np.uint16) for _ in range(2)]
    for p, c in zip(pool, (kc, vc)):
        p[table.ravel()] = c.reshape(b * pages, 128, kvd)
    kp, vp, tb = be.from_numpy(pool[0]), be.from_numpy(pool[1]), be.from_numpy(table)
    be.attention_paged(qb, kp, vp, tb, pages, b * pages + 1, seq_pos=sp, dst=out, **kw)
    check()
    # the merge that ends in 8-bit codes
    n = b * rows
    got, ref = ([be.alloc(n * k), be.alloc(n * k // 256 * 4), be.alloc(n * k // 32 * 4), be.alloc(n * k // 16 * 4)] for _ in range(2))
    be.quantize_q8(256, be.from_numpy(want), n, k, *ref)
    be.attention_q8(qb, kb, vb, *got, seq_stride=ctx * kvd, seq_pos=sp, **kw)
    for g, r in zip(got, ref):
        np.testing.assert_array_equal(be.download(g, np.uint8), be.download(r, np.uint8))
    be.attention_paged(qb, kp, vp, tb, pages, b * pages + 1, seq_pos=sp, q8=got, **kw)
    for g, r in zip(got, ref):
        np.testing.assert_array_equal(be.download(g, np.uint8), be.download(r, np.uint8))
