"""Attention whose operands span more than the exponents of f16: weights far below the largest that meet large or infinite values, query elements far
below the largest that decide the scores, zeros among them.  Reference: softmax and sums in 64 bits.

Scores are at most 40 in magnitude with a relative error of a few 2^-24, so exp() is off by 1e-5 at most; the products keep 22 bits and the sums
24: 1e-4 elementwise."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [  # n_head, n_kv, head_dim, pos, rows, n_seq: a CTA a row (few tiles, many tiles), shared tiles with and without a causal edge in them
    (8, 8, 128, 200, 1, 1), (32, 8, 128, 511, 1, 40), (16, 2, 64, 300, 1, 1), (8, 2, 64, 511, 1, 60), (32, 4, 128, 511, 1, 60),
    (32, 8, 128, 384, 33, 1), (8, 8, 128, 250, 64, 1), (32, 4, 128, 100, 33, 2), (16, 8, 128, 256, 40, 1),
]


def _reference(q, k, v, n_head, n_kv, hd, scale, pos):
    rows, g = q.shape[0], n_head // n_kv
    q, k, v = (a.astype(np.float64).reshape(len(a), -1, hd) for a in (q, k, v))
    out = np.zeros((rows, n_head, hd))
    for r in range(rows):
        n = pos + r + 1
        for h in range(n_head):
            s = (k[:n, h // g] @ q[r, h]) * scale
            w = np.exp(s - s.max())
            out[r, h] = (w / w.sum()) @ v[:n, h // g]
    return out.reshape(rows, -1)


def _run(be, q, k, v, n_head, n_kv, hd, scale, pos, rows, n_seq):
    b = [be.from_numpy(a) for a in (q, k.view(np.uint16), v.view(np.uint16))]
    o = be.alloc(q.nbytes)
    be.attention(*b, o, rows=rows, pos=pos, n_head=n_head, n_kv=n_kv, head_dim=hd, scale=scale, n_seq=n_seq, seq_stride=(pos + rows) * n_kv * hd)
    return be.download(o, np.float32).reshape(q.shape)


@pytest.mark.parametrize("n_head,n_kv,hd,pos,rows,n_seq", SHAPES)
@pytest.mark.parametrize("kind", ["weights", "query"])
def test_small_operands_keep_their_bits(backend, n_head, n_kv, hd, pos, rows, n_seq, kind):
    rng, ctx = np.random.default_rng(pos + rows), pos + rows
    k = np.zeros((n_seq, ctx, n_kv, hd), np.float16)
    v = rng.uniform(1.0, 2.0, k.shape).astype(np.float16)
    q = np.zeros((n_seq, rows, n_head, hd), np.float32)
    if kind == "weights":
        # every 100th key scores 0, the others -20 .. -38: weights down to 2^-55; the values that count belong to those
        scale, q[..., 0] = 1.0, 1.0
        q[..., 1:] = rng.uniform(1.0, 2.0, q[..., 1:].shape)
        k[..., 0] = -rng.uniform(20.0, 38.0, k.shape[:3])
        k[:, ::100, :, 0] = 0.0
        v[:, ::100] = 0.0
        v[:, 1::100] = 6e4
    else:
        # one large element meets zeros, elements of 2^-40 of it the keys
        scale = 2.0**22
        q[..., 0] = 1.0
        q[..., 1:] = rng.uniform(-1.0, 1.0, q[..., 1:].shape) * 2.0**-40
        k[..., 1:] = rng.uniform(-1.0, 1.0, k[..., 1:].shape) * 6e4
    got = _run(backend, q.reshape(n_seq * rows, -1), k.reshape(-1), v.reshape(-1), n_head, n_kv, hd, scale, pos, rows, n_seq)
    for s in {0, n_seq // 2, n_seq - 1}:
        want = _reference(q[s].reshape(rows, -1), k[s].reshape(ctx, -1), v[s].reshape(ctx, -1), n_head, n_kv, hd, scale, pos)
        np.testing.assert_allclose(got[s * rows:(s + 1) * rows], want, rtol=1e-4)


@pytest.mark.parametrize("n_head,n_kv,hd,pos,rows,n_seq", SHAPES)
def test_infinite_value_under_a_small_weight(backend, n_head, n_kv, hd, pos, rows, n_seq):
    """0 < weight * infinity is an infinity, however small the weight."""
    ctx = pos + rows
    q, k, v = (np.zeros((n_seq, n, h, hd), t) for n, h, t in ((rows, n_head, np.float32), (ctx, n_kv, np.float16), (ctx, n_kv, np.float16)))
    q[..., 0] = 1.0
    q[..., 1:] = 0.5
    k[:, 3, :, 0] = -50.0  # a weight of 2^-72
    v[:, 3, :, 1] = np.inf
    got = _run(backend, q.reshape(n_seq * rows, -1), k.reshape(-1), v.reshape(-1), n_head, n_kv, hd, 1.0, pos, rows, n_seq)
    got = got.reshape(n_seq, rows, n_head, hd)
    assert np.isposinf(got[..., 1]).all() and (np.delete(got, 1, axis=-1) == 0.0).all()
