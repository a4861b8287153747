"""One f32 row against Q2_0 weights, quantised inside the GEMV, alone and as a pair, vs the same kernel on rows that the quantiser
prepared (the codes, sums and the order of the additions are the same: the same bits) and vs the CPU restatement."""
import numpy as np
import pytest

import fixtures as fx
import infr_b200
from infr_b200 import ACT_INT8, Q2_0, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    b = infr_b200.CudaBackend(device=0)
    yield b
    b.close()


@pytest.mark.parametrize("in_f,n1,n2", [(64, 1, 3), (192, 37, 16), (704, 300, 41), (14336, 130, 64), (16384, 65, 7), (16448, 20, 300)])
def test_q2_row_is_quantise_then_gemv(be, oracle, in_f, n1, n2):
    w1, w2 = synth.weight(Q2_0, n1, in_f, seed=1), synth.weight(Q2_0, n2, in_f, seed=2)
    x = synth.normal(3, (1, in_f))
    x[0, :32] = 0.0  # a group of zeros
    x[0, 32:64] *= 1e3
    xb, b1, b2 = be.from_numpy(x), be.from_numpy(w1), be.from_numpy(w2)
    qs, d, s, s16 = be.alloc(in_f), be.alloc(in_f // 32 * 4), be.alloc(in_f // 32 * 4), be.alloc(in_f // 16 * 4)
    # the CPU adds in_f / 32 terms of random sign one by one: each rounding is 2^-24 of the sum so far at most, the square root of so many
    # of them together
    tol = max(1e-7, np.sqrt(in_f / 32) * 2.0**-24)
    be.quantize_q8(32, xb, 1, in_f, qs, d, s, s16)
    for w, b, n in ((w1, b1, n1), (w2, b2, n2)):
        y, z = be.alloc(n * 4), be.alloc(n * 4)
        be.linear(Q2_0, b, xb, y, 1, in_f, n)
        be.gemv_q8(Q2_0, b, qs, d, s, s16, z, 1, in_f, n)
        np.testing.assert_array_equal(be.download(y, np.uint32), be.download(z, np.uint32))
        assert fx.rel_l2(be.download(y, np.float32), oracle.linear(Q2_0, w, x, 1, in_f, n).ravel()) < tol
    y1, y2, z1, z2 = (be.alloc(n * 4) for n in (n1, n2, n1, n2))
    be.linear_pair(Q2_0, b1, y1, n1, b2, y2, n2, xb, 1, in_f, ACT_INT8)
    be.linear(Q2_0, b1, xb, z1, 1, in_f, n1)
    be.linear(Q2_0, b2, xb, z2, 1, in_f, n2)
    np.testing.assert_array_equal(be.download(y1, np.uint32), be.download(z1, np.uint32))
    np.testing.assert_array_equal(be.download(y2, np.uint32), be.download(z2, np.uint32))


def test_rope_group_shares_its_rotated_keys(be):
    # two layers rotate their keys through one handle: one launch each; a reader of the handle keeps the ops apart, with the same values
    rows, nh, nkv, hd, pos, base = 3, 8, 2, 64, 5, 10000.0
    kv = nkv * hd

    def run(read_it):
        g = infr_b200.Graph()
        q, k, v = g.input(rows * nh * hd), g.input(rows * kv), g.input(rows * kv)
        p, rot, out = g.input(rows, infr_b200.I32), g.internal(rows * kv), g.output(rows * kv)
        caches = [g.input((pos + rows) * kv, infr_b200.F16) for _ in range(4)]
        for layer in range(2):
            g.rope(k, p, rot, rows, nkv, hd, hd, base)
            g.rope(q, p, q, rows, nh, hd, hd, base)
            g.write_kv(rot, caches[2 * layer], rows, kv, pos)
            g.write_kv(v, caches[2 * layer + 1], rows, kv, pos)
            if read_it:
                g.add(rot, v, out, rows * kv)
        if not read_it:
            g.add(k, v, out, rows * kv)
        bufs = {q: be.from_numpy(synth.normal(1, (rows, nh * hd))), k: be.from_numpy(synth.normal(2, (rows, kv))), v: be.from_numpy(synth.normal(3, (rows, kv))),
                p: be.from_numpy(np.arange(pos, pos + rows, dtype=np.int32)), out: be.alloc(rows * kv * 4)}
        bufs.update({c: be.alloc((pos + rows) * kv * 2) for c in caches})
        n0 = be.launch_count()
        be.execute(be.compile(g), bufs)
        n = be.launch_count() - n0
        return n, [be.download(bufs[h], np.uint16) for h in (*caches, q)], be.download(bufs[out], np.float32)

    n_one, fused, _ = run(False)
    n_ops, apart, out = run(True)
    assert n_one == 3 and n_ops == 10
    for a, b in zip(fused, apart):
        np.testing.assert_array_equal(a, b)
    assert np.abs(out).max() > 0


@pytest.mark.parametrize("v_is,q_is", [("rotated k", "q"), ("q", "q"), ("v", "k"), ("v", "rotated k")])
def test_rope_group_needs_handles_of_its_own(be, v_is, q_is):
    # rope, rope, write_kv, write_kv where a handle stands in two places: the values of the ops one by one
    rows, nh, hd, base = 3, 4, 64, 10000.0
    n = rows * nh * hd
    g = infr_b200.Graph()
    h = {"q": g.input(n), "k": g.input(n), "v": g.input(n), "rotated k": g.internal(n)}
    p, kc, vc = g.input(rows, infr_b200.I32), g.input(n, infr_b200.F16), g.input(n, infr_b200.F16)
    g.rope(h["k"], p, h["rotated k"], rows, nh, hd, hd, base)
    g.rope(h[q_is], p, h[q_is], rows, nh, hd, hd, base)
    g.write_kv(h["rotated k"], kc, rows, nh * hd, 0)
    g.write_kv(h[v_is], vc, rows, nh * hd, 0)
    host = {s: synth.normal(i, (rows, nh * hd)) for i, s in enumerate(("q", "k", "v"))}
    pos = be.from_numpy(np.arange(rows, dtype=np.int32))
    results = []
    for plan in (True, False):
        b = {s: be.from_numpy(a) for s, a in host.items()}
        b["rotated k"], ck, cv = be.alloc(n * 4), be.alloc(n * 2), be.alloc(n * 2)
        if plan:
            be.execute(be.compile(g), {**{h[s]: b[s] for s in host}, p: pos, kc: ck, vc: cv})
        else:
            be.rope(b["k"], pos, b["rotated k"], rows, nh, hd, hd, base)
            be.rope(b[q_is], pos, b[q_is], rows, nh, hd, hd, base)
            be.write_kv(b["rotated k"], ck, rows, nh * hd, 0)
            be.write_kv(b[v_is], cv, rows, nh * hd, 0)
        results.append([be.download(x, np.uint16) for x in (ck, cv, b["q"], b["k"])])
    for x, y in zip(*results):
        np.testing.assert_array_equal(x, y)
