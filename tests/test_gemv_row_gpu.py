"""One row against Q4_K, Q6_K and Q2_0 weights (the GEMV whose matrix-instruction columns are sub-blocks): f32 rows and quantised rows,
one matrix and two, the same bits in every form (the heights are such that the K split of a Q4_K pair, which both heights choose, is that
of two calls), and the CPU restatement's values.

Sizes: rows of one K unit, of as many units as a CTA has warps (16 x 256, 8 x 512, 16 x 512), of one unit more, of several per warp with the
last warp short; heights of part of a 16-row tile, one tile and its neighbours, and more tiles than CTAs (several flushes of partial sums)."""
import numpy as np
import pytest

import fixtures as fx
import infr_b200
from infr_b200 import ACT_INT8, Q2_0, Q4K, Q6K, synth

pytestmark = pytest.mark.gpu

LENGTHS = {Q4K: (256, 4096, 4352, 14336), Q6K: (2048, 4096, 6144, 14336), Q2_0: (512, 8192, 8704, 14336)}
HEIGHTS = ((1, 15), (16, 17), (1030, 16))


@pytest.fixture(scope="module")
def be():
    b = infr_b200.CudaBackend(device=0)
    yield b
    b.close()


def _forms(be, dt, x, in_f, w1, w2, n1, n2):
    """y1, y2 as single calls on f32 rows; every other form has their bits."""
    gran = 32 if dt == Q2_0 else 256
    xb, b1, b2 = be.from_numpy(x), be.from_numpy(w1), be.from_numpy(w2)
    y1, y2, z1, z2 = (be.alloc(n * 4) for n in (n1, n2, n1, n2))
    get = lambda b: be.download(b, np.uint32)
    be.linear(dt, b1, xb, y1, 1, in_f, n1)
    be.linear(dt, b2, xb, y2, 1, in_f, n2)
    be.linear_pair(dt, b1, z1, n1, b2, z2, n2, xb, 1, in_f, ACT_INT8)
    np.testing.assert_array_equal(get(y1), get(z1))
    np.testing.assert_array_equal(get(y2), get(z2))
    q = [be.alloc(n) for n in (in_f, in_f // gran * 4, in_f // 32 * 4, in_f // 16 * 4)]
    be.quantize_q8(gran, xb, 1, in_f, *q)
    z1, z2 = be.alloc(n1 * 4), be.alloc(n2 * 4)
    be.gemv_q8_pair(dt, b1, z1, n1, b2, z2, n2, *q, 1, in_f)
    np.testing.assert_array_equal(get(y1), get(z1))
    np.testing.assert_array_equal(get(y2), get(z2))
    return be.download(y1, np.float32), be.download(y2, np.float32)


@pytest.mark.parametrize("dt", [Q4K, Q6K, Q2_0])
@pytest.mark.parametrize("heights", HEIGHTS)
@pytest.mark.parametrize("i", range(4))
def test_row_forms(be, oracle, dt, heights, i):
    in_f, (n1, n2) = LENGTHS[dt][i], heights
    w1, w2 = synth.weight(dt, n1, in_f, seed=1), synth.weight(dt, n2, in_f, seed=2)
    x = synth.normal(3, (1, in_f))
    x[0, :256] *= 1e3
    x[0, 32:64] = 0.0
    # same block sums, added in another order: each of in_f / 256 (Q2_0: / 32) additions rounds by 2^-24 of the sum so far at most
    tol = max(1e-7, np.sqrt(in_f / (32 if dt == Q2_0 else 256)) * 2.0**-23)
    for got, w, n in zip(_forms(be, dt, x, in_f, w1, w2, n1, n2), (w1, w2), (n1, n2)):
        assert fx.rel_l2(got, oracle.linear(dt, w, x, 1, in_f, n).ravel()) < tol


@pytest.mark.parametrize("dt", [Q4K, Q6K, Q2_0])
def test_row_many_tiles(be, oracle, dt):
    in_f, n1, n2 = 2048, 16 * 148 * 5 + 7, 16 * 148 * 2 + 16  # more flushes than buffers of partial sums; the second matrix's tiles follow mid-CTA
    w1, w2 = synth.weight(dt, n1, in_f, seed=4), synth.weight(dt, n2, in_f, seed=5)
    x = synth.normal(6, (1, in_f))
    for got, w, n in zip(_forms(be, dt, x, in_f, w1, w2, n1, n2), (w1, w2), (n1, n2)):
        assert fx.rel_l2(got, oracle.linear(dt, w, x, 1, in_f, n).ravel()) < 2e-6  # sqrt(64) * 2^-23


@pytest.mark.parametrize("dt", [Q4K, Q6K, Q2_0])
def test_row_infinite_scales(be, oracle, dt):
    """A block with an infinite scale gives what the CPU's whole-block sums give: an infinity, not the NaN that a zero share of the sum would."""
    in_f, n = 2048, 32
    w = synth.weight(dt, n, in_f, seed=7).reshape(-1, {Q4K: 144, Q6K: 210, Q2_0: 18}[dt])
    at = {Q4K: 0, Q6K: 208, Q2_0: 0}[dt]
    w[3, at:at + 2] = np.frombuffer(np.float16(np.inf).tobytes(), np.uint8)
    w = w.reshape(-1)
    x = synth.normal(8, (1, in_f))
    x[0, 1 : 256] = 0.0
    x[0, 512:1024] = 0.0
    x[0, 768] = x[0, 3 * 64] = x[0, 3 * 64 + 40] = 1.0  # block 3 (Q2_0: elements 192..255) meets one sub-block with a non-zero code
    xb, wb, y = be.from_numpy(x), be.from_numpy(w), be.alloc(n * 4)
    be.linear(dt, wb, xb, y, 1, in_f, n)
    got, want = be.download(y, np.float32), oracle.linear(dt, w, x, 1, in_f, n).ravel()
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    np.testing.assert_array_equal(got[~np.isfinite(want)], want[~np.isfinite(want)])
    assert fx.rel_l2(got[np.isfinite(want)], want[np.isfinite(want)]) < 2e-6


@pytest.mark.parametrize("dt,in_f", [(Q4K, 2048), (Q4K, 4352), (Q6K, 4096), (Q2_0, 1024)])
def test_plan_of_independent_rows(be, dt, in_f):
    """Neighbouring one-row Linears that do not depend on each other are one launch per 24, with the bits of single calls; one whose row is
    another's result, or whose result lies in another's buffer, is not grouped with it."""
    count, n = 30, [16 + 37 * (i % 5) for i in range(30)]
    ws = [be.from_numpy(synth.weight(dt, n[i], in_f, seed=i)) for i in range(count)]
    xs = [be.from_numpy(synth.normal(100 + i, (1, in_f))) for i in range(count)]
    want = []
    for i in range(count):
        y = be.alloc(n[i] * 4)
        be.linear(dt, ws[i], xs[i], y, 1, in_f, n[i])
        want.append(be.download(y, np.uint32))

    def run(shared):
        g, bind, outs = infr_b200.Graph(), {}, []
        out = be.alloc(n[0] * 4)
        for i in range(count):
            a, w, c = g.input(in_f), g.weight(n[i] * in_f, dt), g.output(n[i])
            g.linear(a, w, c, 1, in_f, n[i])
            outs.append(out if shared and i in (0, 5) else be.alloc(n[i] * 4))
            bind.update({a: xs[i], w: ws[i], c: outs[i]})
        n0 = be.launch_count()
        be.execute(be.compile(g), bind)
        return be.launch_count() - n0, [be.download(o, np.uint32) for o in outs]

    launches, got = run(False)
    assert launches == 2
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    launches, got = run(True)  # handles 0 and 5 bound to one buffer (same height): in order, the later one stays
    assert launches > 2
    for i, (a, b) in enumerate(zip(got, want)):
        np.testing.assert_array_equal(a, want[5] if i == 0 else b)


@pytest.mark.parametrize("dt,in_f", [(Q4K, 1024), (Q6K, 2048), (Q2_0, 1536)])
def test_plan_of_three_on_one_row(be, dt, in_f):
    """q, k and v of a model in one format: one launch, the bits of single calls."""
    n = (300, 64, 17)
    xb, ws = be.from_numpy(synth.normal(1, (1, in_f))), [be.from_numpy(synth.weight(dt, k, in_f, seed=k)) for k in n]
    g, outs, want = infr_b200.Graph(), [be.alloc(k * 4) for k in n], []
    a, bind = g.input(in_f), {}
    for k, w, o in zip(n, ws, outs):
        wh, oh = g.weight(k * in_f, dt), g.output(k)
        g.linear(a, wh, oh, 1, in_f, k)
        bind.update({wh: w, oh: o})
        y = be.alloc(k * 4)
        be.linear(dt, w, xb, y, 1, in_f, k)
        want.append(be.download(y, np.uint32))
    n0 = be.launch_count()
    be.execute(be.compile(g), {a: xb, **bind})
    assert be.launch_count() - n0 == 1
    for o, y in zip(outs, want):
        np.testing.assert_array_equal(be.download(o, np.uint32), y)
