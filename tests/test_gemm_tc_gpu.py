"""The tensor-memory GEMM (gemm_tc.cu, more than 8 rows) vs the CPU restatement of infr-cpu's production path, at the edges
of its tiles: 32 / 64 / 128 tokens, 128 weight rows, the raw stages and the K splits.

Tolerance: the block sums are the CPU's integers, so a result differs only by f32 rounding, one unit (2^-24) per block and
operation at most: 5e-7 relative L2 for the shapes here (n blocks of random sign: about sqrt(n) of n roundings)."""
import numpy as np
import pytest

import fixtures as fx
import infr_b200
from infr_b200 import Q2_0, Q4K, Q6K, synth

pytestmark = pytest.mark.gpu
TOL = 5e-7


@pytest.fixture(scope="module")
def tc():
    be = infr_b200.CudaBackend(device=0, mmq_kernel=2)
    yield be
    be.close()


@pytest.mark.parametrize("dt", [Q4K, Q6K, Q2_0])
@pytest.mark.parametrize("m,in_f,out_f", [
    (9, 2048, 1),       # one output row
    (32, 2048, 128),    # exactly one tile
    (33, 2048, 129),    # one past it in both dimensions
    (64, 4096, 255),    # a height that is not a multiple of four: the scalar sum over the K splits
    (65, 2048, 130),
    (129, 6144, 384),   # two or three token tiles
    (70, 2048, 38000),  # more tiles than SMs: the persistent loop over tiles
])
def test_gemm_tc_matches_production_cpu(tc, oracle, dt, m, in_f, out_f):
    w = synth.weight(dt, out_f, in_f, seed=m + in_f)
    x = synth.normal(6, (m, in_f))
    x[::3] *= 100.0  # rows of different scale
    got = tc.run_linear(dt, w, x, m, in_f, out_f)
    want = oracle.linear(dt, w, x, m, in_f, out_f)
    assert fx.rel_l2(got, want) < TOL
    if out_f > 1:
        assert max(fx.rel_l2(got[r], want[r]) for r in range(m)) < 2 * TOL


@pytest.mark.parametrize("dt,in_f", [(Q4K, 256), (Q4K, 768), (Q2_0, 512), (Q2_0, 1536)])
def test_gemm_tc_short_rows(tc, oracle, dt, in_f):
    # one stage, and fewer stages than the ring is deep
    w = synth.weight(dt, 100, in_f, seed=3)
    x = synth.normal(4, (70, in_f))
    assert fx.rel_l2(tc.run_linear(dt, w, x, 70, in_f, 100), oracle.linear(dt, w, x, 70, in_f, 100)) < TOL


@pytest.mark.parametrize("dt", [Q6K, Q2_0])
def test_gemm_tc_extreme_codes(tc, oracle, dt):
    # every code bit set, scales at both ends of their range, activations pinned at +/-127
    m, in_f, out_f = 40, 2048, 128
    be, bb = fx.BLOCK[dt]
    blk = np.full(bb, 0xFF, np.uint8)
    if dt == Q6K:
        blk[192:208] = np.tile(np.array([0x80, 0x7F], np.uint8), 8)
    fx.put_f16(blk, fx.D_SLOT[dt], 0.01)
    w = np.tile(blk, out_f * in_f // be)
    x = np.where(np.arange(m * in_f).reshape(m, in_f) % 3 == 0, -1.0, 1.0).astype(np.float32)
    assert fx.rel_l2(tc.run_linear(dt, w, x, m, in_f, out_f), oracle.linear(dt, w, x, m, in_f, out_f)) < TOL


def _q6_rows(rng, out_f, in_f):
    """Codes 60..63 under scales of +127: a weight is 3556..3937 steps, so a block of codes near 127 sums to 1.2e8."""
    blk = rng.integers(0, 256, (out_f * in_f // 256, 210), dtype=np.uint8)
    blk[:, :128] |= 0xCC  # both nibbles 12..15
    blk[:, 128:192] = 0xFF
    blk[:, 192:208] = 127
    blk[:, 208:210] = np.array([0.01], np.float16).view(np.uint8)
    return blk.ravel()


def _q4_rows(rng, out_f, in_f):
    """Every scale and minimum 63, codes 12..15: a weight is 756..945 steps, a block of codes near 127 sums to 2.7e7."""
    blk = rng.integers(0, 256, (out_f * in_f // 256, 144), dtype=np.uint8)
    blk[:, 0:4] = np.array([0.01, 0.02], np.float16).view(np.uint8)
    blk[:, 4:16] = 0xFF
    blk[:, 16:] |= 0xCC
    return blk.ravel()


@pytest.mark.parametrize("m", [20, 40, 100])  # the three token tiles
@pytest.mark.parametrize("x_of", ["same sign", "halves cancel"])
def test_gemm_tc_block_sums_beyond_24_bits(tc, oracle, m, x_of):
    # |block sum|, or what it climbs to half way, is above 2^24: the CPU converts the integer, here the last addition rounds
    # (2^-23 of the sum at most), so the bound stays that of f32
    in_f, out_f, rng = 2048, 130, np.random.default_rng(m)
    x = rng.uniform(0.9, 1.0, (m, in_f)).astype(np.float32)
    if x_of == "halves cancel":
        x[:, np.arange(in_f) % 256 >= 128] *= -1.0
    for dt, w in ((Q4K, _q4_rows(rng, out_f, in_f)), (Q6K, _q6_rows(rng, out_f, in_f))):
        got, want = tc.run_linear(dt, w, x, m, in_f, out_f), oracle.linear(dt, w, x, m, in_f, out_f)
        assert fx.rel_l2(got, want) < TOL


@pytest.mark.parametrize("dt", [Q4K, Q6K, Q2_0])
def test_gemm_tc_two_weights_and_repeat(tc, dt):
    # two matrices against the same rows in one launch; op by op, captured and replayed give the same bits
    m, in_f, n1, n2 = 40, 2048, 200, 130
    w1, w2 = synth.weight(dt, n1, in_f, seed=1), synth.weight(dt, n2, in_f, seed=2)
    x = synth.normal(5, (m, in_f))
    one, two = tc.run_linear(dt, w1, x, m, in_f, n1), tc.run_linear(dt, w2, x, m, in_f, n2)
    g = infr_b200.Graph()
    xi, a, b = g.input(m * in_f), g.weight(n1 * in_f, dt), g.weight(n2 * in_f, dt)
    ya, yb = g.output(m * n1), g.output(m * n2)
    g.linear(xi, a, ya, m, in_f, n1)
    g.linear(xi, b, yb, m, in_f, n2)
    plan = tc.compile(g)
    ba, bb = tc.alloc(m * n1 * 4), tc.alloc(m * n2 * 4)
    bind = {xi: tc.from_numpy(x), a: tc.from_numpy(w1), b: tc.from_numpy(w2), ya: ba, yb: bb}
    runs = []
    for _ in range(3):
        tc.execute(plan, bind)
        runs.append((tc.download(ba, np.float32).reshape(m, n1), tc.download(bb, np.float32).reshape(m, n2)))
    for ga, gb in runs:
        np.testing.assert_array_equal(ga, runs[0][0])
        np.testing.assert_array_equal(gb, runs[0][1])
        # the K splits follow the summed height: rounding order may differ from the single calls
        assert fx.rel_l2(ga, one) < TOL and fx.rel_l2(gb, two) < TOL
    plan.close()


@pytest.mark.parametrize("dt,in_f,n1,n2,m", [
    (Q4K, 4096, 4096, 1024, 24),                                  # the wide GEMV: the bits of two calls
    (Q2_0, 2048, 1000, 256, 16),                                  # its GEMM, each matrix split as it would be alone: the same
    (Q4K, 4096, 4096, 1024, 33), (Q4K, 4096, 4096, 1024, 113),    # K splits of 4 and 16 on their own, another together
    (Q4K, 4096, 8192, 8192, 32),                                  # large together, not each
    (Q4K, 4096, 12288, 12288, 25), (Q4K, 4096, 12288, 200, 32),   # both large; one of them
    (Q6K, 2048, 1024, 256, 300), (Q2_0, 2048, 1000, 256, 300),
])
def test_a_pair_against_two_calls_and_the_cpu(backend, oracle, dt, in_f, n1, n2, m):
    be, bb = fx.BLOCK[dt]
    rows = [synth.weight(dt, 40, in_f, seed=s) for s in (1, 2)]  # the weights repeat with period 40 rows
    w1, w2 = (backend.from_numpy(np.tile(r, n // 40 + 1)[:n * in_f // be * bb]) for r, n in zip(rows, (n1, n2)))
    xh = synth.normal(5, (m, in_f))
    x = backend.from_numpy(xh)
    want = [oracle.linear(dt, r, xh, m, in_f, 40) for r in rows]
    y = [backend.alloc(m * n * 4) for n in (n1, n2, n1, n2)]

    def check():
        single, pair = ([backend.download(b, np.float32).reshape(m, -1) for b in y[i:i + 2]] for i in (0, 2))
        for s, p, cpu in zip(single, pair, want):
            if m <= (16 if dt == Q2_0 else 24):
                np.testing.assert_array_equal(p, s)
            for got in (s, p):
                last = got.shape[1] // 40 * 40 - 40
                assert max(fx.rel_l2(got[:, r:r + 40], cpu) for r in (0, last)) < TOL
    backend.linear(dt, w1, x, y[0], m, in_f, n1)
    backend.linear(dt, w2, x, y[1], m, in_f, n2)
    backend.linear_pair(dt, w1, y[2], n1, w2, y[3], n2, x, m, in_f)
    check()
    if dt == Q6K or (dt == Q4K and m <= 32):  # the same from quantised rows
        q = [backend.alloc(n) for n in (m * in_f, m * in_f // 256 * 4, m * in_f // 32 * 4, m * in_f // 16 * 4)]
        backend.quantize_q8(256, x, m, in_f, *q)
        backend.gemv_q8(dt, w1, *q, y[0], m, in_f, n1)
        backend.gemv_q8(dt, w2, *q, y[1], m, in_f, n2)
        backend.gemv_q8_pair(dt, w1, y[2], n1, w2, y[3], n2, *q, m, in_f)
        check()


@pytest.mark.parametrize("dt,in_f,out_f,rows", [
    (Q6K, 2048, 2048, (33, 48, 49)), (Q6K, 2048, 2080, (33,)), (Q6K, 4096, 1000, (33,)),  # two passes of the wide GEMV, or the GEMM
    (Q2_0, 4096, 12320, (8, 9, 16, 17, 18)), (Q2_0, 4096, 24600, (24, 25)),             # the GEMV, or the GEMM on the warp matrix unit
])
def test_batches_at_the_lines_between_kernels(backend, oracle, dt, in_f, out_f, rows):
    be, bb = fx.BLOCK[dt]
    part = synth.weight(dt, 40, in_f, seed=1)  # the weights repeat with period 40 rows
    w = backend.from_numpy(np.tile(part, out_f // 40 + 1)[:out_f * in_f // be * bb])
    for m in rows:
        x = synth.normal(m, (m, in_f))
        y = backend.alloc(m * out_f * 4)
        backend.linear(dt, w, backend.from_numpy(x), y, m, in_f, out_f)
        got, want = backend.download(y, np.float32).reshape(m, out_f), oracle.linear(dt, part, x, m, in_f, 40)
        for r in (0, out_f // 40 * 40 - 40):
            assert fx.rel_l2(got[:, r:r + 40], want) < TOL


@pytest.mark.parametrize("dt", [Q4K, Q6K, Q2_0])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_gemm_tc_non_finite_activations(tc, oracle, dt, bad):
    m, in_f, out_f = 40, 2048, 128
    w = synth.weight(dt, out_f, in_f, seed=8)
    x = synth.normal(9, (m, in_f))
    x[7, 100] = bad
    got, want = tc.run_linear(dt, w, x, m, in_f, out_f), oracle.linear(dt, w, x, m, in_f, out_f)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want).any(axis=1)
    assert fx.rel_l2(got[ok], want[ok]) < TOL


def test_quantised_rows_above_the_wide_gemv(backend, oracle):
    # gemv_q8 with more Q6_K rows than the wide GEMV takes in a pass: the GEMM from quantised rows
    m, in_f, out_f = 45, 2048, 96
    w, x = synth.weight(Q6K, out_f, in_f, seed=4), synth.normal(5, (m, in_f))
    xb, wb, yb = backend.from_numpy(x), backend.from_numpy(w), backend.alloc(m * out_f * 4)
    qs, d, sums, s16 = (backend.alloc(n) for n in (m * in_f, m * in_f // 256 * 4, m * in_f // 32 * 4, m * in_f // 16 * 4))
    backend.quantize_q8(256, xb, m, in_f, qs, d, sums, s16)
    backend.gemv_q8(Q6K, wb, qs, d, sums, s16, yb, m, in_f, out_f)
    got = backend.download(yb, np.float32).reshape(m, out_f)
    assert fx.rel_l2(got, oracle.linear(Q6K, w, x, m, in_f, out_f)) < TOL


@pytest.mark.parametrize("m,n1,n2", [(25, 12288, 12288), (32, 12288, 0), (32, 12288, 200)])
def test_batches_against_large_q4k_weights(backend, oracle, m, n1, n2):
    # default context, at most 32 rows, enough weights that the GEMM is taken instead of the wide GEMV
    in_f = 4096
    x = synth.normal(5, (m, in_f))
    ws = [np.tile(synth.weight(Q4K, 128, in_f, seed=s), n // 128 + 1)[:n * in_f // 256 * 144] for s, n in ((1, n1), (2, n2)) if n]
    g = infr_b200.Graph()
    xi, bind, outs = g.input(m * in_f), {}, []
    for w in ws:
        n = w.size // (in_f // 256 * 144)
        wi, yi, yb = g.weight(n * in_f, Q4K), g.output(m * n), backend.alloc(m * n * 4)
        g.linear(xi, wi, yi, m, in_f, n)
        bind.update({wi: backend.from_numpy(w), yi: yb})
        outs.append((yb, n, w))
    bind[xi] = backend.from_numpy(x)
    plan = backend.compile(g)
    backend.execute(plan, bind)
    for yb, n, w in outs:
        got = backend.download(yb, np.float32).reshape(m, n)
        want = oracle.linear(Q4K, w[:128 * in_f // 256 * 144], x, m, in_f, 128)  # the rows repeat with period 128
        for r in (0, n // 128 * 128 - 128):
            assert fx.rel_l2(got[:, r:r + 128], want) < TOL
    plan.close()
