"""The batched Q2_0 GEMM (gemm_q2.cu, more than 8 rows) vs the CPU restatement of infr-cpu's production path, at the edges of its
tiles: 256 weight rows, 8 .. 80 tokens, rows of any whole number of 64-element blocks (they start on any even address), the K splits.

Tolerance: the group sums are the CPU's integers, so a result differs only by the order of its f32 additions: 5e-7 relative L2
for the shapes here (as for the other formats' GEMM)."""
import numpy as np
import pytest

import fixtures as fx
import infr_b200
from infr_b200 import Q2_0, synth

pytestmark = pytest.mark.gpu
TOL = 5e-7


@pytest.fixture(scope="module")
def be():
    b = infr_b200.CudaBackend(device=0)
    yield b
    b.close()


@pytest.mark.parametrize("m,in_f,out_f", [
    (9, 64, 1),         # one block, one row
    (16, 192, 257),     # one row past a tile; a stage of three blocks
    (17, 4160, 256),    # rows of 1170 bytes: every other one off a 4-byte boundary
    (40, 576, 255),     # the most tokens that share the blocks of K
    (41, 704, 300),     # the fewest that are split over the warps
    (80, 1088, 130),    # a full token tile
    (81, 640, 512),     # two token tiles of 48
    (100, 14336, 64),   # K split over many CTAs
    (250, 576, 300),    # four token tiles
    (1024, 1024, 70),   # thirteen, the last one short
    (70, 256, 40000),   # more tiles than SMs
])
def test_gemm_q2_matches_production_cpu(be, oracle, m, in_f, out_f):
    w = synth.weight(Q2_0, out_f, in_f, seed=m + in_f)
    x = synth.normal(6, (m, in_f))
    x[::3] *= 100.0
    got, want = be.run_linear(Q2_0, w, x, m, in_f, out_f), oracle.linear(Q2_0, w, x, m, in_f, out_f)
    assert fx.rel_l2(got, want) < TOL
    if out_f > 1:
        assert max(fx.rel_l2(got[r], want[r]) for r in range(m)) < 2 * TOL


def test_gemm_q2_weight_slices(be, oracle):
    # rows of 11 blocks (198 bytes): slices of one weight that start on an even address only, two of them in one launch
    m, in_f, n = 20, 704, 300
    w = synth.weight(Q2_0, n, in_f, seed=2)
    x = synth.normal(3, (m, in_f))
    want = oracle.linear(Q2_0, w, x, m, in_f, n)
    g = infr_b200.Graph()
    xi, wi = g.input(m * in_f), g.weight(n * in_f, Q2_0)
    ya, yb = g.output(m * 37), g.output(m * 250)
    g.linear(xi, wi, ya, m, in_f, 37, w_off=3 * in_f)
    g.linear(xi, wi, yb, m, in_f, 250, w_off=41 * in_f)
    ba, bb = be.alloc(m * 37 * 4), be.alloc(m * 250 * 4)
    be.execute(be.compile(g), {xi: be.from_numpy(x), wi: be.from_numpy(w), ya: ba, yb: bb})
    assert fx.rel_l2(be.download(ba, np.float32).reshape(m, 37), want[:, 3:40]) < TOL
    assert fx.rel_l2(be.download(bb, np.float32).reshape(m, 250), want[:, 41:291]) < TOL


def test_gemm_q2_extreme_codes(be, oracle):
    # code 3 (weight +2) throughout, activations pinned at +/-127, an infinite and a zero activation group
    m, in_f, out_f = 12, 320, 40
    blk = np.full(18, 0xFF, np.uint8)
    blk[0:2] = np.array([0.01], np.float16).view(np.uint8)
    w = np.tile(blk, out_f * in_f // 64)
    x = np.where(np.arange(m * in_f).reshape(m, in_f) % 3 == 0, -1.0, 1.0).astype(np.float32)
    x[2, 64:96] = 0.0
    got, want = be.run_linear(Q2_0, w, x, m, in_f, out_f), oracle.linear(Q2_0, w, x, m, in_f, out_f)
    assert fx.rel_l2(got, want) < TOL
    x[5, 40] = np.inf
    got, want = be.run_linear(Q2_0, w, x, m, in_f, out_f), oracle.linear(Q2_0, w, x, m, in_f, out_f)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))


@pytest.mark.parametrize("m", [9, 12, 16])
@pytest.mark.parametrize("in_f,n1,n2", [
    (4096, 14336, 14336),  # split 2 ways alone, not at all by both heights together
    (4096, 4096, 1024),    # 9 and 15 ways alone, 7 together
    (64, 300, 40),         # one block: neither is split
    (4096, 28672, 515),    # only the second matrix, of a height that is not a multiple of four
])
def test_short_pair_has_the_bits_of_two_calls(be, oracle, m, in_f, n1, n2):
    part = synth.weight(Q2_0, 40, in_f, seed=3)  # the weights repeat with period 40 rows
    w1, w2 = (be.from_numpy(np.tile(part, n // 40 + 1)[:n * in_f // 64 * 18]) for n in (n1, n2))
    xh = synth.normal(7, (m, in_f))
    x, y = be.from_numpy(xh), [be.alloc(m * n * 4) for n in (n1, n2, n1, n2)]
    be.linear(Q2_0, w1, x, y[0], m, in_f, n1)
    be.linear(Q2_0, w2, x, y[1], m, in_f, n2)
    be.linear_pair(Q2_0, w1, y[2], n1, w2, y[3], n2, x, m, in_f)
    want = oracle.linear(Q2_0, part, xh, m, in_f, 40)
    for n, a, b in ((n1, y[0], y[2]), (n2, y[1], y[3])):
        np.testing.assert_array_equal(be.download(a, np.uint32), be.download(b, np.uint32))
        assert fx.rel_l2(be.download(b, np.float32).reshape(m, n)[:, -n % 40 and -(n % 40) - 40 or -40:][:, :40], want) < TOL
