"""The tensor-memory GEMM over several token tiles: whole waves of tiles over all of K, the tiles past them split over K (gemm_tc.cu,
split_of), vs the CPU restatement.  Tolerance as in test_gemm_tc_gpu.py: the block sums are the CPU's integers."""
import numpy as np
import pytest

import fixtures as fx
import infr_b200
from infr_b200 import Q4K, Q6K, synth

pytestmark = pytest.mark.gpu
TOL = 5e-7


@pytest.fixture(scope="module")
def be():
    b = infr_b200.CudaBackend(device=0)
    yield b
    b.close()


@pytest.mark.parametrize("dt", [Q4K, Q6K])
@pytest.mark.parametrize("m,in_f,out_f", [
    (140, 4096, 9590),   # 150 tiles of 128 x 128: two past a wave of 148, the last row tile partial
    (129, 2048, 300),    # fewer tiles than SMs
    (257, 6144, 6273),   # 150 tiles over three token tiles, the last of one token; a height that is not a multiple of four
    (150, 4096, 18944),  # whole waves only
])
def test_gemm_tc_tail_split(be, oracle, dt, m, in_f, out_f):
    w = synth.weight(dt, out_f, in_f, seed=m)
    x = synth.normal(6, (m, in_f))
    x[::3] *= 100.0
    got, want = be.run_linear(dt, w, x, m, in_f, out_f), oracle.linear(dt, w, x, m, in_f, out_f)
    assert fx.rel_l2(got, want) < TOL
    assert max(fx.rel_l2(got[r], want[r]) for r in range(m)) < 2 * TOL


@pytest.mark.parametrize("m", [65, 113, 128])
def test_gemm_tc_q6_halves_share_accumulators(be, oracle, m):
    # 128-token tiles of Q6_K multiply a block in two halves of the tokens, whose accumulators are drained and filled in turn: many blocks
    # through one set of them, the same bits on every run
    in_f, out_f = 28672, 2600  # 21 row tiles: K split 7 ways, 16 blocks a CTA
    part = synth.weight(Q6K, 40, in_f, seed=m)  # the weights repeat with period 40 rows
    w = be.from_numpy(np.tile(part, out_f // 40))
    xh = synth.normal(6, (m, in_f))
    x, y = be.from_numpy(xh), be.alloc(m * out_f * 4)
    runs = set()
    for _ in range(20):
        be.linear(Q6K, w, x, y, m, in_f, out_f)
        runs.add(be.download(y, np.uint32).tobytes())
    assert len(runs) == 1
    got, want = be.download(y, np.float32).reshape(m, out_f // 40, 40), oracle.linear(Q6K, part, xh, m, in_f, 40)
    assert max(fx.rel_l2(got[:, i], want) for i in range(out_f // 40)) < TOL


@pytest.mark.parametrize("dt", [Q4K, Q6K])
@pytest.mark.parametrize("m,in_f,n1,n2", [
    (130, 4096, 4096, 1024),    # fewer tiles than SMs, all of them split
    (300, 2048, 16384, 2600),   # 450 tiles: whole waves in front of the split ones, which lie in the second matrix (its last row tile partial)
    (257, 4096, 300, 6400),     # 159 tiles, the first matrix of three
])
def test_gemm_tc_tail_split_of_a_pair(be, oracle, dt, m, in_f, n1, n2):
    parts = [synth.weight(dt, 40, in_f, seed=s) for s in (1, 2)]  # the weights repeat with period 40 rows
    w1, w2 = (be.from_numpy(np.resize(p, p.size // 40 * n)) for p, n in zip(parts, (n1, n2)))
    xh = synth.normal(6, (m, in_f))
    x, y1, y2 = be.from_numpy(xh), be.alloc(m * n1 * 4), be.alloc(m * n2 * 4)
    be.linear_pair(dt, w1, y1, n1, w2, y2, n2, x, m, in_f)
    for p, y, n in zip(parts, (y1, y2), (n1, n2)):
        want = oracle.linear(dt, p, xh, m, in_f, 40)
        got = be.download(y, np.float32).reshape(m, n)
        assert fx.rel_l2(got, np.tile(want, (1, n // 40 + 1))[:, :n]) < TOL
