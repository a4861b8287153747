"""A Linear whose result lies over its rows (the op list's contract allows it) reads them all before it writes: vs the CPU restatement,
with the tolerance of the same call into a buffer of its own."""
import numpy as np
import pytest

import fixtures as fx
import infr_b200
from infr_b200 import ACT_F32, ACT_INT8, Q2_0, Q4K, Q6K, synth

pytestmark = pytest.mark.gpu
N = 4096  # enough CTAs that some store while others have not begun
TOL = {ACT_INT8: 1e-6, ACT_F32: 1e-5}


@pytest.fixture(scope="module")
def be():
    b = infr_b200.CudaBackend(device=0)
    yield b
    b.close()


def _rows(be, m, seed):
    x = synth.normal(seed, (m, N))
    return x, be.from_numpy(x)


@pytest.mark.parametrize("dt,m,act", [(Q2_0, 1, ACT_INT8), (Q4K, 1, ACT_INT8), (Q4K, 8, ACT_INT8), (Q2_0, 3, ACT_F32), (Q4K, 9, ACT_F32), (Q6K, 1, ACT_F32)])
def test_linear_in_place(be, oracle, dt, m, act):
    w = synth.weight(dt, N, N, seed=1)
    wb = be.from_numpy(w)
    for seed in range(4):
        x, xb = _rows(be, m, seed)
        be.linear(dt, wb, xb, xb, m, N, N, act)
        assert fx.rel_l2(be.download(xb, np.float32).reshape(m, N), oracle.linear(dt, w, x, m, N, N, reference=act == ACT_F32)) < TOL[act]


@pytest.mark.parametrize("dt,m", [(Q2_0, 1), (Q4K, 1), (Q4K, 8)])
@pytest.mark.parametrize("first", [True, False])
def test_pair_with_one_result_over_the_rows(be, oracle, dt, m, first):
    w1, w2 = synth.weight(dt, N, N, seed=1), synth.weight(dt, N, N, seed=2)
    b1, b2, other = be.from_numpy(w1), be.from_numpy(w2), be.alloc(m * N * 4)
    x, xb = _rows(be, m, 9)
    y1, y2 = (xb, other) if first else (other, xb)
    be.linear_pair(dt, b1, y1, N, b2, y2, N, xb, m, N)
    for w, y in ((w1, y1), (w2, y2)):  # both from the rows as they were
        assert fx.rel_l2(be.download(y, np.float32).reshape(m, N), oracle.linear(dt, w, x, m, N, N)) < 1e-6


@pytest.mark.parametrize("dt,m,in_f", [(Q6K, 5, 12544), (Q6K, 8, 14080), (Q4K, 8, 28672), (Q2_0, 8, 14080)])
def test_pair_whose_rows_do_not_fit_a_cta_together(be, oracle, dt, m, in_f):
    # in narrower batches, as a single call takes them
    w1, w2 = synth.weight(dt, 40, in_f, seed=1), synth.weight(dt, 130, in_f, seed=2)
    x, y1, y2 = synth.normal(3, (m, in_f)), be.alloc(m * 40 * 4), be.alloc(m * 130 * 4)
    be.linear_pair(dt, be.from_numpy(w1), y1, 40, be.from_numpy(w2), y2, 130, be.from_numpy(x), m, in_f)
    for w, y, n in ((w1, y1, 40), (w2, y2, 130)):
        assert fx.rel_l2(be.download(y, np.float32).reshape(m, n), oracle.linear(dt, w, x, m, in_f, n)) < 1e-6
