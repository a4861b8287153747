"""Rows of FFN width and beyond: every length that fits some kernel's shared memory runs, in each form, and has the CPU path's values.

Lengths: on both sides of the lines between the one-row kernels (Q4_K 24576, 38912 and 59136, Q6_K 20480, 36864 and 51200) and the longest.
A row's block sums are exact; each of in_f / 256 f32 additions rounds by 2^-24 of the sum so far at most."""
import numpy as np
import pytest

import fixtures as fx
from infr_b200 import Q4K, Q6K, synth

pytestmark = pytest.mark.gpu


LENGTHS = [(Q4K, k) for k in (4352, 24576, 24832, 38912, 39168, 59136, 59392, 65536, 73728, 131072)] + \
          [(Q6K, k) for k in (20480, 22528, 30720, 36864, 38912, 51200, 53248, 65536, 131072)]


@pytest.mark.parametrize("dt,in_f,n", [(dt, k, 33) for dt, k in LENGTHS] + [(dt, k, 2400) for dt, k in LENGTHS if k < 40000])  # more tiles than SMs
def test_one_row(backend, oracle, dt, in_f, n):
    be, n2 = backend, 17
    w, w2, x = synth.weight(dt, n, in_f, seed=1), synth.weight(dt, n2, in_f, seed=2), synth.normal(3, (1, in_f))
    wb, wb2, xb = be.from_numpy(w), be.from_numpy(w2), be.from_numpy(x)
    y, y2 = be.alloc(n * 4), be.alloc(n2 * 4)
    tol = np.sqrt(in_f / 256) * 2.0**-23
    want, want2 = oracle.linear(dt, w, x, 1, in_f, n).ravel(), oracle.linear(dt, w2, x, 1, in_f, n2).ravel()

    def check(one):
        assert fx.rel_l2(be.download(y, np.float32), want) < tol
        if not one:
            assert fx.rel_l2(be.download(y2, np.float32), want2) < tol

    be.linear(dt, wb, xb, y, 1, in_f, n)
    check(True)
    be.linear_pair(dt, wb, y, n, wb2, y2, n2, xb, 1, in_f)
    check(False)
    q = [be.alloc(k) for k in (in_f, in_f // 64, in_f // 8, in_f // 4)]
    be.quantize_q8(256, xb, 1, in_f, *q)
    be.gemv_q8(dt, wb, *q, y, 1, in_f, n)
    check(True)
    be.gemv_q8_pair(dt, wb, y, n, wb2, y2, n2, *q, 1, in_f)
    check(False)


@pytest.mark.parametrize("dt,in_f", [(Q4K, 65536), (Q4K, 131072), (Q6K, 65536)])
def test_three_rows(backend, oracle, dt, in_f):
    """Too long to stage three of them: narrower batches, down to single rows."""
    be, n, m = backend, 20, 3
    w, x = synth.weight(dt, n, in_f, seed=4), synth.normal(5, (m, in_f))
    y = be.alloc(m * n * 4)
    be.linear(dt, be.from_numpy(w), be.from_numpy(x), y, m, in_f, n)
    assert fx.rel_l2(be.download(y, np.float32).reshape(m, n), oracle.linear(dt, w, x, m, in_f, n)) < np.sqrt(in_f / 256) * 2.0**-23


@pytest.mark.parametrize("dt,in_f", [(Q4K, 59392), (Q6K, 53248)])
def test_pushed_row(backend, dt, in_f):
    """A row-parallel result pushed from the GEMV's epilogue (one rank): what the norm reads is gemv_q8's result."""
    be, n = backend, 256
    comm = be.comm_create(0, 1, n)
    w, x = be.from_numpy(synth.weight(dt, n, in_f, seed=6)), be.from_numpy(synth.normal(7, (1, in_f)))
    q = [be.alloc(k) for k in (in_f, in_f // 64, in_f // 8, in_f // 4)]
    be.quantize_q8(256, x, 1, in_f, *q)
    y, zero, s, nw = be.alloc(n * 4), be.from_numpy(np.zeros(n, np.float32)), be.alloc(n * 4), be.from_numpy(np.ones(n, np.float32))
    be.gemv_q8(dt, w, *q, y, 1, in_f, n)
    o = [be.alloc(k) for k in (n, n // 64, n // 8, n // 4)]
    be.gemv_q8_push(comm, dt, w, *q, 1, in_f, n)
    be.add_rms_norm_q8_pull(comm, zero, s, nw, 1, n, 1e-5, *o)
    be.sync()
    np.testing.assert_array_equal(be.download(s, np.float32), be.download(y, np.float32))
    comm.close()
