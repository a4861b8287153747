"""One Q2_0 row: the order in which its blocks are added, which every form of the matvec keeps to the bit.  Block b (64 elements, two groups of 32)
is added to chain b mod 32, one fused multiply-add a group on the product of the two scales; the 32 chains meet along a tree (16 apart, 8, 4, 2, 1).

Sizes: rows of one to four K units of 512, and of more; heights below a CTA's worth of tiles and above; rows too long for the form whose block sums
meet in shared memory (28672 is its longest)."""
import numpy as np
import pytest

from infr_b200 import Q2_0, synth

pytestmark = pytest.mark.gpu


def _want(w, qs, d, n, in_f):
    blk = w.reshape(n, in_f // 64, 18)
    dw = blk[:, :, :2].copy().view(np.float16)[..., 0].astype(np.float32)
    codes = ((blk[:, :, 2:, None] >> np.array([0, 2, 4, 6], np.uint8)) & 3).reshape(n, in_f // 32, 32).astype(np.float32) - 1.0
    sums = np.einsum("ngk,gk->ng", codes, qs.reshape(-1, 32).astype(np.float32)).astype(np.float32)  # whole numbers below 2^13
    chain = np.zeros((n, 32), np.float32)
    for b in range(in_f // 64):
        for g in (2 * b, 2 * b + 1):
            t = (dw[:, b] * d[g]).astype(np.float32)
            # exact product and a 64-bit sum: the one rounding of a fused multiply-add
            chain[:, b % 32] = (t.astype(np.longdouble) * sums[:, g] + chain[:, b % 32]).astype(np.float32)
    while chain.shape[1] > 1:
        h = chain.shape[1] // 2
        chain = chain[:, :h] + chain[:, h:]
    return chain[:, 0]


@pytest.mark.parametrize("in_f,n", [(512, 40), (1024, 2400), (1536, 2500), (2048, 17), (4096, 333), (4096, 5000), (8704, 100), (8704, 2500), (14336, 4800),
                                    (28672, 64), (29184, 48), (29184, 2400)])
def test_order_of_sums(backend, in_f, n):
    be = backend
    w, x = synth.weight(Q2_0, n, in_f, seed=n), synth.normal(in_f, (1, in_f))
    x[0, :64] *= 100.0
    x[0, 96:128] = 0.0
    wb, xb, y = be.from_numpy(w), be.from_numpy(x), be.alloc(n * 4)
    q = [be.alloc(k) for k in (in_f, in_f // 8, in_f // 8, in_f // 4)]
    be.quantize_q8(32, xb, 1, in_f, *q)
    want = _want(w, be.download(q[0], np.int8), be.download(q[1], np.float32), n, in_f)
    be.linear(Q2_0, wb, xb, y, 1, in_f, n)
    np.testing.assert_array_equal(be.download(y, np.float32), want)
    be.gemv_q8(Q2_0, wb, *q, y, 1, in_f, n)
    np.testing.assert_array_equal(be.download(y, np.float32), want)
    y2 = be.alloc(n * 4)
    be.linear_pair(Q2_0, wb, y, n, wb, y2, n, xb, 1, in_f)
    for o in (y, y2):
        np.testing.assert_array_equal(be.download(o, np.float32), want)
