"""Plans whose Linears read rows that the op before them forms (RmsNorm, Add and RmsNorm, GatedAct): where the tensor-memory GEMM takes the
Linear, one launch forms the rows and lays them out.  Every tensor has the bits of the ops called one by one."""
import functools

import numpy as np
import pytest

import infr_b200
from fixtures import Q4K
from infr_b200 import Q6K, synth

pytestmark = pytest.mark.gpu
EPS = 1e-5


@functools.lru_cache(maxsize=None)
def _w(dt, k, dim):
    return synth.weight(dt, k, dim, seed=k)


def _x(seed, rows, dim, special):
    x = synth.normal(seed, (rows, dim))
    if special and rows > 3:
        x[0] = 0.0          # scale zero
        x[1, 5] = 1e30      # one code left
        x[2] *= 1e-30       # small codes' scale
        x[3, :256] = 0.0
    return x


@pytest.mark.parametrize("m", [25, 33, 64, 65, 128, 129])   # token tiles of 32, 64 and 128 rows: with and without empty slots
@pytest.mark.parametrize("dt,dim,n", [(Q4K, 256, (64,)), (Q4K, 4096, (14336, 100)), (Q4K, 8448, (300, 17)), (Q6K, 2048, (130,)), (Q6K, 10240, (64, 200))])
@pytest.mark.parametrize("source", ["norm", "add-norm", "gated"])
def test_rows_formed_for_the_gemm(backend, dt, dim, n, m, source):
    be, up = backend, backend.from_numpy
    g, bind = infr_b200.Graph(), {}
    xa, xb, nw = up(_x(1, m, dim, True)), up(_x(2, m, dim, False)), up((1.0 + 0.1 * synth.normal(3, (dim,))).astype(np.float32))
    a, b, w, s, r = g.input(m * dim), g.input(m * dim), g.input(dim), g.output(m * dim), g.output(m * dim)
    sb, rb = be.alloc(m * dim * 4), be.alloc(m * dim * 4)
    s2, r2 = be.alloc(m * dim * 4), be.alloc(m * dim * 4)
    bind.update({a: xa, b: xb, w: nw, s: sb, r: rb})
    if source == "norm":
        g.rms_norm(a, w, r, m, dim, EPS)
        be.rms_norm(xa, nw, r2, m, dim, EPS)
    elif source == "add-norm":
        g.add(a, b, s, m * dim)
        g.rms_norm(s, w, r, m, dim, EPS)
        be.add_rms_norm(xa, xb, s2, nw, r2, m, dim, EPS)
    else:
        g.gated_act(a, b, r, m, dim)
        be.gated_act(xa, xb, r2, m, dim)
    ws, ys, want = [up(_w(dt, k, dim)) for k in n], [be.alloc(m * k * 4) for k in n], [be.alloc(m * k * 4) for k in n]
    for k, wt, y in zip(n, ws, ys):
        wh, o = g.weight(k * dim, dt), g.output(m * k)
        g.linear(r, wh, o, m, dim, k)
        bind.update({wh: wt, o: y})
    if len(n) == 2:
        be.linear_pair(dt, ws[0], want[0], n[0], ws[1], want[1], n[1], r2, m, dim)
    else:
        be.linear(dt, ws[0], r2, want[0], m, dim, n[0])
    be.execute(be.compile(g), bind)
    np.testing.assert_array_equal(be.download(rb, np.uint32), be.download(r2, np.uint32))
    if source == "add-norm":
        np.testing.assert_array_equal(be.download(sb, np.uint32), be.download(s2, np.uint32))
    for y, v in zip(ys, want):
        np.testing.assert_array_equal(be.download(y, np.uint32), be.download(v, np.uint32))


def test_gated_rows_in_place_and_overlapping(backend):
    """The gate's own buffer as the destination; a destination that starts inside the gate takes the two launches."""
    be, m, dim, k = backend, 40, 512, 96
    x, u, wt = synth.normal(1, (m, dim)), synth.normal(2, (m, dim)), be.from_numpy(synth.weight(Q4K, k, dim, seed=3))
    gb, ub, act, want = be.from_numpy(x), be.from_numpy(u), be.alloc(m * dim * 4), be.alloc(m * k * 4)
    be.gated_act(gb, ub, act, m, dim)
    be.linear(Q4K, wt, act, want, m, dim, k)
    g, y = infr_b200.Graph(), be.alloc(m * k * 4)
    a, b, r, wh, o = g.input(m * dim), g.input(m * dim), g.output(m * dim), g.weight(k * dim, Q4K), g.output(m * k)
    g.gated_act(a, b, r, m, dim)
    g.linear(r, wh, o, m, dim, k)
    n0 = be.launch_count()
    be.execute(be.compile(g), {a: gb, b: ub, r: gb, wh: wt, o: y})
    fused = be.launch_count() - n0
    np.testing.assert_array_equal(be.download(gb, np.uint32), be.download(act, np.uint32))
    np.testing.assert_array_equal(be.download(y, np.uint32), be.download(want, np.uint32))
    big = be.from_numpy(np.concatenate([x.ravel(), np.zeros(dim, np.float32)]))
    lo, hi = be.wrap(big.device_ptr(), m * dim * 4), be.wrap(big.device_ptr() + dim * 4, m * dim * 4)
    n0 = be.launch_count()
    be.execute(be.compile(g), {a: lo, b: ub, r: hi, wh: wt, o: y})
    assert be.launch_count() - n0 == fused + 1
