"""Launches of a stream overlap (a kernel is resident before the one in front of it has finished), so each of them must read what earlier
ones write after its wait.  A chain of every op over shared buffers, called for several inputs without a pause, gives the bits of the
same chain called in the opposite order with a sync after every op: sizes that leave most SMs idle, where the overlap is largest."""
import numpy as np
import pytest

import infr_b200
from infr_b200 import Q2_0, Q4K, Q6K, synth

pytestmark = pytest.mark.gpu
H, FF, HEADS, KV, HD, CALLS = 512, 768, 8, 2, 64, 8


@pytest.fixture(scope="module")
def be():
    b = infr_b200.CudaBackend(device=0)
    yield b
    b.close()


@pytest.mark.parametrize("moe", [False, True])
@pytest.mark.parametrize("dt", [Q4K, Q6K, Q2_0])
@pytest.mark.parametrize("rows", [1, 5, 12, 40])
def test_chain_has_the_bits_of_its_ops_alone(be, rows, dt, moe):
    nx, nu, bank_dt = 12, 3, Q4K if rows == 1 or dt == Q2_0 else dt
    x = [be.from_numpy(synth.normal(10 + i, (rows, H))) for i in range(CALLS)]
    ones, zero = be.from_numpy(np.ones(H, np.float32)), be.from_numpy(np.zeros((rows, H), np.float32))
    wg, wu, wd = (be.from_numpy(synth.weight(dt, o, i, s)) for o, i, s in ((FF, H, 1), (FF, H, 2), (H, FF, 3)))
    router = be.from_numpy(synth.normal(4, (nx, H), H ** -0.5))
    gate, up, down = (be.from_numpy(np.concatenate([synth.weight(bank_dt, o, i, s + e) for e in range(nx)])) for o, i, s in ((FF, H, 20), (FF, H, 40), (H, FF, 60)))
    pos = be.from_numpy(np.arange(rows, dtype=np.int32))
    h, n, a, o, q, m = (be.alloc(rows * w * 4) for w in (H, H, FF, H, H, H))
    g, u = be.alloc(rows * FF * 4), be.alloc(rows * FF * 4)
    kc, vc = be.alloc(rows * KV * HD * 2), be.alloc(rows * KV * HD * 2)
    out = [[be.alloc(rows * H * 4), be.alloc(rows * H * 4), be.alloc(rows * 4)] for _ in range(CALLS)]

    def call(i, sync):
        s, t, ids = out[i]
        be.add(x[i], zero, h, rows * H), sync()
        be.rms_norm(h, ones, n, rows, H, 1e-5), sync()
        be.linear(dt, wg, n, g, rows, H, FF), sync()
        be.linear(dt, wu, n, u, rows, H, FF), sync()
        be.gated_act(g, u, a, rows, FF), sync()
        be.linear(dt, wd, a, o, rows, FF, H), sync()
        be.add_rms_norm(h, o, s, ones, n, rows, H, 1e-5), sync()
        if moe:
            be.moe_ffn(n, n, router, gate, up, down, m, rows=rows, ne=H, n_expert=nx, n_used=nu, n_ff_exp=FF, wdt=bank_dt), sync()
            be.add(n, m, n, rows * H), sync()
        be.linear_pair(dt, wg, g, FF, wu, u, FF, n, rows, H), sync()
        be.gated_act(g, u, a, rows, FF), sync()
        be.linear(dt, wd, a, q, rows, FF, H), sync()
        be.rope_write_kv(q, g, u, pos, kc, vc, rows=rows, pos=0, n_head=HEADS, n_kv=KV, head_dim=HD, theta=1e4), sync()
        be.attention(q, kc, vc, t, rows=rows, pos=0, n_head=HEADS, n_kv=KV, head_dim=HD, scale=HD ** -0.5), sync()
        be.argmax(t, ids, H, rows), sync()

    def results():
        return [[be.download(b, np.uint32) for b in bufs] for bufs in out]

    for i in reversed(range(CALLS)):
        call(i, be.sync)
    want = results()
    assert len({w[1].tobytes() for w in want}) == CALLS
    for _ in range(3):
        for i in range(CALLS):
            call(i, lambda: None)
        for got, w in zip(results(), want):
            for b, c in zip(got, w):
                np.testing.assert_array_equal(b, c)
