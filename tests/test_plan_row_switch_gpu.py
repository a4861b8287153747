"""One-row Linears of a plan that share a launch, with more tiles than CTAs: a CTA goes on to the next matrix and takes that one's row in between, where its
shared memory still serves the last one.  The bits of single calls.

Sizes: one K unit a warp and several (the row in registers, in shared memory), a tile or two a CTA and six; for Q2_0 both ways to share a row."""
import numpy as np
import pytest

import infr_b200
from infr_b200 import Q2_0, Q4K, Q6K, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,in_f,tiles", [(Q4K, 4096, 10), (Q4K, 8192, 10), (Q4K, 5632, 40), (Q6K, 4096, 40), (Q6K, 6144, 10), (Q6K, 10240, 10),
                                           (Q2_0, 1024, 40), (Q2_0, 4096, 10), (Q2_0, 8704, 10), (Q2_0, 8704, 40)])
def test_next_row_in_a_cta(backend, dt, in_f, tiles):
    be, count = backend, 24
    n = [16 * (tiles + i % 3) - 7 * (i % 2) for i in range(count)]
    ws = {k: be.from_numpy(synth.weight(dt, k, in_f, seed=k)) for k in set(n)}
    xs = [be.from_numpy(synth.normal(200 + i, (1, in_f))) for i in range(count)]
    g, bind, ys, want = infr_b200.Graph(), {}, [], []
    for k, x in zip(n, xs):
        y = be.alloc(k * 4)
        be.linear(dt, ws[k], x, y, 1, in_f, k)
        want.append(be.download(y, np.uint32))
        a, w, o = g.input(in_f), g.weight(k * in_f, dt), g.output(k)
        g.linear(a, w, o, 1, in_f, k)
        ys.append(be.alloc(k * 4))
        bind.update({a: x, w: ws[k], o: ys[-1]})
    n0 = be.launch_count()
    be.execute(be.compile(g), bind)
    assert be.launch_count() - n0 == 1
    for y, v in zip(ys, want):
        np.testing.assert_array_equal(be.download(y, np.uint32), v)
