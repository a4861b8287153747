"""Plans of one-row Q4_K Linears: two neighbours on one row have the bits of a pair call (their heights together choose the K split), any other op
those of a call of its own, however many ops share the launch and whether they can share it.

Heights: 4096 and 1024 rows are split otherwise together (320 tiles) than alone (256 and 64)."""
import pytest

import numpy as np

import infr_b200
from infr_b200 import Q4K, synth

pytestmark = pytest.mark.gpu
IN_F = 4096


def _pairs(rows):
    out, k = [], 0
    while k < len(rows):
        n = 2 if k + 1 < len(rows) and rows[k] == rows[k + 1] else 1
        out.append(range(k, k + n))
        k += n
    return out


@pytest.mark.parametrize("rows,alias", [
    ("xx", False), ("xxx", False), ("xxz", False), ("zxx", False), ("xyz", False), ("xxxx", False), ("zxxxy", False),
    ("abcdefghijklmnopqrstuvwxx", False),  # 25 ops: a launch takes 24, the last two are a pair
    ("xxzz", True),                        # the last result lies where the first does: no common launch
])
def test_pairs_in_a_plan(backend, rows, alias):
    be = backend
    h = [(4096, 1024)[k % 2] if len(rows) < 10 else (48, 4096, 1024)[max(0, k - 22)] for k in range(len(rows))]
    if alias:
        h[3] = h[0]
    ws = {n: [be.from_numpy(synth.weight(Q4K, n, IN_F, seed=n + s)) for s in range(2)] for n in set(h)}
    xs = {c: be.from_numpy(synth.normal(ord(c), (1, IN_F))) for c in set(rows)}
    w = [ws[n][k % 2] for k, n in enumerate(h)]
    want = [None] * len(rows)
    for group in _pairs(rows):
        y = [be.alloc(h[k] * 4) for k in group]
        k = group[0]
        if len(group) == 2:
            be.linear_pair(Q4K, w[k], y[0], h[k], w[k + 1], y[1], h[k + 1], xs[rows[k]], 1, IN_F)
        else:
            be.linear(Q4K, w[k], xs[rows[k]], y[0], 1, IN_F, h[k])
        for j, b in zip(group, y):
            want[j] = be.download(b, np.uint32)
    g, bind, ys = infr_b200.Graph(), {}, []
    xh = {c: g.input(IN_F) for c in xs}
    bind.update({xh[c]: xs[c] for c in xs})
    for k, c in enumerate(rows):
        wh, o = g.weight(h[k] * IN_F, Q4K), g.output(h[k])
        ys.append(ys[0] if alias and k == 3 else be.alloc(h[k] * 4))
        bind.update({wh: w[k], o: ys[k]})
        g.linear(xh[c], wh, o, 1, IN_F, h[k])
    be.execute(be.compile(g), bind)
    for k in range(1 if alias else 0, len(rows)):
        np.testing.assert_array_equal(be.download(ys[k], np.uint32), want[k], err_msg=str(k))
