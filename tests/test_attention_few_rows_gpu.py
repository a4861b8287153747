"""A few query rows that share a key / value tile, tiles that they do not fill included: every row has the bits of a call of its own, also
where the last token's values are not finite."""
import numpy as np
import pytest

from infr_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("finite", [True, False])
@pytest.mark.parametrize("n_head,n_kv,rows,pos", [
    (8, 8, 2, 4000),     # two of a tile's sixteen rows, one wave of shared tiles
    (16, 8, 3, 4000),
    (32, 8, 2, 4094),    # the chunk ends on a tile's edge
    (32, 4, 3, 4000),    # two tiles of two rows, the second half empty
    (8, 8, 16, 384),
    (32, 32, 33, 0),     # three shared tiles on 32 heads, one key in the first row
    (32, 8, 8, 1500),
])
def test_rows_equal_single_rows(backend, n_head, n_kv, rows, pos, finite):
    be, hd, kvd = backend, 128, n_kv * 128
    kc = synth.normal(1, (pos + rows, kvd)).astype(np.float16)
    vc = synth.normal(2, (pos + rows, kvd)).astype(np.float16)
    if not finite:
        vc[pos + rows - 1, :] = np.inf
    q = synth.normal(3, (rows, n_head * hd))
    kb, vb = be.from_numpy(kc.view(np.uint16)), be.from_numpy(vc.view(np.uint16))
    qb, ob = be.from_numpy(q), be.alloc(q.nbytes)
    be.attention(qb, kb, vb, ob, rows=rows, pos=pos, n_head=n_head, n_kv=n_kv, head_dim=hd, scale=hd ** -0.5)
    got = be.download(ob, np.float32).reshape(rows, -1)
    assert np.isfinite(got[:-1]).all() and np.isfinite(got[-1]).all() == finite
    for r in range(rows - (0 if finite else 1)):
        q1, o1 = be.from_numpy(q[r:r + 1]), be.alloc(n_head * hd * 4)
        be.attention(q1, kb, vb, o1, rows=1, pos=pos + r, n_head=n_head, n_kv=n_kv, head_dim=hd, scale=hd ** -0.5)
        np.testing.assert_array_equal(got[r], be.download(o1, np.float32))
