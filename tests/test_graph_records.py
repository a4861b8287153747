"""The packed op records of a Graph are the bytes of the ctypes structure that the C ABI reads."""
import numpy as np
import pytest

import infr_b200
from infr_b200 import _OpDesc, _op_record


def _by_fields(tag, tensors, u, f):
    op = _OpDesc()
    op.tag = tag
    for i, t in enumerate(tensors):
        op.t[i] = t
    for i, v in enumerate(u):
        op.u[i] = int(v)
    for i, v in enumerate(f):
        op.f[i] = float(v)
    return bytes(op)


@pytest.mark.parametrize("tag,tensors,u,f", [
    (1, (1, 2, 3), (4, 5, 6, 7), ()),
    (2, tuple(range(7)), tuple(range(9)), (1.5,)),
    (4, (0, 1, 2), (np.int64(3), np.uint32(4), True, False), (np.float32(0.1),)),
    (9, (1, 2), (2.0, 7), ()),                # a float for a count
    (5, (1, 2), (1, 2, -1), ()),              # wraps like the field
    (8, (1, 2, 3), (2**32 + 5,), (1e300,)),   # out of range: wraps, and infinity
    (10, (), (), (1, 2, 3, 4)),
])
def test_record_is_the_structure(tag, tensors, u, f):
    assert _op_record(tag, tensors, u, f) == _by_fields(tag, tensors, u, f)


def test_graph_keeps_its_records():
    g = infr_b200.Graph()
    a, b, c = g.input(256), g.weight(256 * 4, infr_b200.Q4K), g.output(4)
    g.linear(a, b, c, 1, 256, 4, w_off=256)
    op = _OpDesc.from_buffer_copy(g.ops[0])
    assert (op.tag, list(op.t)[:3], list(op.u)[:4]) == (infr_b200.OP_LINEAR, [a, b, c], [1, 256, 4, 256])


@pytest.mark.parametrize("bad", [{"m": 2.5}, {"in_f": 256.0}, {"out_f": "4"}, {"w_off": None}])
def test_linear_refuses_what_is_no_integer(bad):
    g = infr_b200.Graph()
    a, b, c = g.input(256), g.weight(256 * 4, infr_b200.Q4K), g.output(4)
    with pytest.raises(TypeError):
        g.linear(a, b, c, **{**dict(m=1, in_f=256, out_f=4, w_off=0), **bad})
    assert not g.ops
    g.linear(a, b, c, np.int64(1), 256, 2**32 + 4)  # integers of any type; out of range: wraps like the field
    assert list(_OpDesc.from_buffer_copy(g.ops[0]).u)[:3] == [1, 256, 4]


@pytest.mark.parametrize("bad", [{"ne": 256.0}, {"n_used": 1.5}, {"scale": "1"}])
def test_moe_ffn_refuses_what_is_no_number(bad):
    g = infr_b200.Graph()
    t = [g.input(256) for _ in range(7)]
    with pytest.raises(TypeError):
        g.moe_ffn(*t, **{**dict(ne=256, n_expert=4, n_used=2, n_ff_exp=256, scale=1.0), **bad})
    g.moe_ffn(*t, ne=256, n_expert=4, n_used=2, n_ff_exp=256, scale=2)
    assert _OpDesc.from_buffer_copy(g.ops[0]).f[0] == 2.0


def test_ops_can_be_read_and_edited():
    g = infr_b200.Graph()
    a, b, c = g.input(256), g.input(256), g.output(256)
    g.add(a, b, c, 256)
    g.add(c, b, c, 128)
    ops = g.ops
    assert [(o.tag, list(o.t)[:3], o.u[0]) for o in ops] == [(infr_b200.OP_ADD, [a, b, c], 256), (infr_b200.OP_ADD, [c, b, c], 128)]
    ops[1].u[0] = 64
    g.copy(a, 0, c, 0, 8)
    assert g.ops is ops and ops[2].tag == infr_b200.OP_COPY  # what is emitted later shows up as a structure too
    del ops[2]
    ops.append(_OpDesc.from_buffer_copy(ops[0]))
    g.ops = g.ops[:2] + [ops[2]]
    got = []

    class Lib:  # the library's side of compile
        @staticmethod
        def infr_cuda_compile(ctx, desc, out):
            got.extend((desc._obj.ops[i].tag, desc._obj.ops[i].u[0]) for i in range(desc._obj.n_ops))
            return 0

    be = infr_b200.CudaBackend.__new__(infr_b200.CudaBackend)
    be.L, be.ctx = Lib, None
    be.compile(g)
    assert got == [(infr_b200.OP_ADD, 256), (infr_b200.OP_ADD, 64), (infr_b200.OP_ADD, 256)]
