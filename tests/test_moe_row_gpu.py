"""One row of an MoE layer (moe_row.cu: router, gate and up, down in three launches) vs the CPU restatement, where its splits are
uneven: blocks per row against the eight groups of four lanes, ranks against the groups, experts against the lanes.

Tolerance: f32 products of the same dequantised weights, summed in another order: 1e-5 of the output's magnitude, as for every f32 path."""
import numpy as np
import pytest

import infr_b200
from infr_b200 import Q4K, synth
from test_moe_gpu import _banks, _run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    b = infr_b200.CudaBackend(device=0)
    yield b
    b.close()


@pytest.mark.parametrize("ne,n_expert,n_used,nff", [
    (256, 1, 1, 256),      # one block, one expert
    (2304, 33, 5, 768),    # nine blocks a row: one past the groups; five ranks; one expert past a lane's first
    (1280, 60, 6, 512),
    (2048, 8, 2, 2304),    # two ranks: their blocks are split over the groups
    (512, 128, 32, 256),   # the most ranks and experts
    (256, 130, 9, 256),    # one lane too few for the experts: the general launches
])
def test_moe_row_matches_cpu(be, oracle, ne, n_expert, n_used, nff):
    gate, up, down = _banks(n_expert, nff, ne, seed=ne + nff)
    router = synth.normal(17, (n_expert, ne), 1.0 / np.sqrt(ne))
    x = synth.normal(3, (1, ne))
    got, ids, w, lg = _run(be, x, router, gate, up, down, 1, ne, n_expert, n_used, nff)
    want, o_ids, o_w, o_lg = oracle.moe_ffn(x, router, gate, up, down, rows=1, ne=ne, n_expert=n_expert, n_used=n_used, n_ff_exp=nff)
    np.testing.assert_array_equal(lg.view(np.uint32), o_lg.view(np.uint32))
    np.testing.assert_array_equal(ids, o_ids)
    np.testing.assert_allclose(w, o_w, rtol=1e-6)
    assert np.abs(got - want).max() / np.abs(want).max() < 1e-5


def test_moe_row_ties_and_nan(be, oracle):
    # equal logits: the lower expert wins; an infinite activation makes every probability NaN: experts 0 .. k - 1
    ne, n_expert, n_used, nff = 256, 70, 4, 256
    gate, up, down = _banks(n_expert, nff, ne, seed=9)
    router = np.tile(synth.normal(17, (1, ne), 1.0 / np.sqrt(ne)), (n_expert, 1))
    x = synth.normal(3, (1, ne))
    got, ids, w, _ = _run(be, x, router, gate, up, down, 1, ne, n_expert, n_used, nff)
    want, o_ids, o_w, _ = oracle.moe_ffn(x, router, gate, up, down, rows=1, ne=ne, n_expert=n_expert, n_used=n_used, n_ff_exp=nff)
    np.testing.assert_array_equal(ids, o_ids)
    np.testing.assert_allclose(w, o_w, rtol=1e-6)
    assert np.abs(got - want).max() / np.abs(want).max() < 1e-5
    x[0, 7] = np.inf
    _, ids, w, _ = _run(be, x, router, gate, up, down, 1, ne, n_expert, n_used, nff)
    np.testing.assert_array_equal(ids.ravel(), np.arange(n_used))
    assert np.isnan(w).all()


def test_moe_row_takes_the_ids_of_its_own_call(be, oracle):
    # Layers whose gate / up launch leaves SMs idle, so that the down launch is resident while the row is being routed, and ids that change
    # from call to call: neither the ids of the call before nor what the caller's buffer held may be used.
    ne, n_expert, n_used, nff, calls = 512, 60, 4, 256, 24
    gate, up, down = _banks(n_expert, nff, ne, seed=4)
    router = synth.normal(17, (n_expert, ne), 1.0 / np.sqrt(ne))
    x = synth.normal(5, (calls, ne))
    rb, gb, ub, db = (be.from_numpy(a) for a in (router, gate, up, down))
    xs, ys = [be.from_numpy(x[i:i + 1]) for i in range(calls)], [be.alloc(ne * 4) for _ in range(calls)]
    ids, w = be.from_numpy(np.zeros(n_used, np.int32)), be.from_numpy(np.zeros(n_used, np.float32))
    args = dict(rows=1, ne=ne, n_expert=n_expert, n_used=n_used, n_ff_exp=nff)
    for own in (False, True):
        be.sync()
        for xb, yb in zip(xs, ys):
            if own:  # one call at a time
                be.upload(ids, np.zeros(n_used, np.int32))
                be.upload(w, np.zeros(n_used, np.float32))
                be.sync()
            be.moe_ffn(xb, xb, rb, gb, ub, db, yb, **args, **(dict(sel_ids=ids, sel_w=w) if own else {}))
        for i, yb in enumerate(ys):
            want = oracle.moe_ffn(x[i:i + 1], router, gate, up, down, **args)[0].ravel()
            assert np.abs(be.download(yb, np.float32) - want).max() / np.abs(want).max() < 1e-5
            be.upload(yb, np.zeros(ne, np.float32))


@pytest.mark.parametrize("rows,ne,n_expert", [
    (64, 6144, 148), (64, 6144, 149),  # the last whole four waves of the router for a few rows, and one expert more: its tiles
    (5, 2048, 33),                     # rows and experts that are no multiple of four
])
def test_moe_router_kernels_at_the_line(be, oracle, rows, ne, n_expert):
    nff = 256
    gate, up, down = (np.tile(b, n_expert) for b in _banks(1, nff, ne, seed=3))  # (every expert the same)
    router, x = synth.normal(17, (n_expert, ne), 1.0 / np.sqrt(ne)), synth.normal(3, (rows, ne))
    got, ids, _, lg = _run(be, x, router, gate, up, down, rows, ne, n_expert, 1, nff)
    want, o_ids, _, o_lg = oracle.moe_ffn(x, router, gate, up, down, rows=rows, ne=ne, n_expert=n_expert, n_used=1, n_ff_exp=nff)
    np.testing.assert_array_equal(lg.view(np.uint32), o_lg.view(np.uint32))
    np.testing.assert_array_equal(ids, o_ids)
