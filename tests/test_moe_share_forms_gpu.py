"""Grouped expert launches whose CTAs share all items' tiles evenly, Q6_K rows of an odd number of blocks among them: which of the two grids a layer's banks took is
read from the launches (a row of CTAs an item, or one row in all), and the bits are those of calls of three rows."""
import numpy as np
import pytest

import infr_b200
from infr_b200 import Q4K, Q6K
from kernel_trace import launched
from test_moe_shares_gpu import _bank

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,ne,n_expert,n_used,nff,even", [
    (27, 2048, 128, 8, 768, (True, True)),    # rows of three blocks
    (40, 1024, 100, 4, 2304, (True, True)),   # of nine, four warps a CTA
    (64, 1024, 64, 8, 2048, (True, True)),
    (33, 1024, 64, 4, 1280, (False, False)),  # of five: a whole number of CTAs an item
    (100, 2048, 128, 8, 256, (True, False)),  # of one: staging an item costs more than its tiles
])
def test_grids_and_bits(backend, rows, ne, n_expert, n_used, nff, even):
    import torch

    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(rows, ne, device="cuda", generator=g)
    router = torch.randn(n_expert, ne, device="cuda", generator=g) / ne**0.5
    banks = [_bank(torch, dt, n_expert * nff * ne, 4 + i) for i, dt in enumerate((Q4K, Q4K, Q6K))]
    out, parts = torch.zeros(rows, ne, device="cuda"), torch.ones(rows, ne, device="cuda")
    torch.cuda.synchronize()
    wrap = lambda t: backend.wrap(t.data_ptr(), t.numel() * t.element_size(), infr_b200.USAGE_ACTIVATIONS)
    weights = [wrap(t) for t in (router, *banks)]

    def call(dst, r0, n):
        rows_in = wrap(x[r0:r0 + n])
        backend.moe_ffn(rows_in, rows_in, *weights, wrap(dst[r0:r0 + n]), rows=n, ne=ne, n_expert=n_expert, n_used=n_used, n_ff_exp=nff, wdt=Q4K, down_dt=Q6K)

    records = launched(backend, lambda: call(out, 0, rows), ("gemv_q4k_mma_kernel",), ("gemv_q6_mma_grouped_kernel",))
    grids = {name: grid for name, _, grid in records}
    assert (grids["gemv_q4k_mma_kernel"][1] == 1, grids["gemv_q6_mma_grouped_kernel"][1] == 1) == even
    n = rows - (rows % 3 == 1)  # (a single row takes the f32 path)
    for r0 in range(0, n, 3):
        call(parts, r0, min(3, n - r0))
    backend.sync()
    got, want = out.cpu().numpy()[:n], parts.cpu().numpy()[:n]
    np.testing.assert_array_equal(got, want)
    assert np.isfinite(got).all() and np.abs(got).max() > 1e-4
