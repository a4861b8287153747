"""Grouped expert launches whose CTAs share all items' tiles evenly: a CTA goes on from one item to the next, stages its rows anew, and (Q6_K) the
tiles of the next item are on their way while the last ones of this item are multiplied.

A row's result depends on that row alone, so the bits are those of calls of three rows, which have a whole number of CTAs an item and are held
against the CPU path by the other expert-bank tests."""
import numpy as np
import pytest

import infr_b200
from infr_b200 import Q4K, Q6K

pytestmark = pytest.mark.gpu


def _bank(torch, dt, n, seed):
    elems, size = 256, 144 if dt == Q4K else 210
    g = torch.Generator(device="cuda").manual_seed(seed)
    raw = torch.randint(0, 256, (n // elems, size), dtype=torch.uint8, device="cuda", generator=g)
    d = (torch.rand(n // elems, 1, device="cuda", generator=g) + 0.5).half()
    if dt == Q4K:
        raw[:, 0:2] = (d * 1e-4).view(torch.uint8)
        raw[:, 2:4] = (d * 7e-4).view(torch.uint8)
    else:
        raw[:, 208:210] = (d * 2e-5).view(torch.uint8)
    return raw


@pytest.mark.parametrize("rows,ne,n_expert,n_used,nff,down_dt", [
    (27, 2048, 128, 8, 768, Q6K),   # 0.35 items a place, ten slots for eight warps
    (100, 2048, 128, 8, 768, Q4K),  # both banks of Q4_K
    (150, 2048, 128, 8, 256, Q4K),  # items of few tiles: several of them a CTA
    (64, 1024, 64, 8, 2048, Q6K),   # one CTA an SM
    (33, 1024, 64, 4, 1280, Q6K),   # rows of five blocks
])
def test_shares_have_the_bits_of_small_calls(backend, rows, ne, n_expert, n_used, nff, down_dt):
    import torch

    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(rows, ne, device="cuda", generator=g)
    router = torch.randn(n_expert, ne, device="cuda", generator=g) / ne**0.5
    banks = [_bank(torch, dt, n_expert * nff * ne, 4 + i) for i, dt in enumerate((Q4K, Q4K, down_dt))]
    out, parts = torch.zeros(rows, ne, device="cuda"), torch.ones(rows, ne, device="cuda")
    torch.cuda.synchronize()
    wrap = lambda t: backend.wrap(t.data_ptr(), t.numel() * t.element_size(), infr_b200.USAGE_ACTIVATIONS)
    weights = [wrap(t) for t in (router, *banks)]

    def call(dst, r0, n):
        rows_in = wrap(x[r0:r0 + n])
        backend.moe_ffn(rows_in, rows_in, *weights, wrap(dst[r0:r0 + n]), rows=n, ne=ne, n_expert=n_expert, n_used=n_used, n_ff_exp=nff, wdt=Q4K, down_dt=down_dt)

    call(out, 0, rows)
    n = rows - (rows % 3 == 1)  # (a single row takes the f32 path)
    for r0 in range(0, n, 3):
        call(parts, r0, min(3, n - r0))
    backend.sync()
    got, want = out.cpu().numpy()[:n], parts.cpu().numpy()[:n]
    np.testing.assert_array_equal(got, want)
    assert np.isfinite(got).all() and np.abs(got).max() > 1e-4
