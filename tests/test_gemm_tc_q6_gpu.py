"""Q6_K on the tensor-memory GEMM with every code, every 8-bit scale and both block offsets inside a 16-byte unit.

Products and block sums are exact there, so the result differs from the CPU path's by the order of at most eight f32 additions and the
rounding of each block's two products: 2e-6 relative L2."""
import numpy as np
import pytest

import fixtures as fx
import infr_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [33, 64, 65, 128, 129, 300])  # token tiles of 64 and 128 rows, one and several
@pytest.mark.parametrize("in_f,n", [(2048, 130), (4096, 384)])
def test_q6_every_code_and_scale(backend, oracle, m, in_f, n):
    rng = np.random.default_rng(m + in_f)
    w = rng.integers(0, 256, (n * in_f // 256, 210), dtype=np.uint8)
    w[:, 208:] = (rng.choice([-1.0, 1.0], len(w)) * rng.uniform(0.5, 1.0, len(w)) / 4096).astype(np.float16).view(np.uint8).reshape(-1, 2)
    w[:16, 192:208] = np.arange(256, dtype=np.uint8).reshape(16, 16)
    x = rng.standard_normal((m, in_f)).astype(np.float32)
    x[0, :] = np.abs(x[0, :])
    xb, wb, y = backend.from_numpy(x), backend.from_numpy(w.reshape(-1)), backend.alloc(m * n * 4)
    backend.linear(infr_b200.Q6K, wb, xb, y, m, in_f, n)
    want = oracle.linear(infr_b200.Q6K, w.reshape(-1), x, m, in_f, n)
    assert fx.rel_l2(backend.download(y, np.float32).reshape(m, n), want) < 2e-6
