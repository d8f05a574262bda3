"""GPU: precision of f32 results of five to sixteen Q4_K tokens in sizes where the decode kernels (activations of 15 bits, 2.7e-5) need a
second pass or a plan per super-block: the kernels of more pieces have them."""
import numpy as np
import pytest

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, DTYPE_F32, ops

from _util import fetch, to_storage

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x_dtype,M,N,K", [
    (DTYPE_BF16, 6, 1200, 256), (DTYPE_BF16, 8, 1200, 256),
    (DTYPE_F32, 12, 1200, 768), (DTYPE_F32, 12, 1200, 2816), (DTYPE_F32, 8, 1200, 4352), (DTYPE_F32, 12, 14336, 1280),
    (DTYPE_F32, 16, 512, 8192),
])
def test_f32_results(dev, x_dtype, M, N, K):
    rng = np.random.default_rng(M + N + K)
    w = o.gen_q4k_weight(rng, N, K)
    x = o.gen_activation(rng, M, K, x_dtype == DTYPE_BF16)
    d_w, d_x, d_y = dev.htod_sync_copy(w), dev.htod_sync_copy(to_storage(x, x_dtype)), dev.alloc(M * N * 4)
    ops.qmatmul(d_y, d_x, d_w, M, N, K, is_q4k=True, x_dtype=x_dtype, out_dtype=DTYPE_F32, workspace=d_y, ws_bytes=0, stream=dev.stream)
    got = fetch(dev, d_y, DTYPE_F32, (M, N)).astype(np.float64)
    assert dev.device_status() == 0
    want = x.astype(np.float64) @ np.asarray(o.dequant_q4k(w.reshape(-1, 144))).reshape(N, K).astype(np.float64).T
    # two pieces of a weight are within 2^-18 of it and an f32 activation's two within 2^-16: 1.5e-5 at the most, 8e-6 as a 2-norm
    assert np.linalg.norm(got - want) < 1.2e-5 * np.linalg.norm(want)
