"""GPU: rounding of the few-token integer kernel's f32 results (qgemm_unit.cu) for rows of Q6_K, which has the most groups to sum, where
CUDA-core kernels with 6e-8 to 1e-7 took the call otherwise."""
import numpy as np
import pytest

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, DTYPE_F32, ops

from _util import fetch, to_storage

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(8, 1200, 1536), (3, 1200, 1792), (16, 1200, 2304), (6, 20000, 3328)])
def test_q6k_error_of_f32_results(dev, M, N, K):
    rng = np.random.default_rng(M + N + K)
    blob = np.ascontiguousarray(o.gen_q6k_weight(rng, N, K)).reshape(-1)
    x = o.gen_activation(rng, M, K, True)
    d_w, d_x, d_y = dev.htod_sync_copy(blob), dev.htod_sync_copy(to_storage(x, DTYPE_BF16)), dev.alloc(M * N * 4)
    ops.qmatmul_gguf(d_y, d_x, d_w, 14, M, N, K, x_dtype=DTYPE_BF16, out_dtype=DTYPE_F32, workspace=d_y, ws_bytes=0, stream=dev.stream)
    got = fetch(dev, d_y, DTYPE_F32, (M, N)).astype(np.float64)
    assert dev.device_status() == 0
    want = x.astype(np.float64) @ np.asarray(o.dequant_gguf(blob, 14)).reshape(N, K).astype(np.float64).T
    # An addition rounds a sum off by about 2.5e-8 of it (2-norm, 2^-24 over the mantissas).  Four groups, four stages and the exchange of
    # up to eight parts round as much as 2.5, 2.3 and 2 to 3 such additions, the rest is kept: 2.5e-8 * sqrt(8) = 7.1e-8.  One chain
    # of sixteen groups and one of the super-blocks: 8.5 and 3 to 7, 8.5e-8 to 1e-7.
    assert np.linalg.norm(got - want) < 8e-8 * np.linalg.norm(want)
