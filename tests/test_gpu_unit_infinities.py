"""GPU: infinite activations in calls of the few-token integer kernel (qgemm_unit.cu).  The result is that of the plain sum: an infinity with
the weight's sign, NaN where that weight is zero or two infinities meet with opposite signs."""
import numpy as np
import pytest

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, DTYPE_F32, ops

from _util import fetch, to_storage

pytestmark = pytest.mark.gpu

GEN = {2: o.gen_q4_0_weight, 8: o.gen_q8_0_weight, 12: o.gen_q4k_weight, 13: o.gen_q5k_weight, 14: o.gen_q6k_weight}


@pytest.mark.parametrize("x_dtype", [DTYPE_BF16, DTYPE_F32])
@pytest.mark.parametrize("tag,M,N,K", [
    (2, 1, 200, 768), (8, 3, 200, 1280), (12, 6, 200, 13824), (13, 12, 200, 2304), (14, 4, 200, 1280),  # parts of K
    (2, 5, 20000, 256), (13, 20, 20000, 256), (14, 16, 20003, 768),  # whole rows
])
def test_infinities(dev, x_dtype, tag, M, N, K):
    rng = np.random.default_rng(tag + M + N)
    blob = np.ascontiguousarray(GEN[tag](rng, N, K)).reshape(-1)
    if tag in (8, 12):
        w = (o.dequant_q8_0 if tag == 8 else o.dequant_q4k)(blob.reshape(-1, 34 if tag == 8 else 144))
    else:
        w = o.dequant_gguf(blob, tag)
    w = np.asarray(w, np.float32).reshape(N, K)
    x = o.gen_activation(rng, M, K, x_dtype == DTYPE_BF16)
    kinds = [[(100, np.inf)], [(7, -np.inf), (K - 1, np.inf)], [(33, np.inf), (40, np.nan)], [(k, np.inf) for k in range(K)]]
    want = x.astype(np.float64) @ w.T.astype(np.float64)
    for m, places in zip(range(M), kinds):
        with np.errstate(invalid="ignore"):
            want[m] = sum(np.float32(v) * w[:, k] for k, v in places)
        for k, v in places:
            x[m, k] = v
    d_w, d_x, d_y = dev.htod_sync_copy(blob), dev.htod_sync_copy(to_storage(x, x_dtype)), dev.alloc(M * N * 4)
    ops.qmatmul_gguf(d_y, d_x, d_w, tag, M, N, K, x_dtype=x_dtype, out_dtype=DTYPE_F32, workspace=d_y, ws_bytes=0, stream=dev.stream)
    got = fetch(dev, d_y, DTYPE_F32, (M, N))
    assert dev.device_status() == 0
    odd = min(M, len(kinds))
    assert np.array_equal(got[:odd], want[:odd].astype(np.float32), equal_nan=True)
    for m in range(odd, M):
        assert o.rel_l2(got[m], want[m]) < 4e-6
