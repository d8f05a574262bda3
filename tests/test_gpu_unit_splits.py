"""GPU: K splits of the few-token integer kernel (qgemm_unit.cu) on 148 SMs: two, an uneven three, four, an uneven five and six, seven
and an equal eight parts, by the rule that prices a part's super-blocks and one for the exchange; and f32 results of nine to sixteen Q4_K
tokens."""
import numpy as np
import pytest

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, DTYPE_F32, ops

from _util import fetch, to_storage

pytestmark = pytest.mark.gpu

GEN = {2: o.gen_q4_0_weight, 12: o.gen_q4k_weight, 13: o.gen_q5k_weight, 14: o.gen_q6k_weight}
MOST = [0, 296, 148, 93, 71, 56, 45, 37, 33]


def parts(N, K):
    tiles, nsb = (N + 127) // 128, K // 256
    best, cost = 1, -(-tiles // 296) * nsb
    for ks in range(2, min(8, nsb) + 1):
        if tiles > MOST[ks]:
            break
        if -(-nsb // ks) + 1 < cost:
            best, cost = ks, -(-nsb // ks) + 1
    return best


@pytest.mark.parametrize("x_dtype", [DTYPE_BF16, DTYPE_F32])
@pytest.mark.parametrize("tag,M,N,K,ks", [
    (13, 6, 13000, 2304, 2), (13, 7, 11900, 2816, 3), (2, 5, 9000, 3328, 4), (14, 8, 7000, 3328, 5), (2, 16, 5700, 2816, 6),
    (13, 9, 4600, 3328, 7), (14, 12, 4200, 3840, 8), (2, 6, 300, 2304, 5), (12, 4, 4200, 14336, 8), (12, 11, 300, 13824, 8),
])
def test_parts(dev, x_dtype, tag, M, N, K, ks):
    assert parts(N, K) == ks
    rng = np.random.default_rng(N + K)
    blob = np.ascontiguousarray(GEN[tag](rng, N, K)).reshape(-1)
    w = np.asarray(o.dequant_q4k(blob.reshape(-1, 144)) if tag == 12 else o.dequant_gguf(blob, tag)).reshape(N, K)
    x = o.gen_activation(rng, M, K, x_dtype == DTYPE_BF16)
    d_w, d_x, d_y = dev.htod_sync_copy(blob), dev.htod_sync_copy(to_storage(x, x_dtype)), dev.alloc(M * N * 4)
    ops.qmatmul_gguf(d_y, d_x, d_w, tag, M, N, K, x_dtype=x_dtype, out_dtype=DTYPE_F32, workspace=d_y, ws_bytes=0, stream=dev.stream)
    got = fetch(dev, d_y, DTYPE_F32, (M, N)).astype(np.float64)
    assert dev.device_status() == 0
    want = x.astype(np.float64) @ w.astype(np.float64).T
    # f32 rounding of the sums alone: 1e-7 of a token's results (1.2e-7 measured at the most).  Two-piece weights have 2e-6.
    for m in range(M):
        assert np.linalg.norm(got[m] - want[m]) < 5e-7 * np.linalg.norm(want[m]), m
