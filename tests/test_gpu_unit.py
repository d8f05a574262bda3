"""GPU parity of the few-token tensor-core kernel that multiplies the weights' integers (qgemm_unit.cu): every format, the edges
of its tiles, its K splits (one to eight parts, equal or not), more tokens than a tile, f32 and bf16 activations."""
import numpy as np
import pytest

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, DTYPE_F16, DTYPE_F32, ops

from _util import ESIZE, fetch, to_storage

pytestmark = pytest.mark.gpu

GEN = {2: o.gen_q4_0_weight, 8: o.gen_q8_0_weight, 12: o.gen_q4k_weight, 13: o.gen_q5k_weight, 14: o.gen_q6k_weight}


def run(dev, tag, d_w, x, M, N, K, x_dtype, dt):
    d_x, d_y, ws = dev.htod_sync_copy(to_storage(x, x_dtype)), dev.alloc(M * N * ESIZE[dt]), dev.alloc(1 << 16)
    ops.qmatmul_gguf(d_y, d_x, d_w, tag, M, N, K, x_dtype=x_dtype, out_dtype=dt, workspace=ws, ws_bytes=1 << 16,
                     stream=dev.stream)
    got = fetch(dev, d_y, dt, (M, N))
    assert dev.device_status() == 0
    return got


def dequantised(tag, blob, N, K):
    if tag in (8, 12):
        w = (o.dequant_q8_0 if tag == 8 else o.dequant_q4k)(blob.reshape(-1, 34 if tag == 8 else 144))
    else:
        w = o.dequant_gguf(blob, tag)
    return np.asarray(w).reshape(N, K)


@pytest.mark.parametrize("x_dtype", [DTYPE_BF16, DTYPE_F32])
@pytest.mark.parametrize("tag,M,N,K", [
    # one row, one super-block; 16 tokens; a tile of one row behind a whole one
    (13, 3, 1, 256), (2, 16, 129, 256), (14, 4, 257, 256),
    # K splits: two, three (parts of 3, 4, 4), five, seven parts, eight equal ones
    (12, 5, 300, 512), (13, 7, 12000, 2816), (14, 4, 6700, 1280), (2, 2, 4500, 1792), (12, 8, 1000, 13824),
    # no split, more tiles than one round of CTAs
    (2, 4, 40000, 256),
    # Q8_0 rows that are not whole 2048 values, one token to sixteen
    (8, 1, 300, 1280), (8, 4, 129, 2304), (8, 16, 200, 5376),
    # Q6_K: row counts that are no multiple of eight, last bytes off a 16-byte piece
    (14, 8, 1027, 1280), (14, 5, 7, 2304), (14, 16, 4099, 768),
])
def test_few_tokens(dev, x_dtype, tag, M, N, K):
    rng = np.random.default_rng(tag + M + N + K)
    blob = np.ascontiguousarray(GEN[tag](rng, N, K)).reshape(-1)
    x = o.gen_activation(rng, M, K, x_dtype == DTYPE_BF16)
    x[M - 1] *= 0.03125
    want = o.qmatmul_exact(x, dequantised(tag, blob, N, K))
    d_w = dev.htod_sync_copy(blob)
    # Integers and activations are exact, sums are f32: 2^-24 of each of K / 256 partial sums and of every group's, a few 1e-7 as
    # a 2-norm; the widest K split and a cancelling row stay below 4e-6.  Then one rounding of the output.
    for dt, tol in ((DTYPE_F32, 4e-6), (DTYPE_F16, 5e-4), (DTYPE_BF16, 4e-3)):
        got = run(dev, tag, d_w, x, M, N, K, x_dtype, dt)
        if tag == 12:  # some of these are the decode kernels' (15-bit activations), or one-piece weights
            tol = max(tol, 1e-2 if M > 8 else 1e-4)
        for m in range(M):
            assert o.rel_l2(got[m], want[m]) < (tol if N >= 100 else max(tol, 4e-3)), (dt, m)
        assert np.array_equal(got, run(dev, tag, d_w, x, M, N, K, x_dtype, dt))


@pytest.mark.parametrize("x_dtype", [DTYPE_BF16, DTYPE_F32])
@pytest.mark.parametrize("tag,M,N,K", [(2, 17, 300, 768), (13, 33, 130, 2304), (14, 50, 1003, 1280), (14, 18, 129, 6144), (2, 40, 9700, 256)])
def test_f32_results_of_more_tokens(dev, x_dtype, tag, M, N, K):
    rng = np.random.default_rng(tag + M)
    blob = np.ascontiguousarray(GEN[tag](rng, N, K)).reshape(-1)
    x = o.gen_activation(rng, M, K, x_dtype == DTYPE_BF16)
    got = run(dev, tag, dev.htod_sync_copy(blob), x, M, N, K, x_dtype, DTYPE_F32)
    assert o.rel_l2(got, o.qmatmul_exact(x, dequantised(tag, blob, N, K))) < 4e-6


@pytest.mark.parametrize("x_dtype", [DTYPE_BF16, DTYPE_F32])
@pytest.mark.parametrize("tag,M,K", [(12, 6, 13824), (8, 3, 1280), (14, 4, 1280), (13, 12, 2304), (2, 1, 768)])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e34, 1e-30])
def test_extreme_activations(dev, x_dtype, tag, M, K, value):
    """One activation that is not finite: that token's results are not, the others keep their bits.  Large ones do not
    overflow before the weight's scale is applied (a row of them, of either sign), and the smallest keep their value."""
    N = 200
    rng = np.random.default_rng(tag + M)
    blob = np.ascontiguousarray(GEN[tag](rng, N, K)).reshape(-1)
    d_w = dev.htod_sync_copy(blob)
    x = o.gen_activation(rng, M, K, x_dtype == DTYPE_BF16)
    before = run(dev, tag, d_w, x, M, N, K, x_dtype, DTYPE_F32)
    if np.isfinite(value):
        v = o.bf16_bits_to_f32(o.f32_to_bf16_bits(np.float32([value])))[0] if x_dtype == DTYPE_BF16 else np.float32(value)
        x[0] = np.sign(rng.standard_normal(K)) * v
    else:
        x[0, 100] = value
    got = run(dev, tag, d_w, x, M, N, K, x_dtype, DTYPE_F32)
    assert np.array_equal(got[1:], before[1:])
    if not np.isfinite(value):
        assert not np.isfinite(got[0]).any()
        return
    want = x[0].astype(np.float64) @ dequantised(tag, blob, N, K).astype(np.float64).T
    assert np.linalg.norm((got[0].astype(np.float64) - want) / value) < 4e-6 * np.linalg.norm(want / value)
