"""GPU parity of the tensor-core matmul with two-piece weights (qgemm_tc2.cu): every format it takes, f32 and bf16
activations, the edges of its tiles, the K splits and the last bytes of an unaligned matrix."""
import numpy as np
import pytest

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, DTYPE_F16, DTYPE_F32, ops

from _util import ESIZE, fetch, to_storage

pytestmark = pytest.mark.gpu

GEN = {o.GGML_Q4_0: o.gen_q4_0_weight, o.GGML_Q5_K: o.gen_q5k_weight, o.GGML_Q6_K: o.gen_q6k_weight}


@pytest.mark.parametrize("tag", sorted(GEN))
@pytest.mark.parametrize("x_dtype", [DTYPE_BF16, DTYPE_F32])
@pytest.mark.parametrize("M,N,K", [
    (1, 1, 256),        # smallest: one row, one super-block, no K split
    (5, 129, 2048),     # a second weight tile of one row, split in eight... as far as the super-blocks go
    (9, 300, 4352),     # 17 super-blocks over eight ranks: parts of unequal length, last bytes off a 16-byte piece
    (16, 2049, 1280),   # 17 tiles: split in four
    (33, 4300, 768),    # 34 tiles: split in two (three super-blocks: not split at all)
    (64, 4300, 2304),   # the same, nine super-blocks: parts of four and five; the largest tile of 64 tokens
    (65, 9600, 512),    # 75 tiles: no split
    (100, 19100, 512),  # 150 tiles: more than one round of the persistent grid
    (128, 200, 4096), (129, 200, 3072), (256, 130, 1024), (257, 1000, 2048), (333, 500, 4096),
])
def test_two_piece_weights(dev, tag, x_dtype, M, N, K):
    rng = np.random.default_rng(tag + M + N + K)
    blob = np.ascontiguousarray(GEN[tag](rng, N, K)).reshape(-1)
    x = o.gen_activation(rng, M, K, x_dtype == DTYPE_BF16)
    x[M - 1] *= 0.03125
    want = o.qmatmul_exact(x, o.dequant_gguf(blob, tag).reshape(N, K))
    d_w, d_x = dev.htod_sync_copy(blob), dev.htod_sync_copy(to_storage(x, x_dtype))

    def run(dt):
        d_y = dev.alloc(M * N * ESIZE[dt])
        ops.qmatmul_gguf(d_y, d_x, d_w, tag, M, N, K, x_dtype=x_dtype, out_dtype=dt, stream=dev.stream)
        return fetch(dev, d_y, dt, (M, N))

    # Weights are within 2^-18 and f32 activations within 2^-17 of their values, the dropped product below 2^-17: 2e-5 of
    # a term in the worst case, a few 1e-6 as a 2-norm, next to one rounding of the output (f16: 2^-11, bf16: 2^-8).  One
    # output of a token may be a small difference of large terms.  f32 results of most row lengths are not made here.
    for dt, tol in ((DTYPE_F32, 2e-5), (DTYPE_F16, 5e-4), (DTYPE_BF16, 4e-3)):
        got = run(dt)
        assert dev.device_status() == 0
        for m in range(M):
            assert o.rel_l2(got[m], want[m]) < (tol if N >= 100 else max(tol, 4e-3)), (dt, m)
        assert np.array_equal(got, run(dt))  # the parts of a K split are added in a fixed order


def test_half_the_rows_take_no_longer(dev):
    """Every cluster of a K split is on the GPU at once: 2048 rows (sixteen tiles) in one round, as 4096 rows are."""
    import torch

    stream = torch.cuda.ExternalStream(int(getattr(dev.stream, "value", dev.stream)))
    M, K = 8, 4096
    us = {}
    for N in (2048, 4096):
        blob = dev.htod_sync_copy(o.gen_q6k_weight(np.random.default_rng(N), N, K).reshape(-1))
        d_x, d_y = dev.htod_sync_copy(np.zeros((M, K), dtype=np.uint16)), dev.alloc(M * N * 2)
        best = 1e9
        for rep in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            with torch.cuda.stream(stream):
                torch.cuda._sleep(500000)  # the calls below are queued before the first one runs
                a.record(stream)
            for _ in range(20):
                ops.qmatmul_gguf(d_y, d_x, blob, o.GGML_Q6_K, M, N, K, x_dtype=DTYPE_BF16, out_dtype=DTYPE_BF16,
                                 stream=dev.stream)
            b.record(stream)
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 50)
        us[N] = best
    assert us[2048] < 1.1 * us[4096], us


@pytest.mark.parametrize("x_dtype", [DTYPE_BF16, DTYPE_F32])
@pytest.mark.parametrize("tag,M,K", [(o.GGML_Q6_K, 9, 2048), (o.GGML_Q5_K, 70, 768), (12, 6, 5120), (12, 40, 2048), (8, 33, 1280)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_token_that_is_not_finite(dev, x_dtype, tag, M, K, bad):
    """Two pieces and one: that token's results are not finite (an infinity may become NaN: products with the second piece),
    the others keep their bits."""
    N = 200
    gen = dict(GEN)
    gen[12], gen[8] = o.gen_q4k_weight, o.gen_q8_0_weight
    rng = np.random.default_rng(tag + M)
    d_w = dev.htod_sync_copy(np.ascontiguousarray(gen[tag](rng, N, K)).reshape(-1))
    x = o.gen_activation(rng, M, K, x_dtype == DTYPE_BF16)
    y = []
    for value in (x[2, 100], bad):
        x[2, 100] = value
        ws, d_y = dev.alloc(1 << 20), dev.alloc(M * N * 4)
        ops.qmatmul_gguf(d_y, dev.htod_sync_copy(to_storage(x, x_dtype)), d_w, tag, M, N, K, x_dtype=x_dtype,
                         out_dtype=DTYPE_BF16, workspace=ws, ws_bytes=1 << 20, stream=dev.stream)
        y.append(fetch(dev, d_y, DTYPE_BF16, (M, N)))
    others = [m for m in range(M) if m != 2]
    assert np.isfinite(y[0]).all() and not np.isfinite(y[1][2]).any()
    assert np.array_equal(y[0][others], y[1][others])
