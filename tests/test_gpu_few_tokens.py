"""Q4_K and Q8_0 with two to sixteen tokens where the decode kernels need a second pass or do not take the rows, and the
one-piece tensor-core launches at the edges of their ranges."""
import numpy as np
import pytest

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, DTYPE_F16, DTYPE_F32, ops

from _util import ESIZE, fetch, to_storage

pytestmark = pytest.mark.gpu


def _run(dev, w, x, M, N, K, is_q4k, x_dtype, out_dtype):
    ws_bytes = ops.qmatmul_workspace_bytes(M, N, K, is_q4k)
    d_y = dev.alloc(M * N * ESIZE[out_dtype])
    ops.qmatmul(d_y, dev.htod_sync_copy(to_storage(x, x_dtype)), dev.htod_sync_copy(w), M, N, K, is_q4k=is_q4k,
                x_dtype=x_dtype, out_dtype=out_dtype, workspace=dev.alloc(max(ws_bytes, 256)), ws_bytes=ws_bytes,
                stream=dev.stream)
    assert dev.device_status() == 0
    return fetch(dev, d_y, out_dtype, (M, N))


@pytest.mark.parametrize("x_dtype", [DTYPE_BF16, DTYPE_F32])
@pytest.mark.parametrize("is_q4k,M,N,K", [
    (True, 3, 200, 14336), (True, 8, 130, 13824), (True, 5, 300, 1280), (True, 16, 129, 4096), (True, 9, 2100, 256),
    (True, 4, 300, 8960), (True, 4, 300, 9216),  # the longest rows of token pairs in one pass, and the next ones
    (False, 2, 300, 1280), (False, 16, 200, 2304), (False, 16, 300, 4096), (False, 9, 129, 6144), (False, 5, 129, 14336),
])
def test_two_to_sixteen_tokens(dev, x_dtype, is_q4k, M, N, K):
    rng = np.random.default_rng(M + N + K)
    w = (o.gen_q4k_weight if is_q4k else o.gen_q8_0_weight)(rng, N, K)
    x = o.gen_activation(rng, M, K, x_dtype == DTYPE_BF16)
    want = o.c_qmatmul(x, w, N, K, is_q4k)
    # 15-bit activations or two-piece weights: below 1e-4; bf16 results are rounded once, from nine Q4_K tokens in bf16 on
    # the weights as well
    assert o.rel_l2(_run(dev, w, x, M, N, K, is_q4k, x_dtype, DTYPE_F32), want) < 1e-4
    assert o.rel_l2(_run(dev, w, x, M, N, K, is_q4k, x_dtype, DTYPE_BF16), want) < (1e-2 if M > 8 else 4e-3)


@pytest.mark.parametrize("is_q4k,M,N,K", [
    (True, 9, 1, 256), (True, 17, 4300, 2304), (True, 64, 130, 4352), (True, 65, 300, 1280), (True, 128, 9600, 512),
    (True, 129, 1000, 768), (True, 200, 4100, 2304), (True, 384, 5000, 512), (True, 385, 5000, 512), (True, 300, 9600, 256),
    (False, 17, 129, 256), (False, 64, 4300, 1280), (False, 65, 300, 768), (False, 129, 200, 1280),
])
def test_one_piece_launches(dev, is_q4k, M, N, K):
    """K splits of parts of unequal length, one row, ragged tiles, the last and the first token count of each tile size, and
    the line between one round of 128-token tiles (148 of them) and tiles of 256 tokens."""
    rng = np.random.default_rng(M + N + K)
    w = (o.gen_q4k_weight if is_q4k else o.gen_q8_0_weight)(rng, N, K)
    x = o.gen_activation(rng, M, K, True)
    got = _run(dev, w, x, M, N, K, is_q4k, DTYPE_BF16, DTYPE_BF16)
    # weights and results rounded to bf16 (2^-9 each at most); a single row may be a small difference of large terms
    assert o.rel_l2(got, o.c_qmatmul(x, w, N, K, is_q4k)) < (1e-2 if N > 1 else 3e-2)
    assert np.array_equal(got, _run(dev, w, x, M, N, K, is_q4k, DTYPE_BF16, DTYPE_BF16))


@pytest.mark.parametrize("x_dtype", [DTYPE_BF16, DTYPE_F32])
@pytest.mark.parametrize("tag,M,N,K", [
    (o.GGML_Q6_K, 4, 2048, 512), (o.GGML_Q6_K, 4, 1024, 2304), (o.GGML_Q5_K, 1, 2048, 1024), (o.GGML_Q5_K, 2, 1024, 1280),
    (o.GGML_Q4_0, 1, 2048, 1280), (o.GGML_Q4_0, 4, 1024, 512), (8, 2, 2048, 512), (8, 4, 2048, 512),
])
def test_small_matrices_stay_with_the_decode_kernels(dev, x_dtype, tag, M, N, K):
    """A pass of these takes half the time of a tensor-core launch.  Their f32 results are always the decode kernels', so the
    f16 results of the same kernel are those rounded, bit for bit; two-piece weights differ in some of 4000."""
    gen = {o.GGML_Q4_0: o.gen_q4_0_weight, o.GGML_Q5_K: o.gen_q5k_weight, o.GGML_Q6_K: o.gen_q6k_weight, 8: o.gen_q8_0_weight}
    rng = np.random.default_rng(tag + M + N + K)
    d_w = dev.htod_sync_copy(np.ascontiguousarray(gen[tag](rng, N, K)).reshape(-1))
    d_x = dev.htod_sync_copy(to_storage(o.gen_activation(rng, M, K, x_dtype == DTYPE_BF16) * 0.01, x_dtype))
    y = {}
    for dt in (DTYPE_F32, DTYPE_F16):
        d_y = dev.alloc(M * N * 4)
        ops.qmatmul_gguf(d_y, d_x, d_w, tag, M, N, K, x_dtype=x_dtype, out_dtype=dt, stream=dev.stream)
        y[dt] = fetch(dev, d_y, dt, (M, N))
    assert np.array_equal(y[DTYPE_F16], y[DTYPE_F32].astype(np.float16).astype(np.float32))


@pytest.mark.parametrize("is_q4k,M,N,K,x_dtype", [(True, 9, 6144, 4096, DTYPE_F32), (True, 10, 6144, 4096, DTYPE_BF16),
                                                  (False, 9, 12288, 4096, DTYPE_BF16), (True, 9, 1024, 1792, DTYPE_F32)])
def test_a_second_pass_where_it_is_the_faster_way(dev, is_q4k, M, N, K, x_dtype):
    """Eight tokens and the rest through the decode kernels: the bits of two calls."""
    rng = np.random.default_rng(M + N + K)
    w = (o.gen_q4k_weight if is_q4k else o.gen_q8_0_weight)(rng, N, K)
    x = o.gen_activation(rng, M, K, x_dtype == DTYPE_BF16)
    got = _run(dev, w, x, M, N, K, is_q4k, x_dtype, DTYPE_F32)
    assert np.array_equal(got[:8], _run(dev, w, x[:8], 8, N, K, is_q4k, x_dtype, DTYPE_F32))
    assert np.array_equal(got[8:], _run(dev, w, x[8:], M - 8, N, K, is_q4k, x_dtype, DTYPE_F32))
