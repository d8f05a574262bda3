"""Q4_K and Q8_0 with two to sixteen tokens where the decode kernels need a second pass or do not take the rows, and the
one-piece tensor-core launches at the edges of their ranges."""
import numpy as np
import pytest

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, DTYPE_F32, ops

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
