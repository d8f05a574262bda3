"""GPU: weights of the one-piece Q4_K matmul beside very small activations, and super-block scales on either side of where the
producer changes its form, bit by bit.  A token with a single value that is not zero picks a column of W."""
import numpy as np
import pytest

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, ops

from _util import fetch, to_storage

pytestmark = pytest.mark.gpu


def bf16(x):
    m, e = np.frexp(np.asarray(x, dtype=np.float64))
    return np.ldexp(np.rint(m * 256) / 256, e)


def columns(dev, d, value, M, N, K):
    """(what the kernel gives, what it has to give) for tokens that are `value` in one column and zero elsewhere."""
    rng = np.random.default_rng(M + N)
    nb = N * K // 256
    d = np.broadcast_to(d, (nb,)).astype(np.float16)
    sc, mn, q = rng.integers(1, 64, (nb, 8)), rng.integers(0, 64, (nb, 8)), rng.integers(0, 16, (nb, 256))
    dmin = (d.astype(np.float32) * np.float32(0.5)).astype(np.float16)
    w = o.pack_q4k(d, dmin, sc, mn, q)
    s = bf16((d.astype(np.float32)[:, None] * sc.astype(np.float32)).repeat(32, 1)).reshape(N, K)
    m = bf16((dmin.astype(np.float32)[:, None] * mn.astype(np.float32)).repeat(32, 1)).reshape(N, K)
    cols = np.arange(M) * 37 % K
    want = bf16(s * q.reshape(N, K) - m)[:, cols].T * value
    x = np.zeros((M, K), np.float32)
    x[np.arange(M), cols] = value
    ws_bytes = max(256, ops.qmatmul_workspace_bytes(M, N, K, True))
    d_y, ws = dev.alloc(M * N * 2), dev.alloc(ws_bytes)
    d_w, d_x = dev.htod_sync_copy(np.ascontiguousarray(w).reshape(-1)), dev.htod_sync_copy(to_storage(x, DTYPE_BF16))
    ops.qmatmul(d_y, d_x, d_w, M, N, K, is_q4k=True, x_dtype=DTYPE_BF16, out_dtype=DTYPE_BF16, workspace=ws, ws_bytes=ws_bytes,
                stream=dev.stream)
    got = fetch(dev, d_y, DTYPE_BF16, (M, N))
    assert dev.device_status() == 0
    return got, want


SHAPES = [(9, 130, 512), (20, 200, 512), (100, 130, 256), (130, 9600, 256)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("exponent", [-90, -114, 100])
def test_activations_of_any_size(dev, exponent, M, N, K):
    # d = 2^-10, dmin = 2^-11: weights are multiples of 2^-11, at most 2: products are normal numbers, in f32 and (nearly all) in bf16
    got, want = columns(dev, 2.0 ** -10, 2.0 ** exponent, M, N, K)
    normal = (want == 0) | (np.abs(want) >= 2.0 ** -126)
    assert normal.mean() > 0.99 and np.array_equal(got[normal], want[normal])


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_scales_on_either_side(dev, M, N, K):
    # d just below 2^-11, 2^-11 itself, and far from it, in turn: within a warp's rows, and super-block after super-block
    edge = np.float16(2.0 ** -11)
    some = [np.nextafter(edge, np.float16(0)), edge, np.float16(3e-4), -edge, np.float16(40.), np.float16(6e-8)]
    nb = N * K // 256
    for d in (np.resize(some, nb), np.where(np.arange(nb) % 97 == 5, np.float16(1000.), np.float16(1e-4))):
        got, want = columns(dev, d, 1.0, M, N, K)
        assert np.array_equal(got, want)
