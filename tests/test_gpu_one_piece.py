"""GPU: weights of the one-piece tensor-core matmul, bit by bit.  A token with a single one picks a column of W, so what comes
out is the bf16 weight itself; the super-block scales run over the whole range of f16."""
import numpy as np
import pytest

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, ops

from _util import fetch, to_storage

pytestmark = pytest.mark.gpu


def bf16(x):
    """To the nearest bf16, once (by way of f32 it would be twice)."""
    m, e = np.frexp(np.asarray(x, dtype=np.float64))
    return np.ldexp(np.rint(m * 256) / 256, e)


@pytest.mark.parametrize("d,dmin", [(6e-8, 6e-8), (6.1e-5, 0.), (1e-4, 7e-4), (0.5, 3.0), (65504., 65504.), (-65504., 1.), (0., 0.)])
@pytest.mark.parametrize("M,N,K", [(20, 200, 512), (100, 130, 256), (130, 9600, 256)])
def test_q4k_weights(dev, d, dmin, M, N, K):
    rng = np.random.default_rng(M)
    nb = N * K // 256
    sc, mn = rng.integers(0, 64, (nb, 8)), rng.integers(0, 64, (nb, 8))
    sc[0], mn[0] = 63, 63
    sc[1], mn[1] = 0, 0
    q = rng.integers(0, 16, (nb, 256))
    w = o.pack_q4k(np.full(nb, d, np.float16), np.full(nb, dmin, np.float16), sc, mn, q)
    s = bf16((np.float32(np.float16(d)) * sc.astype(np.float32)).repeat(32, 1)).reshape(N, K)
    m = bf16((np.float32(np.float16(dmin)) * mn.astype(np.float32)).repeat(32, 1)).reshape(N, K)
    want = bf16(s * q.reshape(N, K) - m)
    check(dev, w, True, want, M, N, K, 0)


@pytest.mark.parametrize("d", [6e-8, 1e-4, 0.1, 65504., -65504., 0.])
@pytest.mark.parametrize("M,N,K", [(20, 200, 512), (100, 130, 256), (130, 300, 256)])
def test_q8_0_weights(dev, d, M, N, K):
    rng = np.random.default_rng(M)
    q = rng.integers(-128, 128, (N * K // 32, 32)).astype(np.int8)
    q[0, :4] = -128, -127, 0, 127
    w = o.pack_q8_0(np.full(len(q), d, np.float16), q)
    # the scale is two bf16 pieces (within 2^-17): a product may round to the neighbour
    check(dev, w, False, bf16(np.float64(np.float16(d)) * q.reshape(N, K)), M, N, K, 2.0 ** -8)


def check(dev, w, is_q4k, want, M, N, K, tol):
    cols = np.arange(M) * 37 % K
    x = np.zeros((M, K), np.float32)
    x[np.arange(M), cols] = 1.
    d_y, ws = dev.alloc(M * N * 2), dev.alloc(max(256, ops.qmatmul_workspace_bytes(M, N, K, is_q4k)))
    d_w, d_x = dev.htod_sync_copy(np.ascontiguousarray(w).reshape(-1)), dev.htod_sync_copy(to_storage(x, DTYPE_BF16))
    ops.qmatmul(d_y, d_x, d_w, M, N, K, is_q4k=is_q4k, x_dtype=DTYPE_BF16, out_dtype=DTYPE_BF16, workspace=ws,
                ws_bytes=max(256, ops.qmatmul_workspace_bytes(M, N, K, is_q4k)), stream=dev.stream)
    got = fetch(dev, d_y, DTYPE_BF16, (M, N))
    assert dev.device_status() == 0
    ref = want[:, cols].T
    assert np.all(np.abs(got - ref) <= tol * np.abs(ref))
