"""The row-wise kernels between the matmuls with 16-byte accesses: RMSNorm, SiLU.up, strided copy."""
import numpy as np
import pytest

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, DTYPE_F16, DTYPE_F32, ops
from ubridge_b200._lib import UB_QMATMUL_WEIGHTS_FRESH, check, lib

from _util import ESIZE, fetch, to_storage

pytestmark = pytest.mark.gpu
ODT = {DTYPE_F32: o.UB_F32, DTYPE_F16: o.UB_F16, DTYPE_BF16: o.UB_BF16}


@pytest.mark.parametrize("dtype", sorted(ODT))
# one piece; less and more than a round of the CTA; the registers' capacity and beyond; rows that are not whole pieces
@pytest.mark.parametrize("T,H", [(1, 8), (3, 2040), (5, 2056), (2, 8192), (3, 8200), (1, 20000), (4, 1001)])
@pytest.mark.parametrize("in_place", [False, True])
def test_rms_norm_rows(dev, dtype, T, H, in_place):
    rng = np.random.default_rng(T + H)
    x = o.round_through(rng.standard_normal((T, H)).astype(np.float32) * 3, ODT[dtype])
    g = o.round_through(rng.uniform(0.5, 1.5, size=H).astype(np.float32), ODT[dtype])
    d_x = dev.htod_sync_copy(to_storage(x, dtype))
    d_out = d_x if in_place else dev.alloc(T * H * ESIZE[dtype])
    ops.rms_norm(d_out, d_x, dev.htod_sync_copy(to_storage(g, dtype)), T, H, 1e-5, dtype, stream=dev.stream)
    # f32 vs f64 mean and rsqrt: a value on a rounding boundary may fall the other way, by one unit of the type
    assert o.rel_l2(fetch(dev, d_out, dtype, (T, H)), o.rms_norm(x, g, 1e-5, ODT[dtype])) < {
        DTYPE_F32: 1e-6, DTYPE_F16: 1e-3, DTYPE_BF16: 4e-3}[dtype]


@pytest.mark.parametrize("dtype", sorted(ODT))
@pytest.mark.parametrize("rows,D", [(1, 8), (33, 72), (3, 2056), (2, 14336), (5, 77), (40000, 8)])
def test_silu_and_mul_rows(dev, dtype, rows, D):
    rng = np.random.default_rng(rows + D)
    x = o.round_through(rng.standard_normal((rows, 2 * D)).astype(np.float32) * 4, ODT[dtype])
    d_o = dev.alloc(rows * D * ESIZE[dtype])
    ops.silu_and_mul(d_o, dev.htod_sync_copy(to_storage(x, dtype)), rows, D, dtype, stream=dev.stream)
    got, want = fetch(dev, d_o, dtype, (rows, D)), o.silu_and_mul(x, ODT[dtype])
    # expf differs by an ulp between libm and CUDA: one unit of the type on a rounding boundary
    assert np.allclose(got, want, rtol={DTYPE_F32: 2 ** -21, DTYPE_F16: 2 ** -10, DTYPE_BF16: 2 ** -7}[dtype], atol=1e-7)


@pytest.mark.parametrize("rows,width,src_pitch,dst_pitch", [(1, 16, 16, 16), (3, 8192, 12288, 8192), (40000, 32, 48, 64),
                                                            (7, 30, 64, 32), (2, 64, 66, 64)])
def test_copy_rows(dev, rows, width, src_pitch, dst_pitch):
    rng = np.random.default_rng(rows + width)
    src = rng.integers(0, 256, (rows, src_pitch), dtype=np.uint8)
    dst = rng.integers(0, 256, (rows, dst_pitch), dtype=np.uint8)
    d_s, d_d = dev.htod_sync_copy(src), dev.htod_sync_copy(dst)
    check(lib().ub_copy_rows(d_d.ptr, dst_pitch, d_s.ptr, src_pitch, width, rows, dev.stream), "copy_rows")
    dst[:, :width] = src[:, :width]
    assert np.array_equal(dev.dtoh_sync_copy(d_d, np.uint8, (rows, dst_pitch)), dst)


@pytest.mark.parametrize("M,N,K", [(1, 4096, 4096), (1, 4096, 5120), (3, 2048, 14336), (16, 4096, 2048)])
@pytest.mark.parametrize("flag", [0, UB_QMATMUL_WEIGHTS_FRESH])
@pytest.mark.parametrize("between", [False, True])
def test_copied_weights_are_complete(dev, M, N, K, flag, between):
    """Weight rows cut out of a wider matrix by ub_copy_rows, and the matmul that reads them behind it on the stream, directly
    or behind another matmul, with nothing else in between: it must not request them ahead of the copy."""
    rng = np.random.default_rng(M + N + K)
    w = o.gen_q4k_weight(rng, N, K)
    x = o.gen_activation(rng, M, K, True)
    width = K // 256 * 144
    wide = np.zeros((N, 3 * width), dtype=np.uint8)
    wide[:, width:2 * width] = w.reshape(N, width)
    d_wide, d_x, d_y = dev.htod_sync_copy(wide), dev.htod_sync_copy(to_storage(x, DTYPE_BF16)), dev.alloc(M * N * 4)
    d_w = [dev.htod_sync_copy(w), dev.alloc(w.size)]
    d_other = dev.htod_sync_copy(o.gen_q4k_weight(rng, 64, K))
    d_other_y = dev.alloc(M * 64 * 4)

    def matmul(y, w_, n, f=0):
        ops.qmatmul(y, d_x, w_, M, n, K, is_q4k=True, x_dtype=DTYPE_BF16, out_dtype=DTYPE_F32 | f, stream=dev.stream)

    matmul(d_y, d_w[0], N)
    want = fetch(dev, d_y, DTYPE_F32, (M, N))
    assert o.rel_l2(want, o.c_qmatmul(x, w, N, K, True)) < 1e-4
    for rep in range(5):
        d_w[1] = dev.alloc_zeros(w.size)  # stale bytes cannot pass
        dev.synchronize()
        check(lib().ub_copy_rows(d_w[1].ptr, width, d_wide.ptr + width, 3 * width, width, N, dev.stream), "copy_rows")
        if between:
            matmul(d_other_y, d_other, 64)
        matmul(d_y, d_w[1], N, flag)
        assert np.array_equal(fetch(dev, d_y, DTYPE_F32, (M, N)), want)


@pytest.mark.parametrize("dtype", sorted(ODT))
@pytest.mark.parametrize("H", [8, 128, 256, 264, 512, 520, 1024, 2040, 2048, 2056, 3072, 3080])
def test_a_row_is_normalised_alike_whatever_comes_with_it(dev, dtype, H):
    """Rows that a warp takes where there are many, a CTA where there are few; in place as well."""
    T, few = 3001, 5
    rng = np.random.default_rng(H)
    x = o.round_through(rng.standard_normal((T, H)).astype(np.float32) * 3, ODT[dtype])
    d_g = dev.htod_sync_copy(to_storage(o.round_through(rng.uniform(0.5, 1.5, size=H).astype(np.float32), ODT[dtype]), dtype))
    d_x, d_out, d_few = dev.htod_sync_copy(to_storage(x, dtype)), dev.alloc(T * H * 4), dev.alloc(few * H * 4)
    ops.rms_norm(d_few, d_x, d_g, few, H, 1e-5, dtype, stream=dev.stream)
    ops.rms_norm(d_out, d_x, d_g, T, H, 1e-5, dtype, stream=dev.stream)
    got = fetch(dev, d_out, dtype, (T, H))
    assert np.array_equal(got[:few], fetch(dev, d_few, dtype, (few, H)))
    g = fetch(dev, d_g, dtype, (H,))
    assert o.rel_l2(got, o.rms_norm(x, g, 1e-5, ODT[dtype])) < {DTYPE_F32: 1e-6, DTYPE_F16: 1e-3, DTYPE_BF16: 4e-3}[dtype]
    ops.rms_norm(d_x, d_x, d_g, T, H, 1e-5, dtype, stream=dev.stream)
    assert np.array_equal(fetch(dev, d_x, dtype, (T, H)), got)


@pytest.mark.parametrize("pieces", [1, 2, 3, 31, 32, 33, 128, 129, 256, 257])
@pytest.mark.parametrize("rows", [1, 7, 300, 70001])
def test_rows_of_any_number_of_pieces(dev, pieces, rows):
    """Several rows in a CTA, the last of them missing; more rows than the grid is high.  Copy and SiLU.up."""
    if rows * pieces > 300_000:
        rows = 1500
    rng = np.random.default_rng(pieces + rows)
    src = rng.integers(0, 256, (rows, pieces + 1, 16), dtype=np.uint8)
    d_s, d_d = dev.htod_sync_copy(src), dev.alloc(rows * pieces * 16)
    check(lib().ub_copy_rows(d_d.ptr, pieces * 16, d_s.ptr, (pieces + 1) * 16, pieces * 16, rows, dev.stream), "copy_rows")
    assert np.array_equal(dev.dtoh_sync_copy(d_d, np.uint8, (rows, pieces, 16)), src[:, :pieces])
    D = pieces * 8
    x = o.round_through(rng.standard_normal((rows, 2 * D)).astype(np.float32), o.UB_BF16)
    d_o = dev.alloc(rows * D * 2)
    ops.silu_and_mul(d_o, dev.htod_sync_copy(to_storage(x, DTYPE_BF16)), rows, D, DTYPE_BF16, stream=dev.stream)
    assert np.allclose(fetch(dev, d_o, DTYPE_BF16, (rows, D)), o.silu_and_mul(x, o.UB_BF16), rtol=2 ** -7, atol=1e-7)


@pytest.mark.parametrize("tag,M", [(o.GGML_Q6_K, 6), (o.GGML_Q5_K, 9), (o.GGML_Q4_0, 40), (8, 12)])
def test_copied_weights_of_other_formats_are_complete(dev, tag, M):
    """The same for the tensor-core launches of the other formats, which request weights early for rows of whole 2048 values."""
    N, K = 2048, 4096
    gen = {o.GGML_Q4_0: o.gen_q4_0_weight, o.GGML_Q5_K: o.gen_q5k_weight, o.GGML_Q6_K: o.gen_q6k_weight, 8: o.gen_q8_0_weight}
    rng = np.random.default_rng(tag + M)
    w = np.ascontiguousarray(gen[tag](rng, N, K)).reshape(8, -1)  # eight pieces of whole 16 bytes
    wide = np.zeros((8, w.shape[1] + 64), dtype=np.uint8)
    wide[:, 32:-32] = w
    d_wide, d_w = dev.htod_sync_copy(wide), dev.htod_sync_copy(w)
    d_x, d_y = dev.htod_sync_copy(to_storage(o.gen_activation(rng, M, K, True), DTYPE_BF16)), dev.alloc(M * N * 2)

    def matmul():
        ops.qmatmul_gguf(d_y, d_x, d_w, tag, M, N, K, x_dtype=DTYPE_BF16, out_dtype=DTYPE_BF16, stream=dev.stream)

    matmul()
    want = fetch(dev, d_y, DTYPE_BF16, (M, N))
    for rep in range(3):
        d_w = dev.alloc_zeros(w.size)
        dev.synchronize()
        check(lib().ub_copy_rows(d_w.ptr, w.shape[1], d_wide.ptr + 32, wide.shape[1], w.shape[1], 8, dev.stream), "copy_rows")
        matmul()
        assert np.array_equal(fetch(dev, d_y, DTYPE_BF16, (M, N)), want)


@pytest.mark.parametrize("M", [1, 4, 20])
def test_a_chain_gives_the_same_with_and_without_waiting(dev, M):
    """Norm, matmul, copy, matmul, SiLU.up, matmul into the same buffers over and over: every launch overlaps its neighbours,
    the result is that of the chain with a wait behind every call."""
    rng = np.random.default_rng(M)
    H, I = 1024, 1280
    w1, w2, w3 = (dev.htod_sync_copy(o.gen_q4k_weight(rng, n, k)) for n, k in ((H + 512, H), (2 * I, H), (H, I)))
    d_g = dev.htod_sync_copy(to_storage(np.full(H, 0.01, dtype=np.float32), DTYPE_BF16))
    x = to_storage(o.gen_activation(rng, M, H, True), DTYPE_BF16)
    bufs = [dev.alloc(M * n * 2) for n in (H, H + 512, H, 2 * I, I)]
    ws = dev.alloc(1 << 20)

    def chain(wait):
        d_x = dev.htod_sync_copy(x)
        a, b, c, d, e = bufs

        def mm(y, src, w, n, k):
            ops.qmatmul(y, src, w, M, n, k, is_q4k=True, x_dtype=DTYPE_BF16, out_dtype=DTYPE_BF16, workspace=ws,
                        ws_bytes=1 << 20, stream=dev.stream)
            wait()

        for _ in range(6):
            ops.rms_norm(a, d_x, d_g, M, H, 1e-5, DTYPE_BF16, stream=dev.stream)
            wait()
            mm(b, a, w1, H + 512, H)
            check(lib().ub_copy_rows(c.ptr, H * 2, b.ptr, (H + 512) * 2, H * 2, M, dev.stream), "copy_rows")
            wait()
            mm(d, c, w2, 2 * I, H)
            ops.silu_and_mul(e, d, M, I, DTYPE_BF16, stream=dev.stream)
            wait()
            mm(d_x, e, w3, H, I)
        return fetch(dev, d_x, DTYPE_BF16, (M, H))

    want = chain(dev.synchronize)
    assert np.isfinite(want).all()
    for _ in range(3):
        assert np.array_equal(chain(lambda: None), want)
