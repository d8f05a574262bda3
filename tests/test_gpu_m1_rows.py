"""One token on Q4_K rows that are not whole 128-byte lines (K a multiple of 256, not of 2048), and rows of an odd number
of stages on the sixteen-warp kernel."""
import numpy as np
import pytest

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, DTYPE_F16, DTYPE_F32, ops
from ubridge_b200._lib import UbridgeError, check, lib

from _util import fetch, to_storage

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x_dtype", [DTYPE_BF16, DTYPE_F32])
@pytest.mark.parametrize("N,K", [
    (1, 256),        # one super-block: half a box, seven warps without work
    (17, 768),       # an odd super-block at the end of a row
    (5000, 1280),    # more than one tile per CTA
    (300, 5120), (40, 11008),  # last stage of four, of three super-blocks
    (300, 12544),    # sixteen warps, seven stages (an empty one behind them), one super-block in the last
    (5121, 13824), (300, 14336),  # the same with six super-blocks, and rows of whole lines
    (33, 28416),     # fourteen stages, an odd super-block at the end
    (20, 28928),     # longer than the sixteen-warp kernel takes
])
def test_one_token_any_row_length(dev, x_dtype, N, K):
    rng = np.random.default_rng(N + K)
    w = o.gen_q4k_weight(rng, N, K)
    x = o.gen_activation(rng, 1, K, x_dtype == DTYPE_BF16)
    d_w, d_x, d_y = dev.htod_sync_copy(w), dev.htod_sync_copy(to_storage(x, x_dtype)), dev.alloc(N * 4)

    def run():
        ops.qmatmul(d_y, d_x, d_w, 1, N, K, is_q4k=True, x_dtype=x_dtype, out_dtype=DTYPE_F32, stream=dev.stream)
        return fetch(dev, d_y, DTYPE_F32, (1, N))

    got = run()
    # 15-bit activations: 3e-5 as a 2-norm over many outputs; one output may be a small difference of large terms
    assert o.rel_l2(got, o.c_qmatmul(x, w, N, K, True)) < (1e-4 if N >= 300 else 1e-3)
    assert dev.device_status() == 0
    assert np.array_equal(got, run())


@pytest.mark.parametrize("I,K", [(37, 768), (2500, 5120), (264, 12032), (40, 12544)])
def test_gate_up_of_one_token_has_the_bits_of_two_calls(dev, I, K):
    rng = np.random.default_rng(I + K)
    w = o.gen_q4k_weight(rng, 2 * I, K)
    x = o.gen_activation(rng, 1, K, True)
    d_w, d_x = dev.htod_sync_copy(w), dev.htod_sync_copy(to_storage(x, DTYPE_BF16))
    d_y, d_gu, d_y2 = dev.alloc(I * 2), dev.alloc(4 * I), dev.alloc(I * 2)
    ws_bytes = ops.qmatmul_q4k_gate_up_workspace_bytes(1, I, K)
    ops.qmatmul_q4k_gate_up(d_y, d_x, d_w, 1, I, K, out_dtype=DTYPE_BF16, workspace=dev.alloc(ws_bytes),
                            ws_bytes=ws_bytes, stream=dev.stream)
    ops.qmatmul(d_gu, d_x, d_w, 1, 2 * I, K, is_q4k=True, x_dtype=DTYPE_BF16, out_dtype=DTYPE_BF16, stream=dev.stream)
    ops.silu_and_mul(d_y2, d_gu, 1, I, DTYPE_BF16, stream=dev.stream)
    assert np.array_equal(fetch(dev, d_y, DTYPE_BF16, (I,)), fetch(dev, d_y2, DTYPE_BF16, (I,)))


@pytest.mark.parametrize("N,K", [(300, 768), (520, 5120)])
def test_rms_norm_in_front(dev, N, K):
    rng = np.random.default_rng(N + K)
    w = o.gen_q4k_weight(rng, N, K)
    x = o.round_through(o.gen_activation(rng, 1, K, True) * 2.5, o.UB_BF16)
    g = o.round_through(rng.uniform(0.5, 1.5, size=K).astype(np.float32), o.UB_BF16)
    ws_bytes = ops.qmatmul_q4k_rmsnorm_workspace_bytes(1, N, K, False)
    d_y = dev.alloc(N * 2)
    ops.qmatmul_q4k_rmsnorm(d_y, dev.htod_sync_copy(to_storage(x, DTYPE_BF16)), dev.htod_sync_copy(to_storage(g, DTYPE_BF16)),
                            1e-5, dev.htod_sync_copy(w), 1, N, K, gate_up=False, out_dtype=DTYPE_BF16,
                            workspace=dev.alloc(ws_bytes), ws_bytes=ws_bytes, stream=dev.stream)
    want = o.c_qmatmul(o.rms_norm(x, g, 1e-5, o.UB_BF16), w, N, K, True)
    # bf16 activations after the norm (a boundary case may round the other way) and bf16 output
    assert o.rel_l2(fetch(dev, d_y, DTYPE_BF16, (1, N)), want) < 8e-3


def test_what_needs_a_workspace_still_does(dev):
    """Gate/up and RMSNorm forms of one token: without a workspace, and gate/up in f32, for K % 2048 == 0 only."""
    I, K = 64, 1280
    d_w = dev.htod_sync_copy(np.zeros(2 * I * K // 256 * 144, dtype=np.uint8))
    d_x, d_y = dev.htod_sync_copy(np.zeros(K, dtype=np.uint16)), dev.alloc(I * 4)
    with pytest.raises(UbridgeError):
        ops.qmatmul_q4k_gate_up(d_y, d_x, d_w, 1, I, K, out_dtype=DTYPE_BF16, stream=dev.stream)
    with pytest.raises(UbridgeError):
        ops.qmatmul_q4k_rmsnorm(d_y, d_x, d_x, 1e-5, d_w, 1, I, K, gate_up=False, out_dtype=DTYPE_BF16, workspace=None,
                                ws_bytes=0, stream=dev.stream)
    ws_bytes = ops.qmatmul_q4k_gate_up_workspace_bytes(1, I, K)
    with pytest.raises(UbridgeError):
        ops.qmatmul_q4k_gate_up(d_y, d_x, d_w, 1, I, K, out_dtype=DTYPE_F32, workspace=dev.alloc(ws_bytes),
                                ws_bytes=ws_bytes, stream=dev.stream)


@pytest.mark.parametrize("K,bound", [(18944, 1.4e-5), (27648, 1.4e-5), (33024, 5e-6)])
def test_long_rows_keep_their_precision(dev, K, bound):
    """One activation of 256 a hundred times the others.  Rounding these activations in f64 to 16 bits with a scale per 32 values
    leaves 8.3e-6 and 7.4e-6 of the result, to 15 bits with a scale per 256 2.7e-5 and 2.1e-5; f32 throughout far less."""
    N = 600
    rng = np.random.default_rng(K)
    w = o.gen_q4k_weight(rng, N, K)
    x = rng.standard_normal((1, K)).astype(np.float32)
    x[0, 7::256] = 100
    d_y = dev.alloc(N * 4)
    ops.qmatmul(d_y, dev.htod_sync_copy(x), dev.htod_sync_copy(w), 1, N, K, is_q4k=True, x_dtype=DTYPE_F32,
                out_dtype=DTYPE_F32, stream=dev.stream)
    assert o.rel_l2(fetch(dev, d_y, DTYPE_F32, (1, N)), x.astype(np.float64) @ o.c_dequant(w, True).reshape(N, K).T) < bound
    assert dev.device_status() == 0


@pytest.mark.parametrize("N,K", [(300, 768), (520, 5120), (40, 11008), (300, 13824), (300, 17920)])
def test_residual_behind_rows_of_any_length(dev, N, K):
    """The epilogue that adds a residual row, on boxes of two super-blocks, odd ones among them, and in several passes."""
    import ctypes

    rng = np.random.default_rng(N + K)
    w = o.gen_q4k_weight(rng, N, K)
    x, r = o.gen_activation(rng, 1, K, True), o.round_through(rng.standard_normal((1, N)).astype(np.float32), o.UB_BF16)
    d = [dev.htod_sync_copy(v) for v in (to_storage(x, DTYPE_BF16), w, to_storage(r, DTYPE_BF16))]
    d_y = dev.alloc(N * 2)
    check(lib().ub_qmatmul_q4k_allreduce_residual_bf16(ctypes.c_void_p(d_y.ptr), ctypes.c_void_p(d[0].ptr),
                                                       ctypes.c_void_p(d[1].ptr), ctypes.c_void_p(d[2].ptr), 1, N, K, None,
                                                       0, 1, 0, dev.stream), "residual")
    assert o.rel_l2(fetch(dev, d_y, DTYPE_BF16, (1, N)), r + o.c_qmatmul(x, w, N, K, True)) < 5e-3  # one rounding to bf16
    assert dev.device_status() == 0


@pytest.mark.parametrize("N,K", [(300, 768), (300, 5120), (300, 13824), (300, 14336)])
def test_f16_results(dev, N, K):
    """The f32 result rounded once (activations small enough that none overflows)."""
    rng = np.random.default_rng(N + K)
    d_w = dev.htod_sync_copy(o.gen_q4k_weight(rng, N, K))
    x = o.round_through(o.gen_activation(rng, 1, K, True) * 0.0625, o.UB_BF16)
    d_x = dev.htod_sync_copy(to_storage(x, DTYPE_BF16))
    y = {}
    for dt in (DTYPE_F32, DTYPE_F16):
        d_y = dev.alloc(N * 4)
        ops.qmatmul(d_y, d_x, d_w, 1, N, K, is_q4k=True, x_dtype=DTYPE_BF16, out_dtype=dt, stream=dev.stream)
        y[dt] = fetch(dev, d_y, dt, (1, N))
    assert np.array_equal(y[DTYPE_F16], y[DTYPE_F32].astype(np.float16).astype(np.float32))
