"""GPU: the expert layer's grouped launches over token runs of chosen lengths (logits pin every token to its expert): the edges of
the copies' 32-token boxes, of the stages fitted to the longest run, of 128- and 256-token tiles, short runs beside long ones, experts
without a token.  The workspace starts as NaN: rows that pad an alignment block are not written and must not show."""
import numpy as np
import pytest

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, ops

from _util import fetch, to_storage

pytestmark = pytest.mark.gpu


def bf16(x):
    """To the nearest bf16, once (by way of f32 it would be twice)."""
    m, e = np.frexp(np.asarray(x, dtype=np.float64))
    return np.ldexp(np.rint(m * 256) / 256, e).astype(np.float32)


def one_piece(blob, rows, K):
    """The weights these launches multiply: bf16(s q - m) with the group's scale and min rounded to bf16."""
    b = np.ascontiguousarray(blob).view(np.uint8).reshape(-1, 144)
    d, s6 = b[:, :4].copy().view(np.float16).astype(np.float32), b[:, 4:16]
    sc = np.concatenate([s6[:, :4] & 63, s6[:, 8:] & 15 | s6[:, :4] >> 6 << 4], 1).astype(np.float32)
    mn = np.concatenate([s6[:, 4:8] & 63, s6[:, 8:] >> 4 | s6[:, 4:8] >> 6 << 4], 1).astype(np.float32)
    q = np.stack([b[:, 16:].reshape(-1, 4, 32) & 15, b[:, 16:].reshape(-1, 4, 32) >> 4], 2).reshape(-1, 8, 32)
    s, m = bf16(d[:, :1] * sc).astype(np.float64), bf16(d[:, 1:] * mn).astype(np.float64)
    return bf16(s[:, :, None] * q - m[:, :, None]).reshape(rows, K)


@pytest.mark.parametrize("counts,k,block", [
    ((1, 32, 33, 64, 65, 96, 97, 128), 1, 16), ((129, 1, 1, 2, 31, 5, 0, 40), 1, 64),
    ((32, 31, 30, 32), 1, 16), ((33, 30, 28, 31), 1, 16), ((64, 63, 1, 17), 1, 32), ((96, 95, 2, 1), 1, 32), ((97, 90, 3, 4), 1, 64),
    ((127, 128, 5, 1), 1, 128),
    # more than 128 tokens per expert: tiles of 256
    ((129, 257, 300, 1), 1, 64), ((256, 255, 129, 5), 1, 128), ((200, 130, 17, 500), 2, 16), ((128, 127, 0, 513), 2, 64),
])
def test_run_lengths(dev, counts, k, block):
    E, T, H, I = len(counts), sum(counts), 512, 768
    rng = np.random.default_rng(T + block)
    w13, w2 = o.gen_q4k_weight(rng, E * 2 * I, H), o.gen_q4k_weight(rng, E * H, I)
    hidden = o.gen_activation(rng, T, H, True)
    first = rng.permutation(np.repeat(np.arange(E), counts))
    logits = np.zeros((T, E), np.float32)
    logits[np.arange(T), first] = 6.
    if k == 2:  # the second one: mostly the last expert
        second = np.where(rng.random(T) < 0.9, E - 1, 0)
        logits[np.arange(T), np.where(second == first, (first + 1) % E, second)] = 3.
    assert o.rel_l2(one_piece(w2, E * H, I), o.c_dequant(w2, True).reshape(E * H, I)) < 5e-3
    want, _ = o.moe_layer_exact(hidden, logits, one_piece(w13, E * 2 * I, H).reshape(E, 2 * I, H),
                                one_piece(w2, E * H, I).reshape(E, H, I), k, block, True)
    d = [dev.htod_sync_copy(v) for v in (to_storage(hidden, DTYPE_BF16), to_storage(logits, DTYPE_BF16), w13, w2)]
    ws_bytes = ops.moe_layer_q4k_workspace_bytes(T, H, I, E, k, block)
    ws, d_out = dev.htod_sync_copy(np.full(ws_bytes, 0xFF, np.uint8)), dev.alloc(T * H * 2)
    ops.moe_layer_q4k(d_out, d[0], d[1], d[2], d[3], T, H, I, E, k, block, True, ws, ws_bytes, stream=dev.stream)
    got = fetch(dev, d_out, DTYPE_BF16, (T, H))
    assert dev.device_status() == 0
    # with the launches' own weights only a rounding of the 16-bit values between them may differ
    for t in range(T):
        assert o.rel_l2(got[t], want[t]) < 1.5e-2, (t, first[t])
    assert o.rel_l2(got, want) < 1e-2
