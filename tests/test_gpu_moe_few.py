"""Expert layer for a few tokens: a token at a time through the one-token kernels (two launches per token)."""
import numpy as np
import pytest

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, DTYPE_F32, ops
from ubridge_b200._lib import UB_ERR_BAD_INDEX

from _util import fetch, to_storage

pytestmark = pytest.mark.gpu


def _layer(dev, T, H, I, E, k, hidden, logits, w13, w2, emap=None, norm=True):
    ws_bytes = ops.moe_layer_q4k_workspace_bytes(T, H, I, E, k, 64)
    d = [dev.htod_sync_copy(v) for v in (to_storage(hidden, DTYPE_BF16), to_storage(logits, DTYPE_BF16), w13, w2)]
    d_map = None if emap is None else dev.htod_sync_copy(emap)
    d_out = dev.alloc(T * H * 2)
    ops.moe_layer_q4k(d_out, d[0], d[1], d[2], d[3], T, H, I, E, k, 64, norm, dev.alloc(ws_bytes), ws_bytes,
                      expert_map=d_map, stream=dev.stream)
    return fetch(dev, d_out, DTYPE_BF16, (T, H))


@pytest.mark.parametrize("T,H,I,E,k,norm", [
    (1, 256, 256, 4, 1, True),      # one slot, one super-block
    (1, 2048, 4096, 8, 2, True),    # rows of whole lines
    (2, 768, 1280, 5, 3, False),    # boxes of two super-blocks, an odd number of stages over the slots
    (3, 1024, 14336, 4, 2, True),   # two slots of seven stages: the longest the down launch takes
    (2, 512, 1024, 12, 8, True),    # eight slots
    (3, 512, 768, 8, 2, True),      # the most tokens of this size that go one at a time
    (6, 512, 768, 8, 2, True), (7, 512, 768, 8, 2, True),  # more: the grouped kernels
    (2, 512, 28672, 3, 2, True),    # more stages than the down launch takes: the grouped kernels
])
@pytest.mark.parametrize("mapped", [False, True])
def test_few_tokens(dev, T, H, I, E, k, norm, mapped):
    rng = np.random.default_rng(T + H + I + E)
    emap = None
    local = E
    if mapped:  # every other expert is held by another rank
        emap = np.full(E, -1, dtype=np.int32)
        emap[::2] = np.arange((E + 1) // 2)
        local = (E + 1) // 2
    w13, w2 = o.gen_q4k_weight(rng, E * 2 * I, H), o.gen_q4k_weight(rng, E * H, I)
    hidden, logits = o.gen_activation(rng, T, H, True), o.gen_activation(rng, T, E, True)
    got = _layer(dev, T, H, I, E, k, hidden, logits, w13, w2, emap, norm)
    deq13 = o.c_dequant(w13, True).reshape(E, 2 * I, H)[:local]
    deq2 = o.c_dequant(w2, True).reshape(E, H, I)[:local]
    want, _ = o.moe_layer_exact(hidden, logits, deq13, deq2, k, 64, norm, expert_map=emap)
    assert o.rel_l2(got, want) < 1e-2  # activations, each slot's output (in the oracle) and the sum are rounded to bf16
    assert dev.device_status() == 0


@pytest.mark.parametrize("T,H,I,k,own", [(1, 512, 1024, 2, 0), (3, 768, 1280, 2, 0), (2, 512, 1024, 3, 2), (2, 2048, 2304, 2, 1)])
def test_weights_of_other_ranks_are_not_read(dev, T, H, I, k, own):
    """Every matrix but those of this rank (none, some) holds NaN scales: the others' slots add exact zeros."""
    E = 4
    rng = np.random.default_rng(T + H + I + own)
    emap = np.full(E, -1, dtype=np.int32)
    emap[1:1 + own] = np.arange(1, 1 + own)  # matrix 0 is nobody's
    w13, w2 = o.gen_q4k_weight(rng, E * 2 * I, H), o.gen_q4k_weight(rng, E * H, I)
    hidden, logits = o.gen_activation(rng, T, H, True), o.gen_activation(rng, T, E, True)
    want = np.zeros((T, H), dtype=np.float32)
    if own:
        want, _ = o.moe_layer_exact(hidden, logits, o.c_dequant(w13, True).reshape(E, 2 * I, H),
                                    o.c_dequant(w2, True).reshape(E, H, I), k, 64, True, expert_map=emap)
    for w in (w13, w2):
        b = w.reshape(E, -1, 144)
        for e in range(E):
            if e not in emap:
                b[e, :, 0:4] = 0xFF  # d = dmin = NaN
    got = _layer(dev, T, H, I, E, k, hidden, logits, w13, w2, emap)
    if own:
        assert o.rel_l2(got, want) < 1e-2
    else:
        assert np.array_equal(got, want)
    assert dev.device_status() == 0


@pytest.mark.parametrize("H,I", [(512, 1024), (2048, 4096), (768, 1280)])
@pytest.mark.parametrize("what", ["nan", "inf", "gate overflows"])
def test_what_is_not_finite_stays_so(dev, H, I, what):
    """A NaN or an infinity in one token, or a gate whose SiLU is NaN (-inf): that token becomes NaN, as in the grouped
    kernels, the others keep their bits."""
    T, E, k = 3, 4, 2
    rng = np.random.default_rng(H + I)
    w13, w2 = o.gen_q4k_weight(rng, E * 2 * I, H), o.gen_q4k_weight(rng, E * H, I)
    hidden, logits = o.gen_activation(rng, T, H, True), o.gen_activation(rng, T, E, True)
    clean = _layer(dev, T, H, I, E, k, hidden, logits, w13, w2)
    bad = hidden.copy()
    if what == "gate overflows":
        bad[1] = 3e38  # sums beyond the largest float, of either sign
    else:
        bad[1, H // 2 + 3] = np.nan if what == "nan" else np.inf
    got = _layer(dev, T, H, I, E, k, bad, logits, w13, w2)
    assert np.isfinite(clean).all()
    assert np.isnan(got[1]).all()
    assert np.array_equal(got[[0, 2]], clean[[0, 2]])


@pytest.mark.parametrize("K", [2048, 4096, 768, 8192, 14336])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_one_token_that_is_not_finite(dev, K, bad):
    """The one-token matmul itself: short rows, rows in several stages, the sixteen-warp kernel."""
    N = 40
    rng = np.random.default_rng(K)
    x = o.gen_activation(rng, 1, K, True)
    x[0, K - 5] = bad
    d_y = dev.alloc(N * 4)
    ops.qmatmul(d_y, dev.htod_sync_copy(to_storage(x, DTYPE_BF16)), dev.htod_sync_copy(o.gen_q4k_weight(rng, N, K)), 1, N, K,
                is_q4k=True, x_dtype=DTYPE_BF16, out_dtype=DTYPE_F32, stream=dev.stream)
    assert np.isnan(fetch(dev, d_y, DTYPE_F32, (1, N))).all()


@pytest.mark.parametrize("T", [1, 2, 40])
@pytest.mark.parametrize("entry", [-2, 4])
def test_a_map_out_of_range_is_reported(dev, T, entry):
    """Few tokens and the grouped path alike, whether or not a token goes to that expert."""
    H, I, E, k = 256, 256, 4, 1
    rng = np.random.default_rng(T)
    w13, w2 = o.gen_q4k_weight(rng, E * 2 * I, H), o.gen_q4k_weight(rng, E * H, I)
    hidden, logits = o.gen_activation(rng, T, H, True), o.gen_activation(rng, T, E, True)
    logits[:, 0] = 9  # every token to expert 0, the bad entry is expert 3's
    emap = np.array([0, 1, 2, entry], dtype=np.int32)
    _layer(dev, T, H, I, E, k, hidden, logits, w13, w2, emap)
    assert dev.device_status() == UB_ERR_BAD_INDEX
    _layer(dev, T, H, I, E, k, hidden, logits, w13, w2, np.array([0, 1, 2, -1], dtype=np.int32))
    assert dev.device_status() == 0


@pytest.mark.parametrize("T,H,I,mapped,grouped", [(6, 1024, 1024, True, True), (6, 1024, 1024, False, True),
                                                 (2, 1024, 1024, True, False), (3, 1024, 1024, False, False)])
def test_which_way_a_few_tokens_go(dev, T, H, I, mapped, grouped):
    """The grouped kernels give a token the same bits whoever comes with it; one at a time the weights are not rounded.  With
    eight experts on eight ranks (or a small layer) six tokens are faster grouped."""
    E, k, many = 8, 2, 40
    rng = np.random.default_rng(T + mapped)
    emap = None
    if mapped:
        emap = np.full(E, -1, dtype=np.int32)
        emap[3] = 0
    w13, w2 = o.gen_q4k_weight(rng, E * 2 * I, H), o.gen_q4k_weight(rng, E * H, I)
    hidden, logits = o.gen_activation(rng, many, H, True), o.gen_activation(rng, many, E, True)
    logits[0, 3] = 9  # at least one token has work here
    all_ = _layer(dev, many, H, I, E, k, hidden, logits, w13, w2, emap)
    got = _layer(dev, T, H, I, E, k, hidden[:T], logits[:T], w13, w2, emap)
    assert np.array_equal(got, all_[:T]) == grouped
    assert o.rel_l2(got, all_[:T]) < 2e-2
