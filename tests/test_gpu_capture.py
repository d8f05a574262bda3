"""Layers captured in a CUDA graph: every call they make is allowed under capture, and a replay gives the bits of the
eager pass."""
import numpy as np
import pytest
import torch

from oracle import oracle as o
from ubridge_b200 import DTYPE_BF16, ops
from ubridge_b200.parallel import EPMoELayer, TPLinearStack

from _util import to_storage

pytestmark = pytest.mark.gpu


def _check(dev, forward, out, n):
    """forward() once eagerly, then captured and replayed on a cleared output."""
    forward()
    want = dev.dtoh_sync_copy(out.slice(0, n * 2), np.uint16, (n,))
    stream = torch.cuda.ExternalStream(int(getattr(dev.stream, "value", dev.stream)))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        forward()
    for _ in range(2):
        ops.silu_and_mul(out, dev.alloc_zeros(n * 4), 1, n, DTYPE_BF16, stream=dev.stream)  # zeros
        with torch.cuda.stream(stream):
            graph.replay()
        assert np.array_equal(dev.dtoh_sync_copy(out.slice(0, n * 2), np.uint16, (n,)), want)
    assert dev.device_status() == 0


@pytest.mark.parametrize("M", [1, 4, 45, 200])
def test_stack(dev, M):
    rng = np.random.default_rng(M)
    H, I, heads, kv = 1024, 2816, 8, 2
    w = [o.gen_q4k_weight(rng, n, k) for n, k in (((heads + 2 * kv) * 128, H), (H, heads * 128), (2 * I, H), (H, I))]
    stack = TPLinearStack(dev, H, I, heads, kv, 128, 1, *w, M)
    d_x, d_n = dev.htod_sync_copy(to_storage(o.gen_activation(rng, M, H, True), DTYPE_BF16)), dev.alloc(M * H * 2)
    d_g = dev.htod_sync_copy(to_storage(np.ones(H, dtype=np.float32), DTYPE_BF16))

    def forward():
        ops.rms_norm(d_n, d_x, d_g, M, H, 1e-5, DTYPE_BF16, stream=dev.stream)
        stack.forward(d_n, M)

    _check(dev, forward, stack.out, M * H)


@pytest.mark.parametrize("T", [1, 3, 40])
def test_expert_layer(dev, T):
    rng = np.random.default_rng(T)
    H, I, E = 512, 768, 4
    layer = EPMoELayer(dev, T, H, I, E, 2, 64, 0, 1, o.gen_q4k_weight(rng, E * 2 * I, H), o.gen_q4k_weight(rng, E * H, I))
    d_x = dev.htod_sync_copy(to_storage(o.gen_activation(rng, T, H, True), DTYPE_BF16))
    d_l = dev.htod_sync_copy(to_storage(o.gen_activation(rng, T, E, True), DTYPE_BF16))
    _check(dev, lambda: layer.forward(d_x, d_l), layer.out, T * H)
