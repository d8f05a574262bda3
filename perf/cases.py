"""What is timed of this framework: calls a user's program makes, over the sizes it makes them at.

Three kinds of case:

  linear  one quantized linear layer, y = x . W^T, through ``ops.qmatmul`` / ``ops.qmatmul_gguf``
  stack   the linear layers of decoder blocks, an RMSNorm in front of each block: ``ops.rms_norm`` and
          ``parallel.TPLinearStack`` on one GPU (QKV, O, gate and up with SiLU.up, down)
  moe     a mixture-of-experts layer, router logits to combined output, through ``parallel.EPMoELayer``

Weights are synthetic GGUF blocks with the standard deviation that trained weights have (about 0.02), activations and
router logits are N(0, 1).
"""
import math

import torch

import ubridge_b200 as ub
from ubridge_b200 import ops, parallel

DTYPES = {"f32": (ub.DTYPE_F32, torch.float32), "bf16": (ub.DTYPE_BF16, torch.bfloat16)}
# format: GGML type tag, values per block, bytes per block
FORMATS = {"Q4_0": (2, 32, 18), "Q8_0": (8, 32, 34), "Q4_K": (12, 256, 144), "Q5_K": (13, 256, 176),
           "Q6_K": (14, 256, 210)}


def listed():
    return [
        # the smallest call: one token through a small Q8_0 matrix (fused query, key and value rows) with f32
        # activations, as a host that keeps its activations in f32 makes it
        dict(name="q8_0_one_token", kind="linear", format="Q8_0", tokens=1, rows=6144, columns=4096, x="f32", y="f32"),
        # the output matrix of a model: its last linear layer, one token, logits in f32
        dict(name="q6_k_output_matrix", kind="linear", format="Q6_K", tokens=1, rows=32000, columns=4096, x="bf16",
             y="f32"),
        # generating text for one user
        dict(name="decode_1", kind="stack", layers=2, hidden=4096, inner=14336, heads=32, kv_heads=8, tokens=1),
        # the same where rows are not whole multiples of 2048 values
        dict(name="decode_1_odd_rows", kind="stack", layers=2, hidden=5120, inner=13824, heads=40, kv_heads=40, tokens=1),
        # generating for a few users, or checking a few drafted tokens
        dict(name="decode_4", kind="stack", layers=2, hidden=4096, inner=14336, heads=32, kv_heads=8, tokens=4),
        # generating for sixteen users with wide layers
        dict(name="decode_16_wide", kind="stack", layers=1, hidden=8192, inner=28672, heads=64, kv_heads=8, tokens=16),
        # a server's batch while it generates, or a short prompt: a ragged number of tokens
        dict(name="decode_45", kind="stack", layers=2, hidden=4096, inner=14336, heads=32, kv_heads=8, tokens=45),
        # reading a prompt with wide layers
        dict(name="prefill_512_wide", kind="stack", layers=1, hidden=8192, inner=28672, heads=64, kv_heads=8, tokens=512),
        # one layer of a long prompt
        dict(name="q4_k_prefill_2048", kind="linear", format="Q4_K", tokens=2048, rows=14336, columns=4096, x="bf16",
             y="bf16"),
        # mixed-format files keep some matrices (down projections, for instance) in Q6_K: a prompt through one of them
        dict(name="q6_k_prefill_333", kind="linear", format="Q6_K", tokens=333, rows=4096, columns=14336, x="bf16",
             y="bf16"),
        # generating for one user, mixture of experts: two experts of eight are read
        dict(name="moe_1", kind="moe", tokens=1, hidden=4096, inner=14336, experts=8, top_k=2),
        # a server's batch or a prompt, mixture of experts
        dict(name="moe_256", kind="moe", tokens=256, hidden=4096, inner=14336, experts=8, top_k=2),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _blocks(rng, low, high, step=256):
    return step * max(1, _log(rng, low, high) // step)


def draw(rng):
    kind = rng.choice(["linear", "linear", "stack", "stack", "moe"])
    if kind == "linear":
        fmt = rng.choice(["Q4_K", "Q4_K", "Q8_0", "Q6_K", "Q5_K", "Q4_0"])
        rows = _log(rng, 1024, 32000)
        if rng.random() < 0.7:
            rows = rows // 128 * 128
        columns = min(_blocks(rng, 1024, 14336), 4096 * 28672 // rows // 256 * 256)
        tokens = _log(rng, 1, 2048 if fmt in ("Q4_K", "Q8_0") else 333)
        tokens = max(1, min(tokens, 2048 * 14336 * 4096 // (rows * columns)))
        x, y = rng.choice([("bf16", "bf16"), ("bf16", "bf16"), ("bf16", "f32"), ("f32", "f32")])
        return dict(kind=kind, format=fmt, tokens=tokens, rows=rows, columns=columns, x=x, y=y)
    if kind == "stack":
        hidden = _blocks(rng, 1024, 8192)
        heads = hidden // 128
        kv_heads = rng.choice([k for k in (heads, heads // 2, heads // 4, heads // 8) if k and heads % k == 0])
        inner = _blocks(rng, 2 * hidden, 3.5 * hidden)
        layers = 1 if hidden > 5120 else 2
        return dict(kind=kind, layers=layers, hidden=hidden, inner=inner, heads=heads, kv_heads=kv_heads,
                    tokens=_log(rng, 1, 512))
    hidden = _blocks(rng, 1024, 4096)
    return dict(kind=kind, tokens=_log(rng, 1, 256), hidden=hidden, inner=_blocks(rng, hidden, 3.5 * hidden),
                experts=rng.choice([4, 8, 8]), top_k=rng.choice([1, 2, 2]))


# --------------------------------------------------------------------------------------------------- inputs
def _f16_bytes(t):
    return t.to(torch.float16).view(torch.uint8).view(*t.shape, 2)


def _scale(gen, blocks, mean):
    """Block scales, uniform around their mean."""
    return mean * (0.5 + torch.rand(blocks, generator=gen, device="cuda"))


def _weights(gen, fmt, rows, columns):
    """Packed blocks of a rows x columns matrix, flat; values of standard deviation about 0.02."""
    _, per, size = FORMATS[fmt]
    n = rows * columns // per
    b = torch.randint(0, 256, (n, size), dtype=torch.uint8, generator=gen, device="cuda")  # quants: every pattern
    if fmt == "Q8_0":
        b[:, 0:2] = _f16_bytes(_scale(gen, n, 2.7e-4))
    elif fmt == "Q4_0":
        b[:, 0:2] = _f16_bytes(_scale(gen, n, 4.3e-3))
    elif fmt == "Q6_K":
        b[:, 208:210] = _f16_bytes(_scale(gen, n, 1.5e-5))
    else:  # Q4_K, Q5_K: 6-bit scales and mins, the mins at the middle of a sub-block's range as in real files
        d = _scale(gen, n, 1.1e-4 if fmt == "Q4_K" else 5.3e-5)
        b[:, 0:2] = _f16_bytes(d)
        b[:, 2:4] = _f16_bytes(d * (7.5 if fmt == "Q4_K" else 15.5))
        sc = torch.randint(16, 64, (n, 8), dtype=torch.uint8, generator=gen, device="cuda")
        mn = (sc + torch.randint(0, 7, (n, 8), dtype=torch.uint8, generator=gen, device="cuda") - 3).clamp_(0, 63)
        b[:, 4:8] = (sc[:, :4] & 63) | ((sc[:, 4:] >> 4) << 6)
        b[:, 8:12] = (mn[:, :4] & 63) | ((mn[:, 4:] >> 4) << 6)
        b[:, 12:16] = (sc[:, 4:] & 15) | ((mn[:, 4:] & 15) << 4)
    return b.view(-1)


def _normal(gen, shape, dtype):
    return torch.randn(shape, generator=gen, device="cuda").to(dtype)


_device = None


def _dev():
    """The process's device handle: one device, one stream, as a program keeps it."""
    global _device
    if _device is None:
        _device = ub.GcuDevice(torch.cuda.current_device())
    return _device


def _resident(dev, t):
    return ub.GcuSlice(dev, t.data_ptr(), t.numel() * t.element_size(), owner=t)


class _Foreign:
    """A device buffer of the framework, for torch to look at."""

    def __init__(self, buf, shape):
        self.buf = buf
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<i2", data=(buf.ptr, False), version=2)


def _as_tensor(buf, shape):
    return torch.as_tensor(_Foreign(buf, shape), device="cuda").view(torch.bfloat16)


def _inputs(case, seed):
    """Every input of a case, as torch tensors on the GPU."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    if case["kind"] == "linear":
        M, N, K = case["tokens"], case["rows"], case["columns"]
        return dict(w=_weights(gen, case["format"], N, K), x=_normal(gen, (M, K), DTYPES[case["x"]][1]))
    M, H, I = case["tokens"], case["hidden"], case["inner"]
    if case["kind"] == "stack":
        layers = []
        for _ in range(case["layers"]):
            w = [_weights(gen, "Q4_K", n, k) for n, k in _stack_shapes(case)]
            layers.append((w, (0.9 + 0.2 * torch.rand(H, generator=gen, device="cuda")).bfloat16()))
        return dict(layers=layers, x=_normal(gen, (M, H), torch.bfloat16))
    E = case["experts"]
    return dict(w13=_weights(gen, "Q4_K", E * 2 * I, H), w2=_weights(gen, "Q4_K", E * H, I),
                x=_normal(gen, (M, H), torch.bfloat16), logits=_normal(gen, (M, E), torch.bfloat16))


def _stack_shapes(case):
    H, I, h, kv = case["hidden"], case["inner"], case["heads"], case["kv_heads"]
    return [((h + 2 * kv) * 128, H), (H, h * 128), (2 * I, H), (H, I)]


def prepare(case, seed):
    dev = _dev()
    st = dict(case=case, dev=dev)
    made = _inputs(case, seed)
    if case["kind"] == "linear":
        M, N, K = case["tokens"], case["rows"], case["columns"]
        tag, (xd, xt), (yd, yt) = FORMATS[case["format"]][0], DTYPES[case["x"]], DTYPES[case["y"]]
        st["w"], st["x"] = made["w"], made["x"]
        st["y"] = torch.empty((M, N), dtype=yt, device="cuda")
        ws_bytes = ub.lib().ub_qmatmul_gguf_workspace_bytes(tag, M, N, K)
        if case["format"] == "Q8_0":
            ws_bytes = ops.qmatmul_workspace_bytes(M, N, K, False)
        st["ws"] = torch.empty((max(ws_bytes, 256),), dtype=torch.uint8, device="cuda")
        st["pointers"] = (st["y"].data_ptr(), st["x"].data_ptr(), st["w"].data_ptr())
        st["call"] = dict(x_dtype=xd, out_dtype=yd, workspace=st["ws"].data_ptr(), ws_bytes=ws_bytes, stream=dev.stream)
    elif case["kind"] == "stack":
        M, H, I, h, kv = case["tokens"], case["hidden"], case["inner"], case["heads"], case["kv_heads"]
        st["layers"], st["gammas"] = [], []
        for packed, gamma in made["layers"]:
            w = [_resident(dev, t) for t in packed]
            st["layers"].append(parallel.TPLinearStack(dev, H, I, h, kv, 128, 1, w[0], w[1], w[2], w[3], M))
            st["gammas"].append(_resident(dev, gamma))
        st["x"] = _resident(dev, made["x"])
        st["normed"] = dev.alloc(M * H * 2)
        st["y"] = _as_tensor(st["layers"][-1].out, (M, H))
    else:
        T, H, I, E = case["tokens"], case["hidden"], case["inner"], case["experts"]
        w13, w2 = _resident(dev, made["w13"]), _resident(dev, made["w2"])
        st["layer"] = parallel.EPMoELayer(dev, T, H, I, E, case["top_k"], 64, 0, 1, w13, w2)
        st["x"], st["logits"] = _resident(dev, made["x"]), _resident(dev, made["logits"])
        st["y"] = _as_tensor(st["layer"].out, (T, H))
    # the inputs were made on torch's stream, the framework's calls go to the device's own
    torch.cuda.current_stream().synchronize()
    dev.synchronize()
    return st


def run(st):
    case = st["case"]
    if case["kind"] == "linear":
        y, x, w = st["pointers"]
        M, N, K, fmt = case["tokens"], case["rows"], case["columns"], case["format"]
        if fmt == "Q4_K" or fmt == "Q8_0":
            ops.qmatmul(y, x, w, M, N, K, is_q4k=fmt == "Q4_K", **st["call"])
        else:
            ops.qmatmul_gguf(y, x, w, FORMATS[fmt][0], M, N, K, **st["call"])
    elif case["kind"] == "stack":
        M, H, stream, h = case["tokens"], case["hidden"], st["dev"].stream, st["x"]
        for layer, gamma in zip(st["layers"], st["gammas"]):
            ops.rms_norm(st["normed"], h, gamma, M, H, 1e-5, ub.DTYPE_BF16, stream)
            h = layer.forward(st["normed"], M)
    else:
        st["layer"].forward(st["x"], st["logits"])
    return st["y"]


# --------------------------------------------------------------------------------------------------- bounds
def work(case):
    def weight_bytes(fmt, values):
        _, per, size = FORMATS[fmt]
        return values // per * size

    M = case["tokens"]
    if case["kind"] == "linear":
        N, K = case["rows"], case["columns"]
        esz = {"f32": 4, "bf16": 2}
        return dict(bytes=weight_bytes(case["format"], N * K) + M * K * esz[case["x"]] + M * N * esz[case["y"]],
                    flops=2.0 * M * N * K)
    H, I = case["hidden"], case["inner"]
    if case["kind"] == "stack":
        qkv = (case["heads"] + 2 * case["kv_heads"]) * 128
        values = case["layers"] * (qkv * H + H * case["heads"] * 128 + 2 * I * H + H * I)
        return dict(bytes=weight_bytes("Q4_K", values) + 2 * M * H * 2, flops=2.0 * M * values)
    E, k = case["experts"], case["top_k"]
    # experts that at least one token is routed to, on average
    touched = E * (1.0 - (1.0 - k / E) ** M)
    return dict(bytes=int(touched * weight_bytes("Q4_K", 3 * I * H)) + M * (2 * H + E) * 2, flops=2.0 * M * k * 3 * I * H)


def tolerance(case):
    """Measured against the same chain of operations in f64 (2-norm): one linear layer 2.8e-5 where its sums leave in
    f32 (activations carry 15 bits), 1.7e-3 where they are rounded to bf16 once; from nine tokens on Q4_K and Q8_0
    weights are themselves rounded to bf16, which reads 5.0e-3 for Q4_K; 2.4e-2 after two decoder blocks (eight
    matrices one behind the other, bf16 between them); 9.4e-3 for a mixture-of-experts layer."""
    if case["kind"] == "stack":
        return {"rel": 4e-2}
    if case["kind"] == "moe":
        return {"rel": 3e-2}
    if case["format"] in ("Q4_K", "Q8_0") and case["tokens"] > 8:
        return {"rel": 2e-2}
    return {"rel": 7e-3 if case["y"] == "bf16" else 1e-4}


# --------------------------------------------------------------------------------------------------- 64-bit results
def _f16(b, at):
    return b[:, at:at + 2].contiguous().view(torch.float16).double()


def _values(fmt, packed):
    """Packed blocks as f64 values [blocks, values per block]."""
    _, per, size = FORMATS[fmt]
    b = packed.view(-1, size)
    d = _f16(b, 208 if fmt == "Q6_K" else 0)
    if fmt == "Q8_0":
        return d * b[:, 2:].contiguous().view(torch.int8).double()
    if fmt == "Q4_0":
        q = b[:, 2:]
        return d * (torch.cat([q & 15, q >> 4], 1).double() - 8)
    if fmt == "Q6_K":
        sc = b[:, 192:208].contiguous().view(torch.int8).double().repeat_interleave(16, 1)
        q = []
        for half in range(2):
            lo, hi = b[:, 64 * half:64 * half + 64], b[:, 128 + 32 * half:160 + 32 * half]
            for part in range(4):
                nibble = lo[:, 32 * (part & 1):32 * (part & 1) + 32] >> (4 * (part >> 1)) & 15
                q.append(nibble | (hi >> (2 * part) & 3) << 4)
        return d * sc * (torch.cat(q, 1).double() - 32)
    s, dmin = b[:, 4:16], _f16(b, 2)
    sc = torch.cat([s[:, :4] & 63, s[:, 8:] & 15 | s[:, :4] >> 6 << 4], 1).double().repeat_interleave(32, 1)
    mn = torch.cat([s[:, 4:8] & 63, s[:, 8:] >> 4 | s[:, 4:8] >> 6 << 4], 1).double().repeat_interleave(32, 1)
    q4 = b[:, size - 128:]
    q = []
    for sub in range(8):
        v = q4[:, 32 * (sub // 2):32 * (sub // 2) + 32] >> (4 * (sub & 1)) & 15
        if fmt == "Q5_K":
            v = v | (b[:, 16:48] >> sub & 1) << 4
        q.append(v)
    return d * sc * torch.cat(q, 1).double() - dmin * mn


def _linear64(x, fmt, packed, rows):
    """x . W^T in f64, W taken a slice of rows at a time."""
    _, per, size = FORMATS[fmt]
    K = x.shape[1]
    w = packed.view(rows, K // per * size)
    step = max(1, (1 << 26) // K)
    return torch.cat([x @ _values(fmt, w[r:r + step].reshape(-1)).view(-1, K).T for r in range(0, rows, step)], 1)


def _silu_up64(gu, I):
    return torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]


def exact(case, seed):
    made = _inputs(case, seed)
    x = made["x"].double()
    if case["kind"] == "linear":
        return _linear64(x, case["format"], made["w"], case["rows"])
    H, I = case["hidden"], case["inner"]
    if case["kind"] == "stack":
        for w, gamma in made["layers"]:
            x = x * torch.rsqrt(x.square().mean(1, keepdim=True) + 1e-5) * gamma.double()
            for i, (packed, (rows, _)) in enumerate(zip(w, _stack_shapes(case))):
                x = _linear64(x, "Q4_K", packed, rows)
                if i == 0:
                    x = x[:, :case["heads"] * 128]
                elif i == 2:
                    x = _silu_up64(x, I)
        return x
    E, k = case["experts"], case["top_k"]
    p, chosen = torch.softmax(made["logits"].double(), 1).sort(dim=1, descending=True, stable=True)  # ties: lowest
    p, chosen = p[:, :k] / p[:, :k].sum(1, keepdim=True), chosen[:, :k]
    w13, w2 = made["w13"].view(E, -1), made["w2"].view(E, -1)
    y = torch.zeros_like(x)
    for e in range(E):
        t, slot = (chosen == e).nonzero(as_tuple=True)
        if len(t):
            act = _silu_up64(_linear64(x[t], "Q4_K", w13[e], 2 * I), I)
            y.index_add_(0, t, p[t, slot, None] * _linear64(act, "Q4_K", w2[e], H))
    return y
