"""The workloads whose speed this framework is judged by, as a user's program runs them through the `ttnn` API.

listed() names the cases, draw() makes more of the same ranges, prepare() builds what a program holds before the call
(tensors on the device, weights packed once), run() is one pass, work() the bytes and operations a pass cannot do without,
tolerance() how far the results of another correct implementation of the same precision may lie.

Results that stay on the device come back as torch views of their own buffers (tile order, padding included)."""
import os
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "tt-metal_b200")   # imported with the repository's root as the working folder
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)
import ttnn  # noqa: E402

TILE_BYTES = {"bfloat8_b": 1088, "bfloat4_b": 576, "bfloat16": 2048}


def up32(v):
    return (v + 31) // 32 * 32


# ---- the cases -----------------------------------------------------------------------------------------------------------
def _linear(name, rows, k, n, weight, bias=False, activation="", out="bfloat16"):
    c = {"path": "linear", "rows": rows, "k": k, "n": n, "weight": weight, "bias": bias, "activation": activation, "out": out}
    return dict(c, name=name) if name else c


def listed():
    return [
        # The smallest call: one token's activation comes from the host, one linear, the result goes back. Latency only.
        {"name": "serve_one_linear", "path": "serve", "rows": 1, "k": 512, "n": 1024, "weight": "bfloat8_b"},
        # One decode linear of Falcon-7B's MLP, batch 32 (the single-linear benchmark configuration).
        _linear("decode_falcon_h_to_4h", 32, 4544, 18176, "bfloat8_b"),
        # The weight matmuls of one Llama-2-70B decoder layer at batch 32: q/k/v, the output projection, the gated MLP.
        {"name": "decode_layer_llama70b", "path": "layer", "rows": 32, "hidden": 8192, "kv": 1024, "ffn": 28672, "attn": "bfloat8_b",
         "mlp": "bfloat8_b", "down": "bfloat8_b"},
        # The same of one Mistral-7B layer, whose gate and up projections are bfloat4_b.
        {"name": "decode_layer_mistral7b", "path": "layer", "rows": 32, "hidden": 4096, "kv": 1024, "ffn": 14336, "attn": "bfloat8_b",
         "mlp": "bfloat4_b", "down": "bfloat8_b"},
        # Decode with a large batch: 128 sequences through a gate projection with its activation.
        _linear("decode_batch128_gate", 128, 4096, 14336, "bfloat4_b", activation="silu"),
        # A short prompt through Falcon-7B's fused q/k/v projection: ragged row count, a column count with a partial last tile.
        _linear("prompt_350_falcon_qkv", 350, 4544, 4672, "bfloat8_b", bias=True),
        # A prompt through a square projection with bias and activation.
        _linear("prompt_512_square_gelu", 512, 4096, 4096, "bfloat8_b", bias=True, activation="gelu"),
        # Prefill: the Llama-2-70B MLP shape of the benchmark, compute bound.
        _linear("prefill_2048_llama_mlp", 2048, 8192, 28672, "bfloat8_b"),
        # Plain bfloat16 weights (layers a model keeps unquantised), the generic square size.
        _linear("bf16_weight_1024", 1024, 1024, 1024, "bfloat16"),
        # Attention scores of a 512-token prompt, 32 heads of 128: a batched second operand.
        {"name": "scores_32_heads_512", "path": "batched", "batch": 32, "m": 512, "k": 128, "n": 512},
        # Packing on the device, the tensor of the conversion benchmark: fp32 to bfloat8_b tiles.
        {"name": "pack_4096_on_device", "path": "pack", "rows": 4096, "cols": 4096, "src": "float32", "dst": "bfloat8_b"},
        # The conversion benchmark itself: a host tensor to packed tiles on the device and back to the host.
        {"name": "host_round_trip_4096", "path": "host", "rows": 4096, "cols": 4096, "dst": "bfloat8_b"},
    ]


def _size(rng, low, high):
    """Log-uniform; a third each whole 128-column tiles, whole 32-element tiles, anything."""
    v = low * (high / low) ** rng.random()
    step = rng.choice([128, 32, 1])
    return int(min(high, max(low, round(v / step) * step)))


def draw(rng):
    path = rng.choice(["linear"] * 6 + ["layer"] * 2 + ["serve", "batched", "pack", "pack", "host"])
    block_float = rng.choice(["bfloat8_b", "bfloat8_b", "bfloat4_b"])
    if path == "linear":
        weight = rng.choice([block_float] * 5 + ["bfloat16"])
        activation, bias = rng.choice(["", "", "", "relu", "gelu", "silu"]), rng.random() < 0.4
        out = rng.choice(["bfloat16"] * 5 + ["float32"])
        while True:
            rows = int(round(2048 ** rng.random()))
            k, n = _size(rng, 512, 28672), _size(rng, 512, 28672)
            limit = 2048 * 8192 * 28672 if weight != "bfloat16" else 1 << 32
            if up32(rows) * k * n <= limit and k * n <= 8192 * 28672:
                return _linear(None, rows, k, n, weight, bias, activation, out)
    if path == "layer":
        hidden = int(round(_size(rng, 1024, 8192) / 64) * 64)
        return {"path": "layer", "rows": rng.choice([1, 8, 32, 32, 64, 128]), "hidden": hidden, "kv": max(128, hidden // rng.choice([1, 4, 8]) // 32 * 32),
                "ffn": int(hidden * rng.choice([2.6875, 3.5, 4])) // 32 * 32, "attn": "bfloat8_b", "mlp": rng.choice(["bfloat8_b", "bfloat4_b"]),
                "down": "bfloat8_b"}
    if path == "serve":
        return {"path": "serve", "rows": rng.choice([1, 4, 32, 33, 128]), "k": _size(rng, 256, 4096), "n": _size(rng, 256, 4096), "weight": block_float}
    if path == "batched":
        while True:
            c = {"path": "batched", "batch": rng.choice([8, 16, 32]), "m": up32(_size(rng, 32, 1024)), "k": rng.choice([64, 128]), "n": up32(_size(rng, 128, 1024))}
            if rng.random() < 0.5:
                c["k"], c["n"] = c["n"], c["k"]     # probabilities x values
            if c["batch"] * c["m"] * c["k"] * c["n"] <= 32 * 512 * 128 * 512 * 2:
                return c
    if path == "pack":
        return {"path": "pack", "rows": _size(rng, 128, 8192), "cols": _size(rng, 128, 8192), "src": rng.choice(["float32", "bfloat16"]),
                "dst": block_float}
    return {"path": "host", "rows": _size(rng, 64, 4096), "cols": _size(rng, 64, 4096), "dst": block_float}


# ---- inputs --------------------------------------------------------------------------------------------------------------
def _dtype(name):
    return getattr(ttnn, name)


def _on_device(t, dtype, device):
    """A torch tensor on the GPU as a tiled ttnn tensor of `dtype` on the device (packed there for the block-float types)."""
    src = ttnn._ttnn.wrap_device_memory(t.data_ptr(), ttnn.Shape(list(t.shape)), ttnn.float32 if t.dtype == torch.float32 else ttnn.bfloat16,
                                        ttnn.ROW_MAJOR_LAYOUT, device)
    return ttnn.to_layout(src, ttnn.TILE_LAYOUT, dtype=_dtype(dtype))


def _weight(g, k, n, dtype, device):
    w = torch.randn(k, n, generator=g, device="cuda", dtype=torch.float32).mul_(0.02)
    return _on_device(w if dtype != "bfloat16" else w.bfloat16(), dtype, device)


def _activation(g, shape, device):
    return _on_device(torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32).bfloat16(), "bfloat16", device)


def prepare(case, seed):
    torch.cuda.set_device(0)
    device = ttnn.open_device(0)
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = dict(case, device=device)
    path = case["path"]
    if path == "linear":
        s["w"] = _weight(g, case["k"], case["n"], case["weight"], device)
        s["x"] = _activation(g, (1, 1, case["rows"], case["k"]), device)
        s["b"] = _on_device(torch.randn(1, case["n"], generator=g, device="cuda").bfloat16(), "bfloat16", device) if case["bias"] else None
    elif path == "serve":
        s["w"] = _weight(g, case["k"], case["n"], case["weight"], device)
        s["x"] = torch.randn(1, 1, case["rows"], case["k"], generator=g, device="cuda").bfloat16().cpu()
    elif path == "layer":
        h, kv, f = case["hidden"], case["kv"], case["ffn"]
        for name, k, n, dtype in (("wq", h, h, case["attn"]), ("wk", h, kv, case["attn"]), ("wv", h, kv, case["attn"]), ("wo", h, h, case["attn"]),
                                  ("w1", h, f, case["mlp"]), ("w3", h, f, case["mlp"]), ("w2", f, h, case["down"])):
            s[name] = _weight(g, k, n, dtype, device)
        s["x"] = _activation(g, (1, 1, case["rows"], h), device)
    elif path == "batched":
        s["x"] = _activation(g, (1, case["batch"], case["m"], case["k"]), device)
        s["w"] = _activation(g, (1, case["batch"], case["k"], case["n"]), device)
    elif path == "pack":
        t = torch.randn(1, 1, case["rows"], case["cols"], generator=g, device="cuda", dtype=torch.float32).mul_(0.02)
        s["keep"] = t if case["src"] == "float32" else t.bfloat16()
        s["x"] = ttnn._ttnn.wrap_device_memory(s["keep"].data_ptr(), ttnn.Shape(list(t.shape)), _dtype(case["src"]), ttnn.ROW_MAJOR_LAYOUT, device)
    else:
        s["x"] = torch.randn(1, 1, case["rows"], case["cols"], generator=g, device="cuda", dtype=torch.float32).mul_(0.02).cpu()
    torch.cuda.synchronize()
    return s


# ---- one pass ------------------------------------------------------------------------------------------------------------
class _Buffer:
    """A ttnn tensor's device buffer under the CUDA array interface; keeps the tensor."""

    def __init__(self, t):
        self.tensor = t
        self.__cuda_array_interface__ = {"shape": (t.buffer_bytes(),), "typestr": "|u1", "data": (t.buffer_address(), False), "version": 2}


def _view(t, dtype):
    v = torch.as_tensor(_Buffer(t), device="cuda")
    return v if dtype is None else v.view(dtype)


def run(s):
    path = s["path"]
    if path == "linear":
        y = ttnn.linear(s["x"], s["w"], bias=s["b"], activation=s["activation"] or None, dtype=_dtype(s["out"]))
        return _view(y, torch.bfloat16 if s["out"] == "bfloat16" else torch.float32)
    if path == "serve":
        x = ttnn.from_torch(s["x"], layout=ttnn.TILE_LAYOUT, device=s["device"])
        return ttnn.to_torch(ttnn.linear(x, s["w"]))
    if path == "layer":
        q, k, v = ttnn.linear_multi(s["x"], [s["wq"], s["wk"], s["wv"]])
        o = ttnn.linear(q, s["wo"])
        y = ttnn.linear(ttnn.linear_gated(o, s["w1"], s["w3"], activation="silu"), s["w2"])
        return [_view(t, torch.bfloat16) for t in (k, v, y)]
    if path == "batched":
        return _view(ttnn.matmul(s["x"], s["w"]), torch.bfloat16)
    if path == "pack":
        return _view(ttnn.to_layout(s["x"], ttnn.TILE_LAYOUT, dtype=_dtype(s["dst"])), None)
    return ttnn.to_torch(ttnn.from_torch(s["x"], dtype=_dtype(s["dst"]), layout=ttnn.TILE_LAYOUT, device=s["device"]))


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------
def _weight_bytes(k, n, dtype):
    return up32(k) * up32(n) // 1024 * TILE_BYTES[dtype]


def work(case):
    path = case["path"]
    if path in ("linear", "serve"):
        rows, k, n = up32(case["rows"]), case["k"], case["n"]
        out = 4 if case.get("out") == "float32" else 2
        return {"bytes": _weight_bytes(k, n, case["weight"]) + rows * up32(k) * 2 + rows * up32(n) * out, "flops": 2 * rows * k * n}
    if path == "layer":
        rows, h, kv, f = up32(case["rows"]), case["hidden"], case["kv"], case["ffn"]
        shapes = [(h, h, "attn"), (h, kv, "attn"), (h, kv, "attn"), (h, h, "attn"), (h, f, "mlp"), (h, f, "mlp"), (f, h, "down")]
        return {"bytes": sum(_weight_bytes(k, n, case[d]) for k, n, d in shapes) + rows * (2 * h + 2 * kv) * 2,
                "flops": sum(2 * rows * k * n for k, n, _ in shapes)}
    if path == "batched":
        b, m, k, n = case["batch"], case["m"], case["k"], case["n"]
        return {"bytes": 2 * b * (m * k + k * n + m * n), "flops": 2 * b * m * k * n}
    elems = case["rows"] * case["cols"]
    if path == "pack":
        return {"bytes": elems * (4 if case["src"] == "float32" else 2) + _weight_bytes(case["rows"], case["cols"], case["dst"]), "flops": 0}
    return {"bytes": 8 * elems, "flops": 0}


def tolerance(case):
    path = case["path"]
    if path in ("pack", "host"):
        return "exact"                       # the packers' bytes are defined to the bit
    if path == "layer":
        return {"rel": 1.5e-2, "max": 0.07}  # four matmuls in a row, each result rounded to bfloat16; measured against 64 bits: 4.1e-3, 0.018
    if case.get("out") == "float32":
        # fp32 sums of exact products. Tensor cores cut what an addition shifts out instead of rounding it, so the error grows
        # with K: measured against 64 bits 3.4e-6 at K = 8192, 1.7e-5 at 28672 for one chain of additions (bfloat8_b, 512 rows).
        rel = 1e-6 + 2.5e-9 * case["k"]
        return {"rel": rel, "max": 10 * rel}
    return {"rel": 6.5e-3, "max": 0.016}     # one rounding to bfloat16; measured 1.7e-3, 3.9e-3


# ---- the same in 64 bits -------------------------------------------------------------------------------------------------
def _values(w, dtype):
    """The values a weight has after packing: per 16 elements of a row the largest exponent, mantissas of 7 or 3 bits rounded half up."""
    k, n = w.shape
    w = torch.nn.functional.pad(w, (0, up32(n) - n, 0, up32(k) - k)).double()
    if dtype == "bfloat16":
        return w
    bits = 7 if dtype == "bfloat8_b" else 3
    g = w.reshape(w.shape[0], -1, 16)
    e = torch.frexp(g.abs().amax(-1, keepdim=True))[1] - bits
    scale = torch.ldexp(torch.ones_like(g[..., :1]), e)
    return (torch.floor(g.abs() / scale + 0.5).clamp_(max=2 ** bits - 1) * scale * torch.sign(g)).reshape(w.shape)


def _tiled(t):
    """[..., rows, columns], both multiples of 32, in the order of a tiled buffer: 32x32 tiles of four 16x16 faces."""
    t = t.reshape(-1, t.shape[-2] // 32, 2, 16, t.shape[-1] // 32, 2, 16)
    return t.permute(0, 1, 4, 2, 5, 3, 6).reshape(-1)


def _act(v, name):
    return {"": lambda z: z, "relu": torch.relu, "gelu": torch.nn.functional.gelu, "silu": torch.nn.functional.silu}[name](v)


def exact(case, seed):
    path = case["path"]
    if path in ("pack", "host"):
        return None                          # compared to the bit
    g = torch.Generator(device="cuda").manual_seed(seed)

    def weight(k, n, dtype):
        w = torch.randn(k, n, generator=g, device="cuda", dtype=torch.float32).mul_(0.02)
        return _values(w if dtype != "bfloat16" else w.bfloat16(), dtype)

    def activation(*shape):
        x = torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32).bfloat16().double()
        return torch.nn.functional.pad(x, (0, up32(shape[-1]) - shape[-1], 0, up32(shape[-2]) - shape[-2]))

    if path == "linear":
        w = weight(case["k"], case["n"], case["weight"])
        y = activation(case["rows"], case["k"]) @ w
        if case["bias"]:
            y[:, :case["n"]] += torch.randn(1, case["n"], generator=g, device="cuda").bfloat16().double()
        return _tiled(_act(y, case["activation"]))
    if path == "serve":
        w = weight(case["k"], case["n"], case["weight"])
        x = torch.randn(1, 1, case["rows"], case["k"], generator=g, device="cuda").bfloat16().double()
        return (x @ w[:case["k"], :case["n"]]).cpu()
    if path == "layer":
        h, kv, f = case["hidden"], case["kv"], case["ffn"]
        wq, wk, wv, wo = (weight(h, n, case["attn"]) for n in (h, kv, kv, h))
        w1, w3, w2 = weight(h, f, case["mlp"]), weight(h, f, case["mlp"]), weight(f, h, case["down"])
        x = activation(case["rows"], h)
        o = x @ wq @ wo
        return [_tiled(t) for t in (x @ wk, x @ wv, (_act(o @ w1, "silu") * (o @ w3)) @ w2)]
    x = activation(case["batch"], case["m"], case["k"])
    return _tiled(x @ activation(case["batch"], case["k"], case["n"]))


if __name__ == "__main__":
    # How far the results lie from 64 bits: the source of the figures in tolerance().
    for case in [c for c in listed() if c["path"] not in ("pack", "host")] + [
            _linear("fp32 out", 64, 8192, 2048, "bfloat8_b", True, "gelu", "float32"), _linear("fp32 out bf16", 200, 1000, 2048, "bfloat16", out="float32")]:
        got, want = run(prepare(case, 1)), exact(case, 1)
        for y, t in zip(got, want) if case["path"] == "layer" else [(got, want)]:
            d, rms = torch.as_tensor(y).double().to(t.device) - t, t.square().mean().sqrt()
            print(case["name"], "rel %.3e max %.3e" % (float(d.norm() / t.norm()), float((d.abs() / torch.maximum(t.abs(), rms)).max())))
