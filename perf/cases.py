"""Workloads of the quantized matmul path, as programs that serve GGUF models call it.

One inference program keeps one device, one kernel registry and one command encoder; it encodes the products of a step,
commits and waits, because the next step (or the sampler) needs the result.  Weights are GGML blocks in HBM, activations
f32.  Kinds of cases:

  proj    one projection                       quantized_matmul_ggml
  layer   the projections of decoder layers    quantized_matmul_ggml, silu_mul; eager or as a captured graph
  head    the vocabulary projection, logits read by the host-side sampler
  perm    the O-projection on bf16 attention output [n_heads, seq, head_dim]   quantized_matmul_mm_tensor_perm021
  routed  one expert-routed projection         quantized_matmul_id_ggml
  moe     router, routed FFN, weighted sum     moe_softmax_topk, moe_ffn_layer, moe_weighted_reduce
"""
import math

import torch

import mlx_native_b200 as mx
from mlx_native_b200 import DType, GgmlType

# values per block, bytes per block
_GEOMETRY = {"q4_0": (32, 18), "q8_0": (32, 34), "q4_k": (256, 144), "q5_k": (256, 176), "q6_k": (256, 210)}
_TYPES = {"q4_0": GgmlType.Q4_0, "q8_0": GgmlType.Q8_0, "q4_k": GgmlType.Q4_K, "q5_k": GgmlType.Q5_K, "q6_k": GgmlType.Q6_K}
_SIGMA = 0.02  # standard deviation of the weights


def listed():
    return [
        # the smallest call of a decode step: the K or V projection for one token
        {"name": "proj_kv_q4_0_m1", "kind": "proj", "type": "q4_0", "m": 1, "n": 1024, "k": 4096},
        # five sequences decoded together; a width that is a multiple of 32 and not of 256, an odd number of rows
        {"name": "proj_ragged_q8_0_m5", "kind": "proj", "type": "q8_0", "m": 5, "n": 2873, "k": 2880},
        # autoregressive decode of one sequence: four decoder layers, encoded call by call
        {"name": "layers_decode_m1", "kind": "layer", "type": "q4_0", "down": "q6_k", "m": 1, "hidden": 4096, "kv": 1024, "ffn": 12288,
         "layers": 4, "graph": False},
        # a batch of eight sequences: the same layers in 8 bits, recorded once and replayed
        {"name": "layers_decode_m8_graph", "kind": "layer", "type": "q8_0", "down": "q8_0", "m": 8, "hidden": 4096, "kv": 1024, "ffn": 12288,
         "layers": 4, "graph": True},
        # the last product of every decode step: the largest matrix there is
        {"name": "head_q6_k_m1", "kind": "head", "type": "q6_k", "m": 1, "n": 151936, "k": 5120},
        # a prompt chunk of 512 tokens through one decoder layer
        {"name": "layer_prefill_m512", "kind": "layer", "type": "q4_0", "down": "q6_k", "m": 512, "hidden": 4096, "kv": 1024, "ffn": 12288,
         "layers": 1, "graph": False},
        # a long prompt: the down projection of 2048 tokens
        {"name": "proj_down_q6_k_m2048", "kind": "proj", "type": "q6_k", "m": 2048, "n": 4096, "k": 12288},
        # a prompt of ragged length reads the attention output where it lies
        {"name": "perm_o_q4_0_m333", "kind": "perm", "type": "q4_0", "m": 333, "n": 4096, "k": 4096, "head_dim": 128},
        # a short prompt in the K-quant that GGUF files use most
        {"name": "proj_q4_k_m96", "kind": "proj", "type": "q4_k", "m": 96, "n": 4096, "k": 4096},
        # mixture of experts: decode of one sequence, of a batch, and a prompt chunk
        {"name": "moe_decode_t1", "kind": "moe", "gate": "q4_0", "down": "q6_k", "tokens": 1, "experts": 128, "top_k": 8, "hidden": 2048,
         "ffn": 768},
        {"name": "moe_batch_t24", "kind": "moe", "gate": "q4_k", "down": "q8_0", "tokens": 24, "experts": 128, "top_k": 8, "hidden": 2048,
         "ffn": 768},
        {"name": "moe_prefill_t512", "kind": "moe", "gate": "q4_0", "down": "q6_k", "tokens": 512, "experts": 128, "top_k": 8, "hidden": 2048,
         "ffn": 768},
    ]


_MOST_FLOPS = 2.0 * 2048 * 4096 * 12288
_MOST_BYTES = 6.3e8


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rows(rng):
    """Activation rows of a step: decode (one sequence or a few) and prompts are met equally often."""
    return rng.choice((1, 1, 1, 2, 3, 4, 5, 6, 7, 8)) if rng.random() < 0.5 else _log(rng, 9, 2048)


def _width(rng, kind, lo=512, hi=14336):
    """An inner dimension: whole super-blocks for the K-quants; for 32-value blocks every other one is no multiple of 256."""
    k = _log(rng, lo, hi)
    step = 256 if _GEOMETRY[kind][0] == 256 or rng.random() < 0.5 else 32
    return max(step, k // step * step)


def _draw(rng):
    what = rng.choices(("proj", "layer", "moe", "head", "perm", "routed"), (8, 5, 5, 1, 1, 2))[0]
    if what == "proj":
        t = rng.choice(("q4_0", "q8_0", "q6_k", "q4_k"))
        n = _log(rng, 256, 16384)
        return {"kind": what, "type": t, "m": _rows(rng), "n": n if rng.random() < 0.3 else max(64, n // 64 * 64), "k": _width(rng, t)}
    if what == "head":
        t = rng.choice(("q4_0", "q8_0", "q6_k", "q4_k"))
        return {"kind": what, "type": t, "m": rng.choice((1, 1, 1, 2, 4)), "n": rng.choice((32000, 49157, 128256, 151936)),
                "k": rng.choice((1024, 2048, 2560, 4096, 5120))}
    if what == "perm":
        hd = rng.choice((64, 128, 256))
        return {"kind": what, "type": rng.choice(("q4_0", "q6_k")), "m": _log(rng, 9, 2048), "n": rng.choice((2048, 2560, 4096, 5120)),
                "k": rng.choice((2048, 3072, 4096, 5120)), "head_dim": hd}
    if what == "layer":
        t = rng.choice(("q4_0", "q8_0", "q6_k", "q4_k"))
        m, hidden = _rows(rng), rng.choice((1024, 2048, 2560, 3072, 4096, 5120))
        return {"kind": what, "type": t, "down": rng.choice((t, "q6_k")), "m": m, "hidden": hidden,
                "kv": rng.choice((512, 1024)), "ffn": max(512, int(hidden * rng.uniform(2.0, 4.0)) // 512 * 512),
                "layers": rng.choice((1, 2, 4)) if m <= 8 else 1, "graph": rng.random() < 0.4}
    if what == "routed":
        t = rng.choice(("q4_0", "q8_0", "q6_k", "q4_k", "q5_k"))
        return {"kind": what, "type": t, "tokens": _log(rng, 1, 32 if t == "q5_k" else 1024), "experts": rng.choice((16, 32, 64, 128)),
                "top_k": rng.choice((1, 2, 4, 8)), "n": _log(rng, 256, 3072) // 32 * 32, "k": _width(rng, t, 512, 3072)}
    gate, down = rng.choice(("q4_0", "q8_0", "q4_k", "q6_k")), rng.choice(("q4_0", "q8_0", "q6_k"))
    return {"kind": what, "gate": gate, "down": down, "tokens": _log(rng, 1, 1024), "experts": rng.choice((16, 32, 64, 128)),
            "top_k": rng.choice((2, 4, 8)), "hidden": rng.choice((1024, 1536, 2048, 2560)), "ffn": rng.choice((512, 768, 1024, 1536))}


def draw(rng):
    while True:
        case = _draw(rng)
        w = work(case)
        if w["flops"] <= _MOST_FLOPS and w["bytes"] <= _MOST_BYTES and _weight_bytes(case) <= 7e8 and work(case)["bytes"] > 1e5:
            return case


# ---------------------------------------------------------------- sizes
def _matrix_bytes(kind, n, k):
    values, size = _GEOMETRY[kind]
    return n * (k // values) * size


def _layer_shapes(case):
    """(name, type, n, k) of a decoder layer's projections."""
    t, h = case["type"], case["hidden"]
    return [("q", t, h, h), ("k", t, case["kv"], h), ("v", t, case["kv"], h), ("o", t, h, h), ("gate", t, case["ffn"], h),
            ("up", t, case["ffn"], h), ("down", case["down"], h, case["ffn"])]


def _weight_bytes(case):
    """All weights of a case, the experts that no token is routed to included."""
    kind = case["kind"]
    if kind == "layer":
        return case["layers"] * sum(_matrix_bytes(t, n, k) for _, t, n, k in _layer_shapes(case))
    if kind == "moe":
        h, f = case["hidden"], case["ffn"]
        return case["experts"] * (2 * _matrix_bytes(case["gate"], f, h) + _matrix_bytes(case["down"], h, f))
    return case.get("experts", 1) * _matrix_bytes(case["type"], case["n"], case["k"])


def work(case):
    """Weights that are needed read once (of the experts: those that some token is expected to choose), activations read
    once, results written once; two operations for each weight and row."""
    kind = case["kind"]
    if kind in ("moe", "routed"):
        tokens, e = case["tokens"], case["experts"]
        pairs = tokens * case["top_k"]
        used = e * (1 - (1 - case["top_k"] / e) ** tokens) / e
        if kind == "moe":
            h, f = case["hidden"], case["ffn"]
            return {"bytes": used * _weight_bytes(case) + 4 * tokens * (2 * h + e) + 8 * pairs, "flops": 6.0 * pairs * h * f}
        n, k = case["n"], case["k"]
        return {"bytes": used * _weight_bytes(case) + 4 * (tokens * k + pairs * n + pairs), "flops": 2.0 * pairs * n * k}
    m = case["m"]
    if kind == "layer":
        shapes = _layer_shapes(case)
        # read: the layer's input; written: what the caller gets (attention inputs and the layer's result)
        acts = 4 * m * (2 * case["hidden"] + case["hidden"] + 2 * case["kv"])
        return {"bytes": _weight_bytes(case) + case["layers"] * acts, "flops": case["layers"] * 2.0 * m * sum(n * k for _, _, n, k in shapes)}
    n, k = case["n"], case["k"]
    return {"bytes": _weight_bytes(case) + m * k * (2 if kind == "perm" else 4) + 4 * m * n, "flops": 2.0 * m * n * k}


def tolerance(case):
    """Products of up to 8 rows, of up to 32 routed tokens, and those of the K-quant that has no other form, are 32-bit sums of
    exact products; the larger ones round both operands to f16 (11 bits) and add up in 32."""
    kind = case["kind"]
    if kind == "moe":  # the down projection has a row for each (token, slot) pair
        return {"rel": 2e-5} if case["tokens"] * case["top_k"] <= 32 else {"rel": 2e-3}
    if kind == "routed":
        return {"rel": 1e-5} if case["tokens"] <= 32 else {"rel": 1e-3}
    if kind == "layer":
        return {"rel": 2e-5} if case["m"] <= 8 or case["type"] == case["down"] == "q4_k" else {"rel": 2e-3}
    exact = kind != "perm" and (case["m"] <= 8 or case["type"] == "q4_k")
    return {"rel": 1e-5} if exact else {"rel": 1e-3}


# ---------------------------------------------------------------- inputs
def _half_bytes(values):
    return values.to(torch.float16).contiguous().view(torch.uint8).reshape(*values.shape[:-1], 2)


def _codes(gen, blocks, values, centre, sigma, top):
    x = torch.randn(blocks, values, generator=gen, device="cuda")
    return x.mul_(sigma).add_(centre).round_().clamp_(0, top).to(torch.uint8)


def _scales(gen, blocks, middle):
    """One scale for each block, spread as the largest magnitudes of blocks of normal weights are."""
    return (torch.randn(blocks, 1, generator=gen, device="cuda") * 0.12).exp_() * middle


def _k_scales(gen, blocks):
    """Eight 6-bit scales and eight 6-bit minima, packed into 12 bytes as in Q4_K and Q5_K."""
    sc = torch.randint(38, 64, (blocks, 8), generator=gen, device="cuda", dtype=torch.uint8)
    mn = torch.randint(38, 64, (blocks, 8), generator=gen, device="cuda", dtype=torch.uint8)
    lo = torch.cat([sc[:, :4] | (sc[:, 4:] >> 4 << 6), mn[:, :4] | (mn[:, 4:] >> 4 << 6)], dim=1)
    return torch.cat([lo, (sc[:, 4:] & 15) | ((mn[:, 4:] & 15) << 4)], dim=1)


def _blocks(gen, kind, blocks):
    """Random GGML blocks whose weights are close to N(0, _SIGMA)."""
    if kind == "q4_0":
        q = _codes(gen, blocks, 32, 8, 3.4, 15)
        return torch.cat([_half_bytes(_scales(gen, blocks, _SIGMA / 3.4)), q[:, :16] | (q[:, 16:] << 4)], dim=1)
    if kind == "q8_0":
        q = _codes(gen, blocks, 32, 128, 54, 255)
        return torch.cat([_half_bytes(_scales(gen, blocks, _SIGMA / 54)), q ^ 128], dim=1)
    if kind == "q6_k":
        q = _codes(gen, blocks, 256, 32, 16, 63).view(blocks, 2, 4, 32)
        ql = torch.cat([(q[:, :, 0] & 15) | ((q[:, :, 2] & 15) << 4), (q[:, :, 1] & 15) | ((q[:, :, 3] & 15) << 4)], dim=2)
        h = q >> 4
        qh = h[:, :, 0] | (h[:, :, 1] << 2) | (h[:, :, 2] << 4) | (h[:, :, 3] << 6)
        sc = torch.randint(72, 128, (blocks, 16), generator=gen, device="cuda", dtype=torch.int16)
        sign = torch.randint(0, 2, (blocks, 16), generator=gen, device="cuda", dtype=torch.int16) * 2 - 1
        sc = (sc * sign).to(torch.int8).view(torch.uint8)
        return torch.cat([ql.reshape(blocks, 128), qh.reshape(blocks, 64), sc, _half_bytes(_scales(gen, blocks, _SIGMA / 1600))], dim=1)
    five = kind == "q5_k"
    centre = 15.5 if five else 7.5
    q = _codes(gen, blocks, 256, centre, centre / 2, 31 if five else 15).view(blocks, 4, 2, 32)
    d = _scales(gen, blocks, _SIGMA / (centre / 2 * 50))
    parts = [_half_bytes(d), _half_bytes(d * centre), _k_scales(gen, blocks)]
    if five:
        bit = (q >> 4).view(blocks, 8, 32) << torch.arange(8, device="cuda", dtype=torch.uint8).view(1, 8, 1)
        parts.append(bit.sum(dim=1, dtype=torch.uint8))
    parts.append(((q[:, :, 0] & 15) | ((q[:, :, 1] & 15) << 4)).reshape(blocks, 128))
    return torch.cat(parts, dim=1)


def _weights(gen, kind, n, k):
    values, size = _GEOMETRY[kind]
    total = n * (k // values)
    out = torch.empty(total, size, dtype=torch.uint8, device="cuda")
    step = (1 << 26) // values
    for at in range(0, total, step):
        some = min(step, total - at)
        out[at:at + some] = _blocks(gen, kind, some)
    return out


# ---------------------------------------------------------------- the program
_program = {}


def _handles():
    """The device, registry and encoder that an inference program makes once."""
    if not _program:
        device = mx.MlxDevice.new()
        _program.update(device=device, registry=mx.KernelRegistry.new(), encoder=device.command_encoder())
    return _program["device"], _program["registry"], _program["encoder"]


class _State:
    """Tensors of a case and the library's buffers over their memory."""

    def __init__(self, case, seed):
        self.case = case
        self.device, self.registry, self.encoder = _handles()
        self.gen = torch.Generator(device="cuda").manual_seed(seed * 1000003 + 17)
        self.tensors, self.buffers, self.params, self.graph, self.result = {}, {}, {}, None, None

    def add(self, name, tensor, dtype):
        self.tensors[name] = tensor
        self.buffers[name] = self.device.wrap_device_memory(tensor.data_ptr(), tensor.numel() * tensor.element_size(), dtype, list(tensor.shape))

    def weights(self, name, kind, n, k):
        self.add(name, _weights(self.gen, kind, n, k), DType.U8)

    def normal(self, name, *shape):
        self.add(name, torch.randn(*shape, generator=self.gen, device="cuda"), DType.F32)

    def empty(self, name, *shape):
        self.add(name, torch.zeros(*shape, device="cuda"), DType.F32)

    def multiply(self, x, w, y):
        b = self.buffers
        mx.quantized_matmul_ggml(self.encoder, self.registry, self.device, b[x], b[w], b[y], self.params[w])


def prepare(case, seed):
    s = _State(case, seed)
    kind = case["kind"]
    if kind in ("proj", "head", "perm"):
        m, n, k, t = case["m"], case["n"], case["k"], case["type"]
        s.weights("w", t, n, k)
        s.empty("y", m, n)
        if kind == "perm":
            hd = case["head_dim"]
            s.add("x", torch.randn(k // hd, m, hd, generator=s.gen, device="cuda").to(torch.bfloat16), DType.BF16)
            s.params["w"] = mx.GgmlQuantizedMatmulPerm021Params(m, n, k, hd, _TYPES[t])
        else:
            s.normal("x", m, k)
            s.params["w"] = mx.GgmlQuantizedMatmulParams(m, n, k, _TYPES[t])
        if kind == "head":
            s.buffers["y"].as_slice()  # the sampler looks at the logits: every commit brings them back
        s.result = s.tensors["y"]
    elif kind == "layer":
        m = case["m"]
        for i in range(case["layers"]):
            s.normal("x%d" % i, m, case["hidden"])
            for name, t, n, k in _layer_shapes(case):
                s.weights("w_%s%d" % (name, i), t, n, k)
                s.empty("%s%d" % (name, i), m, n)
                s.params["w_%s%d" % (name, i)] = mx.GgmlQuantizedMatmulParams(m, n, k, _TYPES[t])
            s.empty("act%d" % i, m, case["ffn"])
        s.result = {name + str(i): s.tensors[name + str(i)] for i in range(case["layers"]) for name in ("q", "k", "v", "down")}
        if case["graph"]:
            _encode_layers(s)  # eagerly once, then recorded
            s.encoder.commit_and_wait()
            s.encoder.begin_capture()
            _encode_layers(s)
            s.graph = s.encoder.end_capture()
    elif kind == "routed":
        tokens, e, top_k, n, k, t = case["tokens"], case["experts"], case["top_k"], case["n"], case["k"], case["type"]
        s.weights("w", t, e * n, k)
        s.normal("x", tokens, k)
        ids = torch.rand(tokens, e, generator=s.gen, device="cuda").topk(top_k, dim=1).indices
        s.add("ids", ids.to(torch.int32).contiguous(), DType.U32)
        s.empty("y", tokens * top_k, n)
        s.params["w"] = mx.GgmlQuantizedMatmulIdParams(tokens, top_k, n, k, e, _matrix_bytes(t, n, k), _TYPES[t])
        s.result = s.tensors["y"]
    else:
        tokens, e, top_k, h, f = case["tokens"], case["experts"], case["top_k"], case["hidden"], case["ffn"]
        g, d = case["gate"], case["down"]
        s.weights("w_gate", g, e * f, h)
        s.weights("w_up", g, e * f, h)
        s.weights("w_down", d, e * h, f)
        s.normal("x", tokens, h)
        s.normal("logits", tokens, e)
        s.add("ids", torch.zeros(tokens, top_k, dtype=torch.int32, device="cuda"), DType.U32)
        s.empty("shares", tokens, top_k)
        s.empty("gate", tokens * top_k, f)
        s.empty("up", tokens * top_k, f)
        s.empty("down", tokens * top_k, h)
        s.empty("y", tokens, h)
        s.params["ffn"] = mx.MoeFfnLayerParams(tokens, top_k, h, f, e, _TYPES[g], _TYPES[g], _TYPES[d], _matrix_bytes(g, f, h),
                                               _matrix_bytes(g, f, h), _matrix_bytes(d, h, f))
        s.result = {name: s.tensors[name] for name in ("ids", "shares", "y")}
    return s


def _encode_layers(s):
    """The attention and the norms between the products are other kernels of the program: a product reads what it would have
    been given by them, and a barrier stands between layers."""
    case = s.case
    for i in range(case["layers"]):
        at = str(i)
        if i:
            s.encoder.memory_barrier()
        for name in ("q", "k", "v"):
            s.multiply("x" + at, "w_" + name + at, name + at)
        s.multiply("q" + at, "w_o" + at, "o" + at)
        s.multiply("o" + at, "w_gate" + at, "gate" + at)
        s.multiply("o" + at, "w_up" + at, "up" + at)
        b = s.buffers
        mx.silu_mul(s.encoder, s.registry, s.device, b["gate" + at], b["up" + at], b["act" + at], case["m"] * case["ffn"])
        s.multiply("act" + at, "w_down" + at, "down" + at)


def run(state):
    s, case, b = state, state.case, state.buffers
    kind = case["kind"]
    if kind == "layer":
        if s.graph is not None:
            s.graph.launch(s.encoder)
        else:
            _encode_layers(s)
    elif kind in ("proj", "head"):
        s.multiply("x", "w", "y")
    elif kind == "perm":
        mx.quantized_matmul_mm_tensor_perm021(s.encoder, s.registry, s.device, b["x"], b["w"], b["y"], s.params["w"])
    elif kind == "routed":
        mx.quantized_matmul_id_ggml(s.encoder, s.registry, s.device, b["x"], b["w"], b["ids"], b["y"], s.params["w"])
    else:
        mx.moe_softmax_topk(s.encoder, s.registry, s.device, b["logits"], b["ids"], b["shares"], case["tokens"], case["experts"], case["top_k"])
        mx.moe_ffn_layer(s.encoder, s.registry, s.device, b["x"], b["ids"], b["w_gate"], b["w_up"], b["w_down"], b["gate"], b["up"], b["down"],
                         s.params["ffn"])
        mx.moe_weighted_reduce(s.encoder, s.registry, s.device, b["shares"], b["down"], b["y"], case["tokens"], case["top_k"], case["hidden"])
    s.encoder.commit_and_wait()  # the next step starts from these results
    return b["y"].as_slice() if kind == "head" else s.result
