"""The work whose speed counts: what a program that serves a quantized model has this framework do, through its public
entry points (nn.Linear, nn.SparseMoE, DecodeGraph, ops).

A case is one pass of one of five kinds:

    linear      one quantized matrix, nn.Linear.forward
    layer       the matrices of one decoder layer on a batch of tokens: q,k,v as one, o, gate and up as one, the gated
                activation, down.  Formats: GGUF Q4_K_M (down Q6_K), GGUF Q8_0, 4-bit group-128 (GPTQ / AWQ), block FP8
    step        one token of one sequence through DecodeGraph (embedding, layers with attention over a KV cache, lm_head,
                argmax): what a chat session runs per token
    moe         a routed sparse block, nn.SparseMoE.forward: router, top-k, grouped matmuls, combine
    attention   rotary embedding, KV append and attention of a decode step, ops.DecodeAttention

Every kind runs from one token (decode) over batched decode and short, odd-length prompts to long prompts.
"""
import math

import torch

from light_b200 import ops, synth
from light_b200.decode import DecodeGraph, LlamaConfig, LlamaLayer
from light_b200.nn import Linear, SparseMoE

DEVICE = "cuda"
GROUP = 128                       # int4 group, and the FP8 scale block's side
BIAS = 0.05                       # of the sigmoid router's bias per expert: near a top-8 score's 0.9 as much as half a logit
Q4KM, Q80, INT4, FP8 = "q4_k_m", "q8_0", "int4", "fp8"
BITS = {ops.Q4_K: 144 * 8 / 256, ops.Q6_K: 210 * 8 / 256, ops.Q8_0: 34 * 8 / 32}


def listed():
    llama8b = {"hidden": 4096, "inter": 14336, "qkv": 6144}
    qwen7b = {"hidden": 3584, "inter": 18944, "qkv": 4608}
    deepseek = {"format": FP8, "hidden": 7168, "inter": 2048, "experts": 256, "topk": 8}
    return [
        # one projection for one token: the smallest call a program makes, latency and nothing else
        {"name": "linear_q4k_1", "kind": "linear", "format": Q4KM, "n": 4096, "k": 4096, "tokens": 1},
        # one chat session on an 8B-shaped Q4_K_M model (24 of its layers), 1024 tokens into the conversation
        {"name": "step_q4km", "kind": "step", "layers": 24, "hidden": 4096, "inter": 14336, "heads": 32, "kv_heads": 8, "head_dim": 128,
         "vocab": 128256, "position": 1024},
        # batched decode of 32 sessions
        {"name": "layer_q4km_32", "kind": "layer", "format": Q4KM, "tokens": 32, **llama8b},
        # an ordinary prompt, of an odd length
        {"name": "layer_q4km_333", "kind": "layer", "format": Q4KM, "tokens": 333, **llama8b},
        # a long prompt
        {"name": "layer_q4km_2048", "kind": "layer", "format": Q4KM, "tokens": 2048, **llama8b},
        # one token through an 8-bit model
        {"name": "layer_q80_1", "kind": "layer", "format": Q80, "tokens": 1, **llama8b},
        # one token, and a long prompt, through a GPTQ / AWQ model
        {"name": "layer_int4_1", "kind": "layer", "format": INT4, "tokens": 1, **qwen7b},
        {"name": "layer_int4_4096", "kind": "layer", "format": INT4, "tokens": 4096, **qwen7b},
        # a sparse block with block-FP8 experts: eight sessions decoding, and a long prompt
        {"name": "moe_fp8_8", "kind": "moe", "tokens": 8, **deepseek},
        {"name": "moe_fp8_4096", "kind": "moe", "tokens": 4096, **deepseek},
        # a sparse block with GGUF experts on a short prompt
        {"name": "moe_q4km_77", "kind": "moe", "format": Q4KM, "tokens": 77, "hidden": 2048, "inter": 768, "experts": 128, "topk": 8},
        # eight sessions deep into long conversations
        {"name": "attention_bf16_8x8192", "kind": "attention", "dtype": "bf16", "batch": 8, "heads": 32, "kv_heads": 8, "head_dim": 128,
         "context": 8192, "window": 0},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _multiple(rng, step, lo, hi):
    return step * rng.randint(lo // step, hi // step)


def draw(rng):
    kind = rng.choice(["linear", "layer", "layer", "layer", "step", "moe", "moe", "attention"])
    if kind == "linear":
        return {"kind": kind, "format": rng.choice([Q4KM, Q80, INT4, FP8]), "n": _multiple(rng, 128, 1024, 16384), "k": _multiple(rng, 256, 1024, 8192),
                "tokens": _spread(rng, 1, 512)}
    if kind == "layer":
        hidden = _multiple(rng, 256, 1024, 4096)
        return {"kind": kind, "format": rng.choice([Q4KM, Q80, INT4, FP8]), "tokens": _spread(rng, 1, 4096), "hidden": hidden,
                "inter": 256 * round(hidden * rng.uniform(2.5, 4.0) / 256), "qkv": hidden + 256 * rng.randint(1, hidden // 256)}
    if kind == "step":
        head_dim = rng.choice([64, 128])
        hidden = _multiple(rng, 512, 1024, 4096)
        heads = hidden // head_dim
        return {"kind": kind, "layers": rng.randint(2, 24), "hidden": hidden, "inter": _multiple(rng, 256, 2048, 14336), "heads": heads,
                "kv_heads": heads // rng.choice([1, 2, 4]), "head_dim": head_dim, "vocab": 32 * rng.randint(1000, 4008), "position": _spread(rng, 1, 4000)}
    if kind == "moe":
        return {"kind": kind, "format": rng.choice([FP8, FP8, Q4KM]), "tokens": _spread(rng, 1, 4096), "hidden": _multiple(rng, 256, 1024, 4096),
                "inter": _multiple(rng, 256, 512, 2048), "experts": 8 * rng.randint(1, 32), "topk": rng.randint(1, 8)}
    kv_heads = rng.choice([1, 2, 4, 8])
    return {"kind": kind, "dtype": rng.choice(["bf16", "f32"]), "batch": _spread(rng, 1, 16), "heads": kv_heads * rng.choice([1, 2, 4, 8]), "kv_heads": kv_heads,
            "head_dim": rng.choice([64, 128]), "context": _spread(rng, 64, 8192), "window": rng.choice([0, 0, 1024])}


# ---------------------------------------------------------------- inputs


class _Seeds:
    """Seeds of a case's tensors, one after the other, all from the case's own."""

    def __init__(self, seed):
        self.next = seed * 1009

    def __call__(self):
        self.next += 1
        return self.next

    def gen(self):
        return torch.Generator(device=DEVICE).manual_seed(self())

    def normal(self, *shape, dtype=torch.float32):
        return torch.randn(*shape, generator=self.gen(), device=DEVICE).to(dtype)

    def gguf(self, ggml_type, *shape):
        n = math.prod(shape[:-1])
        return ops.QTensor(synth.gaussian_weight(self(), ggml_type, n, shape[-1], device=DEVICE).reshape(-1), ggml_type, tuple(shape))

    def int4(self, n, k):
        g = self.gen()
        codes = torch.randint(-2**31, 2**31, (n, k // 8), generator=g, device=DEVICE, dtype=torch.int32)
        scales = (torch.rand(n, k // GROUP, generator=g, device=DEVICE) * 0.015 + 0.005).half().float()
        zeros = torch.randint(0, 16, (n, k // GROUP), generator=g, device=DEVICE).float()
        return ops.Int4(codes, scales, zeros, GROUP)

    def fp8(self, *shape):
        n, k = math.prod(shape[:-1]), shape[-1]
        codes = torch.empty(n, k, dtype=torch.uint8, device=DEVICE)
        scale = torch.empty(n // GROUP, k // GROUP, device=DEVICE)
        for r in range(0, n, 128 * 512):   # a few hundred MB of f32 at a time
            e = min(n, r + 128 * 512)
            codes[r:e], scale[r // GROUP:e // GROUP] = synth.random_fp8_block(self(), e - r, k, device=DEVICE)
        return codes.view(torch.float8_e4m3fn).reshape(shape), scale.reshape(*shape[:-2], shape[-2] // GROUP, k // GROUP)


def _act(case):
    """The activations' type: GGUF weights take F32, the 4-bit and FP8 ones BF16."""
    return torch.float32 if case["format"] in (Q4KM, Q80) else torch.bfloat16


def _linear(s, fmt, n, k, down=False):
    if fmt == INT4:
        return Linear(k, n, W4=s.int4(n, k))
    if fmt == FP8:
        w, scale = s.fp8(n, k)
        return Linear(k, n, W=w, WBlockScale=scale, WBlock=(GROUP, GROUP))
    return Linear(k, n, W=s.gguf(ops.Q8_0 if fmt == Q80 else ops.Q6_K if down else ops.Q4_K, n, k))


def prepare(case, seed):
    s = _Seeds(seed)
    return {"kind": case["kind"], **globals()["_prepare_" + case["kind"]](case, s)}


def _prepare_linear(c, s):
    return {"linear": _linear(s, c["format"], c["n"], c["k"]), "x": s.normal(c["tokens"], c["k"], dtype=_act(c))}


def _prepare_layer(c, s):
    H, I, f, T = c["hidden"], c["inter"], c["format"], c["tokens"]
    return {"qkv": _linear(s, f, c["qkv"], H), "o": _linear(s, f, H, H), "gate_up": _linear(s, f, 2 * I, H), "down": _linear(s, f, H, I, down=True),
            "x": s.normal(T, H, dtype=_act(c)), "attn": s.normal(T, H, dtype=_act(c)), "normed": s.normal(T, H, dtype=_act(c))}


def _prepare_step(c, s):
    H, I, NH, KH, D = c["hidden"], c["inter"], c["heads"], c["kv_heads"], c["head_dim"]
    norm = lambda: 1.0 + 0.1 * s.normal(H)  # noqa: E731
    layers = [LlamaLayer(q=s.gguf(ops.Q4_K, NH * D, H), k=s.gguf(ops.Q4_K, KH * D, H), v=s.gguf(ops.Q4_K, KH * D, H), o=s.gguf(ops.Q4_K, H, NH * D),
                         gate=s.gguf(ops.Q4_K, I, H), up=s.gguf(ops.Q4_K, I, H), down=s.gguf(ops.Q6_K, H, I), attn_norm=norm(), ffn_norm=norm())
              for _ in range(c["layers"])]
    cap = (c["position"] // 1024 + 1) * 1024
    g = DecodeGraph(LlamaConfig(H, NH, KH, D), layers, norm(), s.gguf(ops.Q6_K, c["vocab"], H), s.gguf(ops.Q4_K, c["vocab"], H), cap, torch.device(DEVICE, 0))
    for buf in g.kbuf + g.vbuf:   # the conversation so far
        buf[:, :, :c["position"]] = s.normal(1, KH, c["position"], D)
    token = s() % c["vocab"]
    g.reset(token, c["position"])
    g.capture()
    return {"graph": g, "token": token, "position": c["position"]}


def _prepare_moe(c, s):
    H, I, E, k, T = c["hidden"], c["inter"], c["experts"], c["topk"], c["tokens"]
    gate = Linear(H, E, W=s.normal(E, H) / math.sqrt(H))
    if c["format"] == FP8:   # sigmoid scores and a bias per expert for the choice, F32 router on BF16 activations
        (gu, gs), (dn, ds) = s.fp8(E, 2 * I, H), s.fp8(E, H, I)
        bias = BIAS * s.normal(E)
        moe = SparseMoE(gate, gu, dn, TopK=k, RouterF32=True, Router=lambda logits: ops.MoERouteSigmoid(logits, bias, k), GateUpScale=gs, DownScale=ds,
                        Block=(GROUP, GROUP))
    else:
        moe = SparseMoE(gate, s.gguf(ops.Q4_K, E, 2 * I, H), s.gguf(ops.Q6_K, E, H, I), TopK=k, NormTopK=True)
    return {"moe": moe, "x": s.normal(T, H, dtype=_act(c))}


def _prepare_attention(c, s):
    dt = torch.bfloat16 if c["dtype"] == "bf16" else torch.float32
    B, NH, KH, D, n = c["batch"], c["heads"], c["kv_heads"], c["head_dim"], c["context"]
    kbuf, vbuf = s.normal(B, KH, n, D, dtype=dt), s.normal(B, KH, n, D, dtype=dt)
    return {"q": s.normal(B, NH, 1, D, dtype=dt), "k": s.normal(B, KH, 1, D, dtype=dt), "v": s.normal(B, KH, 1, D, dtype=dt), "kbuf": kbuf, "vbuf": vbuf,
            "pos": torch.full((1,), n - 1, dtype=torch.int64, device=DEVICE), "scale": 1.0 / math.sqrt(D), "window": c["window"]}


# ---------------------------------------------------------------- one pass


def run(s):
    return globals()["_run_" + s["kind"]](s)


def _run_linear(s):
    return s["linear"].forward(s["x"])


def _run_layer(s):
    qkv = s["qkv"].forward(s["x"])
    o = s["o"].forward(s["attn"])
    return qkv, o, s["down"].forward(ops.MoEGateMul(s["gate_up"].forward(s["normed"])))


def _run_step(s):
    g = s["graph"]
    g.reset(s["token"], s["position"])
    g.step()
    return {"logits": g.logits, "token": g.token, "position": g.pos, "k": g.kbuf, "v": g.vbuf}


def _run_moe(s):
    return s["moe"].forward(s["x"])


def _run_attention(s):
    out = ops.DecodeAttention(s["q"], s["kbuf"], s["vbuf"], s["pos"], s["scale"], s["window"], s["k"], s["v"], rope_base=500000.0)
    return out, s["kbuf"], s["vbuf"]


# ---------------------------------------------------------------- what a pass needs, and how exact it is


def _weight_bytes(fmt, n, k, down=False):
    if fmt == INT4:
        return n * k / 2 + n * (k / GROUP) * 8
    if fmt == FP8:
        return n * k + n * k / GROUP**2 * 4
    return n * k * BITS[ops.Q8_0 if fmt == Q80 else ops.Q6_K if down else ops.Q4_K] / 8


def _experts_used(c):
    """How many experts some token chooses, from a router with scores like the case's."""
    g = torch.Generator().manual_seed(1)
    bias = BIAS * torch.randn(c["experts"], generator=g) if c["format"] == FP8 else 0.0
    scores = torch.randn(c["tokens"], c["experts"], generator=g).sigmoid() + bias
    return scores.topk(c["topk"], -1).indices.unique().numel()


def work(case):
    c = case
    if c["kind"] == "linear":
        n, k, T = c["n"], c["k"], c["tokens"]
        return {"bytes": _weight_bytes(c["format"], n, k) + T * (n + k) * _act(c).itemsize, "flops": 2 * T * n * k}
    if c["kind"] == "layer":
        H, I, T, f = c["hidden"], c["inter"], c["tokens"], c["format"]
        shapes = [(c["qkv"], H, False), (H, H, False), (2 * I, H, False), (H, I, True)]
        weights = sum(_weight_bytes(f, n, k, d) for n, k, d in shapes)
        return {"bytes": weights + T * (5 * H + c["qkv"]) * _act(c).itemsize, "flops": sum(2 * T * n * k for n, k, _ in shapes)}
    if c["kind"] == "step":
        H, I, L = c["hidden"], c["inter"], c["layers"]
        kv = c["kv_heads"] * c["head_dim"]
        per_layer = [(H + 2 * kv, H, False), (H, H, False), (2 * I, H, False), (H, I, True)]
        shapes = per_layer * L + [(c["vocab"], H, True)]
        cache = L * 2 * kv * (c["position"] + 2) * 4
        return {"bytes": sum(_weight_bytes(Q4KM, n, k, d) for n, k, d in shapes) + cache + (2 * L + 1) * H * 4 + c["vocab"] * 4,
                "flops": sum(2 * n * k for n, k, _ in shapes) + L * 4 * H * (c["position"] + 1)}
    if c["kind"] == "moe":
        H, I, E, T, k = c["hidden"], c["inter"], c["experts"], c["tokens"], c["topk"]
        used = _experts_used(c)
        expert = _weight_bytes(c["format"], 2 * I, H) + _weight_bytes(c["format"], H, I, True)
        return {"bytes": used * expert + E * H * 4 + 2 * T * H * _act(c).itemsize, "flops": 2 * T * (k * 3 * I * H + E * H)}
    B, NH, KH, D = c["batch"], c["heads"], c["kv_heads"], c["head_dim"]
    n = min(c["context"], c["window"] or c["context"])
    size = 2 if c["dtype"] == "bf16" else 4
    return {"bytes": B * D * size * (2 * KH * n + 2 * KH + 2 * NH), "flops": 4 * B * NH * n * D}


def tolerance(case):
    c = case
    if c["kind"] == "attention":
        return {"rel": 1e-2} if c["dtype"] == "bf16" else {"rel": 1e-5}
    if c["kind"] == "step":
        return {"rel": 2e-3}     # two dozen layers of F32 arithmetic on the weights, one after the other
    if _act(c) == torch.bfloat16:
        return {"rel": 1e-2}
    if c["tokens"] == 1 and c["kind"] != "moe":
        return {"rel": 2e-4}     # F32 activations against the weights as they are stored
    return {"rel": 2e-3}         # operands rounded to 11 bits for the tensor cores, F32 sums, two matrices one after the other
