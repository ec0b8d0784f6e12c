"""The work this library is measured on: its linears, its attention and a model's step, through the C
ABI and the Python wrappers a program would call.

A case is a dict of plain values whose "path" names one of the ways in:

    fp8_matmul    a 16-bit activation times an e4m3 weight with one scale (fl_fp8_matmul[_add]):
                  what the reference's decoder and UNet layers call; one row while decoding, a
                  prompt's rows in a prefill, an image's rows in a denoise step
    fp8_linear    activation quantised on the fly, per-channel scales (fl_fp8_linear)
    fp8_mlp       two of those, GELU between them, the input added to the result
    nvfp4_linear  block-scaled four-bit weight and activation (fl_nvfp4_linear)
    attention     fl_attention on strided views, with and without a mask
    denoise       MMDiT: the ways in and the blocks over text and image tokens

Weights are quantised once in prepare(), as a program quantises them when it loads a model; outputs
are preallocated where the entry point takes them. All sizes are in elements.
"""
import math

import torch

from libwaifu_b200 import flint as F
from libwaifu_b200.mmdit import FlintBackend, MMDiT, MMDiTConfig

TORCH_TYPE = {"f16": torch.float16, "bf16": torch.bfloat16}
FLINT_TYPE = {"f16": F.DType.FLOAT16, "bf16": F.DType.BFLOAT16}


def listed():
    return [
        # One token through a square projection: the smallest product the decoder asks for.
        {"name": "decode_row", "path": "fp8_matmul", "m": 1, "n": 3072, "k": 3072, "type": "f16", "addend": "none"},
        # A batch of sixteen sequences decoding through the gated MLP's wide projection.
        {"name": "decode_batch", "path": "fp8_matmul", "m": 16, "n": 16384, "k": 3072, "type": "f16", "addend": "bias"},
        # The adaLN modulation of a guided denoise step: two rows against six times the width.
        {"name": "modulation", "path": "fp8_linear", "m": 2, "n": 18432, "k": 3072, "type": "bf16", "bias": True,
         "residual": False, "gelu": False},
        # A 77-token prompt's keys and values for cross attention.
        {"name": "prompt_kv", "path": "fp8_matmul", "m": 77, "n": 2560, "k": 2048, "type": "f16", "addend": "none"},
        # A 512-token prompt's fused q/k/v projection in bfloat16, the stream added.
        {"name": "prefill", "path": "fp8_matmul", "m": 512, "n": 5120, "k": 3072, "type": "bf16", "addend": "residual"},
        # An image's 4096 rows through the MLP's up projection with a bias.
        {"name": "image_ff", "path": "fp8_matmul", "m": 4096, "n": 12288, "k": 3072, "type": "f16", "addend": "bias"},
        # An image's rows through a square projection, activations quantised per token.
        {"name": "image_linear", "path": "fp8_linear", "m": 4096, "n": 3072, "k": 3072, "type": "bf16", "bias": True,
         "residual": False, "gelu": False},
        # The MLP of a joint text and image stream: 4096 + 256 tokens.
        {"name": "joint_mlp", "path": "fp8_mlp", "m": 4352, "hidden": 3072, "inner": 12288, "type": "bf16"},
        # The fused q/k/v projection of the same stream in four bits.
        {"name": "joint_qkv_fp4", "path": "nvfp4_linear", "m": 4352, "n": 9216, "k": 3072, "type": "bf16", "bias": False},
        # A batch of prompts through a decoder's prefill: grouped heads, causal, a ragged length.
        {"name": "attention_prefill", "path": "attention", "batch": 4, "heads": 32, "kv_heads": 8, "q_len": 1000,
         "kv_len": 1000, "head_dim": 128, "causal": True, "type": "f16"},
        # The joint attention of a guided denoise step: two rows of 4096 + 256 tokens.
        {"name": "attention_joint", "path": "attention", "batch": 2, "heads": 24, "kv_heads": 24, "q_len": 4352,
         "kv_len": 4352, "head_dim": 128, "causal": False, "type": "bf16"},
        # A guided denoise step of a 1024 x 1024 image: the ways in and two of its blocks.
        {"name": "denoise", "path": "denoise", "batch": 2, "text_tokens": 256, "image_tokens": 4096, "blocks": 2},
    ]


def _log_int(rng, low, high, step=1):
    """Spread over the logarithm of [low, high], rounded down to a multiple of `step`."""
    value = math.exp(rng.uniform(math.log(low), math.log(high + step)))
    return int(min(high, max(low, int(value) // step * step)))


def draw(rng):
    path = rng.choice(["fp8_matmul", "fp8_matmul", "fp8_linear", "fp8_linear", "fp8_mlp", "nvfp4_linear", "attention", "denoise"])
    kind = rng.choice(["f16", "bf16"])
    if path == "fp8_matmul":
        # (the reference's layers: rows a multiple of 8, k of 16)
        return {"path": path, "m": _log_int(rng, 1, 4096), "n": _log_int(rng, 1280, 16384, 8), "k": _log_int(rng, 640, 4096, 16),
                "type": kind, "addend": rng.choice(["none", "bias", "residual"])}
    if path == "fp8_linear":
        return {"path": path, "m": _log_int(rng, 1, 8704), "n": _log_int(rng, 640, 18432, 8), "k": _log_int(rng, 256, 12288, 16),
                "type": kind, "bias": rng.random() < 0.8, "residual": rng.random() < 0.3, "gelu": rng.random() < 0.3}
    if path == "fp8_mlp":
        hidden = _log_int(rng, 640, 3072, 64)
        return {"path": path, "m": _log_int(rng, 77, 8704), "hidden": hidden, "inner": 4 * hidden, "type": kind}
    if path == "nvfp4_linear":
        return {"path": path, "m": _log_int(rng, 16, 8704), "n": _log_int(rng, 1280, 12288, 8), "k": _log_int(rng, 1024, 12288, 32),
                "type": kind, "bias": rng.random() < 0.5}
    if path == "attention":
        head_dim = rng.choice([64, 128])
        kv_heads = rng.choice([4, 8, 12, 24])
        causal = rng.random() < 0.5
        q_len = _log_int(rng, 77, 4352)
        return {"path": path, "batch": rng.choice([1, 2, 3]), "heads": kv_heads * rng.choice([1, 2]), "kv_heads": kv_heads, "q_len": q_len,
                "kv_len": q_len if rng.random() < 0.6 else min(4352, q_len + _log_int(rng, 1, 2048)), "head_dim": head_dim, "causal": causal,
                "type": kind}
    return {"path": path, "batch": rng.choice([1, 2]), "text_tokens": rng.choice([77, 128, 200, 256]),
            "image_tokens": _log_int(rng, 256, 3840, 16), "blocks": rng.choice([1, 2])}


class _Inputs:
    """Seeded random tensors on the GPU and the library's views of them."""

    def __init__(self, seed):
        self.generator = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, shape, std, kind=torch.float32):
        return (torch.randn(shape, device="cuda", generator=self.generator) * std).to(kind)

    def view(self, t, dtype):
        return F.Tensor.from_device_ptr(t.data_ptr(), tuple(t.shape), dtype, keepalive=t)

    def activation(self, shape, kind):
        t = self.normal(shape, 1.0, TORCH_TYPE[kind])
        return t, self.view(t, FLINT_TYPE[kind])

    def bias(self, n, kind):
        return self.view(self.normal((n,), 0.01, TORCH_TYPE[kind]), FLINT_TYPE[kind])

    def result(self, shape, kind):
        t = torch.zeros(shape, device="cuda", dtype=TORCH_TYPE[kind])
        return t, self.view(t, FLINT_TYPE[kind])

    def fp8_tensor_weight(self, n, k):
        """e4m3 codes with one scale for the whole weight, the reference's format."""
        w = self.normal((n, k), 0.02)
        scale = (w.abs().max() / 448.0).reshape(1)
        codes = (w / scale).to(torch.float8_e4m3fn).view(torch.uint8)
        return self.view(codes, F.DType.FP8E4M3), self.view(scale, F.DType.FLOAT)

    def fp8_channel_weight(self, n, k):
        """e4m3 codes with a scale per output channel."""
        return F.quantize_fp8_rows(self.view(self.normal((n, k), 0.02), F.DType.FLOAT))


def prepare(case, seed):
    new = _Inputs(seed)
    path = case["path"]
    if path == "fp8_matmul":
        m, n, k, kind = case["m"], case["n"], case["k"], case["type"]
        _, a = new.activation((m, k), kind)
        weight, scale = new.fp8_tensor_weight(n, k)
        out, out_view = new.result((m, n), kind)
        addend = {"none": lambda: None, "bias": lambda: new.bias(n, kind), "residual": lambda: new.activation((m, n), kind)[1]}[case["addend"]]()
        return {"path": path, "a": a, "weight": weight, "scale": scale, "addend": addend, "out": out, "out_view": out_view}
    if path == "fp8_linear":
        m, n, k, kind = case["m"], case["n"], case["k"], case["type"]
        _, a = new.activation((m, k), kind)
        weight, scales = new.fp8_channel_weight(n, k)
        out, out_view = new.result((m, n), kind)
        return {"path": path, "a": a, "weight": weight, "scales": scales, "bias": new.bias(n, kind) if case["bias"] else None,
                "residual": new.activation((m, n), kind)[1] if case["residual"] else None,
                "act": F.ACT_GELU_TANH if case["gelu"] else F.ACT_NONE, "out": out, "out_view": out_view}
    if path == "fp8_mlp":
        m, d, h, kind = case["m"], case["hidden"], case["inner"], case["type"]
        _, x = new.activation((m, d), kind)
        up, down = new.fp8_channel_weight(h, d), new.fp8_channel_weight(d, h)
        inner, inner_view = new.result((m, h), kind)
        out, out_view = new.result((m, d), kind)
        return {"path": path, "x": x, "up": up, "up_bias": new.bias(h, kind), "down": down, "down_bias": new.bias(d, kind),
                "inner_view": inner_view, "out": out, "out_view": out_view}
    if path == "nvfp4_linear":
        m, n, k, kind = case["m"], case["n"], case["k"], case["type"]
        _, a = new.activation((m, k), kind)
        codes, block_scales, global_scale = F.quantize_nvfp4(new.view(new.normal((n, k), 0.02), F.DType.FLOAT))
        out, out_view = new.result((m, n), kind)
        return {"path": path, "a": a, "codes": codes, "block_scales": block_scales, "global_scale": global_scale,
                "bias": new.bias(n, kind) if case["bias"] else None, "out": out, "out_view": out_view}
    if path == "attention":
        b, h, hk, lq, lk, d, kind = (case[x] for x in ("batch", "heads", "kv_heads", "q_len", "kv_len", "head_dim", "type"))

        def heads_first(t):
            """(batch, length, heads, head_dim) seen as (batch, heads, length, head_dim), as a model hands it over."""
            p = t.transpose(1, 2)
            return F.Tensor.from_device_ptr(p.data_ptr(), tuple(p.shape), FLINT_TYPE[kind], keepalive=t, stride=tuple(p.stride()))

        q, keys, values = (new.normal(s, 1.0, TORCH_TYPE[kind]) for s in ((b, lq, h, d), (b, lk, hk, d), (b, lk, hk, d)))
        out = torch.zeros((b, lq, h, d), device="cuda", dtype=TORCH_TYPE[kind])
        return {"path": path, "q": heads_first(q), "k": heads_first(keys), "v": heads_first(values), "out": out,
                "out_view": heads_first(out), "mask": F.MaskType.CAUSAL if case["causal"] else F.MaskType.NONE}
    cfg = MMDiTConfig(text_tokens=case["text_tokens"], image_tokens=case["image_tokens"], batch=case["batch"], blocks=case["blocks"])
    return {"path": path, "model": MMDiT(cfg, FlintBackend(), seed=seed),
            "tokens": new.normal((cfg.batch, cfg.image_tokens, cfg.latent_channels), 1.0, torch.bfloat16),
            "context": new.normal((cfg.batch, cfg.text_tokens, cfg.context_size), 1.0, torch.bfloat16),
            "sinusoid": new.normal((cfg.batch, cfg.timestep_embed_dim), 0.7, torch.bfloat16)}


def run(state):
    path = state["path"]
    if path == "fp8_matmul":
        lib = F.lib()
        if state["addend"] is None:
            F.check(lib.fl_fp8_matmul(state["a"].raw(), state["weight"].raw(), state["scale"].raw(), state["out_view"].raw()))
        else:
            F.check(lib.fl_fp8_matmul_add(state["a"].raw(), state["weight"].raw(), state["scale"].raw(), state["addend"].raw(),
                                          state["out_view"].raw()))
        return state["out"]
    if path == "fp8_linear":
        F.fp8_linear(state["a"], state["weight"], state["scales"], state["bias"], state["residual"], state["act"], out=state["out_view"])
        return state["out"]
    if path == "fp8_mlp":
        up, down = state["up"], state["down"]
        F.fp8_linear(state["x"], up[0], up[1], state["up_bias"], None, F.ACT_GELU_TANH, out=state["inner_view"])
        F.fp8_linear(state["inner_view"], down[0], down[1], state["down_bias"], state["x"], F.ACT_NONE, out=state["out_view"])
        return state["out"]
    if path == "nvfp4_linear":
        F.nvfp4_linear(state["a"], state["codes"], state["block_scales"], state["global_scale"], state["bias"], out=state["out_view"])
        return state["out"]
    if path == "attention":
        F.attention(state["q"], state["k"], state["v"], state["mask"], 0, state["out_view"])
        return state["out"]
    model = state["model"]
    stream, embedding = model.embed(state["tokens"], state["context"], state["sinusoid"])
    return {"stream": model.blocks(stream, embedding), "embedding": embedding}


def work(case):
    path = case["path"]
    if path == "attention":
        b, h, hk, lq, lk, d = (case[x] for x in ("batch", "heads", "kv_heads", "q_len", "kv_len", "head_dim"))
        # query i of a causal run sees keys 0 .. i + lk - lq
        pairs = lq * (lk - lq) + lq * (lq + 1) // 2 if case["causal"] else lq * lk
        return {"bytes": 2 * b * d * (2 * h * lq + 2 * hk * lk), "flops": 4 * b * h * pairs * d}
    if path == "denoise":
        cfg = MMDiTConfig(text_tokens=case["text_tokens"], image_tokens=case["image_tokens"], batch=case["batch"], blocks=case["blocks"])
        d, latent = cfg.hidden, cfg.latent_channels
        weights = cfg.blocks * d * (6 * d + 3 * d + d + 2 * cfg.mlp) + d * (cfg.timestep_embed_dim + 2 * d + cfg.context_size + latent)
        activations = 2 * cfg.batch * (cfg.image_tokens * latent + cfg.text_tokens * cfg.context_size + cfg.tokens * d)
        ways_in = 2 * cfg.batch * d * (cfg.text_tokens * (cfg.context_size + d) + cfg.image_tokens * latent)
        return {"bytes": weights + activations, "flops": cfg.block_gemm_flops() * cfg.blocks + ways_in + cfg.attention_flops()}
    m = case["m"]
    if path == "fp8_mlp":
        d, h = case["hidden"], case["inner"]
        return {"bytes": 2 * d * h + 4 * (d + h) + 2 * (d + h) + 4 * m * d, "flops": 4 * m * d * h}
    n, k = case["n"], case["k"]
    operands = 2 * m * k + 2 * m * n
    if path == "fp8_matmul":
        extra = {"none": 0, "bias": 2 * n, "residual": 2 * m * n}[case["addend"]]
        return {"bytes": operands + n * k + extra, "flops": 2 * m * n * k}
    if path == "fp8_linear":
        extra = 4 * n + (2 * n if case["bias"] else 0) + (2 * m * n if case["residual"] else 0)
        return {"bytes": operands + n * k + extra, "flops": 2 * m * n * k}
    return {"bytes": operands + n * k // 2 + n * k // 16 + (2 * n if case["bias"] else 0), "flops": 2 * m * n * k}


def tolerance(case):
    """About four times what each path was seen to differ by from the same arithmetic in 64 bits: of one
    product the rounding of its 16-bit result (2.1e-4 in half, 1.7e-3 in bfloat16); of a quantised
    activation also the codes that fall on the other side of a tie (2.0e-3; 3.7e-3 for two in a row); of
    attention the probabilities' rounding (2.5e-4, 2.3e-3). The blocks quantise six times in a row, each
    turning a difference d of its input into about sqrt(d / 16): twice what exchanging the attention for
    another correct one changes in the stream (1.5e-2)."""
    path = case["path"]
    if path == "denoise":
        return {"rel": 3e-2}
    if path == "fp8_mlp":
        return {"rel": 1.5e-2}
    if path == "fp8_linear":
        return {"rel": 8e-3}
    bf16 = case["type"] == "bf16"
    if path == "attention":
        return {"rel": 1e-2 if bf16 else 1e-3}
    return {"rel": 6.5e-3 if bf16 else 8.5e-4}


def _e4m3(x):
    """x rounded to the nearest e4m3 value, saturating."""
    return x.clamp(-448.0, 448.0).to(torch.float8_e4m3fn).float()


def _quantized_rows(x):
    """x (rows, k) in float32 as e4m3 values times a scale per row (the row's largest magnitude / 448), in 64 bits."""
    scale = x.abs().amax(dim=1, keepdim=True) / 448.0
    return _e4m3(x * (1.0 / torch.where(scale > 0, scale, torch.ones_like(scale)))).double() * scale.double()


def _quantized_blocks(x, scale):
    """x (rows, k) in float32 as e2m1 values times an e4m3 scale per 16 and `scale`, in 64 bits."""
    blocks = x.reshape(x.shape[0], -1, 16)
    factor = _e4m3(blocks.abs().amax(dim=2, keepdim=True) / (6.0 * scale))
    step = factor * scale
    y = blocks * torch.where(step > 0, 1.0 / step, torch.zeros_like(step))
    bounds = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=x.device)  # between the magnitudes, ties to even
    magnitude = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], device=x.device, dtype=torch.float64)
    up, down = torch.bucketize(y.abs(), bounds, right=True), torch.bucketize(y.abs(), bounds)
    code = torch.where(up % 2 == 0, up, down)
    return (magnitude[code] * y.sign().double() * step.double()).reshape(x.shape)


def exact(case, seed):
    """run()'s result from the same inputs with the operands' own quantisation, the arithmetic in 64
    bits. The blocks of a denoise step have none: a rounding moves codes in every quantiser after it."""
    path = case["path"]
    if path == "denoise":
        return None
    new = _Inputs(seed)
    kind = TORCH_TYPE[case["type"]]
    gelu = lambda t: torch.nn.functional.gelu(t, approximate="tanh")
    if path == "attention":
        b, h, hk, lq, lk, d = (case[x] for x in ("batch", "heads", "kv_heads", "q_len", "kv_len", "head_dim"))
        q, keys, values = (new.normal(s, 1.0, kind) for s in ((b, lq, h, d), (b, lk, hk, d), (b, lk, hk, d)))
        out = torch.empty((b, lq, h, d), device="cuda", dtype=torch.float64)
        hidden = torch.ones((lq, lk), device="cuda", dtype=torch.bool).triu(1 + lk - lq) if case["causal"] else None
        for i in range(b):
            for j in range(h):
                g = j // (h // hk)
                scores = q[i, :, j].double() @ keys[i, :, g].double().t() / math.sqrt(d)
                if hidden is not None:
                    scores.masked_fill_(hidden, -math.inf)
                out[i, :, j] = scores.softmax(dim=1) @ values[i, :, g].double()
        return out
    if path == "fp8_mlp":
        m, d, h = case["m"], case["hidden"], case["inner"]
        x = new.normal((m, d), 1.0, kind)
        up, down = _quantized_rows(new.normal((h, d), 0.02)), _quantized_rows(new.normal((d, h), 0.02))
        up_bias, down_bias = (new.normal((n,), 0.01, kind).double() for n in (h, d))
        inner = gelu(_quantized_rows(x.float()) @ up.t() + up_bias).to(kind)
        return _quantized_rows(inner.float()) @ down.t() + down_bias + x.double()
    m, n, k = case["m"], case["n"], case["k"]
    a = new.normal((m, k), 1.0, kind)
    w = new.normal((n, k), 0.02)
    if path == "fp8_matmul":
        scale = w.abs().max() / 448.0
        y = a.double() @ (w / scale).to(torch.float8_e4m3fn).double().t() * scale.double()
        if case["addend"] != "none":
            y += (new.normal((n,), 0.01, kind) if case["addend"] == "bias" else new.normal((m, n), 1.0, kind)).double()
        return y
    if path == "fp8_linear":
        y = _quantized_rows(a.float()) @ _quantized_rows(w).t()
    else:
        y = _quantized_blocks(a.float(), 1.0) @ _quantized_blocks(w, w.abs().max() / (448.0 * 6.0)).t()
    if case["bias"]:
        y += new.normal((n,), 0.01, kind).double()
    if case.get("gelu"):
        y = gelu(y)
    if case.get("residual"):
        y += new.normal((m, n), 1.0, kind).double()
    return y
