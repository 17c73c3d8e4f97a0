"""Timed cases of the framework: what a program that serves a model with it has done on the GPU, one layer or operator call per case.

The quantised cases have the sizes of DeepSeek-V3 (models/modeling_deepseek_v3.DeepseekV3Config: width 7168, 256 experts of 2048, 8 per token,
128 heads of 128 + 64 over latents of 512 + 64); the un-quantised ones those of util/model_bench's "v3-layer" and "2k-wide".  `draw` takes other
sizes from the same ranges.  `exact` is plain torch in 64 bits; the rounding of activations to 8 bits in front of a quantised product (Q8_K, or
e4m3 with a scale per 128) is part of what those operators compute and is done there as their formats define it."""
import contextlib
import math

import torch

Q4_K, Q5_K, Q6_K = 12, 13, 14
BLOCK_BYTES = {Q4_K: 144, Q5_K: 176, Q6_K: 210}
TYPES = {"Q4_K": Q4_K, "Q5_K": Q5_K, "Q6_K": Q6_K}
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
DEV = "cuda"


# ------------------------------------------------------------------------------------------------------------------------- cases
def _moe(tokens, experts=256, top=8, hidden=7168, ff=2048, groups=8, keep=4):
    return {"kind": "moe", "tokens": tokens, "experts": experts, "top": top, "hidden": hidden, "ff": ff, "groups": groups, "keep": keep}


def _experts(tokens, experts=256, top=8, hidden=7168, ff=2048, down="Q6_K"):
    return {"kind": "experts", "tokens": tokens, "experts": experts, "top": top, "hidden": hidden, "ff": ff, "down": down}


def _linear(tokens, n_in, n_out, type="Q4_K", dtype="bf16"):
    return {"kind": "linear", "tokens": tokens, "n_in": n_in, "n_out": n_out, "type": type, "dtype": dtype}


def _fp8(tokens, n_in, n_out, dtype="bf16"):
    return {"kind": "fp8", "tokens": tokens, "n_in": n_in, "n_out": n_out, "dtype": dtype}


def _latent(batch, ctx, heads=128):
    return {"kind": "latent_layer", "batch": batch, "ctx": ctx, "heads": heads, "hidden": 7168, "q_rank": 1536}


def _mla(batch, ctx, heads=128):
    return {"kind": "mla", "batch": batch, "ctx": ctx, "heads": heads}


def _attn(tokens, before, width=7168, heads=64, kv_heads=8, chunk=4096):
    return {"kind": "attention", "tokens": tokens, "before": before, "width": width, "heads": heads, "kv_heads": kv_heads, "dim": 128, "chunk": chunk}


def _dense(tokens, width=2048, ff=1024, experts=32, top=4):
    return {"kind": "dense_experts", "tokens": tokens, "width": width, "ff": ff, "experts": experts, "top": top}


def listed():
    return [
        # one token of one user through a mixture-of-experts layer (router, 8 of 256 experts, shared expert): the step that every decoded
        # token takes 58 times
        dict(_moe(1), name="moe_decode_1"),
        # the same for several users' tokens in one step, an odd number of them
        dict(_moe(7), name="moe_decode_7"),
        # a larger decode batch, beyond what the single-launch block takes
        dict(_moe(24), name="moe_batch_24"),
        # a prompt portion through a layer's routed experts: the largest portion that the experts take at once by default
        dict(_experts(1024), name="experts_prompt_1024"),
        # attention output projection of one decoded token (weights in GGUF blocks)
        dict(_linear(1, 16384, 7168), name="linear_decode_1"),
        # query projection of a prompt portion of odd length
        dict(_linear(777, 1536, 24576), name="linear_prompt_777"),
        # attention output projection of one decoded token (weights in e4m3 with 128 x 128 scales)
        dict(_fp8(1, 16384, 7168), name="fp8_decode_1"),
        # a projection of the dense feed-forward for a prompt portion
        dict(_fp8(2000, 7168, 18432), name="fp8_prompt_2000"),
        # the attention layer of one decoded token with a context of some thousand tokens: projections, rotation, cache, absorbed attention
        dict(_latent(1, 4096), name="latent_layer_decode"),
        # the attention alone at the longest context that the configurations name
        dict(_mla(1, 131072), name="mla_128k"),
        # the second portion of a prompt through a soft-max attention layer with grouped heads
        dict(_attn(2048, 2048), name="attention_prompt_2048"),
        # a prompt portion through un-quantised experts
        dict(_dense(1000), name="dense_experts_prompt_1000"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))


def _int(rng, lo, hi):
    return max(lo, min(hi, int(_log(rng, lo, hi))))


def _of(rng, lo, hi, step):
    return step * _int(rng, lo // step, hi // step)


def draw(rng):
    kind = rng.choice(["moe", "experts", "experts", "linear", "linear", "fp8", "fp8", "latent_layer", "mla", "attention", "dense_experts"])
    if kind == "moe":
        experts, groups, keep = rng.choice([(256, 8, 4), (128, 4, 2), (64, 1, 1), (160, 8, 3)])
        return _moe(_int(rng, 1, 40), experts, rng.choice([4, 6, 8]), _of(rng, 4096, 7168, 256), _of(rng, 512, 2048, 256), groups, keep)
    if kind == "experts":
        experts = rng.choice([256, 160, 64, 16])
        return _experts(_int(rng, 9, 1024), experts, rng.choice([2, 6, 8]), _of(rng, 1024, 7168, 256), _of(rng, 512, 2048, 256), rng.choice(["Q6_K", "Q6_K", "Q4_K"]))
    if kind in ("linear", "fp8"):
        tokens, step = _int(rng, 1, 1024 if kind == "linear" else 2000), 256 if kind == "linear" else 128
        n_in, n_out = _of(rng, 512, 16384, step), rng.choice([_of(rng, 64, 16384, 64), _int(rng, 64, 16384)])
        most = 777 * 1536 * 24576 if kind == "linear" else 2000 * 7168 * 18432 // 2
        if kind == "linear":
            n_out += n_out % 2
        while tokens * n_in * n_out > most and tokens > 64:
            tokens = tokens * 2 // 3
        while tokens * n_in * n_out > most:
            n_out = max(64, n_out // 2 // 2 * 2)
            n_in = max(step, n_in // 2 // step * step)
        dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"])
        return _linear(tokens, n_in, n_out, rng.choice(["Q4_K", "Q4_K", "Q6_K", "Q5_K"]), dtype) if kind == "linear" else _fp8(tokens, n_in, n_out, dtype)
    if kind == "latent_layer":
        return _latent(_int(rng, 1, 8), _int(rng, 64, 16384), rng.choice([128, 64, 16]))
    if kind == "mla":
        batch = _int(rng, 1, 64)
        return _mla(batch, _int(rng, 16, 131072 // batch), rng.choice([128, 64, 32, 16]))
    if kind == "attention":
        heads = rng.choice([64, 32, 16])
        return _attn(_int(rng, 1, 2048), _int(rng, 1, 2048) - 1, rng.choice([7168, 2048]), heads, rng.choice([heads // 8, heads // 4]), rng.choice([4096, 2048, 1024]))
    return _dense(_int(rng, 1, 1024), rng.choice([2048, 1024, 7168]), rng.choice([1024, 512, 2048]), rng.choice([32, 16]), rng.choice([4, 2, 8]))


# ---------------------------------------------------------------------------------------------------------------- inputs of a seed
class _Draws:
    """Tensors in a fixed order from one seed, the same for `prepare` and `exact`."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(int(seed))

    def normal(self, *shape, scale=1.0, dtype=torch.float32):
        return (torch.randn(shape, generator=self.g, device=DEV) * scale).to(dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0, dtype=torch.float32):
        return (torch.rand(shape, generator=self.g, device=DEV) * (hi - lo) + lo).to(dtype)

    def choices(self, rows, n, k):
        """k different numbers below n per row, int64"""
        return torch.rand((rows, n), generator=self.g, device=DEV).argsort(-1)[:, :k].contiguous()

    def blocks(self, type, rows, cols):
        """[rows, cols / 256 * block bytes] of a GGUF type: values of mean about 0 and 2-norm about 1 per row, as in a trained projection"""
        nb = rows * cols // 256
        out = torch.empty((nb, BLOCK_BYTES[type]), dtype=torch.uint8, device=DEV)
        for lo in range(0, nb, 1 << 22):
            out[lo:lo + (1 << 22)].random_(generator=self.g)
        middle = {Q4_K: 7.5, Q5_K: 15.5, Q6_K: 0.0}[type]
        spread = {Q4_K: 4.6 * 36.4, Q5_K: 9.2 * 36.4, Q6_K: 18.5 * 73.9}[type]
        d = self.uniform(nb, lo=0.7, hi=1.3) / (spread * math.sqrt(cols))
        if type == Q6_K:
            out[:, 208:210] = d.to(torch.float16).view(torch.uint8).reshape(nb, 2)
        else:       # minima near the middle of the quants: the six bits of a minimum are those of its scale, their factors differ a little
            out[:, 8:12] = out[:, 4:8]
            out[:, 12:16] = (out[:, 12:16] & 15) * 17
            out[:, 0:2] = d.to(torch.float16).view(torch.uint8).reshape(nb, 2)
            out[:, 2:4] = (d * middle * self.uniform(nb, lo=0.95, hi=1.05)).to(torch.float16).view(torch.uint8).reshape(nb, 2)
        return out.view(rows, -1)


def _inputs(case, seed):
    """every tensor that a case's call reads, by name"""
    r, c = _Draws(seed), case
    k = c["kind"]
    if k in ("moe", "experts"):
        E, H, I, T = c["experts"], c["hidden"], c["ff"], c["tokens"]
        v = {"gate": r.blocks(Q4_K, E * I, H), "up": r.blocks(Q4_K, E * I, H), "down": r.blocks(TYPES[c.get("down", "Q6_K")], E * H, I), "x": r.normal(T, H, dtype=torch.bfloat16)}
        if k == "experts":
            v["ids"], v["weights"] = r.choices(T, E, c["top"]), r.uniform(T, c["top"], lo=0.05, hi=0.5)
        else:
            v["router"], v["correction"] = r.normal(E, H, scale=H ** -0.5), r.uniform(E, lo=-0.2, hi=0.2)
            v["s_gate"], v["s_up"], v["s_down"] = r.blocks(Q4_K, I, H), r.blocks(Q4_K, I, H), r.blocks(Q6_K, H, I)
        return v
    if k == "linear":
        return {"w": r.blocks(TYPES[c["type"]], c["n_out"], c["n_in"]), "x": r.normal(c["tokens"], c["n_in"], dtype=DTYPES[c["dtype"]])}
    if k == "fp8":
        N, K = c["n_out"], c["n_in"]
        return {"w": r.normal(N, K, scale=60.0).clamp_(-448, 448).to(torch.float8_e4m3fn), "scale": r.uniform((N + 127) // 128, K // 128, lo=0.7, hi=1.3) / (60.0 * math.sqrt(K)),
                "x": r.normal(c["tokens"], K, dtype=DTYPES[c["dtype"]])}
    if k == "mla":
        B, L, Hq, page = c["batch"], c["ctx"], c["heads"], 64
        per = (L + page - 1) // page
        kv_len = torch.full((B,), L, dtype=torch.int32, device=DEV)
        if B > 1:       # sequences of different lengths, the longest of them as stated
            kv_len[1:] = (r.uniform(B - 1, lo=0.1, hi=1.0) * L).to(torch.int32).clamp_(min=1)
        return {"q": r.normal(B, Hq, 512, dtype=torch.bfloat16), "q_pe": r.normal(B, Hq, 64, dtype=torch.bfloat16), "kv": r.normal(B * per, page, 576, dtype=torch.bfloat16),
                "pages": r.choices(1, B * per, B * per).view(-1).to(torch.int32), "kv_len": kv_len}
    if k == "latent_layer":
        B, H, R, W = c["batch"], c["heads"], c["q_rank"], c["hidden"]
        return {"q_a": r.blocks(Q4_K, R, W), "q_b": r.blocks(Q4_K, H * 192, R), "kv_a": r.blocks(Q4_K, 576, W), "o": r.blocks(Q4_K, W, H * 128), "q_norm": r.uniform(R, lo=0.8, hi=1.2, dtype=torch.bfloat16),
                "kv_norm": r.uniform(512, lo=0.8, hi=1.2, dtype=torch.bfloat16), "kv_b": r.normal(H * 256, 512, scale=512 ** -0.5, dtype=torch.bfloat16),
                "past": r.normal(B, c["ctx"], 576, dtype=torch.bfloat16), "x": r.normal(B, 1, W, dtype=torch.bfloat16)}
    if k == "attention":
        W, H, G, D = c["width"], c["heads"], c["kv_heads"], c["dim"]
        n_in = (H + 2 * G) * D
        return {"w_in": r.normal(n_in, W, scale=W ** -0.5, dtype=torch.bfloat16), "b_in": r.normal(n_in, scale=0.1, dtype=torch.bfloat16), "q_norm": r.uniform(D, lo=0.8, hi=1.2, dtype=torch.bfloat16),
                "k_norm": r.uniform(D, lo=0.8, hi=1.2, dtype=torch.bfloat16), "o": r.normal(W, H * D, scale=(H * D) ** -0.5, dtype=torch.bfloat16), "past": r.normal(c["before"], G * 2 * D, dtype=torch.bfloat16),
                "h": r.normal(c["tokens"], W, dtype=torch.bfloat16)}
    E, W, F = c["experts"], c["width"], c["ff"]
    return {"gate": r.normal(E, F, W, scale=W ** -0.5, dtype=torch.bfloat16), "up": r.normal(E, F, W, scale=W ** -0.5, dtype=torch.bfloat16), "down": r.normal(E, W, F, scale=F ** -0.5, dtype=torch.bfloat16),
            "x": r.normal(c["tokens"], W, dtype=torch.bfloat16), "ids": r.choices(c["tokens"], E, c["top"]), "weights": r.uniform(c["tokens"], c["top"], lo=0.05, hi=0.5)}


# ------------------------------------------------------------------------------------------------------------ what a program keeps
@contextlib.contextmanager
def _default_dtype(dtype):
    old = torch.get_default_dtype()
    torch.set_default_dtype(dtype)
    try:
        yield
    finally:
        torch.set_default_dtype(old)


class _Weights:
    """A weight loader (the interface of util/custom_loader's loaders) over tensors that are there already."""

    def __init__(self, raw, plain=None):
        self.raw, self.plain, self.tensor_device_map = raw, plain or {}, {}

    def has_tensor(self, name):
        return name in self.raw or name in self.plain

    def get_mmap_tensor(self, name):
        blocks = self.raw[name][0].reshape(-1)
        return blocks if "_exps" in name else blocks.cpu().numpy()

    def get_ggml_type(self, name):
        return self.raw[name][1]

    def load_gguf_tensor(self, name, device="cuda", target_dtype=None):
        t = self.plain[name]
        return t.to(device=device, dtype=target_dtype or t.dtype)


def _kept_moe(c, v):
    from ktransformers_b200.models.modeling_deepseek_v3 import DeepseekV3Config, DeepseekV3MoE
    from ktransformers_b200.operators.experts import KDeepseekV3MoE, KTransformersExperts
    from ktransformers_b200.operators.gate import KMoEGateB200
    from ktransformers_b200.operators.linear import KTransformersLinear
    cfg = DeepseekV3Config(hidden_size=c["hidden"], moe_intermediate_size=c["ff"], n_routed_experts=c["experts"], n_shared_experts=1, num_experts_per_tok=c["top"], n_group=c["groups"],
                           topk_group=c["keep"])
    key = "blk.3"
    raw = {key + ".ffn_%s_exps.weight" % n: (v[n], Q6_K if n == "down" else Q4_K) for n in ("gate", "up", "down")}
    raw.update({key + ".shared_experts.%s_proj.weight" % n: (v["s_" + n], Q6_K if n == "down" else Q4_K) for n in ("gate", "up", "down")})
    weights = _Weights(raw, {key + ".gate.weight": v["router"], key + ".gate.e_score_correction_bias": v["correction"]})
    with _default_dtype(torch.bfloat16):
        with torch.device("meta"):
            plain = DeepseekV3MoE(cfg)
        moe = KDeepseekV3MoE(key, weights, cfg, plain, DEV, DEV)
        plain.gate = KMoEGateB200(key + ".gate", weights, cfg, plain.gate, DEV, DEV)
        plain.experts = KTransformersExperts(key, weights, cfg, plain.experts, prefill_device=DEV, prefill_op=None, generate_device=DEV, generate_op="KExpertsB200", out_device=DEV)
        for n in ("gate", "up", "down"):
            name = n + "_proj"
            setattr(plain.shared_experts, name, KTransformersLinear(key + ".shared_experts." + name, weights, cfg, getattr(plain.shared_experts, name), DEV, "KLinearB200", DEV, None))
        plain.gate.load()
        plain.experts.load(warmup=False)
        for n in ("gate", "up", "down"):
            getattr(plain.shared_experts, n + "_proj").load()
        moe._shared_mlp_handle(plain.experts.generate_experts)
    return moe


def _kept_linear(blocks, type, n_in, n_out, dtype=torch.bfloat16):
    from ktransformers_b200.operators.linear import KLinearB200
    with _default_dtype(dtype):
        with torch.device("meta"):
            plain = torch.nn.Linear(n_in, n_out, bias=False)
        lin = KLinearB200("blk.0.proj", None, None, plain, DEV)
        lin.load(w=(blocks, type))
    return lin


def _kept_latent(c, v):
    from ktransformers_b200.models.custom_cache import StaticCache
    from ktransformers_b200.models.modeling_deepseek_v3 import DeepseekV3Attention, DeepseekV3Config, DeepseekV3RotaryEmbedding
    from ktransformers_b200.operators.attention import KDeepseekV2Attention
    from ktransformers_b200.operators.flashinfer_wrapper import MLAWrapper
    from ktransformers_b200.operators.linear import KTransformersLinear
    B, H, W = c["batch"], c["heads"], c["hidden"]
    cfg = DeepseekV3Config(hidden_size=W, num_attention_heads=H, q_lora_rank=c["q_rank"], num_hidden_layers=1)
    param = lambda t: torch.nn.Parameter(t, requires_grad=False)
    with _default_dtype(torch.bfloat16):
        with torch.device("meta"):
            plain = DeepseekV3Attention(cfg, layer_idx=0)
        for name, blocks in (("q_a_proj", "q_a"), ("q_b_proj", "q_b"), ("kv_a_proj_with_mqa", "kv_a"), ("o_proj", "o")):
            lin = KTransformersLinear("blk.0." + name, _Weights({}), cfg, getattr(plain, name), DEV, "KLinearB200", DEV, None)
            lin.load(w=(v[blocks], Q4_K))
            setattr(plain, name, lin)
        plain.q_a_layernorm.weight, plain.kv_a_layernorm.weight = param(v["q_norm"]), param(v["kv_norm"])
        plain.kv_b_proj.weight = param(v["kv_b"])
        plain.rotary_emb = DeepseekV3RotaryEmbedding(64).to(DEV)
        op = KDeepseekV2Attention("blk.0.self_attn", None, cfg, plain, DEV, DEV)
    cache = StaticCache(cfg, max_batch_size=B, max_cache_len=c["ctx"] + 1, device=DEV)
    rows = cache.key_cache[0].view(B, cache.max_pages * cache.page_size, 576)
    rows[:, :c["ctx"]].copy_(v["past"])
    op.mla_wrapper = MLAWrapper(B, cache.max_pages * B, device=DEV)
    op.get_absorbed()
    return op, cache, torch.full((B, 1), c["ctx"], dtype=torch.int64, device=DEV), torch.tensor([c["ctx"]], device=DEV)


def _kept_attention(c, v):
    from ktransformers_b200.models.configuration_lekapel import RotarySpec
    from ktransformers_b200.models.configuration_lipadra import PlusOneAttentionSpec
    from ktransformers_b200.models.custom_cache import PagedStateCache
    from ktransformers_b200.operators.attention import KPlusOneAttention
    W, H, G, D, T, P = c["width"], c["heads"], c["kv_heads"], c["dim"], c["tokens"], c["before"]
    spec = PlusOneAttentionSpec(heads=H, kv_heads=G, dim=D, vdim=D, scale=D ** -0.5, rot=RotarySpec(10000.0, D // 2, layout="halves"), chunk=c["chunk"])
    op = KPlusOneAttention(W, spec, 1e-6, device=DEV)
    for p, n in ((op.w_in, "w_in"), (op.b_in, "b_in"), (op.q_norm, "q_norm"), (op.k_norm, "k_norm"), (op.o, "o")):
        p.data[:v[n].shape[0]].copy_(v[n])
    cache = PagedStateCache([spec.cache_row_width()], 0, P + T, 1, DEV, page_size=64)
    if P:       # an earlier portion's rows, where its step would have written them
        first = cache.build_batch([("s", [0] * P, [])])
        table, pos = cache.page_table[first.slot.long()[0]].long(), torch.arange(P, device=DEV)
        cache.key_cache[0][table[pos // 64], pos % 64] = v["past"]
        cache.commit()
    batch = cache.build_batch([("s", [0] * T, [])])
    return op, batch, cache


def prepare(case, seed):
    c, v = case, _inputs(case, seed)
    k = c["kind"]
    if k == "moe":
        return {"kind": k, "op": _kept_moe(c, v), "x": v["x"].view(1, c["tokens"], c["hidden"])}
    if k == "experts":
        from ktransformers_b200.models.modeling_deepseek_v3 import DeepseekV3Config
        from ktransformers_b200.operators.experts import KExpertsB200
        cfg = DeepseekV3Config(hidden_size=c["hidden"], moe_intermediate_size=c["ff"], n_routed_experts=c["experts"], num_experts_per_tok=c["top"])
        op = KExpertsB200("blk.3", None, cfg, c["experts"], device=DEV, hidden_dtype=torch.bfloat16)
        op.load(w={"gate": v["gate"], "up": v["up"], "down": v["down"], "gate_type": Q4_K, "up_type": Q4_K, "down_type": TYPES[c["down"]]})
        return {"kind": k, "op": op, "x": v["x"], "ids": v["ids"], "weights": v["weights"]}
    if k == "linear":
        return {"kind": k, "op": _kept_linear(v["w"], TYPES[c["type"]], c["n_in"], c["n_out"], DTYPES[c["dtype"]]), "x": v["x"]}
    if k == "fp8":
        from ktransformers_b200.operators.linear import KLinearFP8
        with _default_dtype(DTYPES[c["dtype"]]):
            with torch.device("meta"):
                plain = torch.nn.Linear(c["n_in"], c["n_out"], bias=False)
            op = KLinearFP8("blk.0.proj", None, None, plain, DEV)
            op.load(w=(v["w"], v["scale"]))
        return {"kind": k, "op": op, "x": v["x"]}
    if k == "mla":
        from ktransformers_b200.operators.flashinfer_wrapper import MLAWrapper
        B, per = c["batch"], v["pages"].numel() // c["batch"]
        op = MLAWrapper(B, per, device=DEV)
        op.plan(None, torch.arange(B + 1, dtype=torch.int32, device=DEV) * per, v["pages"], v["kv_len"], None, c["heads"], 512, 64, 64, 192 ** -0.5, torch.bfloat16, torch.bfloat16)
        return {"kind": k, "op": op, "q": v["q"], "q_pe": v["q_pe"], "ckv": v["kv"][..., :512], "k_pe": v["kv"][..., 512:]}
    if k == "latent_layer":
        op, cache, pos, at = _kept_latent(c, v)
        return {"kind": k, "op": op, "cache": cache, "pos": pos, "at": at, "x": v["x"]}
    if k == "attention":
        op, batch, cache = _kept_attention(c, v)
        return {"kind": k, "op": op, "batch": batch, "cache": cache, "h": v["h"]}
    from ktransformers_b200.operators.experts import KExpertsDense
    op = KExpertsDense(c["width"], c["ff"], c["experts"], device=DEV)
    for p, n in ((op.gate, "gate"), (op.up, "up"), (op.down, "down")):
        p.data.copy_(v[n])
    return {"kind": k, "op": op, "x": v["x"], "ids": v["ids"], "weights": v["weights"]}


@torch.no_grad()
def run(state):
    s, k = state, state["kind"]
    if k in ("moe", "linear", "fp8"):
        return s["op"].forward(s["x"])
    if k in ("experts", "dense_experts"):
        return s["op"].forward(s["x"], s["ids"], s["weights"])
    if k == "mla":
        return s["op"].run(s["q"], s["q_pe"], s["ckv"], s["k_pe"])
    if k == "latent_layer":
        return s["op"](s["x"], position_ids=s["pos"], past_key_value=s["cache"], cache_position=s["at"])[0]
    return s["op"](s["h"], s["batch"], s["cache"], 0)


# ------------------------------------------------------------------------------------------------------------------ work and limits
def work(case):
    c, k = case, case["kind"]
    T = c.get("tokens", 1)
    if k in ("moe", "experts"):
        E, H, I, top = c["experts"], c["hidden"], c["ff"], c["top"]
        per = 2 * I * H // 256 * 144 + H * I // 256 * BLOCK_BYTES[TYPES[c.get("down", "Q6_K")]]
        hit = E * (1.0 - (1.0 - top / E) ** T)
        n_bytes, flops = hit * per + 4 * T * H, 6.0 * T * top * H * I
        if k == "moe":
            n_bytes, flops = n_bytes + per + 4 * E * H, flops + 6.0 * T * H * I + 2.0 * T * E * H
        return {"bytes": n_bytes, "flops": flops}
    if k == "linear":
        size = DTYPES[c["dtype"]].itemsize
        return {"bytes": c["n_in"] * c["n_out"] / 256 * BLOCK_BYTES[TYPES[c["type"]]] + size * T * (c["n_in"] + c["n_out"]), "flops": 2.0 * T * c["n_in"] * c["n_out"]}
    if k == "fp8":
        size = DTYPES[c["dtype"]].itemsize
        return {"bytes": c["n_in"] * c["n_out"] + size * T * (c["n_in"] + c["n_out"]), "flops": 2.0 * T * c["n_in"] * c["n_out"]}
    if k == "mla":
        keys = c["ctx"] * (1.0 if c["batch"] == 1 else (1.0 + 0.55 * (c["batch"] - 1)))
        return {"bytes": keys * 1152 + c["batch"] * c["heads"] * (576 + 512) * 2, "flops": 2.0 * keys * c["heads"] * (576 + 512)}
    if k == "latent_layer":
        B, H, W, R, L = c["batch"], c["heads"], c["hidden"], c["q_rank"], c["ctx"] + 1
        quant = R * W + H * 192 * R + 576 * W + W * H * 128
        return {"bytes": quant * 144 / 256 + H * 256 * 512 * 2 + B * L * 1152, "flops": 2.0 * B * (quant + H * 256 * 512 + L * H * 1088)}
    if k == "attention":
        W, H, G, D, P = c["width"], c["heads"], c["kv_heads"], c["dim"], c["before"]
        pairs, reach = 0, 0
        for i in range(P, P + T):
            pairs += i % c["chunk"] + 1
        reach = P + T - (P - P % c["chunk"])
        n_in = (H + 2 * G) * D
        return {"bytes": 2.0 * (W * n_in + W * H * D + 2 * T * W + (reach + T) * 2 * G * D), "flops": 2.0 * T * W * (n_in + H * D) + 4.0 * pairs * H * D}
    E, W, F, top = c["experts"], c["width"], c["ff"], c["top"]
    hit = E * (1.0 - (1.0 - top / E) ** T)
    return {"bytes": hit * 6.0 * W * F + 6.0 * T * W, "flops": 6.0 * T * top * W * F}


# About four times the distance from `exact` that was measured.  A result in 16 bits is off by 1.7e-3 (bf16) or 2e-4 (fp16) from its last rounding
# alone; behind a second rounding to 8 bits a value at the edge between two steps may fall to either side.
def tolerance(case):
    k, dtype = case["kind"], case.get("dtype", "bf16")
    if k in ("linear", "fp8"):
        return {"rel": {"bf16": 7e-3, "fp16": 1e-3, "fp32": 1e-5}[dtype]}
    return {"rel": {"moe": 3e-2, "experts": 2e-2, "mla": 7e-3, "latent_layer": 5e-2, "attention": 1.3e-2, "dense_experts": 1.4e-2}[k]}


# ------------------------------------------------------------------------------------------------------------------- in 64 bits
def _dequantised(blocks, type, cols):
    """fp64 [rows, cols] of GGUF blocks"""
    b = blocks.reshape(-1, BLOCK_BYTES[type])
    half = lambda lo: b[:, lo:lo + 2].contiguous().view(torch.float16).double()
    if type == Q6_K:
        ql, qh, sc = b[:, :128].view(-1, 2, 2, 32), b[:, 128:192].view(-1, 2, 1, 32), b[:, 192:208].contiguous().view(torch.int8).double()
        low, high = ql & 15, ql >> 4                                    # [blocks, half, 32-group, 32]
        q = torch.cat([low[:, :, :1] | ((qh & 3) << 4), low[:, :, 1:] | ((qh >> 2 & 3) << 4), high[:, :, :1] | ((qh >> 4 & 3) << 4), high[:, :, 1:] | ((qh >> 6 & 3) << 4)], 2)
        v = (q.double() - 32.0).view(-1, 16, 16) * sc.unsqueeze(-1) * half(208).unsqueeze(-1)
        return v.reshape(-1, cols)
    s = b[:, 4:16].int()
    low, mid, top = s[:, 0:4], s[:, 4:8], s[:, 8:12]
    sc = torch.cat([low & 63, (top & 15) | (low >> 6 << 4)], 1).double()
    mn = torch.cat([mid & 63, (top >> 4) | (mid >> 6 << 4)], 1).double()
    qs = b[:, -128:].view(-1, 4, 1, 32)
    q = torch.cat([qs & 15, qs >> 4], 2).reshape(-1, 8, 32)
    if type == Q5_K:
        bits = torch.arange(8, device=b.device, dtype=torch.uint8).view(1, 8, 1)
        q = q + ((b[:, 16:48].unsqueeze(1) >> bits) & 1) * 16
    v = q.double() * (half(0) * sc).unsqueeze(-1) - (half(2) * mn).unsqueeze(-1)
    return v.reshape(-1, cols)


def _q8(x):
    """activations as the Q8_K blocks that K-quant products take: 256 int8 and a scale of their own, from the fp32 values"""
    f = x.float().reshape(-1, 256)
    at = f.abs().argmax(-1, keepdim=True)                # the first largest
    most = f.gather(1, at)
    inv = torch.where(most == 0, most, torch.full_like(most, -127.0) / most)        # (tensor by tensor: one rounding)
    q = (inv.double() * f.double()).round().clamp(max=127.0)
    d = torch.where(most == 0, most, torch.ones_like(inv) / inv)
    return (q * d.double()).reshape(x.shape)


def _gated(x8, gate, up, down, type, H, I):
    """one expert: x8 [n, H] -> fp64 [n, H]"""
    g, u = x8 @ _dequantised(gate, Q4_K, H).T, x8 @ _dequantised(up, Q4_K, H).T
    return _q8((torch.nn.functional.silu(g) * u)) @ _dequantised(down, type, I).T


def _exact_experts(c, v, ids, weights):
    H, I, E, type = c["hidden"], c["ff"], c["experts"], TYPES[c.get("down", "Q6_K")]
    x8 = _q8(v["x"])
    out = torch.zeros((c["tokens"], H), dtype=torch.float64, device=DEV)
    gate, up, down = v["gate"].view(E, -1), v["up"].view(E, -1), v["down"].view(E, -1)
    for e in torch.unique(ids).tolist():
        tok, slot = torch.where(ids == e)
        out.index_add_(0, tok, _gated(x8[tok], gate[e], up[e], down[e], type, H, I) * weights[tok, slot].double().unsqueeze(-1))
    return out


def _rms(x, w, eps=1e-6):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w.double()


def _exact_latent(c, v):
    B, H, R, W, L = c["batch"], c["heads"], c["q_rank"], c["hidden"], c["ctx"]
    lin = lambda x, w, n: _q8(x) @ _dequantised(v[w], Q4_K, n).T
    x = v["x"].view(B, W)
    q = lin(_rms(lin(x, "q_a", W), v["q_norm"]), "q_b", R).view(B, H, 192)
    kv = lin(x, "kv_a", W)
    ckv, k_pe = _rms(kv[:, :512], v["kv_norm"]), kv[:, 512:]
    inv = (1.0 / (10000.0 ** (torch.arange(0, 64, 2, device=DEV).double() / 64)))
    cos, sin = torch.cos(L * inv).repeat(2), torch.sin(L * inv).repeat(2)

    def turned(t):       # pairs of neighbours, written as halves
        t = t.view(*t.shape[:-1], 32, 2).transpose(-1, -2).reshape(*t.shape)
        return t * cos + torch.cat([-t[..., 32:], t[..., :32]], -1) * sin

    kv_b = v["kv_b"].double().view(H, 256, 512)
    keys = torch.cat([v["past"].double(), torch.cat([ckv, turned(k_pe)], -1).unsqueeze(1)], 1)
    q_abs = torch.einsum("bhd,hdr->bhr", q[..., :128], kv_b[:, :128])
    s = torch.einsum("bhr,blr->bhl", torch.cat([q_abs, turned(q[..., 128:])], -1), keys) * 192 ** -0.5
    lat = torch.einsum("bhl,blr->bhr", torch.softmax(s, -1), keys[..., :512])
    o = torch.einsum("bhr,hdr->bhd", lat, kv_b[:, 128:]).reshape(B, H * 128)
    return lin(o, "o", H * 128).view(B, 1, W)


def _exact_attention(c, v):
    W, H, G, D, T, P = c["width"], c["heads"], c["kv_heads"], c["dim"], c["tokens"], c["before"]
    proj = v["h"].double() @ v["w_in"].double().T + v["b_in"].double()
    q, k, val = proj[:, :H * D].view(T, H, D), proj[:, H * D:(H + G) * D].view(T, G, D), proj[:, (H + G) * D:].view(T, G, D)
    pos = torch.arange(P, P + T, device=DEV)
    n = D // 4
    ang = pos.double().view(-1, 1, 1) * (10000.0 ** (-2.0 * torch.arange(n, device=DEV).double() / (2 * n)))

    def turned(t, w):
        t = _rms(t, w)
        a, b = t[..., :n], t[..., n:2 * n]
        return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin(), t[..., 2 * n:]], -1)

    past = v["past"].double()       # a cache row: the keys of every key/value head, then the values
    k = torch.cat([past[:, :G * D].view(P, G, D), turned(k, v["k_norm"])])
    val = torch.cat([past[:, G * D:].view(P, G, D), val])
    q = turned(q, v["q_norm"])
    j = torch.arange(P + T, device=DEV)
    seen = (j <= pos.view(-1, 1)) & (j // c["chunk"] == (pos // c["chunk"]).view(-1, 1))
    out = torch.empty((T, H, D), dtype=torch.float64, device=DEV)
    for h in range(H):
        g = h // (H // G)
        s = (q[:, h] @ k[:, g].T * D ** -0.5).masked_fill(~seen, -math.inf)
        m = s.max(-1, keepdim=True).values.clamp(min=0.0)
        e = torch.exp(s - m)
        out[:, h] = (e @ val[:, g]) / (e.sum(-1, keepdim=True) + torch.exp(-m))
    return out.view(T, H * D) @ v["o"].double().T


@torch.no_grad()
def exact(case, seed):
    c, v = case, _inputs(case, seed)
    k = c["kind"]
    if k == "experts":
        return _exact_experts(c, v, v["ids"], v["weights"])
    if k == "moe":
        T, E, G = c["tokens"], c["experts"], c["groups"]
        score = torch.sigmoid(v["x"].double() @ v["router"].double().T)
        choice = score + v["correction"].double()
        best = choice.view(T, G, -1).topk(2, -1).values.sum(-1).topk(c["keep"], -1).indices
        kept = torch.zeros((T, G), dtype=torch.bool, device=DEV).scatter_(1, best, True)
        ids = choice.masked_fill(~kept.repeat_interleave(E // G, 1), -math.inf).topk(c["top"], -1).indices
        w = score.gather(1, ids)
        w = w / (w.sum(-1, keepdim=True) + 1e-20) * 2.5
        out = _exact_experts(c, v, ids, w) + _gated(_q8(v["x"]), v["s_gate"], v["s_up"], v["s_down"], Q6_K, c["hidden"], c["ff"])
        return out.view(1, T, -1)
    if k == "linear":
        return _q8(v["x"]) @ _dequantised(v["w"], TYPES[c["type"]], c["n_in"]).T
    if k == "fp8":
        f = v["x"].float().view(c["tokens"], -1, 128)
        most = f.abs().amax(-1, keepdim=True)
        s = most / torch.full_like(most, 448.0)         # (tensor by tensor: one rounding)
        x8 = ((f / s).to(torch.float8_e4m3fn).double() * s.double()).view(c["tokens"], -1)
        scale = v["scale"].double().repeat_interleave(128, 0)[:c["n_out"]].repeat_interleave(128, 1)
        return x8 @ (v["w"].double() * scale).T
    if k == "mla":
        B, per = c["batch"], v["pages"].numel() // c["batch"]
        out = torch.empty((B, c["heads"], 512), dtype=torch.float64, device=DEV)
        for b in range(B):
            rows = v["kv"][v["pages"].view(B, per)[b].long()].reshape(-1, 576)[:int(v["kv_len"][b])].double()
            p = torch.softmax(torch.cat([v["q"][b], v["q_pe"][b]], -1).double() @ rows.T * 192 ** -0.5, -1)
            out[b] = p @ rows[:, :512]
        return out
    if k == "latent_layer":
        return _exact_latent(c, v)
    if k == "attention":
        return _exact_attention(c, v)
    T, top = v["ids"].shape
    x, out = v["x"].double(), torch.zeros((T, c["width"]), dtype=torch.float64, device=DEV)
    for e in torch.unique(v["ids"]).tolist():
        tok, slot = torch.where(v["ids"] == e)
        h = torch.nn.functional.silu(x[tok] @ v["gate"][e].double().T) * (x[tok] @ v["up"][e].double().T)
        out.index_add_(0, tok, (h @ v["down"][e].double().T) * v["weights"][tok, slot].double().unsqueeze(-1))
    return out
