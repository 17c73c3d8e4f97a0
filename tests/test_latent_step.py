"""The decode step of KDeepseekV2Attention with its launches fused (`ktb200_mla_step_prep`) against the module-by-module path of the same operator on
the same inputs: the same cache row up to a unit of bf16 in the last place (its products are rounded once instead of three times), the same lengths,
the same output within the reach of those roundings (4 x 2^-8 of the largest value)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bsz,heads,q_rank,pos", [(1, 128, 256, 0), (3, 16, None, 63), (2, 17, 130, 64), (1, 32, 64, 4095)])
def test_step_equals_the_module_path(bsz, heads, q_rank, pos):
    from ktransformers_b200 import native
    from ktransformers_b200.models.custom_cache import StaticCache
    from ktransformers_b200.models.modeling_deepseek_v3 import DeepseekV3Attention, DeepseekV3Config, DeepseekV3RotaryEmbedding
    from ktransformers_b200.operators.attention import KDeepseekV2Attention
    from ktransformers_b200.operators.flashinfer_wrapper import MLAWrapper

    class OtherRotary(DeepseekV3RotaryEmbedding):      # any other module than the plain one takes the module path
        pass

    torch.manual_seed(pos + heads)
    cfg = DeepseekV3Config(hidden_size=512, num_attention_heads=heads, q_lora_rank=q_rank, num_hidden_layers=1)
    plain = DeepseekV3Attention(cfg, layer_idx=0).to(device="cuda", dtype=torch.bfloat16)
    plain.rotary_emb = DeepseekV3RotaryEmbedding(64).to("cuda")
    outs, rows, lens = [], [], []
    x = torch.randn(bsz, 1, 512, device="cuda").to(torch.bfloat16)
    past = torch.randn(bsz, max(pos, 1), 576, device="cuda").to(torch.bfloat16)
    for rot in (DeepseekV3RotaryEmbedding(64).to("cuda"), OtherRotary(64).to("cuda")):
        plain.rotary_emb = rot
        op = KDeepseekV2Attention("blk.0.self_attn", None, cfg, plain, "cuda", "cuda")
        cache = StaticCache(cfg, max_batch_size=bsz, max_cache_len=pos + 2, device="cuda")
        seq = cache.key_cache[0].view(bsz, -1, 576)
        if pos:
            seq[:, :pos].copy_(past)
        op.mla_wrapper = MLAWrapper(bsz, cache.max_pages * bsz)
        where = torch.full((bsz, 1), pos, dtype=torch.int64, device="cuda")
        n0 = native.launch_count()
        with torch.no_grad():
            y, _, _ = op(x, position_ids=where, past_key_value=cache, cache_position=torch.tensor([pos], device="cuda"))
        launches = native.launch_count() - n0
        assert launches == (5 + (q_rank is not None) if type(rot) is DeepseekV3RotaryEmbedding else 5), launches      # prep | cache write, absorb, attention, merge, absorb (+ norm)
        outs.append(y.float()); rows.append(seq[:, pos].float().clone()); lens.append(op.mla_wrapper.kv_len_arr_buf[:bsz].clone())
        assert cache.get_seq_length(0) == 1
    assert torch.equal(lens[0], lens[1]) and (lens[0] == pos + 1).all()
    assert ((rows[0] - rows[1]).abs() <= 2.0 ** -6 * rows[1].abs() + 2.0 ** -7).all()
    assert (outs[0] - outs[1]).abs().max() <= 2.0 ** -6 * outs[1].abs().max()


def test_step_beyond_its_wrapper_is_refused(monkeypatch):
    """The attention's wrapper keeps the sizes of its first caller.  A step of two sequences on one made for one raises, before the prep kernel
    could write two lengths into one place (here that kernel and the attention are replaced by a failure: neither may be reached)."""
    from ktransformers_b200 import native
    from ktransformers_b200.models.custom_cache import StaticCache
    from ktransformers_b200.models.modeling_deepseek_v3 import DeepseekV3Attention, DeepseekV3Config, DeepseekV3RotaryEmbedding
    from ktransformers_b200.operators.attention import KDeepseekV2Attention
    from ktransformers_b200.operators.flashinfer_wrapper import MLAWrapperSingleton

    real = native.lib()

    class Watched:
        def __getattr__(self, name):
            assert name not in ("ktb200_mla_step_prep", "ktb200_mla_decode"), name
            return getattr(real, name)

    monkeypatch.setattr(MLAWrapperSingleton, "wrappers", {})
    cfg = DeepseekV3Config(hidden_size=512, num_attention_heads=16, q_lora_rank=64, num_hidden_layers=1)
    plain = DeepseekV3Attention(cfg, layer_idx=0).to(device="cuda", dtype=torch.bfloat16)
    plain.rotary_emb = DeepseekV3RotaryEmbedding(64).to("cuda")
    for bsz in (1, 2):
        op = KDeepseekV2Attention("blk.0.self_attn", None, cfg, plain, "cuda", "cuda")
        cache = StaticCache(cfg, max_batch_size=bsz, max_cache_len=128, device="cuda")
        step = lambda: op(torch.randn(bsz, 1, 512, device="cuda").to(torch.bfloat16), position_ids=torch.zeros((bsz, 1), dtype=torch.int64, device="cuda"), past_key_value=cache,
                          cache_position=torch.zeros(1, dtype=torch.int64, device="cuda"))
        with torch.no_grad():
            if bsz == 1:
                step()
            else:
                monkeypatch.setattr(native, "lib", lambda: Watched())
                with pytest.raises((RuntimeError, ValueError)):
                    step()


def test_hooks_of_the_modules_between_the_projections_still_run():
    from ktransformers_b200.models.custom_cache import StaticCache
    from ktransformers_b200.models.modeling_deepseek_v3 import DeepseekV3Attention, DeepseekV3Config, DeepseekV3RotaryEmbedding
    from ktransformers_b200.operators.attention import KDeepseekV2Attention
    from ktransformers_b200.operators.flashinfer_wrapper import MLAWrapper
    cfg = DeepseekV3Config(hidden_size=512, num_attention_heads=16, q_lora_rank=64, num_hidden_layers=1)
    plain = DeepseekV3Attention(cfg, layer_idx=0).to(device="cuda", dtype=torch.bfloat16)
    plain.rotary_emb = DeepseekV3RotaryEmbedding(64).to("cuda")
    op = KDeepseekV2Attention("blk.0.self_attn", None, cfg, plain, "cuda", "cuda")
    cache = StaticCache(cfg, max_batch_size=1, max_cache_len=64, device="cuda")
    op.mla_wrapper = MLAWrapper(1, cache.max_pages)
    for name in ("rotary_emb", "kv_a_layernorm", "q_a_layernorm"):
        for register in ("register_forward_hook", "register_forward_pre_hook"):
            seen = []
            handle = getattr(getattr(plain, name), register)(lambda *a: seen.append(name))
            with torch.no_grad():
                op(torch.randn(1, 1, 512, device="cuda").to(torch.bfloat16), position_ids=torch.zeros((1, 1), dtype=torch.int64, device="cuda"), past_key_value=cache,
                   cache_position=torch.zeros(1, dtype=torch.int64, device="cuda"))
            handle.remove()
            assert seen == [name], (name, register)


@pytest.mark.parametrize("bsz,heads,q_rank,pos", [(1, 128, 256, 70), (3, 16, None, 0), (2, 24, 512, 63)])
def test_one_call_equals_the_calls_one_by_one(bsz, heads, q_rank, pos):
    """Projections on GGUF blocks: the step is one host call (`ktb200_latent_step`) unless something wants to see a module's call; the launches, and so all bits, are the same."""
    from ktransformers_b200 import native
    from ktransformers_b200.models.custom_cache import StaticCache
    from ktransformers_b200.models.modeling_deepseek_v3 import DeepseekV3Attention, DeepseekV3Config, DeepseekV3RotaryEmbedding
    from ktransformers_b200.operators.attention import KDeepseekV2Attention
    from ktransformers_b200.operators.flashinfer_wrapper import MLAWrapper
    from ktransformers_b200.operators.linear import KTransformersLinear
    from ktransformers_b200.util.synth import synth_blocks

    torch.manual_seed(pos + heads)
    hidden = 512
    cfg = DeepseekV3Config(hidden_size=hidden, num_attention_heads=heads, q_lora_rank=q_rank, num_hidden_layers=1)
    plain = DeepseekV3Attention(cfg, layer_idx=0).to(device="cuda", dtype=torch.bfloat16)
    plain.rotary_emb = DeepseekV3RotaryEmbedding(64).to("cuda")
    names = (["q_proj"] if q_rank is None else ["q_a_proj", "q_b_proj"]) + ["kv_a_proj_with_mqa", "o_proj"]
    old = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        for i, n in enumerate(names):
            orig = getattr(plain, n)
            lin = KTransformersLinear("blk.0." + n, None, cfg, orig, "cuda", "KLinearB200", "cuda", None)
            lin.load(w=(synth_blocks(12, orig.in_features * orig.out_features, "cuda", i), 12))
            setattr(plain, n, lin)
        op = KDeepseekV2Attention("blk.0.self_attn", None, cfg, plain, "cuda", "cuda")
    finally:
        torch.set_default_dtype(old)
    x = torch.randn(bsz, 1, hidden, device="cuda").to(torch.bfloat16)
    past = torch.randn(bsz, max(pos, 1), 576, device="cuda").to(torch.bfloat16)
    where = torch.full((bsz, 1), pos, dtype=torch.int64, device="cuda")
    got = []
    for watched in (None, "kv_a_proj_with_mqa", "o_proj"):
        cache = StaticCache(cfg, max_batch_size=bsz, max_cache_len=pos + 2, device="cuda")
        rows = cache.key_cache[0].view(bsz, -1, 576)
        if pos:
            rows[:, :pos].copy_(past)
        op.mla_wrapper = MLAWrapper(bsz, cache.max_pages * bsz)
        seen = []
        hook = getattr(plain, watched).register_forward_hook(lambda *a: seen.append(1)) if watched else None
        assert (op._own_linears(x, bsz) is None) == bool(watched)
        n0 = native.launch_count()
        with torch.no_grad():
            y, _, _ = op(x, position_ids=where, past_key_value=cache, cache_position=torch.tensor([pos], device="cuda"))
        got.append((native.launch_count() - n0, y.clone(), rows[:, :pos + 1].clone(), op.mla_wrapper.kv_len_arr_buf[:bsz].clone(), cache.get_seq_length(0)))
        if hook:
            hook.remove()
            assert seen == [1]
    for other in got[1:]:
        assert got[0][0] == other[0] and got[0][4] == other[4] == 1
        assert all(torch.equal(a, b) for a, b in zip(got[0][1:4], other[1:4]))
    assert got[0][1].isfinite().all() and got[0][1].abs().max() > 0


def _layer(bsz, heads, q_rank, pos):
    """(operator on GGUF projections, input, positions, cache(): a new cache with `pos` tokens of a fixed past)"""
    from ktransformers_b200.models.custom_cache import StaticCache
    from ktransformers_b200.models.modeling_deepseek_v3 import DeepseekV3Attention, DeepseekV3Config, DeepseekV3RotaryEmbedding
    from ktransformers_b200.operators.attention import KDeepseekV2Attention
    from ktransformers_b200.operators.linear import KTransformersLinear
    from ktransformers_b200.util.synth import synth_blocks

    torch.manual_seed(pos + heads)
    cfg = DeepseekV3Config(hidden_size=512, num_attention_heads=heads, q_lora_rank=q_rank, num_hidden_layers=1)
    plain = DeepseekV3Attention(cfg, layer_idx=0).to(device="cuda", dtype=torch.bfloat16)
    plain.rotary_emb = DeepseekV3RotaryEmbedding(64).to("cuda")
    old = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        for i, n in enumerate((["q_proj"] if q_rank is None else ["q_a_proj", "q_b_proj"]) + ["kv_a_proj_with_mqa", "o_proj"]):
            orig = getattr(plain, n)
            lin = KTransformersLinear("blk.0." + n, None, cfg, orig, "cuda", "KLinearB200", "cuda", None)
            lin.load(w=(synth_blocks(12, orig.in_features * orig.out_features, "cuda", i), 12))
            setattr(plain, n, lin)
        op = KDeepseekV2Attention("blk.0.self_attn", None, cfg, plain, "cuda", "cuda")
    finally:
        torch.set_default_dtype(old)
    x = torch.randn(bsz, 1, 512, device="cuda").to(torch.bfloat16)
    past = torch.randn(bsz, max(pos, 1), 576, device="cuda").to(torch.bfloat16)

    def cache():
        c = StaticCache(cfg, max_batch_size=bsz, max_cache_len=pos + 2, device="cuda")
        if pos:
            c.key_cache[0].view(bsz, -1, 576)[:, :pos].copy_(past)
        return c

    return op, x, torch.full((bsz, 1), pos, dtype=torch.int64, device="cuda"), cache


@pytest.mark.parametrize("bsz,heads,q_rank,pos", [(1, 128, 256, 70), (2, 16, None, 200)])
def test_wrappers_of_the_callers_own_keep_their_run(bsz, heads, q_rank, pos):
    """A wrapper class or an instance with another `run` is called, and one planned in pages of 32 tokens over the cache's rows reads its table in those: the bits of the one call."""
    from ktransformers_b200.operators.flashinfer_wrapper import MLAWrapper

    op, x, where, new_cache = _layer(bsz, heads, q_rank, pos)
    seen, got = [], []

    class Counting(MLAWrapper):
        def run(self, *args, **kwargs):
            seen.append("class")
            return super().run(*args, **kwargs)

    def replaced(cache):
        w = MLAWrapper(bsz, cache.max_pages * bsz)
        w.run = lambda *a, **k: (seen.append("instance"), MLAWrapper.run(w, *a, **k))[1]
        return w

    def other_pages(cache):
        n = cache.max_pages * cache.page_size // 32
        w = MLAWrapper(bsz, n * bsz)
        w.plan(None, torch.arange(bsz + 1, dtype=torch.int32, device="cuda") * n, torch.arange(n * bsz, dtype=torch.int32, device="cuda"), where[:, 0].int() + 1, None, heads, 512, 64, 32,
               op.softmax_scale, torch.bfloat16, torch.bfloat16)
        return w

    for make in (lambda cache: MLAWrapper(bsz, cache.max_pages * bsz), lambda cache: Counting(bsz, cache.max_pages * bsz), replaced, other_pages):
        cache = new_cache()
        assert cache.page_size == 64
        op.mla_wrapper = make(cache)
        with torch.no_grad():
            got.append(op(x, position_ids=where, past_key_value=cache, cache_position=where[0])[0])
    assert seen == ["class", "instance"]
    assert got[0].abs().max() > 0 and all(torch.equal(got[0], g) for g in got[1:])


def test_a_step_of_another_type_leaves_no_plan_behind():
    """bf16 hidden states whose queries come out as fp16 are refused where the wrapper is planned ("bf16 only"): not run on a plan that the step made before it knew."""
    from ktransformers_b200.operators.flashinfer_wrapper import MLAWrapper

    op, x, where, new_cache = _layer(1, 16, None, 3)
    plain = op.orig_module
    lin = plain.q_proj
    plain.q_proj = type("Half", (torch.nn.Module,), dict(forward=lambda self, x: lin(x).half()))()
    plain.kv_b_proj.half()
    cache = new_cache()
    w = op.mla_wrapper = MLAWrapper(1, cache.max_pages)
    with torch.no_grad(), pytest.raises(AssertionError, match="bf16 only"):
        op(x, position_ids=where, past_key_value=cache, cache_position=where[0])
    assert w.need_plan
