"""Soft-max attention of prompt portions (csrc/softmax_attn_tc.cuh: bf16, head size 128, 256 rows per CTA) against plain torch in 64 bits on the same bf16
queries and cache rows.  Weights reach the second product as bf16 (2^-9 of each, independent of one another) and the result is rounded to bf16: 2^-8 of
the result plus 2^-8 of the values' size at the soft-max's average covers both."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


# portions (tokens before, tokens) per sequence; heads per key/value head 8, 4, 1 and 16; ragged against the tile's tokens and against 128 keys; masks
# whose first key lies inside a key tile; every option of the scores
@pytest.mark.parametrize("heads,kv_heads,portions,opts", [
    (64, 8, [(0, 128)], {}),
    (64, 8, [(5, 300), (1000, 77)], {"sink": 1, "gate": 1}),
    (32, 8, [(129, 513)], {"window": 100}),
    (16, 16, [(200, 600)], {"chunk": 192, "head_scale": 1}),
    (64, 4, [(64, 333), (0, 64), (511, 129)], {"softcap": 20.0, "chunk": 512}),
    (64, 8, [(0, 260)], {"bias": 1, "sink": 1, "out_scale": 0.6}),
])
def test_prompt_portions(heads, kv_heads, portions, opts):
    from ktransformers_b200.models.custom_cache import PagedStateCache
    from ktransformers_b200.operators.attention import paged_softmax_attention
    d, g = 128, torch.Generator(device="cuda").manual_seed(heads + len(portions))
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    cache = PagedStateCache([kv_heads * 2 * d], 0, 4096, 4, "cuda")
    cache.key_cache[0].fill_(float("nan"))        # rows that no sequence has written must not matter
    rows = []
    for stage in (0, 1):
        batch = cache.build_batch([(i, [0] * (p[stage] or 1), []) for i, p in enumerate(portions) if p[stage] or stage])
        if not batch.n_tokens:
            continue
        pos, slot = batch.pos.long(), batch.slot.long()
        r = rnd(batch.n_tokens, kv_heads * 2 * d).to(torch.bfloat16)
        cache.key_cache[0][cache.page_table[slot, pos // 64].long(), pos % 64] = r
        rows.append((r, slot, pos))
        cache.commit()
    T = batch.n_tokens
    q = rnd(T, heads, d).to(torch.bfloat16)
    head_scale = torch.rand(heads, generator=g, device="cuda") * 3 - 1 if opts.get("head_scale") else None      # negative ones among them
    sink = rnd(heads) if opts.get("sink") else None
    bias = (torch.rand(heads, generator=g, device="cuda"), torch.rand(heads, generator=g, device="cuda")) if opts.get("bias") else None
    gate = rnd(T, heads * d + 8).to(torch.bfloat16)[:, 8:] if opts.get("gate") else None
    out = torch.empty((T, heads * d + 2), dtype=torch.bfloat16, device="cuda")[:, :heads * d] if opts.get("gate") else None      # rows that are not 16-byte aligned
    o = paged_softmax_attention(q, cache.key_cache[0], batch, cache, heads, kv_heads, d, d, d ** -0.5, head_scale=head_scale, softcap=opts.get("softcap"), window=opts.get("window"),
                                chunk=opts.get("chunk"), dist_bias=bias, sink=sink, gate=gate, out=out, out_scale=opts.get("out_scale", 1.0))
    all_r, all_slot, all_pos = (torch.cat([x[i] for x in rows]) for i in range(3))
    for s in torch.unique(batch.slot.long()).tolist():
        mine = batch.slot == s
        order = all_pos[all_slot == s].argsort()
        kv = all_r[all_slot == s][order].double()
        p = batch.pos[mine].long()
        k, v = kv[:, :kv_heads * d].view(-1, kv_heads, d).repeat_interleave(heads // kv_heads, 1), kv[:, kv_heads * d:].view(-1, kv_heads, d).repeat_interleave(heads // kv_heads, 1)
        sc = torch.einsum("thd,khd->htk", q[mine].double(), k) * d ** -0.5
        if head_scale is not None:
            sc = sc * head_scale.double().view(-1, 1, 1)
        if opts.get("softcap"):
            sc = opts["softcap"] * torch.tanh(sc / opts["softcap"])
        back = p.view(-1, 1) - torch.arange(kv.shape[0], device="cuda").view(1, -1)
        if bias is not None:
            sc = sc - bias[0].double().view(-1, 1, 1) * torch.log1p(bias[1].double().view(-1, 1, 1) * back.clamp(min=0))
        seen = back >= 0
        if opts.get("window"):
            seen &= back < opts["window"]
        if opts.get("chunk"):
            seen &= (p.view(-1, 1) - back) // opts["chunk"] == p.view(-1, 1) // opts["chunk"]
        sc = sc.masked_fill(~seen, -math.inf)
        if sink is not None:
            w = torch.softmax(torch.cat([sc, sink.double().view(-1, 1, 1).expand(-1, sc.shape[1], 1)], -1), -1)[..., :-1]
        else:
            w = torch.softmax(sc, -1)
        want = torch.einsum("htk,khd->thd", w, v)
        reach = torch.sqrt(torch.einsum("htk,khd->thd", w * w, v * v)) * opts.get("out_scale", 1.0)      # bf16 steps of the weights, added as independent
        want = (want * opts.get("out_scale", 1.0)).reshape(int(mine.sum()), -1)
        if gate is not None:
            want = want * torch.sigmoid(gate[mine].double())
        err = (o[mine].double() - want).abs()
        assert (err <= 2.0 ** -8 * want.abs() + 6 * 2.0 ** -9 * reach.reshape(want.shape) + 1e-6).all(), err.max().item()



# steps that mix portions of every length run the 256-row tiles as a whole (a portion of one token among them); few short portions, and keys cut into parts, do not
@pytest.mark.parametrize("heads,kv_heads,portions,opts,tiles", [
    (64, 8, [(0, 128)], {}, 1),
    (64, 8, [(5, 300), (1000, 1), (70, 15), (200, 16)], {"sink": 1, "gate": 1}, 1),
    (64, 8, [(3, 10), (100, 12), (0, 15), (64, 9)], {}, 1),
    (32, 8, [(77, 1), (129, 513), (900, 33), (64, 31)], {"window": 100}, 1),
    (16, 16, [(200, 600), (5, 127), (9, 128)], {"chunk": 192, "head_scale": 1}, 1),
    (64, 4, [(100, 8), (511, 7), (64, 333), (0, 1)], {"softcap": 20.0, "bias": 1, "out_scale": 0.5}, 1),
    (16, 8, [(0, 100)], {}, 0),
    (64, 8, [(900, 1)] * 4, {}, 0),
    (64, 8, [(900, 7)], {}, 0),
])
def test_steps_of_mixed_portions(monkeypatch, heads, kv_heads, portions, opts, tiles):
    from ktransformers_b200 import native
    real, seen = native.seq_lib(), []

    class Watched:
        def __getattr__(self, name):
            if name != "ktb200_softmax_attn":
                return getattr(real, name)
            return lambda a, T, splits, *rest: seen.append(real.ktb200_softmax_attn_prompt_tiles(a, T, splits)) or real.ktb200_softmax_attn(a, T, splits, *rest)

    monkeypatch.setattr(native, "seq_lib", lambda **kw: Watched())
    test_prompt_portions(heads, kv_heads, portions, opts)
    assert seen == [tiles]
