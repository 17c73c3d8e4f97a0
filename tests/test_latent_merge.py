"""Latent decode attention (csrc/mla.cu): queries that come as boxes of 64 heads, and the merge of the splits in parts, against plain torch in 64 bits."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


# heads that end inside a box (whose other rows are the next sequence's, here not numbers, or lie beyond the last); splits around the ten that a part of the merge loads at once and its
# four parts; more splits than tiles, and than the merge takes; a sequence without keys; a page of 32 and of 64
@pytest.mark.parametrize("heads,splits,page,lens", [(16, 1, 64, [33, 700]), (63, 9, 32, [300, 1, 2000]), (100, 10, 64, [4000, 0, 31]), (128, 11, 64, [1500]), (64, 21, 32, [3000, 900]),
                                                    (130, 40, 64, [5000, 64]), (16, 74, 64, [9000]), (128, 128, 64, [9000, 4097]), (16, 129, 64, [9000]), (16, 200, 32, [20000, 64, 8191]), (8, 0, 64, [2500, 65, 640])])
def test_queries_and_splits(heads, splits, page, lens):
    from ktransformers_b200 import native
    B, g = len(lens), torch.Generator(device="cuda").manual_seed(heads + splits)
    pages = [(n + page - 1) // page for n in lens]
    most = max(pages)
    kv = torch.randn((sum(pages) + 1, page, 576), generator=g, device="cuda").bfloat16()
    order = torch.randperm(sum(pages), generator=g, device="cuda").to(torch.int32) + 1
    table, at = torch.zeros((B, most), dtype=torch.int32, device="cuda"), 0
    for b, n in enumerate(pages):
        table[b, :n] = order[at:at + n]
        at += n
    q, pe = torch.randn((B, heads, 512), generator=g, device="cuda").bfloat16(), torch.randn((B, heads, 64), generator=g, device="cuda").bfloat16()
    if B > 1:
        q[1] = float("nan")        # (a box of the sequence before it may bring these along)
    kv_len = torch.tensor(lens, dtype=torch.int32, device="cuda")
    out, lse = torch.full((B, heads, 512), 9.0, dtype=torch.bfloat16, device="cuda"), torch.zeros((B, heads), device="cuda")
    lib = native.lib()
    need = lib.ktb200_mla_workspace_bytes(B, heads, 0)
    work = torch.full((need // 4,), float("nan"), device="cuda")
    p = native.MlaParams(B, heads, page, most, splits, 192 ** -0.5, q.data_ptr(), pe.data_ptr(), kv.data_ptr(), table.data_ptr(), kv_len.data_ptr(), out.data_ptr(), lse.data_ptr(), work.data_ptr(), need)
    native.check(lib.ktb200_mla_decode(C.byref(p), torch.cuda.current_stream().cuda_stream))
    for b, n in enumerate(lens):
        if n == 0:
            assert (out[b] == 0).all() and (lse[b] == float("-inf")).all()
            continue
        if b == 1:
            continue
        rows = kv[table[b, :pages[b]].long()].reshape(-1, 576)[:n].double()
        s = torch.cat([q[b], pe[b]], -1).double() @ rows.T * 192 ** -0.5
        want = torch.softmax(s, -1) @ rows[:, :512]
        # probabilities reach the product as bf16 (2^-9 of each) and the result is rounded to bf16
        assert ((out[b].double() - want).norm() / want.norm()).item() < 4e-3
        assert (lse[b].double() - torch.logsumexp(s, -1)).abs().max() < 1e-3


# Scores are sums of 36 products of 16 columns in the tensor core's accumulators, which drop what does not fit at every step: 1.35e-7 (2-norm) in four sums of nine steps that are
# added up in fp32, 5.3e-7 in one of 36.  With one key a head the log-sum-exp is the score (times log2 e and back: three more roundings of 2^-25 on average)
def test_scores_are_four_sums():
    from ktransformers_b200 import native
    B, heads, g, lib = 64, 64, torch.Generator(device="cuda").manual_seed(3), native.lib()
    q, pe, kv = (torch.randn(s, generator=g, device="cuda").bfloat16() for s in ((B, heads, 512), (B, heads, 64), (B, 64, 576)))
    table, kv_len = torch.arange(B, dtype=torch.int32, device="cuda").view(B, 1), torch.ones(B, dtype=torch.int32, device="cuda")
    out, lse, need = torch.zeros_like(q), torch.zeros((B, heads), device="cuda"), lib.ktb200_mla_workspace_bytes(B, heads, 0)
    work = torch.zeros(need // 4, device="cuda")
    p = native.MlaParams(B, heads, 64, 1, 1, 1.0, q.data_ptr(), pe.data_ptr(), kv.data_ptr(), table.data_ptr(), kv_len.data_ptr(), out.data_ptr(), lse.data_ptr(), work.data_ptr(), need)
    native.check(lib.ktb200_mla_decode(C.byref(p), torch.cuda.current_stream().cuda_stream))
    want = (torch.cat([q, pe], -1).double() @ kv[:, 0].double()[:, :, None])[..., 0]
    assert ((lse.double() - want).norm() / want.norm()).item() < 2.5e-7
