"""The router's and the rotation's kernels for batches: against the same library's calls for one token, and for rows that only its general kernel takes."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
F32, F16, BF16 = 0, 1, 30
TORCH = {F32: torch.float32, F16: torch.float16, BF16: torch.bfloat16}


def _stream():
    return torch.cuda.current_stream().cuda_stream


# one tile of 8 tokens, a ragged second, more tiles than the grid is deep (16), more tokens than there are selectors (64); rows that do not begin at a whole vector;
# a batch whose live size is on the device.  A token's partial sums and their order do not depend on its batch: the same bits
@pytest.mark.parametrize("T,E,H,hid,shift", [(8, 256, 7168, BF16, 0), (9, 64, 2048, F32, 0), (24, 256, 7168, BF16, 1), (33, 160, 5120, F16, 0), (70, 256, 1028, F32, 1), (131, 128, 512, BF16, 0),
                                             (200, 384, 256, F16, 1)])
def test_router_batches(T, E, H, hid, shift):
    from ktransformers_b200 import native
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T * H + shift, generator=g, device="cuda").to(TORCH[hid])[shift:].view(T, H)
    W, bias = torch.randn((E, H), generator=g, device="cuda") * H ** -0.5, torch.rand(E, generator=g, device="cuda")
    k, lib = 6, native.lib()
    cfg = native.GateConfig(E, H, k, 8, 4, 0, 0, 1, 2.5, W.data_ptr(), bias.data_ptr(), hid)

    def call(lo, hi, bsz=None):
        idx, w, logits = torch.full((hi - lo, k), -1, dtype=torch.int64, device="cuda"), torch.zeros((hi - lo, k), device="cuda"), torch.zeros((hi - lo, E), device="cuda")
        native.check(lib.ktb200_moe_gate_forward(C.byref(cfg), hi - lo, x[lo:].data_ptr(), idx.data_ptr(), w.data_ptr(), logits.data_ptr(), bsz.data_ptr() if bsz is not None else None, _stream()))
        return idx, w, logits

    got = call(0, T)
    for a, b in zip(got, zip(*[call(t, t + 1) for t in range(T)])):
        assert torch.equal(a, torch.cat(b))
    assert (got[2].double() - x.double() @ W.double().T).abs().max() < 1e-4
    live = call(0, T, torch.tensor([T - 3], dtype=torch.int32, device="cuda"))
    assert torch.equal(live[0][:T - 3], got[0][:T - 3]) and (live[0][T - 3:] == -1).all()
    none = call(0, T, torch.zeros(1, dtype=torch.int32, device="cuda"))
    assert (none[0] == -1).all() and torch.equal(call(0, T)[0], got[0])        # (the tickets are back at zero)
