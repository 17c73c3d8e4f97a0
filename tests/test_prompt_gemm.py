"""Tensor-core products of prompt-sized batches (csrc/fp8_linear.cu) through the C-ABI, at the edges of their tiles, against plain torch in 64 bits
on the same quantised operands.  The operands' products are exact, so a result is off by its fp32 sums (n ~ 100 terms of one rounding each: well
below 4e-6 of the largest value) and its last rounding (half a unit: 2^-9 of a bf16, 2^-12 of an fp16)."""
import ctypes as C

import pytest
import torch

from ktransformers_b200 import native

pytestmark = pytest.mark.gpu

F32, F16, BF16 = 0, 1, 30
TORCH = {F32: torch.float32, F16: torch.float16, BF16: torch.bfloat16}
HALF_UNIT = {F32: 2.0 ** -24, F16: 2.0 ** -11, BF16: 2.0 ** -8}      # twice the half unit: a sum at the edge may fall to the other side


def _check(got, want, hid):
    got, want = got.double(), want.double()
    assert ((got - want).abs() <= HALF_UNIT[hid] * want.abs() + 4e-6 * want.abs().max()).all(), (got - want).abs().max().item()


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _rows_untouched(call, y, live, full):
    """rows at or beyond the device-side batch size keep what they held"""
    held = torch.full_like(y, 7.0)
    call(held, torch.tensor([live], dtype=torch.int32, device="cuda"))
    assert torch.equal(held[:live], full[:live]) and (held[live:] == 7.0).all()


# 17 rows: the first batch of this path; 128 / 129: one tile of tokens and a ragged second; N ragged against every tile width, against the scale
# blocks of 128 and against 16-byte stores; 4100: two passes
@pytest.mark.parametrize("T,K,N,hid", [(17, 128, 64, BF16), (128, 1152, 515, BF16), (129, 256, 4096, F16), (300, 2048, 2307, F32), (1000, 384, 20000, BF16), (40, 9216, 200, F32),
                                       (4100, 256, 136, F16)])
def test_fp8_prompt_batches(T, K, N, hid):
    g = torch.Generator(device="cuda").manual_seed(T + K + N)
    x = torch.randn((T, K), generator=g, device="cuda").to(TORCH[hid])
    w = (torch.randn((N, K), generator=g, device="cuda") * 50).clamp_(-448, 448).to(torch.float8_e4m3fn)
    ws = torch.rand(((N + 127) // 128, K // 128), generator=g, device="cuda") * 0.01 + 1e-3
    lib, h = native.lib(), C.c_void_p()
    native.check(lib.ktb200_fp8_linear_create(K, N, w.data_ptr(), ws.data_ptr(), hid, 0, C.byref(h)))

    def call(y, bsz=None):
        native.check(lib.ktb200_fp8_linear_forward(h, T, x.data_ptr(), y.data_ptr(), bsz.data_ptr() if bsz is not None else None, _stream()))

    y = torch.zeros((T, N), dtype=TORCH[hid], device="cuda")
    call(y)
    f = x.float().view(T, -1, 128)
    most = f.abs().amax(-1, keepdim=True)
    s = most / torch.full_like(most, 448.0)
    x8 = ((f / s).to(torch.float8_e4m3fn).double() * s.double()).view(T, K)
    want = x8 @ (w.double() * ws.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)).T
    _check(y, want, hid)
    _rows_untouched(call, y, T - 5, y)
    lib.ktb200_fp8_linear_destroy(h)
