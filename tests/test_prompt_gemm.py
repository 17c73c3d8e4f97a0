"""Tensor-core products of prompt-sized batches (csrc/fp8_linear.cu, csrc/kq_gemm.cu) through the C-ABI, at the edges of their tiles, against plain torch in 64 bits
on the same quantised operands.  The operands' products are exact, so a result is off by its fp32 sums (n ~ 100 terms of one rounding each: well
below 4e-6 of the largest value) and its last rounding (half a unit: 2^-9 of a bf16, 2^-12 of an fp16)."""
import ctypes as C

import pytest
import torch

from ktransformers_b200 import native
from ktransformers_b200.util.synth import synth_blocks
from oracle.bindings import Oracle

pytestmark = pytest.mark.gpu

F32, F16, BF16 = 0, 1, 30
Q4_K, Q5_K, Q6_K = 12, 13, 14
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


def _q8(x):
    """Q8_K rounding of activations, in 64 bits: 256 int8 and the fp32 scale of their block"""
    f = x.float().reshape(-1, 256)
    most = f.gather(1, f.abs().argmax(-1, keepdim=True))
    inv = torch.full_like(most, -127.0) / most
    q = (inv.double() * f.double()).round().clamp(max=127.0)
    return (q * (torch.ones_like(inv) / inv).double()).reshape(x.shape)


# 9 rows: the first batch of this path; 64 / 65: one tile of tokens and a ragged second; R ragged against the 128 rows of a matrix and the 256 of a
# tile; one block of K, two blocks (no parts), many (K in parts); every weight type and, for Q6_K, its 8-row groups; 4100: two passes
@pytest.mark.parametrize("type,T,K,R,hid", [(Q4_K, 9, 256, 64, BF16), (Q4_K, 64, 7168, 300, F32), (Q4_K, 65, 512, 40002, BF16), (Q4_K, 200, 1536, 2051, F16), (Q5_K, 16, 2560, 129, F32),
                                            (Q5_K, 130, 256, 38000, BF16), (Q6_K, 17, 768, 1000, F32), (Q6_K, 257, 3072, 520, BF16), (Q6_K, 33, 256, 38400, F16), (Q4_K, 4100, 256, 272, BF16)])
def test_k_quant_prompt_batches(type, T, K, R, hid):
    blocks = synth_blocks(type, R * K, "cuda", T + K + R)
    dense = torch.from_numpy(Oracle().to_float(blocks.cpu().numpy(), type, R * K)).cuda().view(R, K)
    g = torch.Generator(device="cuda").manual_seed(T + R)
    x = torch.randn((T, K), generator=g, device="cuda").to(TORCH[hid])
    bias = torch.randn(R, generator=g, device="cuda")
    lib, h = native.lib(), C.c_void_p()
    native.check(lib.ktb200_linear_create(K, R, blocks.data_ptr(), type, hid, T, 0, C.byref(h)))
    native.check(lib.ktb200_linear_load_weights(h, _stream()))

    def call(y, bsz=None):
        native.check(lib.ktb200_linear_forward(h, T, x.data_ptr(), y.data_ptr(), bias.data_ptr(), bsz.data_ptr() if bsz is not None else None, _stream()))

    y = torch.zeros((T, R), dtype=TORCH[hid], device="cuda")
    call(y)
    _check(y, _q8(x) @ dense.double().T + bias.double(), hid)
    _rows_untouched(call, y, T - 3, y)
    lib.ktb200_linear_destroy(h)


# results that are infinite, not numbers or subnormal leave as ggml rounds fp32 to bf16 (subnormals to zero, a NaN keeps its upper bits): the same sums in fp32, rounded here.
# 17 and 70 tokens: a partly filled group of eight at a tile's end, in the first tile and in a second; 1538 rows: two in the last tile
@pytest.mark.parametrize("T", [17, 70])
def test_k_quant_prompt_batches_round_special_results(T):
    K, R = 256, 1538
    blocks = synth_blocks(Q4_K, R * K, "cuda", T).view(R, 144)
    d = blocks[:, 0:2].view(torch.int16)
    d[0], d[1], d[2], d[R - 2], d[R - 1] = 0x7c00, 0x7e01, 1, 0x7c00, 1        # infinity, NaN, the smallest subnormal scale
    blocks[torch.tensor([2, R - 1]), 2:4] = 0
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn((T, K), generator=g, device="cuda").bfloat16()
    x[3], x[T - 1] = x[3] * 2.0 ** -112, x[T - 1] * 2.0 ** -112
    lib, ys = native.lib(), {}
    for hid in (F32, BF16):
        h, xt = C.c_void_p(), x.to(TORCH[hid])
        y = ys[hid] = torch.zeros((T, R), dtype=TORCH[hid], device="cuda")
        native.check(lib.ktb200_linear_create(K, R, blocks.data_ptr(), Q4_K, hid, T, 0, C.byref(h)))
        native.check(lib.ktb200_linear_load_weights(h, _stream()))
        native.check(lib.ktb200_linear_forward(h, T, xt.data_ptr(), y.data_ptr(), None, None, _stream()))
        torch.cuda.synchronize()
        lib.ktb200_linear_destroy(h)
    i = ys[F32].view(torch.int32).long() & 0xffffffff
    size = i & 0x7fffffff
    want = torch.where(size > 0x7f800000, (i >> 16) | 64, torch.where(size < 0x00800000, (i >> 31) << 15, (i + 0x7fff + ((i >> 16) & 1)) >> 16))
    assert (size > 0x7f800000).any() and (size == 0x7f800000).any() and ((size > 0) & (size < 0x00800000)).any()
    assert torch.equal(ys[BF16].view(torch.int16).long() & 0xffff, want)


# experts with no token, one token, 64, 65 and all tokens; an expert named twice by a token and ids beyond the experts; gate and up of one
# 128-row tile and of several; down in both layouts
@pytest.mark.parametrize("gu,down,H,I,T", [(Q4_K, Q6_K, 256, 256, 48), (Q4_K, Q4_K, 512, 256, 131), (Q4_K, Q6_K, 1024, 768, 200), (Q4_K, Q6_K, 2048, 512, 1100), (Q5_K, Q5_K, 768, 512, 100),
                                           (Q6_K, Q6_K, 512, 256, 70)])
def test_experts_of_a_prompt_at_tile_edges(gu, down, H, I, T):
    import gpu_util as G
    E, k = 6, 3
    gate, up, dn = synth_blocks(gu, E * I * H, "cuda", 1), synth_blocks(gu, E * I * H, "cuda", 2), synth_blocks(down, E * H * I, "cuda", 3)
    orc = Oracle()
    dense = [torch.from_numpy(orc.to_float(t.cpu().numpy(), q, t_n)).cuda().view(E, r, c) for t, q, t_n, r, c in
             ((gate, gu, E * I * H, I, H), (up, gu, E * I * H, I, H), (dn, down, E * H * I, H, I))]
    gen = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn((T, H), generator=gen, device="cuda") / 10
    w = torch.rand((T, k), generator=gen, device="cuda")
    ids = torch.full((T, k), 0, dtype=torch.int64, device="cuda")      # expert 0: every token
    ids[:, 1] = 1 + (torch.arange(T, device="cuda") >= min(65, T - 1)).long() * 4      # expert 1: 65 tokens, expert 5: the others
    ids[:, 2] = -1
    ids[:min(64, T), 2] = 3                                             # expert 3: 64 tokens
    ids[T - 1, 2] = 4                                                   # expert 4: one token; expert 2: none
    ids[0, 1] = 0                                                       # twice the same expert
    ids[1, 2] = E + 7
    m = G.Moe(E, k, H, I, gate, up, dn, gu, gu, down, F32, max_tokens=T)
    got = torch.from_numpy(m.forward(ids.cpu().numpy(), w.cpu().numpy(), x.cpu().numpy())).cuda()
    x8, want = _q8(x), torch.zeros((T, H), dtype=torch.float64, device="cuda")
    for e in range(E):
        tok, slot = torch.where(ids == e)
        if len(tok):
            a = torch.nn.functional.silu(x8[tok] @ dense[0][e].double().T) * (x8[tok] @ dense[1][e].double().T)
            want.index_add_(0, tok, (_q8(a) @ dense[2][e].double().T) * w[tok, slot].double().unsqueeze(-1))
    # an activation at the edge of two int8 steps may fall to either side: a unit of 1/127 of its block's largest, in a few values of a row
    assert (got.double() - want).norm() <= 1e-3 * want.norm()
    assert (got.double() - want).abs().max() <= 2e-2 * want.abs().max()
    m.close()


# an MLP of a prompt portion against the CPU oracle (its bounds are those of the decode kernels: an activation whose rounding falls to the other side moves a
# quantised value by one step), with the rounded sum of `accumulate` and a device-side batch size
@pytest.mark.parametrize("gate,up,down,H,I,T", [(Q4_K, Q4_K, Q6_K, 512, 256, 9), (Q4_K, Q5_K, Q4_K, 1024, 768, 64), (Q6_K, Q6_K, Q6_K, 768, 512, 65), (Q5_K, Q5_K, Q5_K, 256, 1280, 130),
                                                (Q4_K, Q4_K, Q6_K, 2048, 512, 1100)])
@pytest.mark.parametrize("hid", [F32, BF16])
def test_mlp_of_a_prompt(gate, up, down, H, I, T, hid):
    g, u, d = (synth_blocks(t, n, seed=i + 3) for i, (t, n) in enumerate(((gate, I * H), (up, I * H), (down, H * I))))
    rnd = torch.Generator().manual_seed(T)
    x, y0 = (torch.randn(T, H, generator=rnd) / 100).to(TORCH[hid]), torch.randn(T, H, generator=rnd).to(TORCH[hid])
    host = lambda t: (t.view(torch.int16).numpy().view("uint16") if hid == BF16 else t.numpy())
    want = torch.from_numpy(Oracle().mlp_forward(H, I, g.cpu().numpy(), u.cpu().numpy(), d.cpu().numpy(), gate, up, down, hid, host(x)).copy().view("int16" if hid == BF16 else "float32"))
    want = want.view(TORCH[hid]).view(T, H)
    lib, h, w = native.lib(), C.c_void_p(), [t.cuda() for t in (g, u, d)]
    native.check(lib.ktb200_mlp_create(H, I, *[t.data_ptr() for t in w], gate, up, down, hid, T, 0, C.byref(h)))
    native.check(lib.ktb200_mlp_load_weights(h, _stream()))
    xd, live = x.cuda(), torch.tensor([T - 5], dtype=torch.int32, device="cuda")
    for accumulate in (0, 1):
        y = y0.cuda()
        native.check(lib.ktb200_mlp_forward(h, T, xd.data_ptr(), y.data_ptr(), accumulate, live.data_ptr(), _stream()))
        got, ref = y.cpu(), (y0 + want if accumulate else want)
        assert torch.equal(got[T - 5:], y0[T - 5:])
        diff, size = (got[:T - 5].double() - ref[:T - 5].double()).abs(), want.double().abs().max()
        # bf16: the MLP's rows are rounded, then their sum with what was there; each may fall to the other side, one unit (at most 2^-7) of either
        units = 2.0 ** -7 * (ref.double().abs() + want.double().abs())[:T - 5] if hid == BF16 else 0
        assert (diff <= units + 1e-3 * size).all(), (diff / size).max().item()
    lib.ktb200_mlp_destroy(h)


# Activations of one sign and about one size: an ordinary Q5_K block then sums to about 20 million, beyond the 2^24 of an fp32 accumulator, and its minima take most of
# it away again; and blocks at the largest sums their format has.  The decode kernels, 8 rows at a time, round a block's sum once: the prompt's may not be further
# from 64 bits than they are, or than two units of fp32.  Rows in between are ordinary ones (marked and other blocks beside each other), and the order of the rows must not matter
@pytest.mark.parametrize("type", [Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("K,R,T", [(256, 3000, 9), (512, 520, 65), (7168, 1024, 130), (4096, 20000, 320)])
@pytest.mark.parametrize("weights", ["ordinary", "largest"])
def test_k_quant_sums_beyond_an_fp32_accumulator(type, K, R, T, weights):
    b = synth_blocks(type, R * K, "cuda", T + K).view(R * K // 256, -1)
    if weights == "largest":
        b[:, 4 if type != Q6_K else 0:208] = 255      # (d and dmin of the first, d of the second lie outside)
        if type == Q6_K:
            b[:, 192:208] = 127
        b[::7, 20:60] = 170
    elif type != Q6_K:       # minima like the scales times the middle quant: values about 0
        b[:, 8:12] = b[:, 4:8]
        b[:, 12:16] = (b[:, 12:16] & 15) * 17
        d = b[:, 0:2].contiguous().view(torch.float16).float()
        b[:, 2:4] = (d * (7.5 if type == Q4_K else 15.5)).to(torch.float16).view(torch.uint8)
    blocks = b.reshape(-1)
    dense = torch.from_numpy(Oracle().to_float(blocks.cpu().numpy(), type, R * K)).cuda().view(R, K)
    g = torch.Generator(device="cuda").manual_seed(K)
    x = torch.randn((T, K), generator=g, device="cuda")
    flat = torch.arange(T, device="cuda") % 3 != 1
    x[flat] = 1 + 0.01 * x[flat]
    lib, h = native.lib(), C.c_void_p()
    native.check(lib.ktb200_linear_create(K, R, blocks.data_ptr(), type, F32, T, 0, C.byref(h)))
    native.check(lib.ktb200_linear_load_weights(h, _stream()))

    def call(x):
        y = torch.zeros((x.shape[0], R), device="cuda")
        native.check(lib.ktb200_linear_forward(h, x.shape[0], x.data_ptr(), y.data_ptr(), None, None, _stream()))
        return y

    want = _q8(x) @ dense.double().T
    y, rows = call(x), torch.cat([call(x[t:t + 8].contiguous()) for t in range(0, T, 8)])
    for part in (flat, ~flat):
        off, off_rows = (((v[part].double() - want[part]).norm() / want[part].norm()).item() for v in (y, rows))
        assert off <= max(1.1 * off_rows, 2.0 ** -23), (off, off_rows)
    order = torch.randperm(T, generator=g, device="cuda")
    assert torch.equal(call(x[order].contiguous()), y[order])
    lib.ktb200_linear_destroy(h)


# matrices so small that the launches of the GEMM cost more than the row kernels (the FP8 passes) take: (path, K, R or N, rows, launches)
@pytest.mark.parametrize("kind,K,R,T,launches", [("linear", 512, 512, 32, 1), ("linear", 512, 512, 41, 2), ("linear", 4096, 64, 11, 1), ("linear", 4096, 64, 12, 3), ("q6", 512, 512, 20, 1),
                                                 ("q6", 512, 512, 24, 2), ("fp8", 7168, 576, 24, 4), ("fp8", 7168, 576, 25, 2), ("fp8", 16384, 72, 48, 6), ("fp8", 512, 512, 17, 2),
                                                 ("mlp", 512, 512, 17, 2), ("mlp", 512, 512, 18, 6), ("mlp", 512, 256, 39, 2), ("mlp", 512, 256, 40, 6)])
def test_small_matrices_keep_the_kernels_of_few_rows(kind, K, R, T, launches):
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn((T, K), generator=g, device="cuda").to(torch.bfloat16)
    lib, h = native.lib(), C.c_void_p()
    out = K if kind == "mlp" else R
    if kind == "fp8":
        w, ws = (torch.randn((R, K), generator=g, device="cuda") * 50).to(torch.float8_e4m3fn), torch.rand(((R + 127) // 128, K // 128), generator=g, device="cuda")
        native.check(lib.ktb200_fp8_linear_create(K, R, w.data_ptr(), ws.data_ptr(), BF16, 0, C.byref(h)))
        run = lambda x, y: lib.ktb200_fp8_linear_forward(h, x.shape[0], x.data_ptr(), y.data_ptr(), None, _stream())
    elif kind == "mlp":
        keep = [synth_blocks(t, R * K, "cuda", i) for i, t in enumerate((Q4_K, Q4_K, Q6_K))]
        native.check(lib.ktb200_mlp_create(K, R, *[t.data_ptr() for t in keep], Q4_K, Q4_K, Q6_K, BF16, T, 0, C.byref(h)))
        native.check(lib.ktb200_mlp_load_weights(h, _stream()))
        run = lambda x, y: lib.ktb200_mlp_forward(h, x.shape[0], x.data_ptr(), y.data_ptr(), 0, None, _stream())
    else:
        q = Q6_K if kind == "q6" else Q4_K
        keep = synth_blocks(q, R * K, "cuda", 1)
        native.check(lib.ktb200_linear_create(K, R, keep.data_ptr(), q, BF16, T, 0, C.byref(h)))
        native.check(lib.ktb200_linear_load_weights(h, _stream()))
        run = lambda x, y: lib.ktb200_linear_forward(h, x.shape[0], x.data_ptr(), y.data_ptr(), None, None, _stream())
    y, few = (torch.zeros((T, out), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    n0 = native.launch_count()
    native.check(run(x, y))
    assert native.launch_count() - n0 == launches
    for t in range(0, T, 8):
        native.check(run(x[t:t + 8], few[t:t + 8]))
    # the same sums in another order: a value at the edge of two bf16 steps falls to the other; an activation of the MLP at the edge of two int8 steps moves a row by 1e-3
    size = few.double().abs().max()
    assert ((y.double() - few.double()).abs() <= 2.0 ** -7 * few.double().abs() + (1e-3 if kind == "mlp" else 4e-6) * size).all()
    (lib.ktb200_fp8_linear_destroy if kind == "fp8" else lib.ktb200_mlp_destroy if kind == "mlp" else lib.ktb200_linear_destroy)(h)


# the same through routed experts: rows in between with marked blocks, against the per-pair kernels (8 tokens at a time)
@pytest.mark.parametrize("gu,down", [(Q4_K, Q6_K), (Q5_K, Q5_K), (Q6_K, Q4_K)])
def test_experts_with_flat_activations(gu, down):
    import gpu_util as G
    E, k, H, I, T = 4, 2, 1024, 512, 200
    w = synth_blocks(gu, E * I * H, "cuda", 1), synth_blocks(gu, E * I * H, "cuda", 2), synth_blocks(down, E * H * I, "cuda", 3)
    gen = torch.Generator().manual_seed(T)
    x = torch.randn((T, H), generator=gen) / 10
    x[::3] = 0.1 + 0.001 * x[::3]
    ids, wt = torch.stack([torch.randperm(E, generator=gen)[:k] for _ in range(T)]).numpy(), torch.rand((T, k), generator=gen).numpy()
    m = G.Moe(E, k, H, I, *w, gu, gu, down, F32, max_tokens=T)
    got = torch.from_numpy(m.forward(ids, wt, x.numpy()))
    want = torch.cat([torch.from_numpy(m.forward(ids[t:t + 8], wt[t:t + 8], x[t:t + 8].numpy())) for t in range(0, T, 8)])
    assert torch.isfinite(got).all() and (got - want).norm() <= 1e-3 * want.norm()
    m.close()


# fp32 results of long rows: no further from 64 bits than the row kernels, whose lanes add short chains of blocks (parts, and many tiles without parts of their own)
@pytest.mark.parametrize("type", [Q4_K, Q6_K])
@pytest.mark.parametrize("K,R,T", [(16384, 256, 64), (4096, 8192, 260)])
def test_k_quant_long_rows_in_fp32(type, K, R, T):
    blocks = synth_blocks(type, R * K, "cuda", K)
    dense = torch.from_numpy(Oracle().to_float(blocks.cpu().numpy(), type, R * K)).cuda().view(R, K)
    x = torch.randn((T, K), generator=torch.Generator(device="cuda").manual_seed(R), device="cuda")
    lib, h = native.lib(), C.c_void_p()
    native.check(lib.ktb200_linear_create(K, R, blocks.data_ptr(), type, F32, T, 0, C.byref(h)))
    native.check(lib.ktb200_linear_load_weights(h, _stream()))

    def call(x):
        y = torch.zeros((x.shape[0], R), device="cuda")
        native.check(lib.ktb200_linear_forward(h, x.shape[0], x.data_ptr(), y.data_ptr(), None, None, _stream()))
        return y

    want = _q8(x) @ dense.double().T
    off, off_rows = ((v.double() - want).norm().item() for v in (call(x), torch.cat([call(x[t:t + 8].contiguous()) for t in range(0, T, 8)])))
    assert off <= 1.05 * off_rows, (off, off_rows)
    lib.ktb200_linear_destroy(h)


# decode batches between the row kernels' 8 tokens and the prompt sizes: what the rule sends to the GEMMs agrees with the row kernels (8 tokens at a time); a shared expert
# whose handle takes fewer tokens keeps the batch with the row kernels, where it rides along
@pytest.mark.parametrize("T", [9, 24, 47])
def test_decode_batches_as_gemms(T):
    import gpu_util as G
    E, k, H, I = 32, 6, 2048, 1536
    gate, up, down = synth_blocks(Q4_K, E * I * H, "cuda", 1), synth_blocks(Q4_K, E * I * H, "cuda", 2), synth_blocks(Q6_K, E * H * I, "cuda", 3)
    shared = [synth_blocks(t, I * H, "cuda", 4 + i) for i, t in enumerate((Q4_K, Q4_K, Q6_K))]
    m = G.Moe(E, k, H, I, gate, up, down, Q4_K, Q4_K, Q6_K, BF16, max_tokens=64)
    lib, handles = native.lib(), []
    for most in (64, 8):
        h, keep = C.c_void_p(), [t.clone() for t in shared]
        native.check(lib.ktb200_mlp_create(H, I, *[t.data_ptr() for t in keep], Q4_K, Q4_K, Q6_K, BF16, most, 0, C.byref(h)))
        native.check(lib.ktb200_mlp_load_weights(h, _stream()))
        handles.append((h, keep))
    (big, _), (small, _) = handles
    g = torch.Generator(device="cuda").manual_seed(T)
    x = (torch.randn((T, H), generator=g, device="cuda") / 10).bfloat16()
    w = torch.rand((T, k), generator=g, device="cuda")
    ids = torch.rand((T, E), generator=g, device="cuda").argsort(-1)[:, :k].contiguous()
    assert [lib.ktb200_moe_takes_gemms(m.h, None, t, k) for t in (1, 8, T, 48)] == [0, 0, 1, 1]
    assert lib.ktb200_moe_takes_gemms(m.h, big, T, k) == 1 and lib.ktb200_moe_takes_gemms(m.h, small, T, k) == 0

    def call(sh, n0, n1, y, bsz=None):
        native.check(lib.ktb200_moe_forward_shared(m.h, sh, n1 - n0, k, ids[n0:n1].data_ptr(), w[n0:n1].data_ptr(), x[n0:n1].data_ptr(), y[n0:n1].data_ptr(),
                                                   bsz.data_ptr() if bsz is not None else None, _stream()))

    for sh in (None, big, small):
        y, few = (torch.zeros((T, H), dtype=torch.bfloat16, device="cuda") for _ in range(2))
        n0 = native.launch_count()
        call(sh, 0, T, y)
        assert (native.launch_count() - n0 >= 10) == (sh is not small)
        for t in range(0, T, 8):
            call(sh, t, min(t + 8, T), few)
        # the same sums in another order: to the last bf16 place (two with a shared term), and an activation at the edge of two int8 steps moves a row by 1e-3
        size = few.double().abs().max()
        assert ((y.double() - few.double()).abs() <= 2.0 ** (-6 if sh else -7) * few.double().abs() + 2e-3 * size).all()
        held = torch.full_like(y, 7.0)
        call(sh, 0, T, held, torch.tensor([T - 2], dtype=torch.int32, device="cuda"))
        assert torch.equal(held[:T - 2], y[:T - 2]) and (held[T - 2:] == 7.0).all()
    for h, _ in handles:
        lib.ktb200_mlp_destroy(h)
    m.close()
