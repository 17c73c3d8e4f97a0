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
    assert (none[0] == -1).all() and torch.equal(call(0, T)[0], got[0])


# a captured call keeps its scratch whatever is called after it, and calls that overlap on two streams share none: the bits of calls one by one
def test_router_calls_share_nothing():
    from ktransformers_b200 import native
    E, H, k, big, lib = 256, 2048, 8, 4096, native.lib()
    g = torch.Generator(device="cuda").manual_seed(1)
    x, W, bias = (torch.randn(s, generator=g, device="cuda") for s in ((big, H), (E, H), (E,)))
    W *= H ** -0.5
    cfg = native.GateConfig(E, H, k, 8, 4, 0, 0, 1, 2.5, W.data_ptr(), bias.data_ptr(), F32)
    outs = lambda n: (torch.full((n, k), -1, dtype=torch.int64, device="cuda"), torch.zeros((n, k), device="cuda"))
    run = lambda lo, n, o: native.check(lib.ktb200_moe_gate_forward(C.byref(cfg), n, x[lo:].data_ptr(), o[0].data_ptr(), o[1].data_ptr(), None, None, _stream()))
    few, graph = outs(5), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(7, 5, few)
    whole = outs(big)
    run(0, big, whole)
    graph.replay()
    for a, b in zip(few, whole):
        assert torch.equal(a, b[7:12])
    streams, got = [torch.cuda.Stream(), torch.cuda.Stream()], []
    torch.cuda.synchronize()
    for i in range(200):
        with torch.cuda.stream(streams[i & 1]):
            got.append((i, outs(24)))
            run(16 * i, 24, got[-1][1])
    torch.cuda.synchronize()
    for i, o in got:
        for a, b in zip(o, whole):
            assert torch.equal(a, b[16 * i:16 * i + 24])


def _turned(x, heads, pos, inv_freq, rot, layout, norm, w, eps=1e-6):
    """[T][heads * d] in 64 bits: the rows turned and normed, and how large a value's terms are"""
    T, d = x.shape[0], x.shape[1] // heads
    x = x.double().view(T, heads, d)
    whole = (x.square().mean((1, 2), keepdim=True) + eps).rsqrt()
    inv, w = {0: torch.ones_like(whole), 2: whole}.get(norm, (x.square().mean(2, keepdim=True) + eps).rsqrt()), w.double()
    if norm == 3:
        x = x * w
    first = torch.arange(rot // 2, device=x.device) * (1 if layout else 2)
    second = first + (rot // 2 if layout else 1)
    a, b, angle, y, size = x[..., first], x[..., second], pos.double()[:, None, None] * inv_freq, x.clone(), x.abs()
    if rot:
        y[..., first], y[..., second] = a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()
        size[..., first] = size[..., second] = (a.square() + b.square()).sqrt()
    scale = inv * (w.view(heads, d) if norm == 2 else 1.0)
    return (y * scale).view(T, -1), (size * scale.abs()).view(T, -1)


# heads of 64, 128 and 256 columns in both types and layouts, every norm, part of the columns and none turned, one token and many (blocks of units, and fewer units than
# a block's warps); the general kernel takes the same rows at an odd offset.  Both against 64 bits: some ten roundings of fp32 of a value's terms, and of sums of squares of up to 8192
# columns in order of lanes, and half a place of bf16; between the two, sums in another order may move a bf16 by one place
@pytest.mark.parametrize("T,H,G,d,rot,layout,norm,unit_v,dtype", [(1, 64, 8, 128, 64, 1, 1, 0, BF16), (300, 16, 2, 128, 128, 1, 3, 1, BF16), (2100, 4, 4, 64, 32, 0, 1, 0, BF16), (37, 6, 3, 256, 64, 1, 2, 0, BF16),
                                                                  (5, 40, 8, 128, 0, 0, 1, 1, F32), (65, 8, 2, 64, 64, 0, 3, 0, F32), (700, 3, 1, 256, 256, 1, 0, 0, F32), (16, 8, 8, 128, 32, 0, 2, 1, F32)])
def test_rotated_rows(T, H, G, d, rot, layout, norm, unit_v, dtype):
    from ktransformers_b200 import native
    dt, g, n = TORCH[dtype], torch.Generator(device="cuda").manual_seed(T + H), (H + 2 * G) * d
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    proj, inv_freq = rnd(T, n).to(dt), (10000.0 ** (-torch.arange(max(rot // 2, 1), device="cuda").double() / max(rot // 2, 1)))
    q_w, k_w = ((rnd(H * d) if norm == 2 else rnd(d)).to(dt), (rnd(G * d) if norm == 2 else rnd(d)).to(dt))
    page, pages = 64, (T + 63) // 64 + 1
    pos = torch.arange(T, dtype=torch.int32, device="cuda") + 11
    slot, table = torch.zeros(T, dtype=torch.int32, device="cuda"), torch.randperm(pages, generator=g, device="cuda").to(torch.int32)
    lib, out = native.seq_lib(), []
    for pad in (0, 1):      # a row stride of n + 1 and q one column in: no whole vectors
        p = torch.zeros((T, n + pad), dtype=dt, device="cuda")
        p[:, pad:] = proj
        q, cache = torch.zeros((T, H * d), dtype=dt, device="cuda"), torch.full((pages * page, 2 * G * d), 7.0, dtype=dt, device="cuda")
        native.check_seq(lib.ktb200_rope_norm_cache_write(p.data_ptr(), n + pad, pad, pad + H * d, pad + (H + G) * d, H, G, d, d, rot, layout, inv_freq.data_ptr(), norm, q_w.data_ptr(), k_w.data_ptr(), unit_v,
                                                          1e-6, None, 0, None, pos.data_ptr(), slot.data_ptr(), table.data_ptr(), pages, page, cache.data_ptr(), q.data_ptr(), T, dtype, _stream()))
        out.append((q, cache))
    row = table[(pos.long() // page) % pages].long() * page + pos.long() % page
    parts = list(proj.split((H * d, G * d, G * d), 1))
    wq, wk = _turned(parts[0], H, pos, inv_freq, rot, layout, norm, q_w), _turned(parts[1], G, pos, inv_freq, rot, layout, norm, k_w)
    wv = _turned(parts[2], G, pos, inv_freq, 0, layout, 1 if unit_v else 0, k_w)
    for q, cache in out:
        for got, (want, size) in ((q, wq), (cache[row][:, :G * d], wk), (cache[row][:, G * d:], wv)):
            assert ((got.double() - want).abs() <= (2.0 ** -8 if dtype == BF16 else 0.0) * want.abs() + 2.0 ** -20 * size).all()
    for a, b in zip(*out):
        assert torch.isfinite(a.float()).all() and ((a.double() - b.double()).abs() <= (2.0 ** -7 if dtype == BF16 else 2.0 ** -20) * b.double().abs() + 1e-6).all()
        assert dtype != BF16 or (a != b).double().mean() < 0.01
    assert (out[0][1] == 7.0).all(1).sum() == pages * page - T        # (only the tokens' rows were written)


# results in whole sectors (rows and address multiples of 32 bytes), in vectors of 16 and value by value: the same values wherever they go; blocks of K that are no multiple of the
# four whose scales are under way; tiles of 256, 128 and 64 columns, the last one ragged
@pytest.mark.parametrize("T,K,N,hid", [(130, 128, 4096, BF16), (300, 640, 19000, F16), (257, 1152, 19208, BF16), (129, 384, 2064, F32), (1030, 896, 515, BF16), (64, 2048, 1032, F16),
                                         (300, 512, 2068, F32), (200, 256, 19001, F32), (4200, 128, 131, BF16)])
def test_fp8_batches_wherever_results_go(T, K, N, hid):
    from ktransformers_b200 import native
    g = torch.Generator(device="cuda").manual_seed(N)
    w, ws = (torch.randn((N, K), generator=g, device="cuda") * 50).to(torch.float8_e4m3fn), torch.rand(((N + 127) // 128, K // 128), generator=g, device="cuda") / K
    x, dt = torch.randn((T, K), generator=g, device="cuda").to(TORCH[hid]), TORCH[hid]
    lib, h, live = native.lib(), C.c_void_p(), torch.tensor([T - 5], dtype=torch.int32, device="cuda")
    native.check(lib.ktb200_fp8_linear_create(K, N, w.data_ptr(), ws.data_ptr(), hid, 0, C.byref(h)))
    out = []
    for shift in (0, 16 // x.element_size(), 1):
        room = torch.full((T * N + 32,), 7.0, dtype=dt, device="cuda")
        native.check(lib.ktb200_fp8_linear_forward(h, T, x.data_ptr(), room[shift:].data_ptr(), None, _stream()))
        assert (room[:shift] == 7.0).all() and (room[shift + T * N:] == 7.0).all()
        out.append(room[shift:shift + T * N].clone())
        native.check(lib.ktb200_fp8_linear_forward(h, T, x.data_ptr(), room.fill_(7.0)[shift:].data_ptr(), live.data_ptr(), _stream()))
        assert torch.equal(room[shift:shift + (T - 5) * N], out[-1][:(T - 5) * N]) and (room[shift + (T - 5) * N:] == 7.0).all()
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
    f = x.float().view(T, -1, 128)
    s = f.abs().amax(-1, keepdim=True) / 448.0
    x8 = ((f / s).to(torch.float8_e4m3fn).double() * s.double()).view(T, K)
    want = x8 @ (w.double() * ws.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)).T
    off = (out[0].view(T, N).double() - want).norm() / want.norm()
    assert off < {F32: 1e-5, F16: 1e-3, BF16: 4e-3}[hid], off.item()
    lib.ktb200_fp8_linear_destroy(h)


# fp32 results of up to 16 rows: the error against 64 bits is that of sums of four blocks of K (one chain of 12 and 16 blocks: 9.5e-8 to 9.9e-8 and 1.01e-7 to 1.05e-7)
@pytest.mark.parametrize("K,N,most", [(1536, 24576, 9.25e-8), (2048, 20480, 9.5e-8)])
@pytest.mark.parametrize("T", [1, 3, 16])
def test_fp8_rows_in_fp32(T, K, N, most):
    from ktransformers_b200 import native
    g = torch.Generator(device="cuda").manual_seed(5)
    w = (torch.randn((N, K), generator=g, device="cuda") * 60).clamp_(-448, 448).to(torch.float8_e4m3fn)
    ws, x = (torch.rand(((N + 127) // 128, K // 128), generator=g, device="cuda") * 0.6 + 0.7) / 5000, torch.randn((T, K), generator=g, device="cuda")
    y, lib, h = torch.zeros((T, N), device="cuda"), native.lib(), C.c_void_p()
    native.check(lib.ktb200_fp8_linear_create(K, N, w.data_ptr(), ws.data_ptr(), F32, 0, C.byref(h)))
    native.check(lib.ktb200_fp8_linear_forward(h, T, x.data_ptr(), y.data_ptr(), None, _stream()))
    f = x.view(T, -1, 128)
    s = f.abs().amax(-1, keepdim=True) / 448.0
    want = ((f / s).to(torch.float8_e4m3fn).double() * s.double()).view(T, K) @ (w.float().double() * ws.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)).T
    assert ((y.double() - want).norm() / want.norm()).item() < most
    lib.ktb200_fp8_linear_destroy(h)


# 12 and more rows split K by the time of CTAs taken in order (11 splits with a short last one for 10; 3 for 5; 2 for 3); 11 rows as one.  The sums are the same up to their order
@pytest.mark.parametrize("K,N", [(18432, 7168), (4224, 12864), (2944, 19904)])
@pytest.mark.parametrize("T,hid", [(12, BF16), (16, F16), (16, F32)])
def test_fp8_rows_in_other_splits(T, K, N, hid):
    from ktransformers_b200 import native
    g = torch.Generator(device="cuda").manual_seed(T)
    w = (torch.randn((N, K), generator=g, device="cuda") * 60).clamp_(-448, 448).to(torch.float8_e4m3fn)
    ws, x = (torch.rand(((N + 127) // 128, K // 128), generator=g, device="cuda") * 0.6 + 0.7) / 5000, torch.randn((T, K), generator=g, device="cuda").to(TORCH[hid])
    y, few, lib, h = torch.zeros((T, N), dtype=x.dtype, device="cuda"), torch.zeros((T, N), dtype=x.dtype, device="cuda"), native.lib(), C.c_void_p()
    native.check(lib.ktb200_fp8_linear_create(K, N, w.data_ptr(), ws.data_ptr(), hid, 0, C.byref(h)))
    for _ in range(2):      # (the workspace is zero again after a call)
        native.check(lib.ktb200_fp8_linear_forward(h, T, x.data_ptr(), y.data_ptr(), None, _stream()))
        for t in range(0, T, 11):
            native.check(lib.ktb200_fp8_linear_forward(h, min(11, T - t), x[t:].data_ptr(), few[t:].data_ptr(), None, _stream()))
        a, b = y.double(), few.double()
        assert ((a - b).abs() <= {BF16: 2.0 ** -7, F16: 2.0 ** -10, F32: 2.0 ** -20}[hid] * b.abs() + 4e-6 * b.abs().max()).all()
    lib.ktb200_fp8_linear_destroy(h)


# linears of two to eight rows on either side of the line between the row kernels and the GEMM: one row at a time gives the same sums in another order (half a place of the result and
# 4e-6 of the largest), and the launches tell which one ran
@pytest.mark.parametrize("type,K,R,T,hid,launches", [(12, 16384, 7168, 8, BF16, 1), (14, 7168, 18432, 2, BF16, 3), (14, 7168, 18432, 1, BF16, 1), (14, 7168, 18432, 8, F32, 1), (14, 2048, 2048, 8, BF16, 1),
                                                     (14, 1536, 24584, 5, F16, 2), (14, 1536, 24577, 5, F16, 1), (13, 512, 40002, 7, BF16, 2), (13, 4096, 8200, 3, BF16, 3), (13, 10240, 16000, 8, F16, 3)])
def test_few_rows_as_gemms(type, K, R, T, hid, launches):
    from ktransformers_b200 import native
    from ktransformers_b200.util.synth import synth_blocks
    g = torch.Generator(device="cuda").manual_seed(T + R)
    blocks, x = synth_blocks(type, R * K, "cuda", T), torch.randn((T, K), generator=g, device="cuda").to(TORCH[hid])
    bias, lib, h = torch.randn(R, generator=g, device="cuda"), native.lib(), C.c_void_p()
    native.check(lib.ktb200_linear_create(K, R, blocks.data_ptr(), type, hid, T, 0, C.byref(h)))
    native.check(lib.ktb200_linear_load_weights(h, _stream()))
    y, one = (torch.full((T, R), 7.0, dtype=TORCH[hid], device="cuda") for _ in range(2))
    run = lambda x, y, n, bsz=None: native.check(lib.ktb200_linear_forward(h, n, x.data_ptr(), y.data_ptr(), bias.data_ptr(), bsz.data_ptr() if bsz is not None else None, _stream()))
    n0 = native.launch_count()
    run(x, y, T)
    assert native.launch_count() - n0 == launches
    for t in range(T):
        run(x[t:], one[t:], 1)
    a, b = y.double(), one.double()
    assert ((a - b).abs() <= {BF16: 2.0 ** -7, F16: 2.0 ** -10, F32: 2.0 ** -20}[hid] * b.abs() + 4e-6 * b.abs().max()).all()
    held = torch.full_like(y, 7.0)
    run(x, held, T, torch.tensor([T - 1], dtype=torch.int32, device="cuda"))
    assert torch.equal(held[:T - 1], y[:T - 1]) and (held[T - 1:] == 7.0).all()
    lib.ktb200_linear_destroy(h)


# such calls take no scratch where they are captured (the row kernels run: one launch, the bits of the rows one by one), and give the same as ever beside a capture
@pytest.mark.parametrize("type,K,R,T,hid", [(14, 7168, 18432, 2, BF16), (13, 10240, 7168, 8, F16), (14, 2048, 32000, 6, BF16), (14, 7168, 8192, 8, F32)])
def test_few_rows_captured(type, K, R, T, hid):
    from ktransformers_b200 import native
    from ktransformers_b200.util.synth import synth_blocks
    g = torch.Generator(device="cuda").manual_seed(T + R)
    blocks, x = synth_blocks(type, R * K, "cuda", T), torch.randn((T, K), generator=g, device="cuda").to(TORCH[hid])
    lib, h = native.lib(), C.c_void_p()
    native.check(lib.ktb200_linear_create(K, R, blocks.data_ptr(), type, hid, T, 0, C.byref(h)))
    native.check(lib.ktb200_linear_load_weights(h, _stream()))
    one, eager, held = (torch.zeros((T, R), dtype=x.dtype, device="cuda") for _ in range(3))
    run = lambda x, y, n: native.check(lib.ktb200_linear_forward(h, n, x.data_ptr(), y.data_ptr(), None, None, _stream()))
    for t in range(T):
        run(x[t:], one[t:], 1)
    n0 = native.launch_count()
    run(x, eager, T)
    assert (native.launch_count() - n0 > 1) == (hid != F32)        # (fp32 results keep the row kernels everywhere)
    graph, n0 = torch.cuda.CUDAGraph(), native.launch_count()
    with torch.cuda.graph(graph):
        run(x, held, T)
    assert native.launch_count() - n0 == 1
    graph.replay()
    assert torch.equal(held, one)
    assert ((eager.double() - one.double()).abs() <= {BF16: 2.0 ** -7, F16: 2.0 ** -10, F32: 0.0}[hid] * one.double().abs() + (hid != F32) * 4e-6 * one.double().abs().max()).all()
    lib.ktb200_linear_destroy(h)


def _without_memory_for_scratch():
    """Takes what the device has, in pieces down to 1 MB.  A linear and the router run all the same, in other kernels, with the bits of rows one by one and of the usual ones."""
    from ktransformers_b200 import native
    from ktransformers_b200.util.synth import synth_blocks
    T, K, R, g = 4, 7168, 18432, torch.Generator(device="cuda").manual_seed(2)
    blocks, x = synth_blocks(14, R * K, "cuda", T), torch.randn((T, K), generator=g, device="cuda").bfloat16()
    lib, h, stream = native.lib(), C.c_void_p(), _stream()
    native.check(lib.ktb200_linear_create(K, R, blocks.data_ptr(), 14, BF16, T, 0, C.byref(h)))
    native.check(lib.ktb200_linear_load_weights(h, stream))
    few, y = (torch.zeros((T, R), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    for t in range(T):
        native.check(lib.ktb200_linear_forward(h, 1, x[t:].data_ptr(), few[t:].data_ptr(), None, None, stream))
    many = torch.zeros((16, R), dtype=torch.bfloat16, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):      # (the row kernels for as many rows)
        native.check(lib.ktb200_linear_forward(h, T, x.data_ptr(), y.data_ptr(), None, None, _stream()))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, few)
    y.zero_()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    E, k, Tr = 256, 8, 24
    W, xr = torch.randn((E, K), generator=g, device="cuda") * K ** -0.5, torch.randn((Tr, K), generator=g, device="cuda").bfloat16()
    cfg = native.GateConfig(E, K, k, 8, 4, 0, 0, 1, 2.5, W.data_ptr(), None, BF16)
    routed = [(torch.full((Tr, k), -1, dtype=torch.int64, device="cuda"), torch.zeros((Tr, k), device="cuda"), torch.zeros((Tr, E), device="cuda")) for _ in range(2)]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    rt, p, held, taken = C.CDLL("libcudart.so.12"), C.c_void_p(), 1 << 36, []
    while held >= 1 << 20:
        if rt.cudaMalloc(C.byref(p), C.c_size_t(held)):
            held >>= 1
        else:
            taken.append(p.value)
    rt.cudaGetLastError()
    before, n0 = lib.ktb200_last_error(), native.launch_count()
    native.check(lib.ktb200_linear_forward(h, T, x.data_ptr(), y.data_ptr(), None, None, stream))
    assert native.launch_count() - n0 == 1 and lib.ktb200_last_error() == before == b""
    assert lib.ktb200_linear_forward(h, 16, many.data_ptr(), many.data_ptr(), None, None, stream) not in (0, native.EINVAL) and b"scratch" in lib.ktb200_last_error()      # a prompt's size is refused as ever
    for o in routed:
        n0 = native.launch_count()
        native.check(lib.ktb200_moe_gate_forward(C.byref(cfg), Tr, xr.data_ptr(), *[t.data_ptr() for t in o], None, stream))
        torch.cuda.synchronize()
        assert native.launch_count() - n0 == (1 if o is routed[0] else 2)
        while taken:
            rt.cudaFree(C.c_void_p(taken.pop()))
    assert torch.equal(y, few)
    for a, b in zip(*routed):
        assert torch.equal(a, b)


def test_without_memory_for_scratch():
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], capture_output=True, text=True, timeout=300, env=dict(os.environ, PYTHONPATH=root, CUDA_MODULE_LOADING="EAGER"))
    assert r.returncode == 0, r.stdout + r.stderr


if __name__ == "__main__":
    _without_memory_for_scratch()
