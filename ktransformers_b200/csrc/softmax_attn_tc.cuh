// Soft-max attention of prompt portions on tcgen05 (bf16, one map, head sizes 128): the prompt-sized twin of window_softmax_attn_mma_kernel
// (softmax_attn.cu), with its masks, scores, sink and gate.
//
// A CTA owns 256 rows = (token, query head) pairs of one sequence portion and one key/value head as two tiles of 128 (RH heads of 128 / RH consecutive
// tokens each); keys run in tiles of 128 from the 128-aligned position at or below the first visible key.
//     warp 0       TMA: Q once (3-D boxes: 64 columns x RH heads x 128 / RH tokens), then K and V tiles, two stages each; a tile is two runs of 64
//                  keys, each inside one page (pages are multiples of 64 tokens)
//     warp 1       MMAs: S = Q K^T from shared memory, O += P V with P in tensor memory.  The tiles take turns, S of the next key tile
//                  right behind PV of this one, so that one tile's soft-max runs beside the other's products
//     warps 4-7    soft-max of the first tile, 8-11 of the second: a thread owns a row, so that maximum and sum need no exchange.  P (bf16) replaces
//                  its S in tensor memory; the reference maximum is raised, and O scaled in tensor memory, only when a row's maximum grows by
//                  more than 2^8 (P <= 256 in between, where bf16 and fp32 are as exact as below 1)
// TMEM: [S0 | O0 | S1 | O1], 128 columns each.  Shared memory: Q 64 KB, K and V 2 x 32 KB each.
// Bounds: 16 products of 64 cycles per (row tile, key tile), 2,050 cycles of tensor pipe for two tiles, 95-105 us for 2048 tokens behind 2048, 64 heads over 8; beside them
// 128 exponentials per thread at 4 per cycle and scheduler, 1,024 cycles a warp and as much as the products for the two warps that share a scheduler.  It takes 247 us: a row's
// maximum, exponentials, conversions and stores run one after the other in its thread, the tile's next product waits for all of them, and there is one score buffer a tile (tensor
// pipe 48 % active, issue slots 35 %).
#pragma once
#include <cuda.h>

#include "key_runs.h"
#include "umma.cuh"

namespace ktb {

constexpr int kTcThreads = 384, kTcKeys = 128, kTcTile = 128 * 128 * 2, kTcSmem = 6 * kTcTile + 1024 + 256;
// CTAs from which this kernel is taken: at 40 (600 tokens, 16 heads over 2) the layer took 70 us against 85 us with the 64-row tiles, which spread
// shorter portions over more SMs
constexpr int kTcMinCtas = 32;
struct TcMisc {
    unsigned long long q_full, k_full[2], k_free[2], v_full[2], v_free[2], s_full[2], p_full[2], o_done[2];
    uint32_t tmem_base;
    int info[3];
};

__device__ __forceinline__ float tc_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__global__ void __launch_bounds__(kTcThreads, 1) softmax_attn_tc_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kvmap, const SmAttn a) {
    using namespace umma;
    extern __shared__ __align__(16) uint8_t tc_smem[];
    const uint32_t raw = smem_u32(tc_smem), base = (raw + 1023u) & ~1023u;
    uint8_t* smem = tc_smem + (base - raw);
    const uint32_t kbase = base + 2 * kTcTile, vbase = base + 4 * kTcTile;
    TcMisc& misc = *reinterpret_cast<TcMisc*>(smem + 6 * kTcTile);
    const int tid = threadIdx.x, lane = tid & 31, warp = uniform(tid >> 5);
    const int RH = a.RH, TOKS = 128 / RH, R = a.H / a.G, hblocks = R / RH;
    if (tid == 0) {      // which sequence portion and which of its tokens this CTA covers; the last tiles, which see most keys, come first
        int b = gridDim.y - 1 - blockIdx.y, found = -1, off = 0, len = 0;
        for (int s = 0; s < a.n_seqs; s++) {
            len = a.seqs[a.seqs_stride + s];
            const int nt = (len + 2 * TOKS - 1) / (2 * TOKS);
            if (b < nt) { found = s; off = b * 2 * TOKS; break; }
            b -= nt;
        }
        misc.info[0] = found;
        misc.info[1] = found >= 0 ? a.seqs[found] + off : 0;
        misc.info[2] = found >= 0 ? min(2 * TOKS, len - off) : 0;
        bar_init(smem_u32(&misc.q_full), 1);
        for (int i = 0; i < 2; i++) {
            bar_init(smem_u32(&misc.k_full[i]), 1); bar_init(smem_u32(&misc.k_free[i]), 1); bar_init(smem_u32(&misc.v_full[i]), 1); bar_init(smem_u32(&misc.v_free[i]), 1);
            bar_init(smem_u32(&misc.s_full[i]), 1); bar_init(smem_u32(&misc.p_full[i]), 4); bar_init(smem_u32(&misc.o_done[i]), 1);
        }
        bar_fence_init();
    }
    __syncthreads();
    if (misc.info[0] < 0) return;
    if (warp == 1) tmem_alloc(smem_u32(&misc.tmem_base), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = uniform(misc.tmem_base);
    const int tok0 = misc.info[1], ntok = misc.info[2];
    const int g = blockIdx.x / hblocks, h0 = g * R + (blockIdx.x % hblocks) * RH;
    const int pos0 = a.pos[tok0], max_pos = pos0 + ntok - 1, lo = first_visible(pos0, a.window, a.chunk);
    const int t0 = lo / kTcKeys, n = max_pos / kTcKeys - t0 + 1;

    // registers: 168 a thread at launch; a soft-max thread holds a row of 128 scores (2 x 208 + 88 = 3 x 168)
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    if (warp == 0) {
        // ================================================================ copies
        if (lane == 0) {
            const uint32_t qf = smem_u32(&misc.q_full);
            bar_expect_tx(qf, 2 * kTcTile);
#pragma unroll
            for (int t = 0; t < 2; t++)
#pragma unroll
                for (int c = 0; c < 2; c++) tma_load_3d(base + t * kTcTile + c * (kTcTile / 2), &qmap, qf, 64 * c, h0, tok0 + t * TOKS);
            const int* pt = a.page_table + (long)a.slot[tok0] * a.max_pages;
            for (int j = 0; j < n; j++) {
                const int st = j & 1, ph = ((j >> 1) & 1) ^ 1;
                int row[2];
#pragma unroll
                for (int i = 0; i < 2; i++) {      // (keys outside [lo, max_pos] that come along are masked, and their values zeroed)
                    const int kp = key_run((t0 + j) * kTcKeys, i, lo, max_pos);
                    row[i] = pt[(kp / a.page_size) % a.max_pages] * a.page_size + kp % a.page_size;
                }
                const uint32_t kf = smem_u32(&misc.k_full[st]), vf = smem_u32(&misc.v_full[st]);
                bar_wait(smem_u32(&misc.k_free[st]), ph);
                bar_expect_tx(kf, kTcTile);
#pragma unroll
                for (int i = 0; i < 4; i++) tma_load_2d(kbase + st * kTcTile + (i & 1) * (kTcTile / 2) + (i >> 1) * (kTcTile / 4), &kvmap, kf, g * 128 + 64 * (i & 1), row[i >> 1]);
                bar_wait(smem_u32(&misc.v_free[st]), ph);
                bar_expect_tx(vf, kTcTile);
#pragma unroll
                for (int i = 0; i < 4; i++) tma_load_2d(vbase + st * kTcTile + (i & 1) * (kTcTile / 2) + (i >> 1) * (kTcTile / 4), &kvmap, vf, (a.G + g) * 128 + 64 * (i & 1), row[i >> 1]);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ================================================================ products (converged warp)
        constexpr uint32_t idesc_qk = instr_desc(1, 1, 1, 0, 0, 128, 128), idesc_pv = instr_desc(1, 1, 1, 0, 1, 128, 128);      // V [key][column]: B MN-major
        auto scores = [&](int t, int j) {
            const uint32_t qb = base + t * kTcTile, kb = kbase + (j & 1) * kTcTile;
#pragma unroll
            for (int k = 0; k < 2; k++)
                mma_f16_x4(tmem + t * 256, smem_desc(qb + k * (kTcTile / 2), 16, 1024, kLayoutSw128), smem_desc(kb + k * (kTcTile / 2), 16, 1024, kLayoutSw128), idesc_qk, k != 0,
                           k ? smem_u32(&misc.s_full[t]) : 0);
        };
        bar_wait(smem_u32(&misc.q_full), 0);
        bar_wait(smem_u32(&misc.k_full[0]), 0);
        tc_fence_after();
        scores(0, 0);
        scores(1, 0);
        mma_commit(smem_u32(&misc.k_free[0]));
        for (int j = 0; j < n; j++) {
            const int st = j & 1;
            const uint32_t vb = vbase + st * kTcTile;
            bar_wait(smem_u32(&misc.v_full[st]), (j >> 1) & 1);
            const int k0 = (t0 + j) * kTcKeys;
            if (k0 < lo || k0 + kTcKeys - 1 > max_pos) {      // the first and last tiles: values that no row sees are not of this sequence and may be anything (0 x NaN)
                for (int i = lane; i < kTcKeys * 16; i += 32) {
                    const int r = i >> 4, c = i & 15;
                    if (k0 + r < lo || k0 + r > max_pos)
                        *reinterpret_cast<uint4*>(smem + (vb - base) + (c >> 3) * (kTcTile / 2) + r * 128 + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
                }
                fence_async_smem();
                __syncwarp();
            }
            if (j + 1 < n) bar_wait(smem_u32(&misc.k_full[st ^ 1]), ((j + 1) >> 1) & 1);
#pragma unroll 1
            for (int t = 0; t < 2; t++) {
                bar_wait(smem_u32(&misc.p_full[t]), j & 1);
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < 8; k++)
                    mma_f16_ta(tmem + t * 256 + 128, tmem + t * 256 + 8 * k, smem_desc(vb + k * 2048, kTcTile / 2, 1024, kLayoutSw128), idesc_pv, (j | k) != 0);
                if (t == 1) mma_commit(smem_u32(&misc.v_free[st]));
                if (j + 1 < n) {
                    scores(t, j + 1);
                    if (t == 1) mma_commit(smem_u32(&misc.k_free[st ^ 1]));
                } else {
                    mma_commit(smem_u32(&misc.o_done[t]));
                }
            }
        }
    }
    } else {
        // ================================================================ soft-max
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        const int t = (warp - 4) >> 2, sp = warp & 3, r = 32 * sp + lane;
        const uint32_t ts = tmem + ((uint32_t)(32 * sp) << 16) + t * 256, to = ts + 128;
        const int tok = t * TOKS + r / RH, h = h0 + r % RH;
        const bool valid = tok < ntok;
        const int p = pos0 + tok, first = first_visible(p, a.window, a.chunk);
        constexpr float kLog2e = 1.4426950408889634f;
        const float scale = a.head_scale ? a.scale * a.head_scale[h] : a.scale, softcap = a.softcap, two_over_cap = softcap > 0.f ? 2.0f / softcap : 0.f;
        const float b1 = a.r1 ? a.r1[h] * 0.6931471805599453f : 0.f, b2 = a.r1 ? a.r2[h] : 0.f;      // r1 ln(1 + r2 n) = (r1 ln 2) log2(1 + r2 n)
        // scores that are only scaled (by a positive number) go to the exponential as they are
        const bool direct = __all_sync(0xffffffffu, softcap <= 0.f && !a.r1 && scale > 0.f);
        const float c = direct ? scale * kLog2e : 1.f;
        const int w_tok0 = t * TOKS + 32 * sp / RH, w_tok1 = t * TOKS + (32 * sp + 31) / RH;      // the warp's first and last token
        const bool w_full = w_tok1 < ntok;
        const int w_last_first = first_visible(pos0 + w_tok1, a.window, a.chunk);
        float m_ref = -INFINITY, l = 0.f;
        for (int j = 0; j < n; j++) {
            const int k0 = (t0 + j) * kTcKeys;
            bar_wait(smem_u32(&misc.s_full[t]), j & 1);      // (also: PV of the tile before this one is complete)
            tc_fence_after();
            float s[kTcKeys];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                uint32_t v[32];
                tmem_ld32(ts + 32 * q, v);
#pragma unroll
                for (int i = 0; i < 32; i++) s[32 * q + i] = __uint_as_float(v[i]);
            }
            tmem_wait_ld();
            // (the loads above are in registers only now)
#pragma unroll
            for (int i = 0; i < kTcKeys; i++) asm volatile("" : "+f"(s[i]));
            if (!direct) {
#pragma unroll
                for (int i = 0; i < kTcKeys; i++) {
                    float x = s[i] * scale;
                    if (softcap > 0.f) x = cap_score_fast(x, two_over_cap, softcap);
                    if (a.r1) x = fmaf(-b1, __log2f(fmaf(b2, (float)(p - k0 - i), 1.0f)), x);      // (masked below where the key lies ahead)
                    s[i] = x * kLog2e;
                }
            }
            if (!(w_full && k0 + kTcKeys - 1 <= pos0 + w_tok0 && k0 >= w_last_first)) {
                const int i0 = first - k0, i1 = valid ? p - k0 : -1;
#pragma unroll
                for (int i = 0; i < kTcKeys; i++)
                    if (i < i0 || i > i1) s[i] = -INFINITY;
            }
            float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
            for (int i = 4; i < kTcKeys; i += 4)
#pragma unroll
                for (int u = 0; u < 4; u++) mx[u] = fmaxf(mx[u], s[i + u]);
            const float m_new = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * c;
            const bool raise = m_new > m_ref + 8.f || (m_ref == -INFINITY && m_new > -INFINITY);
            if (__any_sync(0xffffffffu, raise)) {
                const float alpha = raise ? tc_ex2(m_ref - m_new) : 1.f;      // (2^-inf = 0: nothing was summed yet)
                if (raise) { m_ref = m_new; l *= alpha; }
                if (j > 0) {
#pragma unroll 1
                    for (int q = 0; q < 4; q++) {
                        uint32_t v[32];
                        tmem_ld32(to + 32 * q, v);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
                        tmem_st32(to + 32 * q, v);
                    }
                }
            }
            const float u = m_ref == -INFINITY ? 0.f : m_ref;
            const f32x2 c2 = pack2(c, c), nu2 = pack2(-u, -u);
            f32x2 sum[2] = {0, 0};
#pragma unroll
            for (int q = 0; q < 2; q++) {
                uint32_t pk[32];
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    float e0, e1;
                    unpack2(fma2(pack2(s[64 * q + 2 * i], s[64 * q + 2 * i + 1]), c2, nu2), e0, e1);
                    e0 = tc_ex2(e0);
                    e1 = tc_ex2(e1);
                    pk[i] = pack_bf16(e0, e1);
                    // the sum is of the weights as they are used: what rounding takes from a weight it takes from its share of the sum too
                    sum[i & 1] = add2(sum[i & 1], pack2(__uint_as_float(pk[i] << 16), __uint_as_float(pk[i] & 0xffff0000u)));
                }
                tmem_st32(ts + 32 * q, pk);
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(smem_u32(&misc.p_full[t]));
            float a0, a1, a2, a3;
            unpack2(sum[0], a0, a1);
            unpack2(sum[1], a2, a3);
            l += (a0 + a1) + (a2 + a3);
        }
        bar_wait(smem_u32(&misc.o_done[t]), 0);
        tc_fence_after();
        float inv = 1.0f / l;
        if (a.sink) {
            const float sink = a.sink[h], m_nat = m_ref * 0.6931471805599453f, mn = fmaxf(m_nat, sink), k = __expf(m_nat - mn);
            inv = k / (l * k + __expf(sink - mn));
        }
        inv *= a.out_scale;
        const __nv_bfloat16* gate = a.gate ? (const __nv_bfloat16*)a.gate + (long)(tok0 + tok) * a.gate_stride + (long)h * 128 : nullptr;
        __nv_bfloat16* out = (__nv_bfloat16*)a.out + (long)(tok0 + tok) * a.out_stride + (long)h * 128;
        const bool vec = ((reinterpret_cast<uintptr_t>(a.out) | (uintptr_t)(a.out_stride * 2)) & 15) == 0;
#pragma unroll 1
        for (int q = 0; q < 4; q++) {
            uint32_t v[32], o[16];
            tmem_ld32(to + 32 * q, v);
            tmem_wait_ld();
            if (valid) {
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    float x = __uint_as_float(v[2 * i]) * inv, y = __uint_as_float(v[2 * i + 1]) * inv;
                    if (gate) {
                        const uint32_t w = *reinterpret_cast<const uint32_t*>(gate + 32 * q + 2 * i);
                        x *= sm_sigmoid(__uint_as_float(w << 16));
                        y *= sm_sigmoid(__uint_as_float(w & 0xffff0000u));
                    }
                    o[i] = pack_bf16(x, y);
                }
                if (vec) {
#pragma unroll
                    for (int i = 0; i < 4; i++) *reinterpret_cast<uint4*>(out + 32 * q + 8 * i) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
                } else {
#pragma unroll
                    for (int i = 0; i < 16; i++) *reinterpret_cast<uint32_t*>(out + 32 * q + 2 * i) = o[i];
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// CTAs of softmax_attn_tc_kernel per key/value head and head block (an upper bound)
static int softmax_tc_tiles(int RH, int n_tokens, int n_seqs) { return n_seqs + n_tokens / (2 * (128 / RH)); }

static int launch_softmax_tc(const SmAttn& a, int n_tokens, cudaStream_t s) {
    umma::EncodeTiledFn enc = umma::encode_tiled();
    if (!enc) { set_error("softmax_attn: cuTensorMapEncodeTiled is not available from this driver"); return KTB200_ECUDA; }
    CUtensorMap qmap, kvmap;
    const cuuint32_t estr[3] = {1, 1, 1};
    const cuuint64_t qd[3] = {128, (cuuint64_t)a.H, (cuuint64_t)n_tokens}, qs[2] = {256, (cuuint64_t)a.H * 256};
    const cuuint32_t qb[3] = {64, (cuuint32_t)a.RH, (cuuint32_t)(128 / a.RH)};
    // (rows come from the page table's columns of pages that hold a visible key, which bounds them: the map itself does not know how many pages there are)
    const cuuint64_t kd[2] = {(cuuint64_t)a.G * 256, 1u << 30}, ks[1] = {(cuuint64_t)a.G * 512};
    const cuuint32_t kb[2] = {64, 64};
    CUresult cr = enc(&qmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(a.q), qd, qs, qb, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr == CUDA_SUCCESS)
        cr = enc(&kvmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(a.cache), kd, ks, kb, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                 CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) { set_error("softmax_attn: cuTensorMapEncodeTiled failed (%d)", (int)cr); return KTB200_ECUDA; }
    KTB_CUDA_CHECK(cudaFuncSetAttribute(softmax_attn_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem));
    const dim3 grid(a.H / a.RH, softmax_tc_tiles(a.RH, n_tokens, a.n_seqs));
    softmax_attn_tc_kernel<<<grid, kTcThreads, kTcSmem, s>>>(qmap, kvmap, a);
    KTB_LAUNCH_CHECK();
    return KTB200_OK;
}

}  // namespace ktb
