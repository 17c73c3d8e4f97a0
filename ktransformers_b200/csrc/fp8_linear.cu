// FP8 (e4m3, 128 x 128 block scales) linear for decode batches — KLinearFP8 (archive/ktransformers/operators/linear.py:388-435)
// = act_quant (fp8gemm.py:10-47) -> fp8_gemm (fp8gemm.py:104-192), DeepSeek-V3's native checkpoint format:
//     s[t][kb] = max|x[t][128 kb .. +128]| / 448,   xq = e4m3(x / s)                         (per token and 128 of K)
//     acc[t][n] += dot_e4m3(xq[t][kb], W[n][kb]) * s[t][kb] * scale_inv[n / 128][kb]          fp32, kb ascending
//     y = cast(acc)
// One byte per weight: a pure HBM stream.  The weights never pass through registers: TMA drops [128 rows x 128 bytes] boxes of W
// into shared memory in the 128-byte-swizzle layout, which IS the K-major A operand of tcgen05.mma.kind::f8f6f4; the quantised
// activations (16 token rows, padded) are the B operand; the products of two e4m3 values are exact in the fp32 accumulator (TMEM).
// After every 128 of K (4 MMAs) the epilogue takes the partial dot out of TMEM and applies the two scales in the reference's order.
//     grid = (ceil(N / 128) row tiles, K splits), two CTAs per SM; 192 threads: warp 0 TMA producer (4-stage ring), warp 1 issuer,
//     warps 2-5 quantise x for the CTA's K range while the first weight boxes are in flight, then run the epilogue.
// K splits add their fp32 partial sums with atomics into a zeroed workspace; the last CTA of a row tile converts and re-zeroes.
// Most batches of more than kFT tokens take fp8_gemm_kernel below: tokens on the MMA's rows, so that the weights are read once per 128 of them.
#include <cuda.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <climits>
#include <new>

#include "common.cuh"
#include "handles.cuh"
#include "umma.cuh"

namespace ktb {
using namespace umma;

constexpr int kFT = 16;                    // token rows per pass (the MMA's N)
constexpr int kFStages = 4, kFA = 128 * 128, kFB = kFT * 128, kFMaxKb = 16;   // 64 + 32 KB: two CTAs per SM, 128 KB of weight boxes in flight
constexpr int kFOffB = kFStages * kFA, kFOffS = kFOffB + kFMaxKb * kFB, kFOffMisc = kFOffS + kFT * kFMaxKb * 4;
struct Fp8Misc {
    unsigned long long a_full[kFStages], a_free[kFStages], d_full[2], d_free[2], b_ready;
    uint32_t tmem_base;
    int last;
};
constexpr int kFSmem = kFOffMisc + (int)sizeof(Fp8Misc) + 1024;

struct Fp8Params {
    const void* x;            // [T][K] hidden type
    void* y;                  // [T][N]
    const float* scale_inv;   // [ceil(N/128)][nkb]
    float* ws;                // [kFT][N] fp32, zero between calls (K splits only)
    unsigned* tickets;        // [row tiles], zero between calls
    const int* bsz;
    const uint8_t* xq;        // [kFT][K] e4m3 and
    const float* xs;          // [kFT][nkb] scales from fp8_act_quant_kernel (batches of more than 2 tokens), else null
    int hidden_type, T, K, N, nkb, kb_per_split, ksplit, t0;
};

// act_quant (fp8gemm.py:10-27) for one (token, 128 values) block held 4 values per lane: returns the scale, packs the 4 e4m3 bytes
__device__ __forceinline__ float fp8_quant_block(const float (&v)[4], uint32_t& packed) {
    float am = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    const float s = __fdiv_rn(am, 448.f);
    packed = 0;
#pragma unroll
    for (int e = 0; e < 4; e++)   // x / s in IEEE fp32, round to nearest even into e4m3 (0 / 0 = NaN like the reference)
        packed |= (uint32_t)__nv_cvt_float_to_fp8(__fdiv_rn(v[e], s), __NV_SATFINITE, __NV_E4M3) << (8 * e);
    return s;
}
__device__ __forceinline__ void fp8_load4(const void* x, long off, int hidden_type, float (&v)[4]) {
    if (hidden_type == KTB200_TYPE_F32) {
        const float4 f = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + off);
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    } else {
        const uint2 w2 = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(x) + off);
        const uint32_t ww[2] = {w2.x, w2.y};
#pragma unroll
        for (int e = 0; e < 2; e++) {
            if (hidden_type == KTB200_TYPE_BF16) { v[2 * e] = __uint_as_float(ww[e] << 16); v[2 * e + 1] = __uint_as_float(ww[e] & 0xffff0000u); }
            else { v[2 * e] = fp16_bits_to_f32((uint16_t)(ww[e] & 0xffff)); v[2 * e + 1] = fp16_bits_to_f32((uint16_t)(ww[e] >> 16)); }
        }
    }
}
// batches of more than 2 tokens: quantise x ONCE (one warp per block) instead of once per row tile
// (scales [token][block], or with spitch > 0 [block][spitch] for the GEMM)
__global__ void __launch_bounds__(256) fp8_act_quant_kernel(const void* x, int hidden_type, int T, int K, uint8_t* xq, float* xs, int spitch) {
    const int lane = threadIdx.x & 31, blk = blockIdx.x * 8 + (threadIdx.x >> 5), nkb = K / 128;
    griddep_launch_dependents();
    if (blk >= T * nkb) return;
    const int t = blk / nkb, kb = blk - t * nkb;
    float v[4];
    fp8_load4(x, (long)t * K + (long)kb * 128 + lane * 4, hidden_type, v);
    uint32_t packed;
    const float s = fp8_quant_block(v, packed);
    reinterpret_cast<uint32_t*>(xq + (long)t * K + (long)kb * 128)[lane] = packed;
    if (lane == 0) xs[spitch ? (long)kb * spitch + t : (long)t * nkb + kb] = s;
}

// TWO (fp32 results): the sum is cut every 4 blocks into a second accumulator.  2-norm error against 64 bits, 3 rows, one chain / in fours: 1536 -> 24576 9.5e-8 / 8.6e-8, 2048 -> 20480
// 1.01e-7 / 8.7e-8 (splits of 4 blocks that atomics add up are as close), 18432 -> 7168 1.21e-7 / 1.10e-7; the same time.  Results of 16 bits round more away
template <bool TWO>
__global__ void __launch_bounds__(192, 2) fp8_linear_kernel(const __grid_constant__ CUtensorMap wmap, const Fp8Params p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    Fp8Misc& misc = *reinterpret_cast<Fp8Misc*>(smem + kFOffMisc);
    float* a_s = reinterpret_cast<float*>(smem + kFOffS);   // [kFT][kb_per_split]
    const int tid = threadIdx.x, lane = tid & 31, warp = uniform(tid >> 5);
    const int row0 = blockIdx.x * 128;
    const int kb0 = blockIdx.y * p.kb_per_split, nk = min(p.kb_per_split, p.nkb - kb0);
    if (tid == 0) {
        for (int s = 0; s < kFStages; s++) { bar_init(smem_u32(&misc.a_full[s]), 1); bar_init(smem_u32(&misc.a_free[s]), 1); }
        for (int b = 0; b < 2; b++) { bar_init(smem_u32(&misc.d_full[b]), 1); bar_init(smem_u32(&misc.d_free[b]), 4); }
        bar_init(smem_u32(&misc.b_ready), 4);
        bar_fence_init();
        tma_prefetch_desc(&wmap);
    }
    if (warp == 1) tmem_alloc(smem_u32(&misc.tmem_base), 32);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = uniform(misc.tmem_base);
    griddep_launch_dependents();   // a PDL-launched successor may set up and prefetch its own weights while this grid streams

    if (warp == 0) {
        // ---------------------------------------------------------------- weight boxes: independent of x, start at once
        if (lane == 0) {
            for (int i = 0; i < nk; i++) {
                const int s = i % kFStages;
                bar_wait(smem_u32(&misc.a_free[s]), ((i / kFStages) & 1) ^ 1);
                bar_expect_tx(smem_u32(&misc.a_full[s]), kFA);
                tma_load_2d(base + s * kFA, &wmap, smem_u32(&misc.a_full[s]), (kb0 + i) * 128, row0);
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- issuer (converged warp)
        constexpr uint32_t idesc = instr_desc(1, 0, 0, 0, 0, 128, kFT);   // f32 += e4m3 . e4m3, K-major both
        bar_wait(smem_u32(&misc.b_ready), 0);
        for (int i = 0; i < nk; i++) {
            const int s = i % kFStages, buf = i & 1;
            bar_wait(smem_u32(&misc.a_full[s]), (i / kFStages) & 1);
            bar_wait(smem_u32(&misc.d_free[buf]), ((i >> 1) & 1) ^ 1);
            tc_fence_after();
#pragma unroll
            for (int j = 0; j < 4; j++)
                mma_f8(tmem + buf * kFT, smem_desc(base + s * kFA + j * 32, 16, 1024, kLayoutSw128), smem_desc(base + kFOffB + i * kFB + j * 32, 16, 1024, kLayoutSw128), idesc,
                       j != 0);
            mma_commit(smem_u32(&misc.a_free[s]));
            mma_commit(smem_u32(&misc.d_full[buf]));
        }
    } else {
        // ---------------------------------------------------------------- act_quant for this K range, then the epilogue
        const int ew = warp - 2;
        // rows T .. 15 of the B tiles: zeros (their accumulator columns are never read)
        for (int i = (tid - 64); i < nk * (kFB / 16); i += 128) {
            const int r = (i >> 3) & (kFT - 1);
            if (r >= p.T) *reinterpret_cast<uint4*>(smem + kFOffB + i * 16) = make_uint4(0, 0, 0, 0);
        }
        griddep_wait();   // x (or its quantised copy) comes from the kernel before this one; the weight boxes above did not wait
        if (p.xq) {
            // already quantised by fp8_act_quant_kernel: copy this CTA's K range into the swizzled B tiles (16-byte pieces)
            for (int i = tid - 64; i < p.T * nk * 8; i += 128) {
                const int pc = i & 7, kb = (i >> 3) % nk, t = (i >> 3) / nk;
                *reinterpret_cast<uint4*>(smem + kFOffB + kb * kFB + t * 128 + ((pc ^ (t & 7)) << 4)) =
                    *reinterpret_cast<const uint4*>(p.xq + (long)t * p.K + (long)(kb0 + kb) * 128 + pc * 16);
            }
            for (int i = tid - 64; i < p.T * nk; i += 128) a_s[(i / nk) * p.kb_per_split + (i % nk)] = p.xs[(i / nk) * p.nkb + kb0 + (i % nk)];
        } else {
            // one warp per (token, 128 of K), lane owns 4 consecutive values; 8 blocks' loads are issued before the first is reduced
            for (int g0 = ew; g0 < p.T * nk; g0 += 4 * 8) {
                float v[8][4];
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int blk = g0 + 4 * u;
                    if (blk < p.T * nk) {
                        const int t = blk / nk, kb = blk - t * nk;
                        fp8_load4(p.x, (long)t * p.K + (long)(kb0 + kb) * 128 + lane * 4, p.hidden_type, v[u]);
                    }
                }
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int blk = g0 + 4 * u;
                    if (blk < p.T * nk) {   // warp-uniform
                        const int t = blk / nk, kb = blk - t * nk;
                        uint32_t packed;
                        const float s = fp8_quant_block(v[u], packed);
                        *reinterpret_cast<uint32_t*>(smem + kFOffB + kb * kFB + t * 128 + (((lane >> 2) ^ (t & 7)) << 4) + (lane & 3) * 4) = packed;
                        if (lane == 0) a_s[t * p.kb_per_split + kb] = s;
                    }
                }
            }
        }
        fence_async_smem();
        asm volatile("bar.sync 1, 128;" ::: "memory");   // a_s is read by all four epilogue warps
        if (lane == 0) bar_arrive(smem_u32(&misc.b_ready));

        const int sp = warp & 3, row = 32 * sp + lane;
        float acc[kFT], sum[TWO ? kFT : 1];
#pragma unroll
        for (int t = 0; t < kFT; t++) {
            acc[t] = 0.f;
            if (TWO) sum[t] = 0.f;
        }
        const float* sinv = p.scale_inv + (long)blockIdx.x * p.nkb + kb0;
        for (int i = 0; i < nk; i++) {
            const int buf = i & 1;
            const float bs = __ldg(sinv + i);
            bar_wait(smem_u32(&misc.d_full[buf]), (i >> 1) & 1);
            tc_fence_after();
            uint32_t d[kFT];
            tmem_ld16(tmem + ((uint32_t)(32 * sp) << 16) + buf * kFT, d);
            tmem_wait_ld();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(smem_u32(&misc.d_free[buf]));
#pragma unroll
            for (int t = 0; t < kFT; t++)
                if (t < p.T) acc[t] = __fadd_rn(acc[t], __fmul_rn(__fmul_rn(__uint_as_float(d[t]), a_s[t * p.kb_per_split + i]), bs));   // (dot * a_s) * b_s, then +=
            if (TWO && ((i & 3) == 3 || i + 1 == nk)) {
#pragma unroll
                for (int t = 0; t < kFT; t++) { sum[t] += acc[t]; acc[t] = 0.f; }
            }
        }
        if (TWO) {
#pragma unroll
            for (int t = 0; t < kFT; t++) acc[t] = sum[t];
        }
        const int n = row0 + row;
        const int live = p.bsz ? max(0, min(p.T, *p.bsz - p.t0)) : p.T;   // rows at or beyond the live batch size stay untouched
        if (p.ksplit == 1) {
            if (n < p.N)
#pragma unroll
                for (int t = 0; t < kFT; t++)
                    if (t < live) store_hidden(p.y, (long)t * p.N + n, p.hidden_type, acc[t]);
        } else {
            if (n < p.N)
#pragma unroll
                for (int t = 0; t < kFT; t++)
                    if (t < p.T) atomicAdd(p.ws + (long)t * p.N + n, acc[t]);
            __threadfence();
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (tid == 64) misc.last = atomicAdd(p.tickets + blockIdx.x, 1u) == (unsigned)(p.ksplit - 1);
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (misc.last) {
                __threadfence();
                if (n < p.N)
                    for (int t = 0; t < p.T; t++) {
                        const float v = __ldcg(p.ws + (long)t * p.N + n);
                        p.ws[(long)t * p.N + n] = 0.f;
                        if (t < live) store_hidden(p.y, (long)t * p.N + n, p.hidden_type, v);
                    }
                if (tid == 64) p.tickets[blockIdx.x] = 0;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 32);
    }
}

// Prompt portions (more than kFT tokens): y = xq . W^T as a persistent GEMM.  The pass kernel above streams all of W again for every 16
// tokens (2000 tokens, 7168 -> 18432: 125 passes, 7.9 ms); here a tile is 128 tokens x BN weight rows, both operands come by TMA in the
// 128-byte-swizzle layout.  A K block of a 128 x 256 tile takes 735 cycles (its products alone 524; they read 48 KB of shared memory while the copies bring 48 KB in).
// 2000 tokens, 7168 -> 18432: 8 rounds of 56 blocks and 8 outputs of 4,000 cycles are 361 k of the 368 k cycles counted, 214 us at the 1.72 GHz of one launch (tensor pipe 64 % active);
// the quantisation before it 24 us; a call 245 us by itself, and 277-289 in a long row of them, where the power limit takes the clock to 1.48 GHz.  A pair of CTAs on one tile would halve the
// reading of W.
//     warp 0 TMA ring (4 to 8 stages, 192 KB), warp 1 issuer, warps 4-19 epilogue: a thread owns one token and a quarter of the tile's columns;
//     lanes are tokens, so the token scale is a register and acc += dot * (a_s * b_s) is ONE fma per value and 128 of K.
//     Two TMEM buffers of BN columns: the MMAs of one K block run while the block before it is promoted.
// BN: 256 where that gives every SM a tile; 128 and 64 keep the chip full when there are few tiles.
// The same call 338 -> 317 us by scales that are fetched four blocks ahead (a load takes about 1,000 cycles beside the copies; one block ahead each block waited 400 of
// them), four epilogue warps a scheduler instead of two (a drain's chain of loads and sums: 720 cycles a block), a tile's output without branches in whole sectors (12,800 -> 4,000
// cycles) and one election for a block's products and barriers.  The roles are known to be uniform (umma.cuh): 351 -> 333 us (the kernel above, one token 16384 -> 7168: 34.1 -> 32.7).
// Tiles run token tile fastest inside groups of kFGroupM, so that the CTAs of a wave share the weight rows and the tokens through L2.
constexpr int kFGemmThreads = 640, kFGroupM = 16, kFGemmRing = 192 * 1024, kFGemmTokens = 4096;
struct Fp8GemmMisc {
    unsigned long long full[8], free[8], d_full[2], d_free[2];
    uint32_t tmem_base;
};
constexpr int kFGemmTurn = 16 * 33;      // floats of an epilogue warp: 16 columns of 32 tokens
constexpr int kFGemmSmem = kFGemmRing + (int)sizeof(Fp8GemmMisc) + 1024, kFGemmSmemTurn = kFGemmSmem + 16 * kFGemmTurn * 4;
static_assert(kFGemmSmemTurn <= 232448, "shared memory budget");

struct Fp8GemmParams {
    const float* xs;          // [nkb][tpad] token scales, token fastest
    const float* scale_inv;   // [ceil(N/128)][nkb]
    void* y;                  // [T][N]
    const int* bsz;
    int hidden_type, T, N, nkb, tpad, mt, nt, t0, vec;      // vec: result rows begin at whole sectors (2), at 16 bytes (1), anywhere (0)
};

// TWO: fp32 results, where the order of a long fp32 chain shows (K = 12032: 2.0e-7 off in one chain, 1.2e-7 with K splits): the chain is cut
// every 8 blocks into a second accumulator.
// TURN: result rows that begin anywhere, and fp32 ones that do not begin at a sector.  A thread's columns of its token would be scattered values; the warp turns 16 columns of its 32 tokens
// around in shared memory, and 16 threads write 16 columns of one row (a kernel of its own: in one with the other form aligned rows took 7 % longer).  Value by value / like this (us):
// 1200 tokens, 1536 -> 9001 fp32 91 / 44, fp16 150 / 38; 64 tokens, 4096 -> 4101 bf16 22.2 / 19.7; in vectors of 16 bytes / like this: fp32 1200 tokens 1024 -> 16388 62.1 / 56.7, 500 tokens
// 4096 -> 4100 31.9 / 30.1, 1200 tokens 7168 -> 3004 60.7 / 62.5; bf16 1200 tokens 2048 -> 8200 40.3 / 56.6.
template <int BN, bool TWO, bool TURN>
__global__ void __launch_bounds__(kFGemmThreads, 1) fp8_gemm_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const Fp8GemmParams p) {
    constexpr int kStageB = 128 * 128 + BN * 128, kStages = kFGemmRing / kStageB, kCols = 2 * BN;
    static_assert(kStages <= 8, "barriers");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    Fp8GemmMisc& misc = *reinterpret_cast<Fp8GemmMisc*>(smem_raw + (base - raw) + kFGemmRing);
    const int tid = threadIdx.x, lane = tid & 31, warp = uniform(tid >> 5);
    if (tid == 0) {
        for (int s = 0; s < kStages; s++) { bar_init(smem_u32(&misc.full[s]), 1); bar_init(smem_u32(&misc.free[s]), 1); }
        for (int b = 0; b < 2; b++) { bar_init(smem_u32(&misc.d_full[b]), 1); bar_init(smem_u32(&misc.d_free[b]), 16); }
        bar_fence_init();
        tma_prefetch_desc(&xmap);
        tma_prefetch_desc(&wmap);
    }
    if (warp == 1) tmem_alloc(smem_u32(&misc.tmem_base), kCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = uniform(misc.tmem_base);
    const int tiles = p.mt * p.nt;
    auto place = [&](int tile, int& m0, int& n0) {      // groups of kFGroupM token tiles; inside a group the token tile is fastest
        const int per = kFGroupM * p.nt, g = tile / per, r = tile - g * per, gm = min(kFGroupM, p.mt - g * kFGroupM);
        n0 = (r / gm) * BN;
        m0 = (g * kFGroupM + r % gm) * 128;
    };
    griddep_wait();      // the quantised tokens and their scales come from the kernel before this one

    // registers: 96 a thread at launch, of which the copies and the issuer need a third (32 + 4 x 112 = 5 x 96)
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        __syncwarp();
    }
    if (warp == 0) {
        if (lane == 0) {
            int s = 0, ph = 1;
            for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
                int m0, n0;
                place(tile, m0, n0);
                for (int kb = 0; kb < p.nkb; kb++) {
                    bar_wait(smem_u32(&misc.free[s]), ph);
                    const uint32_t bar = smem_u32(&misc.full[s]), dst = base + s * kStageB;
                    bar_expect_tx(bar, kStageB);
                    tma_load_2d(dst, &xmap, bar, kb * 128, m0);
                    tma_load_2d(dst + 128 * 128, &wmap, bar, kb * 128, n0);
                    if (++s == kStages) { s = 0; ph ^= 1; }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        constexpr uint32_t idesc = instr_desc(1, 0, 0, 0, 0, 128, BN);   // f32 += e4m3 . e4m3, K-major both
        int s = 0, ph = 0;
        unsigned it = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x)
            for (int kb = 0; kb < p.nkb; kb++, it++) {
                const int buf = it & 1;
                bar_wait(smem_u32(&misc.full[s]), ph);
                bar_wait(smem_u32(&misc.d_free[buf]), ((it >> 1) & 1) ^ 1);
                tc_fence_after();
                const uint32_t a = base + s * kStageB, b = a + 128 * 128;
                mma_f8_x4(tmem + buf * BN, smem_desc(a, 16, 1024, kLayoutSw128), smem_desc(b, 16, 1024, kLayoutSw128), idesc, 0, smem_u32(&misc.free[s]), smem_u32(&misc.d_full[buf]));
                if (++s == kStages) { s = 0; ph ^= 1; }
            }
    } else if (warp >= 4) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
        constexpr int kPart = BN / 4, kAhead = 4, kLoad = kPart < 32 ? kPart : 32;
        const int sp = warp & 3, ch = (warp - 4) >> 2;
        const uint32_t tcol = tmem + ((uint32_t)(32 * sp) << 16) + ch * kPart;
        const int live = p.bsz ? max(0, min(p.T, *p.bsz - p.t0)) : p.T;
        unsigned it = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            int m0, n0;
            place(tile, m0, n0);
            const int t = m0 + 32 * sp + lane, nb = n0 + ch * kPart;
            const float* xs = p.xs + t;                                                     // t < tpad
            const float* sinv = p.scale_inv + (long)min(nb / 128, (p.N - 1) / 128) * p.nkb;
            float acc[kPart], sum[TWO ? kPart : 1];
#pragma unroll
            for (int i = 0; i < kPart; i++) {
                acc[i] = 0.f;
                if (TWO) sum[i] = 0.f;
            }
            // The scales of kAhead blocks are under way: a load takes about 1,000 cycles beside the tiles' copies, and one block ahead each block waited 400 of them
            float a_s[kAhead], b_s[kAhead];
            auto scales = [&](int i, int kb) {
                const int k = min(kb, p.nkb - 1);
                a_s[i] = __ldg(xs + (long)k * p.tpad);
                b_s[i] = __ldg(sinv + k);
            };
#pragma unroll
            for (int i = 0; i < kAhead; i++) scales(i, i);
            for (int kb0 = 0; kb0 < p.nkb; kb0 += kAhead)
#pragma unroll
                for (int i = 0; i < kAhead; i++) {
                    const int kb = kb0 + i, buf = it & 1;
                    if (kb >= p.nkb) break;
                    const float f = a_s[i] * b_s[i];
                    scales(i, kb + kAhead);
                    bar_wait(smem_u32(&misc.d_full[buf]), (it >> 1) & 1);
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < kPart; c += kLoad) {
                        uint32_t d[kLoad];
                        if constexpr (kLoad == 32) tmem_ld32(tcol + buf * BN + c, d); else tmem_ld16(tcol + buf * BN + c, d);
                        tmem_wait_ld();
#pragma unroll
                        for (int u = 0; u < kLoad; u++) acc[c + u] = __fmaf_rn(__uint_as_float(d[u]), f, acc[c + u]);
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) bar_arrive(smem_u32(&misc.d_free[buf]));
                    if (TWO && ((kb & 7) == 7 || kb + 1 == p.nkb)) {
#pragma unroll
                        for (int u = 0; u < kPart; u++) { sum[u] += acc[u]; acc[u] = 0.f; }
                    }
                    it++;
                }
            if (TWO) {
#pragma unroll
                for (int i = 0; i < kPart; i++) acc[i] = sum[i];
            }
            if (TURN) {
                float* turn = reinterpret_cast<float*>(smem_raw + (base - raw) + kFGemmRing + sizeof(Fp8GemmMisc)) + (warp - 4) * kFGemmTurn;
                const int t1 = m0 + 32 * sp + (lane >> 4);
#pragma unroll
                for (int c = 0; c < kPart; c += 16) {
                    const int col = nb + c + (lane & 15);
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 16; i++) turn[33 * i + lane] = acc[c + i];
                    __syncwarp();
#pragma unroll 4
                    for (int k = 0; k < 32; k += 2)
                        if (t1 + k < live && col < p.N) store_hidden(p.y, (long)(t1 + k) * p.N + col, p.hidden_type, turn[33 * (lane & 15) + (lane >> 4) + k]);
                }
            } else if (t < live) {
                const long o = (long)t * p.N + nb;
#pragma unroll
                for (int c = 0; c < kPart; c += 16) {
                    if (p.vec && nb + c + 16 <= p.N) {
                        // (a thread's row is its own: whole sectors where the rows allow them)
                        auto sector = [&](uint8_t* y, const uint32_t (&w)[8]) {
                            if (p.vec == 2) {
                                asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(y), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
                            } else {
                                reinterpret_cast<uint4*>(y)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                                reinterpret_cast<uint4*>(y)[1] = make_uint4(w[4], w[5], w[6], w[7]);
                            }
                        };
                        uint32_t w[8];
                        if (p.hidden_type == KTB200_TYPE_F32) {
                            uint8_t* y = reinterpret_cast<uint8_t*>(reinterpret_cast<float*>(p.y) + o + c);
#pragma unroll
                            for (int q = 0; q < 2; q++) {
#pragma unroll
                                for (int i = 0; i < 8; i++) w[i] = __float_as_uint(acc[c + 8 * q + i]);
                                sector(y + 32 * q, w);
                            }
                        } else {
#pragma unroll
                            for (int i = 0; i < 8; i++) w[i] = pack16(acc[c + 2 * i], acc[c + 2 * i + 1], p.hidden_type == KTB200_TYPE_BF16);
                            sector(reinterpret_cast<uint8_t*>(reinterpret_cast<uint16_t*>(p.y) + o + c), w);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; i++)
                            if (nb + c + i < p.N) store_hidden(p.y, o + c + i, p.hidden_type, acc[c + i]);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kCols);
    }
}

}  // namespace ktb

struct ktb200_fp8_linear {
    int K, N, hidden_type, device, nkb, row_tiles, kb_per_split, kb_many;      // (kb_many: for kFp8Many and more rows)
    const void* w;
    const float* scale_inv;
    CUtensorMap map;
    float* ws;
    unsigned* tickets;
    uint8_t* xq;   // [kFT][K] e4m3
    float* xs;     // [kFT][nkb]
};

namespace ktb {
// Blocks of K a CTA of the pass kernel takes: at most kFMaxKb, at least as many as fill its ring, and of these the number whose CTAs, two an SM, take least one after the other; kFp8Round is what
// a CTA costs beside its blocks, in blocks: set-up, quantisation, the atomics of its sums.  Against as many splits as give four CTAs an SM (us, weights from memory, one and 16 rows):
// 1536 -> 24576 16.3 -> 10.9, 35 -> 20 (no splits, no atomics); 7168 -> 4096 13.7 -> 10.4, 28 -> 23; 10240 -> 14000 39.5 -> 35.5, 68 -> 60; 16384 -> 7168 33.3 -> 32.0, 56 -> 52; matrices of
// few tiles as before.
// From kFp8Many rows on, where the CTAs do not run all at once, a block takes longer (kFp8RoundMany) and the last split's CTAs, which have what is left of K, fill the gaps: the least time of
// CTAs taken in order by whichever place is free.  16 rows: 18432 -> 7168 54.9 -> 52.6, 4224 -> 12864 37.1 -> 32.4, 5120 -> 19456 51.7 -> 49.1, 9728 -> 11136 50.0 -> 47.7, 7680 -> 19904
// 66.8 -> 68.4; at 9 rows as often slower as faster.
constexpr int kFp8Round = 8, kFp8RoundMany = 4, kFp8Many = 12;
static long fp8_span(int tiles, int nkb, int kb, int places) {
    const int splits = (nkb + kb - 1) / kb, full = tiles * (splits - 1), whole = full / places, rest = full % places;
    const long c = kb + kFp8RoundMany, d = nkb - kb * (splits - 1) + kFp8RoundMany;      // a whole CTA, one of the last split
    long at[2] = {whole * c, (whole + 1) * c}, end = at[rest > 0];
    const int free[2] = {places - rest, rest};
    for (int left = tiles; left > 0;) {
        const int i = free[1] > 0 && at[1] < at[0];
        at[i] += d;
        left -= free[i];
        end = std::max(end, at[i]);
    }
    return end;
}
static int fp8_blocks(int tiles, int nkb, int places, bool many) {
    int best = std::min(nkb, 4);
    long least = LONG_MAX;
    for (int kb = best; kb <= std::min(nkb, kFMaxKb); kb++) {
        const long cost = (long)((tiles * ((nkb + kb - 1) / kb) + places - 1) / places) * (kb + kFp8Round);
        if (cost < least) { least = cost; best = kb; }
    }
    if (!many || best == nkb || tiles * ((nkb + best - 1) / best) <= places) return best;      // (one split needs no atomics)
    least = LONG_MAX;
    for (int kb = std::min(nkb, 4); kb <= std::min(nkb, kFMaxKb); kb++) {
        const long cost = fp8_span(tiles, nkb, kb, places);
        if (cost < least) { least = cost; best = kb; }
    }
    return best;
}
// Whether a batch of more than kFT tokens is still faster in passes of kFT.  The GEMM has no K splits, so a matrix of few rows is one serial chain of
// K / 128 steps a tile.  The line was fitted to former kernels, 10 us + 0.48 us a step and round of tiles against 17.5 us + 1 us per 2.9 MB of weights a pass, a last one of a few tokens
// less.  Measured again (40 matrices, graphs): 4 us + 0.25 us a step, and 12 us + 1 us per 5 MB, a last pass of up to 2 tokens 0.6, of up to 8 tokens 0.85 of one.  Where the matrix is
// narrow and long both lines agree (20480 -> 256, 24 tokens: passes 27, GEMM 47 us); near the line the GEMM is now the faster one by up to 1.45 (7168 -> 576: 24 tokens 26.6 / 19.6; 5120 -> 1024,
// 18 tokens 22.6 / 15.3), 2 % on the average of all.  The choice stays where callers and tests have it.
static bool fp8_passes_win(const ktb200_fp8_linear* l, int T, int sms) {
    if (T > 64) return false;
    const int rest = T % kFT, rounds = ((l->N + 63) / 64 + sms - 1) / sms;      // (few tiles: 64 weight rows each)
    const float pass = 17.5f + (float)l->N * l->K / 2.9e6f, last = rest == 0 ? 0.f : rest <= 2 ? -10.f : rest <= 8 ? -4.f : 0.f;
    return (T + kFT - 1) / kFT * pass + last < 10.f + 0.48f * l->nkb * rounds;
}
// one box of `rows` x 128 bytes of a row-major byte matrix [n][K]
static int fp8_map(CUtensorMap* map, const void* ptr, int K, int n, int rows) {
    const cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)n};
    const cuuint64_t gstr[1] = {(cuuint64_t)K};
    const cuuint32_t box[2] = {128, (cuuint32_t)rows}, estr[2] = {1, 1};
    const CUresult cr = encode_tiled()(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) { set_error("fp8_linear: cuTensorMapEncodeTiled failed (%d)", (int)cr); return KTB200_ECUDA; }
    return KTB200_OK;
}
template <int BN, bool TWO, bool TURN>
static cudaError_t launch_fp8_gemm_as(const CUtensorMap& xmap, const CUtensorMap& wmap, const Fp8GemmParams& p, int grid, cudaStream_t s) {
    constexpr int smem = TURN ? kFGemmSmemTurn : kFGemmSmem;
    const cudaError_t e = cudaFuncSetAttribute(fp8_gemm_kernel<BN, TWO, TURN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return e != cudaSuccess ? e : launch_pdl(fp8_gemm_kernel<BN, TWO, TURN>, dim3(grid), dim3(kFGemmThreads), (size_t)smem, s, xmap, wmap, p);
}
template <int BN, bool TWO>
static cudaError_t launch_fp8_gemm(const CUtensorMap& xmap, const CUtensorMap& wmap, const Fp8GemmParams& p, int grid, cudaStream_t s) {
    return p.vec > TWO ? launch_fp8_gemm_as<BN, TWO, false>(xmap, wmap, p, grid, s) : launch_fp8_gemm_as<BN, TWO, true>(xmap, wmap, p, grid, s);
}
static int fp8_forward_gemm(ktb200_fp8_linear* l, int qlen, const void* x, void* y, const int* bsz, cudaStream_t s) {
    const size_t hb = type_size(l->hidden_type);
    for (int t0 = 0; t0 < qlen; t0 += kFGemmTokens) {
        Fp8GemmParams p{};
        p.T = qlen - t0 < kFGemmTokens ? qlen - t0 : kFGemmTokens;
        p.N = l->N; p.nkb = l->nkb; p.t0 = t0; p.bsz = bsz; p.hidden_type = l->hidden_type; p.scale_inv = l->scale_inv;
        p.mt = (p.T + 127) / 128; p.tpad = p.mt * 128;
        p.y = reinterpret_cast<uint8_t*>(y) + (size_t)t0 * l->N * hb;
        p.vec = (size_t)l->N * hb % 16 || (uintptr_t)y % 16 ? 0 : (size_t)l->N * hb % 32 || (uintptr_t)y % 32 ? 1 : 2;
        ScratchBlock mem(s);
        const size_t xs_bytes = (size_t)l->nkb * p.tpad * sizeof(float);
        KTB_CUDA_CHECK(mem.take(l->device, (size_t)p.T * l->K + xs_bytes));
        float* xs = reinterpret_cast<float*>(mem.ptr);
        uint8_t* xq = reinterpret_cast<uint8_t*>(mem.ptr) + xs_bytes;
        p.xs = xs;
        const void* xc = reinterpret_cast<const uint8_t*>(x) + (size_t)t0 * l->K * hb;
        fp8_act_quant_kernel<<<(unsigned)(((long)p.T * l->nkb + 7) / 8), 256, 0, s>>>(xc, l->hidden_type, p.T, l->K, xq, xs, p.tpad);
        // the widest tile that still gives every SM one
        const int sms = num_sms(l->device);
        const bool two = l->hidden_type == KTB200_TYPE_F32;      // (twice the accumulators: no room for 256 columns)
        int bn = two ? 128 : 256;
        while (bn > 64 && (long)p.mt * ((l->N + bn - 1) / bn) < sms) bn >>= 1;
        p.nt = (l->N + bn - 1) / bn;
        CUtensorMap xmap, wmap;
        int rc = fp8_map(&xmap, xq, l->K, p.T, 128);
        if (rc == KTB200_OK) rc = fp8_map(&wmap, l->w, l->K, l->N, bn);
        if (rc) return rc;
        const int grid = p.mt * p.nt < sms ? p.mt * p.nt : sms;
        const auto go = two ? (bn == 128 ? launch_fp8_gemm<128, true> : launch_fp8_gemm<64, true>)
                            : (bn == 256 ? launch_fp8_gemm<256, false> : bn == 128 ? launch_fp8_gemm<128, false> : launch_fp8_gemm<64, false>);
        KTB_CUDA_CHECK(go(xmap, wmap, p, grid, s));
        count_launch(2);
    }
    return KTB200_OK;
}
}  // namespace ktb

extern "C" {

int ktb200_fp8_linear_create(int in_features, int out_features, const void* weight_e4m3, const float* weight_scale_inv, int hidden_type, int device,
                             ktb200_fp8_linear** out) {
    using namespace ktb;
    if (!out || !weight_e4m3 || !weight_scale_inv) { set_error("fp8_linear: null argument"); return KTB200_EINVAL; }
    if (in_features <= 0 || out_features <= 0 || in_features % 128) { set_error("fp8_linear: in_features %d must be a positive multiple of 128 (act_quant block)", in_features); return KTB200_EINVAL; }
    if (!is_hidden_type(hidden_type)) { set_error("fp8_linear: bad hidden_type %d", hidden_type); return KTB200_EINVAL; }
    if ((uintptr_t)weight_e4m3 & 15) { set_error("fp8_linear: weight must be 16-byte aligned"); return KTB200_EINVAL; }
    DeviceGuard g(device);
    if (!g.ok) { set_error("cudaSetDevice(%d) failed", device); return KTB200_ECUDA; }
    EncodeTiledFn enc = encode_tiled();
    if (!enc) { set_error("fp8_linear: cuTensorMapEncodeTiled is not available from this driver"); return KTB200_ECUDA; }
    ktb200_fp8_linear* l = new (std::nothrow) ktb200_fp8_linear();
    if (!l) return KTB200_ENOMEM;
    l->K = in_features; l->N = out_features; l->hidden_type = hidden_type; l->device = device; l->w = weight_e4m3; l->scale_inv = weight_scale_inv;
    l->nkb = in_features / 128; l->row_tiles = (out_features + 127) / 128;
    const int places = 2 * num_sms(device);
    l->kb_per_split = fp8_blocks(l->row_tiles, l->nkb, places, false);
    l->kb_many = fp8_blocks(l->row_tiles, l->nkb, places, true);
    const cuuint64_t gdim[2] = {(cuuint64_t)in_features, (cuuint64_t)out_features};
    const cuuint64_t gstr[1] = {(cuuint64_t)in_features};
    const cuuint32_t box[2] = {128, 128}, estr[2] = {1, 1};
    const CUresult cr = enc(&l->map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(weight_e4m3), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) { set_error("fp8_linear: cuTensorMapEncodeTiled failed (%d)", (int)cr); delete l; return KTB200_ECUDA; }
    l->ws = nullptr; l->tickets = nullptr; l->xq = nullptr; l->xs = nullptr;
    scratch_prepare(device);
    cudaError_t e = cudaMalloc(&l->ws, (size_t)kFT * out_features * sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(l->ws, 0, (size_t)kFT * out_features * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&l->tickets, (size_t)l->row_tiles * sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMemset(l->tickets, 0, (size_t)l->row_tiles * sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMalloc(&l->xq, (size_t)kFT * in_features);
    if (e == cudaSuccess) e = cudaMalloc(&l->xs, (size_t)kFT * l->nkb * sizeof(float));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fp8_linear_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fp8_linear_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFSmem);
    if (e != cudaSuccess) { set_error("fp8_linear: %s", cudaGetErrorString(e)); cudaFree(l->ws); cudaFree(l->tickets); cudaFree(l->xq); cudaFree(l->xs); delete l; return KTB200_ENOMEM; }
    *out = l;
    return KTB200_OK;
}

void ktb200_fp8_linear_destroy(ktb200_fp8_linear* l) {
    if (!l) return;
    DeviceGuard g(l->device);
    cudaFree(l->ws); cudaFree(l->tickets); cudaFree(l->xq); cudaFree(l->xs);
    delete l;
}

int ktb200_fp8_linear_forward(ktb200_fp8_linear* l, int qlen, const void* x, void* y, const int* bsz, void* stream) {
    using namespace ktb;
    if (!l || !x || !y) { set_error("fp8_linear: null pointer"); return KTB200_EINVAL; }
    if (qlen <= 0) return KTB200_OK;
    DeviceGuard g(l->device);
    if (qlen > kFT && !fp8_passes_win(l, qlen, num_sms(l->device))) return fp8_forward_gemm(l, qlen, x, y, bsz, (cudaStream_t)stream);
    const size_t hb = type_size(l->hidden_type);
    const auto kernel = l->hidden_type == KTB200_TYPE_F32 ? fp8_linear_kernel<true> : fp8_linear_kernel<false>;
    for (int t0 = 0; t0 < qlen; t0 += kFT) {
        Fp8Params p{};
        p.x = reinterpret_cast<const uint8_t*>(x) + (size_t)t0 * l->K * hb;
        p.y = reinterpret_cast<uint8_t*>(y) + (size_t)t0 * l->N * hb;
        p.scale_inv = l->scale_inv; p.ws = l->ws; p.tickets = l->tickets; p.bsz = bsz; p.t0 = t0;
        p.hidden_type = l->hidden_type; p.T = qlen - t0 < kFT ? qlen - t0 : kFT; p.K = l->K; p.N = l->N; p.nkb = l->nkb;
        p.kb_per_split = p.T < kFp8Many ? l->kb_per_split : l->kb_many; p.ksplit = (l->nkb + p.kb_per_split - 1) / p.kb_per_split;
        if (p.T > 2) {   // quantise once, then the GEMM as a programmatic dependent launch: its weight boxes stream while the quantiser drains
            p.xq = l->xq; p.xs = l->xs;
            fp8_act_quant_kernel<<<(p.T * l->nkb + 7) / 8, 256, 0, (cudaStream_t)stream>>>(p.x, l->hidden_type, p.T, l->K, l->xq, l->xs, 0);
            KTB_CUDA_CHECK(launch_pdl(kernel, dim3(l->row_tiles, p.ksplit), dim3(192), (size_t)kFSmem, (cudaStream_t)stream, l->map, p));
            count_launch(2);
        } else {
            KTB_CUDA_CHECK(launch_pdl(kernel, dim3(l->row_tiles, p.ksplit), dim3(192), (size_t)kFSmem, (cudaStream_t)stream, l->map, p));
            count_launch(1);
        }
    }
    return KTB200_OK;
}

}  // extern "C"
