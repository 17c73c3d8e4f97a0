// Un-quantised experts of a prompt portion (KExpertsDense, bf16): the (token, choice) pairs sorted by expert, then per expert
//     a = act(W_gate x, W_up x)  (or relu(W_up x)^2)        y = W_down a        out[t] = sum_j w_j y_tj
// as two persistent tcgen05 GEMMs over tiles of the sorted pairs (the reference loops over experts in torch:
// archive/ktransformers/operators/experts.py:562-678).  The weights' rows are the M side of the products and the pairs the N side, so that a tile costs what its
// pairs need in steps of 16 and an expert's pairs are dealt evenly to its tiles; with the pairs on the M side a tile of 20 took as long as one of 128.  Both products
// of a gated expert share a tile's accumulators [gate | up], so the activation is applied to the fp32 sums in the epilogue and the pre-activations never reach
// memory; y stays fp32 up to the weighted sum.
// Bounds: each expert's weights once per tile of its pairs from HBM or L2, so the second tile's reading shows where experts have more than one.  1000 tokens, 32
// experts of 1024 x 2048, 4 choices (403 MB of weights, 62 us at 6.5 TB/s): 149 us with the pairs on the M side, 133 like this (products 65 and 34, sort 10, gather 7,
// weighted sum 10); 1200 tokens 176 -> 139; 2400 tokens, 128 experts of 768 x 2048, 8 choices 512 -> 385; 128 tokens, 64 experts of 1536 x 4096, 6 choices (2.4 GB)
// 430 -> 420, 5.8 TB/s; 1000 tokens, 8 experts of 512 x 1024 (one round of CTAs, latency) 43 -> 43.  Half tiles of weights (M = 64): 170 us, the pairs are read twice.
//     kernel: warp 0 TMA (32 KB of weights, 16 KB of pairs and 4 stages, or 32 KB and 3; 128-byte swizzle; of the pairs only pieces of 32 that the tile has), warp 1
//     issuer, warps 4-19 epilogue (neighbouring threads write neighbouring columns of a result row); two sets of accumulators where a tile has up to 128 pairs, so
//     that its epilogue runs beside the next one's products.  The launches are chained (programmatic dependent launch): each waits for all of its predecessor before
//     it touches the workspace.
#include <cuda.h>

#include "common.cuh"
#include "seq_common.cuh"
#include "umma.cuh"

namespace ktb {
using namespace umma;

constexpr int kEgThreads = 640, kEgRing = 192 * 1024, kEgMaxExperts = 1024, kEgWide = 256;
enum EgMode { EG_GATED, EG_RELU2, EG_DOWN };
struct EgMisc {
    unsigned long long full[4], free[4], d_full[2], d_free[2];
    uint32_t tmem_base, pad;
    int prefix[kEgMaxExperts + 2];      // pair tiles before every expert; whether a tile has up to kEgWide pairs (else 128)
};
constexpr int kEgSmem = kEgRing + (int)sizeof(EgMisc) + 1024;
static_assert(kEgSmem <= 232448, "shared memory budget");

struct EgParams {
    const int *counts, *offsets, *prefix;
    int E, nk, rows, cols, act;          // 64-wide steps of K; rows of an expert's matrix; columns of the result
    float limit;
    const float* row_scale;              // per sorted pair, multiplies the pre-activations (weights on the input); null: 1
    void* out;                           // [pairs][cols]: bf16, EG_DOWN fp32
};

// One CTA sorts the pairs by expert (counting sort: their order inside an expert does not matter, every row is a result of its own).  place: where a
// pair's row goes among the sorted rows; -1: its id names no expert.  One launch of ~6 us for 4000 pairs instead of three (clear, count, scan) and the
// gather's atomics; beyond that ~1 us per 1000 pairs, 1-2% of what their products take.
__global__ void __launch_bounds__(1024) eg_sort_kernel(const int64_t* __restrict__ ids, int n, int E, int* __restrict__ counts, int* __restrict__ offsets, int* __restrict__ prefix,
                                                       int64_t* __restrict__ place, int col_tiles, int ctas) {
    __shared__ int cursor[kEgMaxExperts];
    __shared__ int2 part[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    griddep_launch_dependents();
    cursor[tid] = 0;
    __syncthreads();
    // adds a warp's pairs to their experts' counters, one atomic per expert present; the value before, per pair
    auto add = [&](int e) {
        const unsigned same = __match_any_sync(0xffffffffu, e);
        const int leader = __ffs(same) - 1;
        int before = 0;
        if (e >= 0 && lane == leader) before = atomicAdd(&cursor[e], __popc(same));
        return __shfl_sync(0xffffffffu, before, leader) + __popc(same & ((1u << lane) - 1));
    };
    auto expert = [&](long i) {
        const long e = i < n ? (long)ids[i] : -1;
        return e >= 0 && e < E ? (int)e : -1;
    };
    for (long i = tid; i - tid < n; i += 4096) {
        int e[4];
#pragma unroll
        for (int j = 0; j < 4; j++) e[j] = expert(i + 1024 * j);
#pragma unroll
        for (int j = 0; j < 4; j++) add(e[j]);
    }
    __syncthreads();
    const int own = tid < E ? cursor[tid] : 0;
    // Tiles of up to 256 pairs where every expert has one and they save a third of the CTAs' rounds, else of 128.  The weights are read once, but the tile has no second
    // set of accumulators for the next one, and takes ~1.4 times as long.  128 pairs / 256, us, rounds: 32 experts of 1024 x 2048, 4 choices, 1000 tokens 137 / 133 (3 / 2),
    // 1200 152 / 139 (4 / 2), 900 123 / 127 (2 / 2); 128 of 768 x 2048, 8 choices, 2400 399 / 385 (11 / 6), 2000 346 / 354 (8 / 6); 8 of 512 x 1024 (one round) 43 / 49.
    const int one = __syncthreads_count(own > 0), two = __syncthreads_count(own > 128), more = __syncthreads_or(own > kEgWide);
    const bool wide = two && !more && 2 * (((long)(one + two) * col_tiles + ctas - 1) / ctas) >= 3 * (((long)one * col_tiles + ctas - 1) / ctas);
    const int tiles = wide ? own > 0 : (own + 127) / 128;
    int2 v = make_int2(own, tiles);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, v.x, o), y = __shfl_up_sync(0xffffffffu, v.y, o);
        if (lane >= o) { v.x += x; v.y += y; }
    }
    if (lane == 31) part[warp] = v;
    __syncthreads();
    for (int w = 0; w < warp; w++) { v.x += part[w].x; v.y += part[w].y; }
    if (tid < E) {
        counts[tid] = own;
        offsets[tid] = cursor[tid] = v.x - own;
        prefix[tid] = v.y - tiles;
        if (tid == E - 1) { prefix[E] = v.y; prefix[E + 1] = wide; }
    }
    __syncthreads();
    for (long i = tid; i - tid < n; i += 4096) {
        int e[4];
#pragma unroll
        for (int j = 0; j < 4; j++) e[j] = expert(i + 1024 * j);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int at = add(e[j]);
            if (i + 1024 * j < n) place[i + 1024 * j] = e[j] < 0 ? -1 : at;
        }
    }
}
// one CTA per pair: its row (and weight) to its place
__global__ void __launch_bounds__(128) eg_gather_kernel(const uint4* __restrict__ x, const float* __restrict__ weights, int top, int row16, const int64_t* __restrict__ place,
                                                        float* __restrict__ scale, uint4* __restrict__ xs) {
    griddep_launch_dependents();
    griddep_wait();
    const long p = blockIdx.x, at = place[p];
    if (at < 0) return;
    if (scale && threadIdx.x == 0) scale[at] = weights[p];
    const uint4* src = x + p / top * row16;
    uint4* dst = xs + at * row16;
    for (int i = threadIdx.x; i < row16; i += 128) dst[i] = src[i];
}

template <int MODE>
__global__ void __launch_bounds__(kEgThreads, 1) eg_gemm_kernel(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap, const __grid_constant__ CUtensorMap umap,
                                                               const EgParams p) {
    extern __shared__ uint8_t eg_smem[];
    const uint32_t raw = smem_u32(eg_smem), base = (raw + 1023u) & ~1023u;
    EgMisc& misc = *reinterpret_cast<EgMisc*>(eg_smem + (base - raw) + kEgRing);
    const int tid = threadIdx.x, lane = tid & 31, warp = uniform(tid >> 5);
    if (tid == 0) {
        for (int s = 0; s < 4; s++) { bar_init(smem_u32(&misc.full[s]), 1); bar_init(smem_u32(&misc.free[s]), 1); }
        for (int b = 0; b < 2; b++) { bar_init(smem_u32(&misc.d_full[b]), 1); bar_init(smem_u32(&misc.d_free[b]), 16); }
        bar_fence_init();
        tma_prefetch_desc(&amap);
        tma_prefetch_desc(&bmap);
        if (MODE == EG_GATED) tma_prefetch_desc(&umap);
    }
    griddep_launch_dependents();
    griddep_wait();
    for (int i = tid; i <= p.E + 1; i += kEgThreads) misc.prefix[i] = p.prefix[i];
    if (warp == 1) tmem_alloc(smem_u32(&misc.tmem_base), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = uniform(misc.tmem_base);
    const bool wide = uniform(misc.prefix[p.E + 1]);
    const int sets = wide ? 1 : 2, stages = wide ? 3 : 4, stage = kEgRing / stages, wofs = wide ? 256 * 128 : 128 * 128;
    const uint32_t second = wide ? 256 : 128;            // accumulator columns: [first matrix | second], a set of 256 each; a wide tile takes all 512
    constexpr int kTileCols = MODE == EG_GATED ? 128 : 256;
    const int nt = (p.cols + kTileCols - 1) / kTileCols, total = misc.prefix[p.E] * nt;
    struct Tile { int e, at, n, n0; };
    auto place = [&](int tile) {      // expert, then column tile, then pair tile fastest: neighbouring CTAs share the weights.  An expert's tiles have the same number of pairs
        int lo = 0, hi = p.E;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (misc.prefix[mid] * nt <= tile) lo = mid; else hi = mid;
        }
        const int local = tile - misc.prefix[lo] * nt, mt = misc.prefix[lo + 1] - misc.prefix[lo], count = p.counts[lo], per = (count + mt - 1) / mt, m0 = (local % mt) * per;
        return Tile{uniform(lo), uniform(p.offsets[lo] + m0), uniform(min(per, count - m0)), uniform((local / mt) * kTileCols)};
    };

    if (warp == 0) {
        int s = 0, ph = 1;
        for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
            const Tile t = place(tile);
            const int brow = t.e * p.rows + t.n0, pieces = (t.n + 31) / 32;      // (of 32 pairs; a pair's sums need no other pair)
            for (int k = 0; k < p.nk; k++) {
                bar_wait(smem_u32(&misc.free[s]), ph);
                if (lane == 0) {
                    const uint32_t bar = smem_u32(&misc.full[s]), dst = base + s * stage, wdst = dst + wofs;
                    bar_expect_tx(bar, 256 * 128 + pieces * 32 * 128);
                    for (int i = 0; i < pieces; i++) tma_load_2d(dst + i * 32 * 128, &amap, bar, k * 64, t.at + i * 32);
                    for (int i = 0; i < 128; i += 64) tma_load_2d(wdst + i * 128, &bmap, bar, k * 64, brow + i);
                    for (int i = 0; i < 128; i += 64) tma_load_2d(wdst + (128 + i) * 128, MODE == EG_GATED ? &umap : &bmap, bar, k * 64, (MODE == EG_GATED ? brow : brow + 128) + i);
                }
                __syncwarp();
                if (++s == stages) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        int s = 0, ph = 0;
        unsigned it = 0;
        for (int tile = blockIdx.x; tile < total; tile += gridDim.x, it++) {
            const Tile t = place(tile);
            const uint32_t idesc = instr_desc(1, 1, 1, 0, 0, 128, (t.n + 15) & ~15);      // f32 += bf16 . bf16, K-major both
            const int buf = it % sets;
            const uint32_t d = tmem + buf * 256;
            bar_wait(smem_u32(&misc.d_free[buf]), ((it / sets) & 1) ^ 1);
            for (int k = 0; k < p.nk; k++) {
                bar_wait(smem_u32(&misc.full[s]), ph);
                tc_fence_after();
                const uint32_t b = base + s * stage, a = b + wofs;
                const uint64_t bd = smem_desc(b, 16, 1024, kLayoutSw128);
                mma_f16_x4(d, smem_desc(a, 16, 1024, kLayoutSw128), bd, idesc, k != 0);
                mma_f16_x4(d + second, smem_desc(a + 128 * 128, 16, 1024, kLayoutSw128), bd, idesc, k != 0, smem_u32(&misc.free[s]), k + 1 == p.nk ? smem_u32(&misc.d_full[buf]) : 0);
                if (++s == stages) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp >= 4) {
        // epilogue: a thread owns a row of either matrix and every fourth run of 16 pairs
        const int sp = warp & 3, part = (warp - 4) >> 2;
        unsigned it = 0;
        for (int tile = blockIdx.x; tile < total; tile += gridDim.x, it++) {
            const Tile t = place(tile);
            const int buf = it % sets, col = t.n0 + 32 * sp + lane;
            const uint32_t tc = tmem + ((uint32_t)(32 * sp) << 16) + buf * 256;
            bar_wait(smem_u32(&misc.d_full[buf]), (it / sets) & 1);
            tc_fence_after();
#pragma unroll 1
            for (int c = 16 * part; c < t.n; c += 64) {
                uint32_t v[16], u[16];
                tmem_ld16(tc + c, v);
                tmem_ld16(tc + second + c, u);
                tmem_wait_ld();
                const long pos = (long)t.at + c;
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    if (c + i >= t.n) break;
                    const float a = __uint_as_float(v[i]), b = __uint_as_float(u[i]);
                    if (MODE == EG_DOWN) {
                        float* o = (float*)p.out + (pos + i) * p.cols;
                        if (col < p.cols) o[col] = a;
                        if (col + 128 < p.cols) o[col + 128] = b;
                    } else {
                        const float sc = p.row_scale ? p.row_scale[pos + i] : 1.f;
                        __nv_bfloat16* o = (__nv_bfloat16*)p.out + (pos + i) * p.cols;
                        if (MODE == EG_GATED) {
                            if (col < p.cols) o[col] = __float2bfloat16_rn(gated_act(a * sc, b * sc, p.act, p.limit));
                        } else {
                            const float ra = fmaxf(a * sc, 0.f), rb = fmaxf(b * sc, 0.f);
                            if (col < p.cols) o[col] = __float2bfloat16_rn(ra * ra);
                            if (col + 128 < p.cols) o[col + 128] = __float2bfloat16_rn(rb * rb);
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(smem_u32(&misc.d_free[buf]));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

static int eg_map(CUtensorMap* map, const void* ptr, long cols, long rows, int box_rows) {      // boxes of so many rows x 64 bf16
    EncodeTiledFn enc = encode_tiled();
    if (!enc) { set_error("experts_prompt: cuTensorMapEncodeTiled is not available from this driver"); return KTB200_ECUDA; }
    const cuuint64_t dim[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, stride[1] = {(cuuint64_t)cols * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows}, estr[2] = {1, 1};
    const CUresult cr = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dim, stride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) { set_error("experts_prompt: cuTensorMapEncodeTiled failed (%d)", (int)cr); return KTB200_ECUDA; }
    return KTB200_OK;
}
template <int MODE>
static int eg_gemm(const void* a, long a_rows, int K, const void* b, const void* u, long b_rows, const EgParams& p, int grid, cudaStream_t s) {
    CUtensorMap am, bm, um;
    int rc = eg_map(&am, a, K, a_rows, 32);
    if (rc == KTB200_OK) rc = eg_map(&bm, b, K, b_rows, 64);
    if (rc == KTB200_OK) rc = eg_map(&um, u ? u : b, K, b_rows, 64);
    if (rc) return rc;
    KTB_CUDA_CHECK(cudaFuncSetAttribute(eg_gemm_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kEgSmem));
    KTB_CUDA_CHECK(launch_pdl(eg_gemm_kernel<MODE>, dim3(grid), dim3(kEgThreads), (size_t)kEgSmem, s, am, bm, um, p));
    KTB_LAUNCH_CHECK();
    return KTB200_OK;
}
static size_t up256(size_t n) { return (n + 255) / 256 * 256; }
}  // namespace ktb

using namespace ktb;

extern "C" int ktb200_experts_combine(const void* rows, const int64_t* place, const int64_t* ids, int n_experts, const float* weights, int top, float* out, int n_tokens, int width, int dtype,
                                      void* stream);

extern "C" size_t ktb200_experts_prompt_workspace(int n_tokens, int top, int n_experts, int width, int ff) {
    const size_t P = (size_t)n_tokens * top;
    return up256((3 * (size_t)n_experts + 2) * sizeof(int)) + up256(P * 8) + up256(P * 4) + up256(P * width * 2) + up256(P * ff * 2) + up256(P * width * 4);
}

extern "C" int ktb200_experts_prompt(const void* x, const int64_t* ids, const float* weights, int weights_on_input, int top, int n_experts, const void* w_gate, const void* w_up,
                                     const void* w_down, float* out, int n_tokens, int width, int ff, int act_kind, float limit, void* workspace, void* stream) {
    if (!x || !ids || !weights || !w_up || !w_down || !out || !workspace || top <= 0 || n_experts <= 0 || width <= 0 || ff <= 0) { set_error("experts_prompt: bad argument"); return KTB200_EINVAL; }
    if (width % 8 || ff % 8 || n_experts > kEgMaxExperts) { set_error("experts_prompt: widths in multiples of 8, at most %d experts", kEgMaxExperts); return KTB200_EINVAL; }
    if (((uintptr_t)x | (uintptr_t)w_gate | (uintptr_t)w_up | (uintptr_t)w_down | (uintptr_t)workspace) & 15) { set_error("experts_prompt: 16-byte aligned rows"); return KTB200_EINVAL; }
    if (n_tokens <= 0) return KTB200_OK;
    const size_t P = (size_t)n_tokens * top;
    if (P > (1u << 30)) { set_error("experts_prompt: too many pairs"); return KTB200_EINVAL; }
    cudaStream_t s = (cudaStream_t)stream;
    int dev = 0;
    KTB_CUDA_CHECK(cudaGetDevice(&dev));
    uint8_t* at = (uint8_t*)workspace;
    auto take = [&](size_t n) { uint8_t* p = at; at += up256(n); return p; };
    int* counts = (int*)take((3 * (size_t)n_experts + 2) * sizeof(int));
    int *offsets = counts + n_experts, *prefix = offsets + n_experts;
    int64_t* place = (int64_t*)take(P * 8);
    float* scale = (float*)take(P * 4);
    void *xs = take(P * width * 2), *a = take(P * ff * 2), *y = take(P * width * 4);
    eg_sort_kernel<<<1, 1024, 0, s>>>(ids, (int)P, n_experts, counts, offsets, prefix, place, (ff + (w_gate ? 127 : 255)) / (w_gate ? 128 : 256), num_sms(dev));
    KTB_LAUNCH_CHECK();
    KTB_CUDA_CHECK(launch_pdl(eg_gather_kernel, dim3((unsigned)P), dim3(128), 0, s, (const uint4*)x, weights, top, width / 8, (const int64_t*)place, weights_on_input ? scale : nullptr,
                              (uint4*)xs));
    KTB_LAUNCH_CHECK();
    const int grid = num_sms(dev);
    EgParams p{counts, offsets, prefix, n_experts, (width + 63) / 64, ff, ff, act_kind, limit, weights_on_input ? scale : nullptr, a};
    int rc;
    if (w_gate) rc = eg_gemm<EG_GATED>(xs, (long)P, width, w_gate, w_up, (long)n_experts * ff, p, grid, s);
    else rc = eg_gemm<EG_RELU2>(xs, (long)P, width, w_up, nullptr, (long)n_experts * ff, p, grid, s);
    if (rc) return rc;
    EgParams d{counts, offsets, prefix, n_experts, (ff + 63) / 64, width, width, 0, 0.f, nullptr, y};
    rc = eg_gemm<EG_DOWN>(a, (long)P, ff, w_down, nullptr, (long)n_experts * width, d, grid, s);
    if (rc) return rc;
    return ktb200_experts_combine(y, place, ids, n_experts, weights_on_input ? nullptr : weights, top, out, n_tokens, width, KTB200_TYPE_F32, stream);
}
