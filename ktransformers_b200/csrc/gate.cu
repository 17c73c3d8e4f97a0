// DeepSeek MoEGate routing on the GPU.  Replaces MoEGate.forward
// (archive/ktransformers/models/modeling_deepseek_v3.py:430-481 for V3 sigmoid/noaux_tc,
//  archive/ktransformers/models/modeling_deepseek.py:411-459 for V2 softmax greedy/group_limited_greedy),
// which the reference runs as ~10 ATen kernels per layer (fp32 F.linear, sigmoid, two topk, scatter,
// masked_fill, gather, sum, div, mul).
//
// Two kernels, the second a programmatic dependent launch of the first:
//   gate_dot_kernel     fp32 GEMV  logits[t][e] = x_t(fp32) . W[e]   (HBM-bound: E*H*4 bytes).  A CTA of 4 warps owns 4
//            expert rows x one column split; each warp streams its row slice with 16-byte loads (8 in flight
//            per lane) against the token slice staged in shared memory, and writes one partial sum per
//            (token, expert, split).  Partials are added in fixed split order: deterministic, no float atomics.
//   gate_select_kernel  one CTA of 128 threads per token: scoring, bias, group top-2 / max, group top-k, expert top-k by
//            iterative arg-max with REDUX max/min (ties -> lowest index), gather, normalise, scale.
// The partial sums are scratch of the call (common.cuh): calls on several streams or threads and replays of captured ones share nothing, and no CTA waits for another.
#include <algorithm>

#include "gate.cuh"

namespace ktb {

// Bound for batches by chains of loads: CTAs of their own for every tile of 8 tokens (they share the rows through L2), a tile's columns in one round of loads while the rows are on
// their way to L2 (256 x 7168, 24 tokens: 77.6 us with one CTA per rows and columns that took tile after tile, value by value, and 16 selectors).  The selection as a launch of its own, against
// the dots' last CTAs selecting behind a counter (us, calls in a graph, weights from memory, 256 x 7168): one token 13.1 -> 10.9, 8 tokens 16.9 -> 15.7, 24 tokens 29.3 -> 26.5,
// 200 tokens 154 -> 137; 64 x 2048, 24 tokens 11.3 -> 9.7.
// 5 CTAs an SM (96 registers) where there are more than two an SM and more than two tokens, else all the registers a thread's loads in flight want.
constexpr int kGateTiles = 16;
// a tile's columns in fp32: four values a load, eight loads of a thread in flight before the first is looked at
__device__ __forceinline__ float4 gate_floats(uint4 w, int) { return make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w)); }
__device__ __forceinline__ float4 gate_floats(uint2 w, int hidden_type) {
    if (hidden_type == KTB200_TYPE_BF16)
        return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u));
    return make_float4(fp16_bits_to_f32((uint16_t)(w.x & 0xffff)), fp16_bits_to_f32((uint16_t)(w.x >> 16)), fp16_bits_to_f32((uint16_t)(w.y & 0xffff)), fp16_bits_to_f32((uint16_t)(w.y >> 16)));
}
template <typename V>
__device__ __forceinline__ void gate_stage(const V* x, int row, int nt, int nc4, int hidden_type, float4* xs) {
    for (int i0 = threadIdx.x; i0 < nt * nc4; i0 += 8 * kGateThreads) {
        V v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int i = min(i0 + u * kGateThreads, nt * nc4 - 1), tt = i / nc4;
            v[u] = __ldg(x + (long)tt * row + (i - tt * nc4));
        }
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (i0 + u * kGateThreads < nt * nc4) xs[i0 + u * kGateThreads] = gate_floats(v[u], hidden_type);
    }
}

template <int PER_SM>      // CTAs an SM that its registers leave room for (1: as many as the compiler wants)
__global__ void __launch_bounds__(kGateThreads, PER_SM) gate_dot_kernel(const GateParams p) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    float* xs = reinterpret_cast<float*>(smem_raw);   // [tok tile][slice cols]
    griddep_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int Teff = p.T;
    if (p.bsz) Teff = min(p.T, *p.bsz);
    const int s = blockIdx.y, S = p.S;
    const int n4 = p.H / 4;
    const int c0 = (int)((long)n4 * s / S), c1 = (int)((long)n4 * (s + 1) / S);   // float4 column range of this split
    const int nc4 = c1 - c0;
    const int e = blockIdx.x * kGateWarps + warp;
    const float4* wrow = reinterpret_cast<const float4*>(p.W + (long)(e < p.E ? e : 0) * p.H) + c0;

    // the rows are under way to L2 while the tokens are fetched
    if (e < p.E)
        for (int c = 8 * lane; c < nc4; c += 256) asm volatile("prefetch.global.L2 [%0];" ::"l"(wrow + c));
    const bool vec = (reinterpret_cast<uintptr_t>(p.x) & (p.hidden_type == KTB200_TYPE_F32 ? 15 : 7)) == 0;
    for (int t0 = blockIdx.z * kGateTokTile; t0 < Teff; t0 += gridDim.z * kGateTokTile) {
        const int nt = min(kGateTokTile, Teff - t0);
        __syncthreads();
        if (vec) {
            const long x0 = (long)t0 * p.H + 4L * c0;
            if (p.hidden_type == KTB200_TYPE_F32) gate_stage(reinterpret_cast<const uint4*>(reinterpret_cast<const float*>(p.x) + x0), p.H / 4, nt, nc4, p.hidden_type, reinterpret_cast<float4*>(xs));
            else gate_stage(reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(p.x) + x0), p.H / 4, nt, nc4, p.hidden_type, reinterpret_cast<float4*>(xs));
        } else {
            for (int tt = 0; tt < nt; tt++)
                for (int c = threadIdx.x; c < nc4 * 4; c += kGateThreads) xs[tt * nc4 * 4 + c] = load_hidden(p.x, (long)(t0 + tt) * p.H + 4L * c0 + c, p.hidden_type);
        }
        __syncthreads();
        if (e < p.E) {
            switch (nt) {   // compile-time token counts: no predicated-off FMAs for the common bs=1 decode
                case 1: gate_dot<1>(p, wrow, xs, nc4, lane, t0, e, s, S); break;
                case 2: gate_dot<2>(p, wrow, xs, nc4, lane, t0, e, s, S); break;
                case 3: case 4: gate_dot<4>(p, wrow, xs, nc4, lane, t0, e, s, S, nt); break;
                default: gate_dot<kGateTokTile>(p, wrow, xs, nc4, lane, t0, e, s, S, nt); break;
            }
        }
    }
}

// From the partial sums (S of them) or from logits that a GEMM has already made (S = 1): one CTA per token (grid-stride)
__global__ void __launch_bounds__(kGateThreads) gate_select_kernel(const GateParams p) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    griddep_wait();
    const int T = p.bsz ? min(p.T, *p.bsz) : p.T;
    for (int t = blockIdx.x; t < T; t += gridDim.x)
        gate_select_token<0>(p, t, reinterpret_cast<float*>(smem_raw), p.idx + (long)t * p.top_k, p.w + (long)t * p.top_k, p.logits_out);
}
// Both for a token in one CTA, its partial sums (the same, in the same order) in shared memory: where the pool has no memory for them.  Every CTA reads all of W through L2 (256 x 7168, one to 148 tokens: 584 us)
__global__ void __launch_bounds__(kGateThreads) gate_alone_kernel(const GateParams p) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    GateParams own = p;
    own.partial = reinterpret_cast<float*>(smem_raw);
    float *sel = own.partial + (size_t)p.S * p.E, *xs = sel + 2 * p.E + 32 + 4 * kGateWarps;
    xs = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(xs) + 15) & ~(uintptr_t)15);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n4 = p.H / 4, T = p.bsz ? min(p.T, *p.bsz) : p.T;
    for (int t = blockIdx.x; t < T; t += gridDim.x) {
        for (int s = 0; s < p.S; s++) {
            const int c0 = (int)((long)n4 * s / p.S), nc4 = (int)((long)n4 * (s + 1) / p.S) - c0;
            __syncthreads();
            for (int c = threadIdx.x; c < nc4 * 4; c += kGateThreads) xs[c] = load_hidden(p.x, (long)t * p.H + 4L * c0 + c, p.hidden_type);
            __syncthreads();
            for (int e = warp; e < p.E; e += kGateWarps) gate_dot<1>(own, reinterpret_cast<const float4*>(p.W + (long)e * p.H) + c0, xs, nc4, lane, 0, e, s, p.S);
        }
        __syncthreads();
        gate_select_token<0, true>(own, 0, sel, p.idx + (long)t * p.top_k, p.w + (long)t * p.top_k, p.logits_out ? p.logits_out + (long)t * p.E : nullptr);
    }
}
static size_t gate_select_smem(int E) { return ((size_t)2 * E + 32 + 4 * kGateWarps) * sizeof(float); }
static int gate_select_ctas(int T) { return std::min(T, 148 * 16); }

}  // namespace ktb

extern "C" int ktb200_moe_gate_forward(const ktb200_gate_config* c, int qlen, const void* x, int64_t* idx, float* w,
                                       float* logits, const int* bsz, void* stream) {
    using namespace ktb;
    if (!c || !x || !idx || !w) { set_error("null pointer"); return KTB200_EINVAL; }
    if (qlen <= 0) return KTB200_OK;
    if (c->n_experts > kGateThreads * kGateEPT) { set_error("gate: at most %d experts", kGateThreads * kGateEPT); return KTB200_EINVAL; }
    if (c->n_experts <= 0 || c->hidden_size <= 0 || c->hidden_size % 4 || c->top_k <= 0 || c->top_k > 32 || c->top_k > c->n_experts) {
        set_error("gate: bad shape (E=%d H=%d top_k=%d; top_k<=32, H%%4==0)", c->n_experts, c->hidden_size, c->top_k);
        return KTB200_EINVAL;
    }
    if (c->n_group < 1 || c->n_group > 32 || c->n_experts % c->n_group || c->topk_group < 1 || c->topk_group > c->n_group) {
        set_error("gate: bad grouping (n_group=%d topk_group=%d)", c->n_group, c->topk_group);
        return KTB200_EINVAL;
    }
    if (c->scoring < 0 || c->scoring > 2 || c->topk_method < 0 || c->topk_method > 3) { set_error("gate: bad scoring/topk_method"); return KTB200_EINVAL; }
    if (!is_hidden_type(c->hidden_type) || !c->weight) { set_error("gate: bad hidden_type or null weight"); return KTB200_EINVAL; }
    int dev = 0;
    KTB_CUDA_CHECK(cudaGetDevice(&dev));
    cudaStream_t s = (cudaStream_t)stream;
    const int row_ctas = (c->n_experts + kGateWarps - 1) / kGateWarps;
    const int S = gate_splits(c->n_experts, c->hidden_size, num_sms(dev));
    ScratchBlock partial(s);
    const bool alone = partial.take(dev, (size_t)qlen * c->n_experts * S * sizeof(float)) != cudaSuccess;
    GateParams p{c->weight, x, c->hidden_type, c->n_experts, c->hidden_size, qlen, S, c->top_k, c->n_group, c->topk_group,
                 c->scoring, c->topk_method, c->norm_topk_prob, c->routed_scaling_factor, c->bias, (float*)partial.ptr, logits,
                 idx, w, bsz};
    const int nc4_max = c->hidden_size / 4 / S + 1;
    if (alone) {
        const size_t smem = (size_t)S * c->n_experts * sizeof(float) + gate_select_smem(c->n_experts) + (size_t)nc4_max * 16 + 16;
        if (smem > 48 * 1024) KTB_CUDA_CHECK(raise_smem_limit((const void*)gate_alone_kernel, smem));
        gate_alone_kernel<<<gate_select_ctas(qlen), kGateThreads, smem, s>>>(p);
        KTB_LAUNCH_CHECK();
        return KTB200_OK;
    }
    const int nt = qlen < kGateTokTile ? qlen : kGateTokTile;
    const size_t smem = (size_t)nt * nc4_max * 16;
    const int tiles = std::min((qlen + kGateTokTile - 1) / kGateTokTile, kGateTiles);
    auto kernel = qlen > 2 && row_ctas * S * tiles > 2 * num_sms(dev) ? gate_dot_kernel<5> : gate_dot_kernel<1>;
    if (smem > 48 * 1024) KTB_CUDA_CHECK(raise_smem_limit((const void*)kernel, smem));
    kernel<<<dim3(row_ctas, S, tiles), kGateThreads, smem, s>>>(p);
    KTB_LAUNCH_CHECK();
    KTB_CUDA_CHECK(launch_pdl(gate_select_kernel, dim3(gate_select_ctas(qlen)), dim3(kGateThreads), gate_select_smem(c->n_experts), s, p));
    count_launch();
    return KTB200_OK;
}

/* The selection of ktb200_moe_gate_forward on logits [qlen][E] fp32 computed elsewhere (c->weight and c->hidden_* are not read). */
extern "C" int ktb200_moe_gate_select(const ktb200_gate_config* c, int qlen, const float* logits, int64_t* idx, float* w, void* stream) {
    using namespace ktb;
    if (!c || !logits || !idx || !w) { set_error("null pointer"); return KTB200_EINVAL; }
    if (qlen <= 0) return KTB200_OK;
    if (c->n_experts <= 0 || c->n_experts > kGateThreads * kGateEPT || c->top_k <= 0 || c->top_k > 32 || c->top_k > c->n_experts) {
        set_error("gate: bad shape (E=%d top_k=%d; E<=%d, top_k<=32)", c->n_experts, c->top_k, kGateThreads * kGateEPT);
        return KTB200_EINVAL;
    }
    if (c->n_group < 1 || c->n_group > 32 || c->n_experts % c->n_group || c->topk_group < 1 || c->topk_group > c->n_group) {
        set_error("gate: bad grouping (n_group=%d topk_group=%d)", c->n_group, c->topk_group);
        return KTB200_EINVAL;
    }
    if (c->scoring < 0 || c->scoring > 2 || c->topk_method < 0 || c->topk_method > 3) { set_error("gate: bad scoring/topk_method"); return KTB200_EINVAL; }
    GateParams p{nullptr, nullptr, c->hidden_type, c->n_experts, c->hidden_size, qlen, 1, c->top_k, c->n_group, c->topk_group,
                 c->scoring, c->topk_method, c->norm_topk_prob, c->routed_scaling_factor, c->bias, const_cast<float*>(logits), nullptr,
                 idx, w, nullptr};
    gate_select_kernel<<<gate_select_ctas(qlen), kGateThreads, gate_select_smem(c->n_experts), (cudaStream_t)stream>>>(p);
    KTB_LAUNCH_CHECK();
    return KTB200_OK;
}
