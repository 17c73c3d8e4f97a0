// Routed experts of a prompt portion — MOE::forward_many
// (archive/csrc/ktransformers_ext/operators/llamafile/moe.cpp:248-365 = kt-kernel/operators/llamafile/moe.hpp:461-746):
//     count tokens per expert -> per-token Q8_K quantisation, stored in per-expert contiguous order ->
//     per-expert GEMMs (gate and up in one launch) -> silu * mul -> requantise -> per-expert GEMM (down) -> per-token weighted gather.
// The decode kernels stream every (token, expert) pair's weights; here an expert's weights are read once per 64 of its tokens.  The GEMMs are
// kq_gemm.cu; this file sorts the pairs and puts the tokens' results together.
#include <cstdlib>

#include "act_quant.cuh"
#include "common.cuh"
#include "handles.cuh"
#include "kq_gemm.cuh"

namespace ktb {

// tile table: tile -> {expert, first weight row, first sorted position, tokens}, token tile fastest so that CTAs running side by side share the
// weight tile through L2.  One thread per tile; tiles beyond the data-dependent total are left alone.
__device__ __forceinline__ void grp_tile(int tile, const int* nt_prefix, const int* offsets, const int* counts, int E, int MT, int rows, int4* tinfo) {
    if (tile >= nt_prefix[E] * MT) return;
    int lo = 0, hi = E;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (nt_prefix[mid] * MT <= tile) lo = mid; else hi = mid;
    }
    const int local = tile - nt_prefix[lo] * MT, ntile_e = nt_prefix[lo + 1] - nt_prefix[lo];
    const int mt = local / ntile_e, nt = local - mt * ntile_e;
    tinfo[tile] = make_int4(lo, mt * rows, offsets[lo] + nt * kKqN, min(kKqN, counts[lo] - nt * kKqN));
}

// ---------------------------------------------------------------------------------------------------------------
// bookkeeping kernels (moe.cpp:250-290: m_local_num_, m_local_pos_, prefix offsets)
__global__ void grp_count_kernel(const int64_t* ids, int npairs, int k, int id_offset, int n_local, const int* bsz, int t0, int* counts) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npairs) return;
    if (bsz && t0 + i / k >= *bsz) return;
    const long e = (long)ids[i] - id_offset;
    if (e >= 0 && e < n_local) atomicAdd(counts + e, 1);
}
// one CTA of 1024 threads, a thread per expert: an expert's rows start at a multiple of 4 (16-byte aligned token scales)
__global__ void __launch_bounds__(1024) grp_scan_kernel(const int* counts, int E, int* offsets, int* nt_prefix, int* cursor) {
    __shared__ int2 part[32];
    const int e = threadIdx.x, lane = e & 31, warp = e >> 5, n = e < E ? counts[e] : 0;
    const int2 own = make_int2((n + 3) & ~3, (n + kKqN - 1) / kKqN);
    int2 v = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, v.x, o), y = __shfl_up_sync(0xffffffffu, v.y, o);
        if (lane >= o) { v.x += x; v.y += y; }
    }
    if (lane == 31) part[warp] = v;
    __syncthreads();
    for (int w = 0; w < warp; w++) { v.x += part[w].x; v.y += part[w].y; }
    if (e < E) {
        offsets[e] = cursor[e] = v.x - own.x;
        nt_prefix[e] = v.y - own.y;
        if (e == E - 1) nt_prefix[E] = v.y;
    }
}
// what the offsets are for, in one launch: a thread per pair (its place), then a thread per tile of gate and up, then of down
__global__ void grp_place_kernel(const int64_t* ids, int npairs, int k, int id_offset, int n_local, const int* bsz, int t0, int* cursor, int* pos, const int* nt_prefix, const int* offsets,
                                 const int* counts, int mt_gu, int ub_gu, int4* tinfo_gu, int mt_d, int rows_d, int4* tinfo_d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < npairs) {
        const long e = (long)ids[i] - id_offset;
        if ((bsz && t0 + i / k >= *bsz) || e < 0 || e >= n_local) { pos[i] = -1; return; }
        const int s = atomicAdd(cursor + e, 1);   // order inside an expert is irrelevant: every pair's result is independent
        pos[i] = s;
        return;
    }
    i -= npairs;
    if (i < ub_gu) grp_tile(i, nt_prefix, offsets, counts, n_local, mt_gu, 128, tinfo_gu);
    else grp_tile(i - ub_gu, nt_prefix, offsets, counts, n_local, mt_d, rows_d, tinfo_d);
}
// out[t] = sum_j w[t][j] * down[pos[t][j]] in expert_ids order, one FMA per expert (moe.cpp:340-358), rounded like from_float
// Four columns a thread, the loads of four choices in flight: bound by the rows' bytes (1024 tokens of 8 choices and 7168 columns, 235 MB: 60 us column by column, 40 like this).
__global__ void __launch_bounds__(256) grp_combine_kernel(const float* dd, const int* pos, const float* weights, int T, int k, int H, const int* bsz, int t0, void* out,
                                                          int hidden_type) {
    const int t = blockIdx.y;
    if (bsz && t0 + t >= *bsz) return;
    const int h = (blockIdx.x * blockDim.x + threadIdx.x) * 4;      // (H is a multiple of 256)
    if (h >= H) return;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j0 = 0; j0 < k; j0 += 4) {
        float4 v[4];
        int s[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            s[j] = j0 + j < k ? pos[t * k + j0 + j] : -1;
            if (s[j] >= 0) v[j] = __ldcs(reinterpret_cast<const float4*>(dd + (long)s[j] * H + h));
        }
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (s[j] >= 0) {
                const float w = weights[t * k + j0 + j];
                acc.x = __fmaf_rn(v[j].x, w, acc.x); acc.y = __fmaf_rn(v[j].y, w, acc.y); acc.z = __fmaf_rn(v[j].z, w, acc.z); acc.w = __fmaf_rn(v[j].w, w, acc.w);
            }
    }
    const long at = (long)t * H + h;
    store_hidden(out, at, hidden_type, acc.x); store_hidden(out, at + 1, hidden_type, acc.y); store_hidden(out, at + 2, hidden_type, acc.z); store_hidden(out, at + 3, hidden_type, acc.w);
}

// true when ktb200_moe_forward may take the grouped tensor-core path for this handle: gate and up of one type, every matrix in a layout of kq_gemm.cu
static KqFmt grp_gate_up(const ktb200_moe* m) {
    const KqFmt g = kq_fmt(pick_fmt(m->cfg.gate_type, m->gu_soa));
    return g == kq_fmt(pick_fmt(m->cfg.up_type, m->gu_soa)) ? g : KQ_NONE;
}
bool grouped_ok(const ktb200_moe* m, int k) {
    const ktb200_moe_config& c = m->cfg;
    return grp_gate_up(m) != KQ_NONE && kq_fmt(pick_fmt(c.down_type, m->down_layout)) != KQ_NONE && c.hidden_size % 256 == 0 && c.intermediate_size % 256 == 0 && c.expert_num <= 1023 &&
           k <= 32;
}

int moe_forward_grouped(ktb200_moe* m, int qlen, int k, const int64_t* ids, const float* weights, const void* input, void* output, const int* bsz, cudaStream_t s) {
    const ktb200_moe_config& c = m->cfg;
    const int E = c.expert_num, H = c.hidden_size, I = c.intermediate_size, dev = m->device;
    static const int chunk_cap = [] { const char* e = getenv("KTB200_GROUPED_CHUNK"); return e ? atoi(e) : 1024; }();
    const int Tc = qlen < chunk_cap ? qlen : chunk_cap;
    const KqFmt fg = grp_gate_up(m), fd = kq_fmt(pick_fmt(c.down_type, m->down_layout));
    const size_t hb = type_size(c.hidden_type);
    // scratch of one chunk: bookkeeping | quantised tokens, gate and up rows (then the down rows in their place) | quantised activations
    const size_t P = (size_t)Tc * k, rows = P + 3 * (size_t)E;
    const int ub_gu = (int)(P / kKqN + E) * (I / 128), ub_d = (int)(P / kKqN + E) * (H / kKqRows);      // upper bounds of the tile counts
    auto up = [](size_t n) { return (n + 255) / 256 * 256; };
    const size_t n_ints = up((4 * (size_t)(E + 1) + P) * 4), n_tab = up((size_t)(ub_gu + ub_d) * sizeof(int4));
    const size_t n_x = up(KqActs::bytes(rows, H)), n_g = up(rows * I * 4), n_d = up(rows * H * 4), n_a = up(KqActs::bytes(rows, I));
    const size_t n_mid = n_x + 2 * n_g > n_d ? n_x + 2 * n_g : n_d;
    ScratchBlock mem(s);
    if (!mem.taken(dev, n_ints + n_tab + n_mid + n_a)) return kNoScratch;
    uint8_t* at = reinterpret_cast<uint8_t*>(mem.ptr);
    int *counts = reinterpret_cast<int*>(at), *offsets = counts + E + 1, *nt_prefix = offsets + E + 1, *cursor = nt_prefix + E + 1, *pos = cursor + E + 1;
    int4 *tinfo_gu = reinterpret_cast<int4*>(at + n_ints), *tinfo_d = tinfo_gu + ub_gu;
    uint8_t* mid = at + n_ints + n_tab;
    const KqActs xa(mid, (long)rows, H), aa(mid + n_mid, (long)rows, I);
    float *g = reinterpret_cast<float*>(mid + n_x), *u = reinterpret_cast<float*>(mid + n_x + n_g), *dd = reinterpret_cast<float*>(mid);
    for (int t0 = 0; t0 < qlen; t0 += Tc) {
        const int T = qlen - t0 < Tc ? qlen - t0 : Tc, n = T * k;
        const int64_t* ids_c = ids + (size_t)t0 * k;
        const uint8_t* x_c = reinterpret_cast<const uint8_t*>(input) + (size_t)t0 * H * hb;
        uint8_t* o_c = reinterpret_cast<uint8_t*>(output) + (size_t)t0 * H * hb;
        KTB_CUDA_CHECK(cudaMemsetAsync(counts, 0, (size_t)E * sizeof(int), s));
        grp_count_kernel<<<(n + 255) / 256, 256, 0, s>>>(ids_c, n, k, c.expert_id_offset, E, bsz, t0, counts);
        grp_scan_kernel<<<1, 1024, 0, s>>>(counts, E, offsets, nt_prefix, cursor);
        grp_place_kernel<<<(n + ub_gu + ub_d + 255) / 256, 256, 0, s>>>(ids_c, n, k, c.expert_id_offset, E, bsz, t0, cursor, pos, nt_prefix, offsets, counts, I / 128, ub_gu, tinfo_gu,
                                                                        H / kKqRows, kKqRows, tinfo_d);
        int rc = kq_quant(x_c, c.hidden_type, T, H, pos, k, kq_is_q6(fg), kq_limit(fg), xa, s);
        if (rc) return rc;
        KqGemm gp{};
        gp.fmt = fg; gp.w[0] = c.gate_proj; gp.w[1] = c.up_proj; gp.pair = true; gp.expert_bytes = (long)I * row_bytes(H, c.gate_type); gp.experts = E; gp.R = I; gp.K = H; gp.acts = &xa;
        gp.tinfo = tinfo_gu; gp.n_tiles_dev = nt_prefix + E; gp.tiles_mul = I / 128; gp.splits = 1; gp.out[0] = g; gp.out[1] = u;
        rc = kq_gemm(gp, dev, s);
        if (rc) return rc;
        rc = kq_act_quant(g, u, pos, n, I, c.use_silu, kq_is_q6(fd), kq_limit(fd), aa, s);
        if (rc) return rc;
        KqGemm gd{};
        gd.fmt = fd; gd.w[0] = gd.w[1] = c.down_proj; gd.expert_bytes = (long)H * row_bytes(I, c.down_type); gd.experts = E; gd.R = H; gd.K = I; gd.acts = &aa;
        gd.tinfo = tinfo_d; gd.n_tiles_dev = nt_prefix + E; gd.tiles_mul = H / kKqRows; gd.splits = 1; gd.out[0] = gd.out[1] = dd;
        rc = kq_gemm(gd, dev, s);
        if (rc) return rc;
        grp_combine_kernel<<<dim3((H + 1023) / 1024, T), 256, 0, s>>>(dd, pos, weights + (size_t)t0 * k, T, k, H, bsz, t0, o_c, c.hidden_type);
        KTB_LAUNCH_CHECK();
        count_launch(3);      // 10 launches per chunk: the 6 that kq_* and the 1 that the check counts, and the 3 bookkeeping kernels
    }
    return KTB200_OK;
}

}  // namespace ktb
