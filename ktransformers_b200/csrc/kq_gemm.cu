// Prompt-sized products against GGUF K-quant matrices — the per-expert GEMMs of MOE::forward_many (archive/csrc/ktransformers_ext/operators/
// llamafile/moe.cpp:248-365) and the dense linears of a prompt portion (operators/llamafile/linear.cpp:37-70) — on tcgen05 with the weights
// as the tensor-memory operand.
//
// Arithmetic: the reference's dot of a 256-block is an exact integer, sum_j sc_j * sum_i q_ij * x8_ij, scaled in fp32.  Here a weight enters the
// tensor core as the fp16 integer sc * q (Q4_K: at most 63 * 15; Q5_K: 63 * 31, halved; Q6_K: two terms, sc * (low four bits) and
// sc * (16 * high two bits - 32), both quartered), an activation as the fp16 integer x8; the products are exact, the fp32 accumulator of a
// 256-block holds integers (or halves, quarters) that stay below 2^24 short of inputs built for it, and the epilogue applies
// dx * (d * isum - dmin * msum) once per block in fp32, the decode kernels' formula; msum (minima x 16-value activation sums) is one K = 16 MMA.
//
// What bounds it: an expert's weights are read from HBM once per 64 of its tokens (1024 tokens of 256 experts: about once), so the routed
// experts are HBM-bound, and the work per weight has to stay under what an SM has per weight byte that arrives (24 B per cycle):
//   * the weights go registers -> tensor memory (tcgen05.st, a thread = a weight row = a lane) and never to shared memory as operands.  Through
//     shared memory, 2 B per weight written and 2 B read by the MMA would take 128 B per cycle to 21 weights per cycle, half of what HBM brings;
//     and an MMA of 128 x 64 x 16 runs in 32 cycles with A in tensor memory against 48 with A in shared memory (measured; N = 32: 17 and 40).
//   * nibbles become fp16 by or-ing them into the mantissa of 1024 and one fused multiply-add with (sc, -1024 sc): 9 instructions for 8
//     weights.  The pairs come out as (0, 2), (1, 3) of four; the activations are stored in that order (kq_pos4).
//   * a scale per 256-block needs the accumulator drained per 256-block: two matrices of 128 rows per CTA (gate and up of the same experts, or
//     256 rows of one) take turns, one drained while the other multiplies, and share the activation tiles.
// CTA: 20 warps.  0-3 / 4-7 producers of matrix 0 / 1: cp.async ring of raw blocks private to the warp (32 rows) -> registers -> TMEM;
//      8 TMA of activations, 9 / 10 MMA issuers of matrix 0 / 1; 12-15 / 16-19 epilogue of matrix 0 / 1.
// TMEM: [accumulator | minima] x 2 matrices, then 64-column operand stages, 2 per matrix.
#include <cuda_fp16.h>

#include "act_quant.cuh"
#include "kq_gemm.cuh"
#include "umma.cuh"

namespace ktb {

using namespace umma;

template <int FMT>
struct KqCfg {
    static constexpr bool kQ6 = FMT == KQ_Q6K_T4 || FMT == KQ_Q6K_SOA8;
    static constexpr int kRow = FMT == KQ_Q4K ? 144 : FMT == KQ_Q5K ? 176 : 208;      // bytes of a row's block in a ring slot: 16-byte words, an odd number of them (conflict-free)
    static constexpr int kTail = kQ6 ? 4 : 0;                                         // + the word that holds a Q6_K block's d
    static constexpr int kRing = FMT == KQ_Q4K ? 3 : 2;
    static constexpr int kWarpSlot = 32 * (kRow + kTail);
    static constexpr int kStages = kQ6 ? 4 : 2;                                       // operand stages per block
    static constexpr float kScale = FMT == KQ_Q4K ? 1.f : FMT == KQ_Q5K ? 2.f : 4.f;  // what the fp16 integers were divided by
    // registers: producers, issuers, epilogue.  They draw on the launch's 5 x 96 per warp group
    static constexpr int kRegsP = 88, kRegsI = 64, kRegsE = 120;
    static_assert(2 * kRegsP + kRegsI + 2 * kRegsE == 5 * 96, "register split");
    // shared memory
    static constexpr int kB = kKqN * 512, kOffSums = 2 * kB, kSums = kQ6 ? 0 : kKqN * 32;
    static constexpr int kOffMins = kOffSums + 2 * kSums, kMins = kQ6 ? 0 : 128 * 32;                            // [matrix][2]
    static constexpr int kOffRing = kOffMins + 4 * kMins, kOffMisc = kOffRing + kRing * 8 * kWarpSlot;
};
struct KqMisc {
    unsigned long long b_full[2], b_free[2], dx_full[4], dx_free[4], a_full[2][2], a_free[2][2], acc_full[2], acc_free[2], hdr_free[2][2];
    uint32_t tmem_base, pad[3];
    float dx[4][kKqN];
    uint32_t hdr[2][2][128];      // half2 (d, dmin) of a row's block
};
constexpr int kKqThreads = 640;
template <int FMT>
constexpr int kq_smem() { return KqCfg<FMT>::kOffMisc + (int)sizeof(KqMisc) + 1024; }
static_assert(kq_smem<KQ_Q4K>() <= 232448 && kq_smem<KQ_Q5K>() <= 232448 && kq_smem<KQ_Q6K_T4>() <= 232448, "shared memory budget");

struct KqParams {
    const uint8_t* w[2];
    long expert_bytes, dpitch;
    int pair, R, nblk, T, rt, nt, splits, total, tiles_mul, hidden_type, t0;
    const float* dx;
    const int4* tinfo;
    const int* n_tiles;
    float* out[2];
    void* y;
    const float* bias;
    const int* bsz;
};

// where element e of a 256-block sits among the fp16 activations: the order in which the producers unpack the weights
__device__ __forceinline__ int kq_pos4(int e0, bool q6) {      // first of the places of e0 .. e0 + 3 (e0 a multiple of 4), themselves in the order 0, 2, 1, 3
    const int j = (e0 & 31) >> 2;
    if (q6) return 64 * (2 * (e0 >> 7) + ((e0 >> 5) & 1)) + 8 * j + 4 * ((e0 >> 6) & 1);
    return 64 * (e0 >> 6) + 8 * j + 4 * ((e0 >> 5) & 1);
}

__device__ __forceinline__ void kq_cp16(uint32_t dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void kq_cp4(uint32_t dst, const void* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void kq_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void kq_cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
template <int N>
__device__ __forceinline__ void regs_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void regs_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
__device__ __forceinline__ void kq_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// D[tmem] (+)= A[tmem] . B[smem], fp16: A's lane = row, a 32-bit column = two consecutive K; K = 16 per instruction.  Eight of them on consecutive
// 8-column slices of A, against the four 32-byte steps of a 64-wide B tile and of the tile `next` (in descriptor units) behind it.  One election.
__device__ __forceinline__ void mma_f16_ta8(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint64_t next, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p, q, t;\n"
        ".reg .b32 r, a;\n"
        ".reg .b64 b;\n"
        "elect.sync r|q, 0xffffffff;\n"
        "setp.ne.b32 p, %5, 0;\n"
        "setp.eq.b32 t, 0, 0;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %4, p;\n"
        "add.u32 a, %1, 8;\n"
        "add.u64 b, %2, 2;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %4, t;\n"
        "add.u32 a, %1, 16;\n"
        "add.u64 b, %2, 4;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %4, t;\n"
        "add.u32 a, %1, 24;\n"
        "add.u64 b, %2, 6;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %4, t;\n"
        "add.u32 a, %1, 32;\n"
        "add.u64 b, %2, %3;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %4, t;\n"
        "add.u32 a, %1, 40;\n"
        "add.u64 b, b, 2;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %4, t;\n"
        "add.u32 a, %1, 48;\n"
        "add.u64 b, b, 2;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %4, t;\n"
        "add.u32 a, %1, 56;\n"
        "add.u64 b, b, 2;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %4, t;\n"
        "}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(desc_b), "l"(next), "r"(idesc), "r"(accumulate)
        : "memory");
}
// bar_wait (umma.cuh) with a long suspension per poll: 18 warps that poll at the default rate take a third of the issue slots
__device__ __forceinline__ bool kq_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t it = 0; it < (1u << 19); it++) {
        uint32_t done;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    atomicAdd(&g_bar_wait_gave_up, 1u);
    return false;
}

__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }
constexpr uint32_t kMagic = 0x64006400u;      // fp16 1024, 1024: a small integer or-ed into the mantissa adds itself
// (a & mask) | 1024, 1024 in one instruction (both constants in registers)
template <uint32_t MASK>
__device__ __forceinline__ __half2 magic_and(uint32_t a) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(MASK), "r"(kMagic));
    return as_h2(d);
}
// packed fp32: two products or fused multiply-adds per instruction, each rounded as the scalar one
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ f32x2 pack2(uint32_t lo, uint32_t hi) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float half_of(f32x2 v, int hi) { return __uint_as_float((uint32_t)(hi ? v >> 32 : v)); }
__device__ __forceinline__ __half2 h2_of(int small) { return __hsub2(as_h2(kMagic | (uint32_t)small * 0x10001u), as_h2(kMagic)); }      // 0 <= small < 1024

// the 6-bit scales and minima of a Q4_K / Q5_K header (words 1-3 of the block) as bytes: sub-blocks 0-3 | 4-7 (get_scale_min_k4)
struct KqScales { uint32_t sc[2], mn[2]; };
__device__ __forceinline__ KqScales kq_scales(uint32_t w0, uint32_t w1, uint32_t w2) {
    KqScales k;
    k.sc[0] = w0 & 0x3f3f3f3fu;
    k.mn[0] = w1 & 0x3f3f3f3fu;
    k.sc[1] = (w2 & 0x0f0f0f0fu) | ((w0 >> 2) & 0x30303030u);
    k.mn[1] = ((w2 >> 4) & 0x0f0f0f0fu) | ((w1 >> 2) & 0x30303030u);
    return k;
}
__device__ __forceinline__ int byte_of(uint32_t w, int i) { return (int)((w >> (8 * i)) & 0xffu); }

struct KqTile { int e, row0, p0, n, sb0, nsb, split; };
__device__ __forceinline__ KqTile kq_tile(const KqParams& p, int tile) {
    KqTile t;
    if (p.tinfo) {
        const int4 i = __ldg(p.tinfo + tile);
        t.e = i.x; t.row0 = i.y; t.p0 = i.z; t.n = i.w; t.sb0 = 0; t.nsb = p.nblk; t.split = 0;
    } else {      // token tile fastest: the CTAs of a wave share the weight rows through L2
        const int nt = tile % p.nt, r = tile / p.nt;
        t.e = 0; t.row0 = (r % p.rt) * kKqRows; t.split = r / p.rt;
        t.p0 = nt * kKqN; t.n = min(kKqN, p.T - t.p0);
        t.sb0 = (int)((long)p.nblk * t.split / p.splits);
        t.nsb = (int)((long)p.nblk * (t.split + 1) / p.splits) - t.sb0;
    }
    return t;
}

// 32 columns (64 weights of a row) of an operand stage from 8 words of quants; sl / sh: scales of the low / high nibbles' values
__device__ __forceinline__ void kq_unpack4(const uint32_t (&w)[8], __half2 sl, __half2 sh, uint32_t (&o)[32]) {
    const __half2 cl = __hmul2(sl, __float2half2_rn(-1024.f)), s16 = __hmul2(sh, __float2half2_rn(1.f / 16.f)), ch = __hmul2(sh, __float2half2_rn(-64.f));
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const uint32_t a = w[j], b = a >> 8;
        o[4 * j] = as_u32(__hfma2(magic_and<0x000f000fu>(a), sl, cl));
        o[4 * j + 1] = as_u32(__hfma2(magic_and<0x000f000fu>(b), sl, cl));
        o[4 * j + 2] = as_u32(__hfma2(magic_and<0x00f000f0u>(a), s16, ch));
        o[4 * j + 3] = as_u32(__hfma2(magic_and<0x00f000f0u>(b), s16, ch));
    }
}
// Q5_K, halved: the fifth bits are bits 0 (low nibbles) and 1 (high nibbles) of the bytes of t
__device__ __forceinline__ void kq_unpack5(const uint32_t (&w)[8], const uint32_t (&q)[8], int shift, __half2 sl, __half2 sh, uint32_t (&o)[32]) {
    const __half2 s2 = __hmul2(sl, __float2half2_rn(0.5f)), cl = __hmul2(sl, __float2half2_rn(-512.f)), s32 = __hmul2(sh, __float2half2_rn(1.f / 32.f)), ch = __hmul2(sh, __float2half2_rn(-32.f));
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const uint32_t a = w[j], b = a >> 8, t = q[j] >> shift;
        o[4 * j] = as_u32(__hfma2(as_h2((a & 0x000f000fu) | ((t << 4) & 0x00100010u) | kMagic), s2, cl));
        o[4 * j + 1] = as_u32(__hfma2(as_h2((b & 0x000f000fu) | ((t >> 4) & 0x00100010u) | kMagic), s2, cl));
        o[4 * j + 2] = as_u32(__hfma2(as_h2((a & 0x00f000f0u) | ((t << 7) & 0x01000100u) | kMagic), s32, ch));
        o[4 * j + 3] = as_u32(__hfma2(as_h2((b & 0x00f000f0u) | ((t >> 1) & 0x01000100u) | kMagic), s32, ch));
    }
}
__device__ __forceinline__ void kq_words8(const uint8_t* src, uint32_t (&w)[8]) {
    const uint4 a = reinterpret_cast<const uint4*>(src)[0], b = reinterpret_cast<const uint4*>(src)[1];
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
}

template <int FMT>
__global__ void __launch_bounds__(kKqThreads, 1) kq_gemm_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap smap, const KqParams p) {
    using C = KqCfg<FMT>;
    constexpr bool Q6 = C::kQ6;
    constexpr int kAccCols = Q6 ? kKqN : 2 * kKqN, kColA = 2 * kAccCols;      // per matrix: accumulator (and minima); then the operand stages
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    KqMisc& misc = *reinterpret_cast<KqMisc*>(smem + C::kOffMisc);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int i = 0; i < 2; i++) {
            bar_init(smem_u32(&misc.b_full[i]), 1); bar_init(smem_u32(&misc.b_free[i]), 2);
            bar_init(smem_u32(&misc.acc_full[i]), 1); bar_init(smem_u32(&misc.acc_free[i]), 4);
            for (int j = 0; j < 2; j++) { bar_init(smem_u32(&misc.a_full[i][j]), 4); bar_init(smem_u32(&misc.a_free[i][j]), 1); bar_init(smem_u32(&misc.hdr_free[i][j]), 4); }
        }
        for (int i = 0; i < 4; i++) { bar_init(smem_u32(&misc.dx_full[i]), 1); bar_init(smem_u32(&misc.dx_free[i]), 8); }
        bar_fence_init();
        tma_prefetch_desc(&qmap);
        if (!Q6) tma_prefetch_desc(&smap);
    }
    if (warp == 9) tmem_alloc(smem_u32(&misc.tmem_base), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = misc.tmem_base;
    const int total = p.n_tiles ? *p.n_tiles * p.tiles_mul : p.total;

    if (warp < 8) {
        // ========================================================================== producers
        regs_down<C::kRegsP>();
        const int mat = warp >> 2, r = tid & 127;                  // weight row of the tile's matrix = TMEM lane
        const uint32_t ring = base + C::kOffRing + warp * C::kWarpSlot;
        const uint8_t* ring_p = smem + C::kOffRing + warp * C::kWarpSlot;
        constexpr int kSlot = 8 * C::kWarpSlot;
        // fetch cursor, kRing blocks ahead of the conversion and across tile boundaries
        int ftile = blockIdx.x, fs = 0, fn = 0, fslot = 0, fblk = 0;
        const uint8_t* fbase = nullptr;
        int frow = 0;                                              // warp's first row (matrix coordinates)
        auto enter = [&]() {
            if (ftile >= total) return;
            const KqTile t = kq_tile(p, ftile);
            fbase = p.w[p.pair ? mat : 0] + (long)t.e * p.expert_bytes;
            frow = t.row0 + (p.pair ? 0 : 128 * mat) + 32 * (warp & 3);
            fs = 0; fn = t.nsb; fblk = t.sb0;
        };
        auto fetch = [&]() {
            if (ftile < total) {
                const uint32_t dst = ring + fslot * kSlot;
                const int last = p.R - 1;                          // rows beyond the matrix read its last row and are never stored
                if (!Q6) {
                    constexpr int kCh = C::kRow / 16, kDr = 32 / kCh, kDp = 32 - kDr * kCh;
                    int rr = lane / kCh, part = lane - rr * kCh;
#pragma unroll 3
                    for (int i = 0; i < kCh; i++) {                // 16-byte words of the warp's 32 blocks, a row's words on consecutive lanes
                        kq_cp16(dst + (i * 32 + lane) * 16, fbase + ((uint32_t)(min(frow + rr, last) * p.nblk + fblk) * (unsigned long long)C::kRow + part * 16));
                        rr += kDr; part += kDp;
                        if (part >= kCh) { part -= kCh; rr++; }
                    }
                } else if (FMT == KQ_Q6K_T4) {                     // 4-row items of 16-byte planes (repack_q6k4t): a lane fetches its row's 13 words
                    const int row = min(frow + lane, last), f = (row & 3) * p.nblk + fblk, plane = 4 * p.nblk * 16;
                    const uint8_t* item = fbase + (long)(row >> 2) * 4 * p.nblk * SZ_Q6_K;
                    const uint8_t* src = item + f * 16;
#pragma unroll 4
                    for (int c = 0; c < 13; c++, src += plane) kq_cp16(dst + lane * C::kRow + c * 16, src);
                    kq_cp4(dst + 32 * C::kRow + lane * 4, item + 13L * plane + (f >> 1) * 4);
                } else {                                           // 8-row groups of ql | qh | scales | d (repack_q6k)
                    auto group = [&](int row) { return fbase + (long)(row >> 3) * 8 * p.nblk * SZ_Q6_K; };
                    auto at = [&](int row) { return (row & 7) * p.nblk + fblk; };
#pragma unroll 2
                    for (int i = 0; i < 8; i++) {
                        const int rr = 4 * i + (lane >> 3), c = lane & 7, row = min(frow + rr, last);
                        kq_cp16(dst + rr * C::kRow + c * 16, group(row) + at(row) * 128 + c * 16);
                    }
#pragma unroll 2
                    for (int i = 0; i < 4; i++) {
                        const int rr = 8 * i + (lane >> 2), c = lane & 3, row = min(frow + rr, last);
                        kq_cp16(dst + rr * C::kRow + 128 + c * 16, group(row) + 1024 * p.nblk + at(row) * 64 + c * 16);
                    }
                    const int row = min(frow + lane, last);
                    kq_cp16(dst + lane * C::kRow + 192, group(row) + 1536 * p.nblk + at(row) * 16);
                    kq_cp4(dst + 32 * C::kRow + lane * 4, group(row) + 1664 * p.nblk + (at(row) >> 1) * 4);
                }
                fslot = fslot == C::kRing - 1 ? 0 : fslot + 1;
                fblk++;
                if (++fs == fn) { ftile += gridDim.x; enter(); }
            }
            kq_cp_commit();
        };
        enter();
        for (int i = 0; i < C::kRing; i++) fetch();
        int slot = 0;
        unsigned it = 0, stage = 0;      // blocks and operand stages so far
        for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
            const KqTile t = kq_tile(p, tile);
            const int row = min(t.row0 + (p.pair ? 0 : 128 * mat) + r, p.R - 1);
            for (int s = 0; s < t.nsb; s++, it++) {
                kq_cp_wait<C::kRing - 1>();
                __syncwarp();
                const uint8_t* src = ring_p + slot * kSlot + lane * C::kRow;
                kq_wait(smem_u32(&misc.hdr_free[mat][it & 1]), ((it >> 1) & 1) ^ 1);
                KqScales k{};
                uint32_t qh[8];
                if (!Q6) {
                    const uint4 head = *reinterpret_cast<const uint4*>(src);
                    k = kq_scales(head.y, head.z, head.w);
                    misc.hdr[mat][it & 1][r] = head.x;
                    // minima, each twice, against the sixteen 16-value activation sums: K-major core matrices of 8 rows x 16 bytes
                    uint8_t* m = smem + C::kOffMins + (mat * 2 + (it & 1)) * C::kMins + (r >> 3) * 256 + (r & 7) * 16;
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        *reinterpret_cast<uint4*>(m + h * 128) = make_uint4(as_u32(h2_of(byte_of(k.mn[h], 0))), as_u32(h2_of(byte_of(k.mn[h], 1))), as_u32(h2_of(byte_of(k.mn[h], 2))),
                                                                            as_u32(h2_of(byte_of(k.mn[h], 3))));
                    fence_async_smem();
                    if (FMT == KQ_Q5K) kq_words8(src + 16, qh);
                } else {
                    const uint32_t tail = *reinterpret_cast<const uint32_t*>(ring_p + slot * kSlot + 32 * C::kRow + lane * 4);
                    const int f = FMT == KQ_Q6K_T4 ? (row & 3) * p.nblk + t.sb0 + s : (row & 7) * p.nblk + t.sb0 + s;
                    misc.hdr[mat][it & 1][r] = (f & 1) ? tail >> 16 : tail & 0xffffu;
                }
                // (rolled: four roles of fully unrolled code overran the instruction cache, 10,000 cycles a block where this takes less than 2,000)
#pragma unroll 1
                for (int h = 0; h < C::kStages; h++, stage++) {
                    kq_wait(smem_u32(&misc.a_free[mat][stage & 1]), ((stage >> 1) & 1) ^ 1);
                    tc_fence_after();
                    const uint32_t dst = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + kColA + (mat * 2 + (stage & 1)) * 64;
                    uint32_t w[8], o[32];
                    if (!Q6) {      // chunk c = 2h + part: low nibbles are sub-block 2c, high nibbles sub-block 2c + 1
#pragma unroll 1
                        for (int part = 0; part < 2; part++) {
                            const uint32_t sc = (h ? k.sc[1] : k.sc[0]) >> (16 * part);
                            kq_words8(src + C::kRow - 128 + 32 * (2 * h + part), w);
                            if (FMT == KQ_Q4K) kq_unpack4(w, h2_of(sc & 0xff), h2_of((sc >> 8) & 0xff), o);
                            else kq_unpack5(w, qh, 2 * (2 * h + part), h2_of(sc & 0xff), h2_of((sc >> 8) & 0xff), o);
                            tmem_st32(dst + 32 * part, o);
                        }
                    } else {
                        // quarter (hh, pp) of the block: elements 128 hh + 32 pp + l (ql low nibbles, qh bits 2 pp) and + 64 (high nibbles, bits 4 + 2 pp), l < 32;
                        // first 32 columns sc * low four bits / 4, last 32 columns sc * (16 * high two bits - 32) / 4; a scale per 16 elements
                        const int hh = h >> 1, pp = h & 1;
                        const uint2 sc = *reinterpret_cast<const uint2*>(src + 192 + 8 * hh);
                        const __half2 quarter = __float2half2_rn(0.25f);
                        __half2 sl[2], sh[2];
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            sl[i] = __hmul2(__half2half2(__int2half_rn((int)(int8_t)((sc.x >> (16 * pp + 8 * i)) & 0xff))), quarter);
                            sh[i] = __hmul2(__half2half2(__int2half_rn((int)(int8_t)((sc.y >> (16 * pp + 8 * i)) & 0xff))), quarter);
                        }
                        kq_words8(src + 32 * h, w);
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            const __half2 cl = __hmul2(sl[i], __float2half2_rn(-1024.f)), s16 = __hmul2(sh[i], __float2half2_rn(1.f / 16.f)), ch = __hmul2(sh[i], __float2half2_rn(-64.f));
#pragma unroll
                            for (int j = 4 * i; j < 4 * i + 4; j++) {
                                const uint32_t a = w[j], b = a >> 8;
                                o[4 * j] = as_u32(__hfma2(magic_and<0x000f000fu>(a), sl[i], cl));
                                o[4 * j + 1] = as_u32(__hfma2(magic_and<0x000f000fu>(b), sl[i], cl));
                                o[4 * j + 2] = as_u32(__hfma2(magic_and<0x00f000f0u>(a), s16, ch));
                                o[4 * j + 3] = as_u32(__hfma2(magic_and<0x00f000f0u>(b), s16, ch));
                            }
                        }
                        tmem_st32(dst, o);
                        kq_words8(src + 128 + 32 * hh, w);
                        const __half2 m = as_h2(0x64206420u);      // 1024 + 32
                        const int up = 4 - 2 * pp, down = 2 * pp;   // the two bits moved to bits 4 and 5 of their byte
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            const uint32_t lo = w[j] << up, hi = w[j] >> down;
                            o[4 * j] = as_u32(__hmul2(__hsub2(magic_and<0x00300030u>(lo), m), sl[j >> 2]));
                            o[4 * j + 1] = as_u32(__hmul2(__hsub2(magic_and<0x00300030u>(lo >> 8), m), sl[j >> 2]));
                            o[4 * j + 2] = as_u32(__hmul2(__hsub2(magic_and<0x00300030u>(hi), m), sh[j >> 2]));
                            o[4 * j + 3] = as_u32(__hmul2(__hsub2(magic_and<0x00300030u>(hi >> 8), m), sh[j >> 2]));
                        }
                        tmem_st32(dst + 32, o);
                    }
                    tmem_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) bar_arrive(smem_u32(&misc.a_full[mat][stage & 1]));
                }
                fetch();                                           // refills the slot just read (every lane is past its reads: the __syncwarp above)
                slot = slot == C::kRing - 1 ? 0 : slot + 1;
            }
        }
        kq_cp_wait<0>();
    } else if (warp < 12) {
        regs_down<C::kRegsI>();
        if (warp == 8) {
            // ====================================================================== activations
            if (lane == 0) {
                unsigned it = 0;
                for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
                    const KqTile t = kq_tile(p, tile);
                    const int groups = (t.n + 31) >> 5;
                    for (int s = 0; s < t.nsb; s++, it++) {
                        const int b = it & 1, sb = t.sb0 + s;
                        kq_wait(smem_u32(&misc.b_free[b]), ((it >> 1) & 1) ^ 1);
                        const uint32_t full = smem_u32(&misc.b_full[b]);
                        bar_expect_tx(full, groups * 32 * (Q6 ? 512 : 544));
                        for (int g = 0; g < groups; g++) {
#pragma unroll
                            for (int c = 0; c < 4; c++) tma_load_2d(base + b * C::kB + c * (kKqN * 128) + g * 4096, &qmap, full, sb * 256 + c * 64, t.p0 + 32 * g);
                            if (!Q6) tma_load_2d(base + C::kOffSums + b * C::kSums + g * 1024, &smap, full, sb * 16, t.p0 + 32 * g);
                        }
                        const int d = it & 3;
                        kq_wait(smem_u32(&misc.dx_free[d]), ((it >> 2) & 1) ^ 1);
                        bar_expect_tx(smem_u32(&misc.dx_full[d]), kKqN * 4);
                        kq_bulk(smem_u32(&misc.dx[d][0]), p.dx + (long)sb * p.dpitch + t.p0, kKqN * 4, smem_u32(&misc.dx_full[d]));
                    }
                }
            }
            __syncwarp();
        } else if (warp < 11) {
            // ====================================================================== tensor-core issuers (converged warps), one per matrix
            const int mat = warp - 9;
            const uint32_t acc = tmem + mat * kAccCols, a0 = tmem + kColA + mat * 128;
            unsigned it = 0, stage = 0;
            for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
                const KqTile t = kq_tile(p, tile);
                const uint32_t idesc = instr_desc(1, 0, 0, 0, 0, 128, (t.n + 15) & ~15);      // f32 += f16 . f16
                for (int s = 0; s < t.nsb; s++, it++) {
                    const int b = it & 1;
                    kq_wait(smem_u32(&misc.b_full[b]), (it >> 1) & 1);
                    kq_wait(smem_u32(&misc.acc_free[mat]), (it & 1) ^ 1);
                    uint64_t bd = smem_desc(base + b * C::kB, 16, 1024, kLayoutSw128);
#pragma unroll 1
                    for (int h = 0; h < C::kStages; h++, stage++) {
                        kq_wait(smem_u32(&misc.a_full[mat][stage & 1]), (stage >> 1) & 1);
                        tc_fence_after();
                        // (the address field of a descriptor counts 16 bytes, and nothing carries out of it)
                        mma_f16_ta8(acc, a0 + (stage & 1) * 64, bd, Q6 ? 0 : kKqN * 128 >> 4, idesc, h);      // Q6_K: both terms of the quarter's 64 weights
                        bd += (Q6 ? 1 : 2) * (kKqN * 128 >> 4);
                        if (!Q6 && h == 0)
                            mma_f16(acc + kKqN, smem_desc(base + C::kOffMins + (mat * 2 + b) * C::kMins, 128, 256, kLayoutNone),
                                    smem_desc(base + C::kOffSums + b * C::kSums, 16, 256, kLayoutSw32), idesc, 0);
                        mma_commit(smem_u32(&misc.a_free[mat][stage & 1]));
                    }
                    mma_commit(smem_u32(&misc.acc_full[mat]));
                    mma_commit(smem_u32(&misc.b_free[b]));
                }
            }
        }
    } else {
        // ========================================================================== epilogue: a thread owns one weight row and the tile's tokens
        regs_up<C::kRegsE>();
        const int mat = (warp - 12) >> 2, sp = warp & 3, r = 32 * sp + lane;
        const uint32_t tacc = tmem + ((uint32_t)(32 * sp) << 16) + mat * kAccCols;
        unsigned it = 0;
        for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
            const KqTile t = kq_tile(p, tile);
            f32x2 acc[kKqN / 2];
#pragma unroll
            for (int n = 0; n < kKqN / 2; n++) acc[n] = 0;
            for (int s = 0; s < t.nsb; s++, it++) {
                kq_wait(smem_u32(&misc.dx_full[it & 3]), (it >> 2) & 1);
                kq_wait(smem_u32(&misc.acc_full[mat]), it & 1);
                tc_fence_after();
                const __half2 dm = as_h2(misc.hdr[mat][it & 1][r]);
                const float dw = __low2float(dm) * C::kScale, dmin = -__high2float(dm);
                const f32x2 dw2 = pack2(dw, dw), dmin2 = pack2(dmin, dmin);
                const ulonglong2* dx = reinterpret_cast<const ulonglong2*>(misc.dx[it & 3]);
#pragma unroll
                for (int c = 0; c < kKqN / 16; c++) {
                    if (16 * c < t.n) {
                        uint32_t v[16], m[16];
                        tmem_ld16(tacc + 16 * c, v);
                        if (!Q6) tmem_ld16(tacc + kKqN + 16 * c, m);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const ulonglong2 x = dx[4 * c + i];
#pragma unroll
                            for (int u = 0; u < 2; u++) {
                                f32x2 q = mul2(dw2, pack2(v[4 * i + 2 * u], v[4 * i + 2 * u + 1]));
                                if (!Q6) q = fma2(dmin2, pack2(m[4 * i + 2 * u], m[4 * i + 2 * u + 1]), q);
                                f32x2& a = acc[8 * c + 2 * i + u];
                                a = fma2(u ? x.y : x.x, q, a);
                            }
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    bar_arrive(smem_u32(&misc.acc_free[mat]));
                    bar_arrive(smem_u32(&misc.hdr_free[mat][it & 1]));
                    bar_arrive(smem_u32(&misc.dx_free[it & 3]));
                }
            }
            const int row = t.row0 + (p.pair ? 0 : 128 * mat) + r;
            if (row < p.R) {
                if (p.y) {
                    const float b = p.bias ? p.bias[row] : 0.f;
                    const int n = p.bsz ? min(t.n, *p.bsz - p.t0 - t.p0) : t.n;
                    const long at = (long)t.p0 * p.R + row;
                    auto put = [&](int type) {
#pragma unroll
                        for (int i = 0; i < kKqN; i++)
                            if (i < n) store_hidden(p.y, at + (long)i * p.R, type, half_of(acc[i >> 1], i & 1) + b);
                    };
                    if (p.hidden_type == KTB200_TYPE_BF16) put(KTB200_TYPE_BF16);
                    else if (p.hidden_type == KTB200_TYPE_F16) put(KTB200_TYPE_F16);
                    else put(KTB200_TYPE_F32);
                } else {
                    float* out = p.out[mat] + ((long)t.split * p.T + t.p0) * p.R + row;
#pragma unroll
                    for (int i = 0; i < kKqN; i++)
                        if (i < t.n) out[(long)i * p.R] = half_of(acc[i >> 1], i & 1);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// ---------------------------------------------------------------------------------------------------------------- activations
__device__ __forceinline__ void kq_store_block(const KqActs& a, long row, int b, int K, int lane, bool q6, uint32_t w0, uint32_t w1, float d, int s2) {
    const uint32_t w[2] = {w0, w1};
#pragma unroll
    for (int h = 0; h < 2; h++) {
        __half v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = __int2half_rn((int)(int8_t)byte_of(w[h], i));
        *reinterpret_cast<uint2*>(a.q + row * K + b * QK_K + kq_pos4(8 * lane + 4 * h, q6)) =
            make_uint2(as_u32(__halves2half2(v[0], v[2])), as_u32(__halves2half2(v[1], v[3])));
    }
    if (!q6 && (lane & 1) == 0) a.sums[row * (K / 16) + b * 16 + (lane >> 1)] = __int2half_rn((int)(int16_t)s2);
    if (lane == 0) a.d[(long)b * a.pitch + row] = d;
}
// one warp per (token, 256-block): quantised once, stored for every row the token has
__global__ void __launch_bounds__(256) kq_quant_kernel(const void* x, int hidden_type, int T, int K, const int* pos, int k, int q6, const KqActs a) {
    const int lane = threadIdx.x & 31, nblk = K / QK_K;
    const long gw = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (gw >= (long)T * nblk) return;
    const int t = (int)(gw / nblk), b = (int)(gw - (long)t * nblk);
    float v[8], d;
    uint32_t w0, w1;
    int s;
    load_block8(x, (long)t * K + (long)b * QK_K + lane * 8, hidden_type, v);
    warp_q8k_words(v, w0, w1, d, s);
    const int s2 = s + __shfl_xor_sync(0xffffffffu, s, 1);
    if (!pos) kq_store_block(a, t, b, K, lane, q6, w0, w1, d, s2);
    else
        for (int j = 0; j < k; j++) {
            const int row = pos[t * k + j];
            if (row >= 0) kq_store_block(a, row, b, K, lane, q6, w0, w1, d, s2);
        }
}
__global__ void __launch_bounds__(256) kq_act_quant_kernel(const float* g, const float* u, const int* pos, int n, int K, int use_silu, int q6, const KqActs a) {
    const int lane = threadIdx.x & 31, nblk = K / QK_K;
    const long gw = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (gw >= (long)n * nblk) return;
    const int i = (int)(gw / nblk), b = (int)(gw - (long)i * nblk), row = pos[i];
    if (row < 0) return;
    const long o = (long)row * K + (long)b * QK_K + lane * 8;
    const float4 g0 = *reinterpret_cast<const float4*>(g + o), g1 = *reinterpret_cast<const float4*>(g + o + 4);
    const float4 u0 = *reinterpret_cast<const float4*>(u + o), u1 = *reinterpret_cast<const float4*>(u + o + 4);
    const float gv[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w}, uv[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
    float v[8], d;
    uint32_t w0, w1;
    int s;
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = (use_silu ? act_silu(gv[j]) : act_relu(gv[j])) * uv[j];
    warp_q8k_words(v, w0, w1, d, s);
    const int s2 = s + __shfl_xor_sync(0xffffffffu, s, 1);
    kq_store_block(a, row, b, K, lane, q6, w0, w1, d, s2);
}
// y = sum of the K parts + bias, in the hidden type
__global__ void __launch_bounds__(256) kq_finish_kernel(const float* part, int splits, int T, int R, void* y, int hidden_type, const float* bias, const int* bsz, int t0) {
    const long i = (long)blockIdx.x * 256 + threadIdx.x, n = (long)(bsz ? max(0, min(T, *bsz - t0)) : T) * R;
    if (i >= n) return;
    float v = part[i];
    for (int s = 1; s < splits; s++) v += part[(long)s * T * R + i];
    if (bias) v += bias[i % R];
    store_hidden(y, i, hidden_type, v);
}

int kq_quant(const void* x, int hidden_type, int T, int K, const int* pos, int k, bool q6, const KqActs& a, cudaStream_t s) {
    kq_quant_kernel<<<(unsigned)(((long)T * (K / QK_K) + 7) / 8), 256, 0, s>>>(x, hidden_type, T, K, pos, k, q6, a);
    KTB_LAUNCH_CHECK();
    return KTB200_OK;
}
int kq_act_quant(const float* g, const float* u, const int* pos, int n, int K, int use_silu, bool q6, const KqActs& a, cudaStream_t s) {
    kq_act_quant_kernel<<<(unsigned)(((long)n * (K / QK_K) + 7) / 8), 256, 0, s>>>(g, u, pos, n, K, use_silu, q6, a);
    KTB_LAUNCH_CHECK();
    return KTB200_OK;
}

// ---------------------------------------------------------------------------------------------------------------- launch
typedef CUresult (*EncodeTiledFnKq)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                    CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFnKq encode_tiled_kq() {
    static EncodeTiledFnKq fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
        return (EncodeTiledFnKq)f;
    }();
    return fn;
}
// boxes of 32 rows x `cols` fp16 of a row-major matrix
static int kq_map(CUtensorMap* map, const void* ptr, long width, long rows, int cols, CUtensorMapSwizzle sw) {
    EncodeTiledFnKq enc = encode_tiled_kq();
    if (!enc) { set_error("kq_gemm: cuTensorMapEncodeTiled is not available from this driver"); return KTB200_ECUDA; }
    const cuuint64_t gdim[2] = {(cuuint64_t)width, (cuuint64_t)rows};
    const cuuint64_t gstr[1] = {(cuuint64_t)width * 2};
    const cuuint32_t box[2] = {(cuuint32_t)cols, 32}, estr[2] = {1, 1};
    const CUresult cr = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) { set_error("kq_gemm: cuTensorMapEncodeTiled failed (%d)", (int)cr); return KTB200_ECUDA; }
    return KTB200_OK;
}
template <int FMT>
static int kq_launch(const CUtensorMap& qmap, const CUtensorMap& smap, const KqParams& p, int grid, cudaStream_t s) {
    KTB_CUDA_CHECK(cudaFuncSetAttribute(kq_gemm_kernel<FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kq_smem<FMT>()));
    kq_gemm_kernel<FMT><<<grid, kKqThreads, kq_smem<FMT>(), s>>>(qmap, smap, p);
    KTB_LAUNCH_CHECK();
    return KTB200_OK;
}

int kq_gemm(const KqGemm& g, int device, cudaStream_t s) {
    KqParams p{};
    for (int i = 0; i < 2; i++) { p.w[i] = reinterpret_cast<const uint8_t*>(g.w[i]); p.out[i] = g.out[i]; }
    p.expert_bytes = g.expert_bytes; p.dpitch = g.acts->pitch; p.pair = g.pair; p.R = g.R; p.nblk = g.K / QK_K; p.dx = g.acts->d;
    p.tinfo = g.tinfo; p.n_tiles = g.n_tiles_dev; p.tiles_mul = g.tiles_mul; p.y = g.y; p.hidden_type = g.hidden_type; p.bias = g.bias; p.bsz = g.bsz;
    p.t0 = g.t0; p.T = g.T; p.splits = g.splits; p.rt = (g.R + kKqRows - 1) / kKqRows; p.nt = (g.T + kKqN - 1) / kKqN; p.total = p.rt * p.nt * g.splits;
    CUtensorMap qmap, smap;
    int rc = kq_map(&qmap, g.acts->q, g.K, g.acts->rows, 64, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc == KTB200_OK) rc = kq_map(&smap, g.acts->sums, g.K / 16, g.acts->rows, 16, CU_TENSOR_MAP_SWIZZLE_32B);
    if (rc) return rc;
    const int sms = num_sms(device), grid = g.tinfo || p.total > sms ? sms : p.total;
    switch (g.fmt) {
        case KQ_Q4K: return kq_launch<KQ_Q4K>(qmap, smap, p, grid, s);
        case KQ_Q5K: return kq_launch<KQ_Q5K>(qmap, smap, p, grid, s);
        case KQ_Q6K_T4: return kq_launch<KQ_Q6K_T4>(qmap, smap, p, grid, s);
        case KQ_Q6K_SOA8: return kq_launch<KQ_Q6K_SOA8>(qmap, smap, p, grid, s);
        default: set_error("kq_gemm: unsupported weight type"); return KTB200_EINVAL;
    }
}

int kq_linear(FmtId fmt, const void* w, int R, int K, const void* x, int hidden_type, int T, void* y, const float* bias, const int* bsz, int device, cudaStream_t s) {
    const KqFmt f = kq_fmt(fmt);
    if (f == KQ_NONE || (uintptr_t)w % 16) return 1;
    constexpr int kChunk = 4096;      // rows per pass: bounds the scratch
    const size_t hb = type_size(hidden_type);
    for (int t0 = 0; t0 < T; t0 += kChunk) {
        const int n = T - t0 < kChunk ? T - t0 : kChunk, sms = num_sms(device);
        const int tiles = ((R + kKqRows - 1) / kKqRows) * ((n + kKqN - 1) / kKqN), nblk = K / QK_K;
        // K in parts when the tiles leave SMs idle, two blocks or more each
        int splits = sms / tiles;
        if (splits > nblk / 2) splits = nblk / 2;
        if (splits < 1) splits = 1;
        ScratchBlock mem(s);
        const size_t act = (KqActs::bytes(n, K) + 255) / 256 * 256;
        KTB_CUDA_CHECK(mem.take(device, act + (splits > 1 ? (size_t)splits * n * R * 4 : 0)));
        const KqActs a(mem.ptr, n, K);
        int rc = kq_quant(reinterpret_cast<const uint8_t*>(x) + (size_t)t0 * K * hb, hidden_type, n, K, nullptr, 1, kq_is_q6(f), a, s);
        if (rc) return rc;
        KqGemm g{};
        g.fmt = f; g.w[0] = g.w[1] = w; g.R = R; g.K = K; g.acts = &a; g.T = n; g.splits = splits; g.hidden_type = hidden_type; g.bias = bias; g.t0 = t0;
        void* yc = reinterpret_cast<uint8_t*>(y) + (size_t)t0 * R * hb;
        float* part = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(mem.ptr) + act);
        if (splits == 1) { g.y = yc; g.bsz = bsz; }
        else g.out[0] = g.out[1] = part;
        rc = kq_gemm(g, device, s);
        if (rc) return rc;
        if (splits > 1) {
            kq_finish_kernel<<<(unsigned)(((long)n * R + 255) / 256), 256, 0, s>>>(part, splits, n, R, yc, hidden_type, bias, bsz, t0);
            KTB_LAUNCH_CHECK();
        }
    }
    return KTB200_OK;
}

}  // namespace ktb
