// Prompt-sized products against GGUF K-quant matrices — the per-expert GEMMs of MOE::forward_many (archive/csrc/ktransformers_ext/operators/
// llamafile/moe.cpp:248-365) and the dense linears of a prompt portion (operators/llamafile/linear.cpp:37-70) — on tcgen05 with the weights
// as the tensor-memory operand.
//
// Arithmetic: the reference's dot of a 256-block is an exact integer, sum_j sc_j * sum_i q_ij * x8_ij, scaled in fp32.  Here a weight enters the
// tensor core as the fp16 integer sc * q (Q4_K: at most 63 * 15; Q5_K: 63 * 31, halved; Q6_K: two terms, sc * (low four bits) and
// sc * (16 * high two bits - 32), both quartered), an activation as the fp16 integer x8; the products are exact, and the epilogue applies
// dx * (d * isum - dmin * msum) once per block in fp32, the decode kernels' formula; msum (minima x 16-value activation sums) is one K = 16 MMA.
// The fp32 accumulator of a 256-block holds integers (or halves, quarters), exact while they stay within 2^24 of their unit.  A full block can reach 31, 63 and
// 133 million (Q4_K, Q5_K, Q6_K), and an ordinary Q5_K block under activations of one sign and size 20 million, of which the minima then take most away again.  So a block
// of activations that might get there (kq_limit in kq_gemm.cuh, marked by the quantiser) is summed stage by stage: each stage's 128 values (Q6_K: 64), at most
// 16 (Q4_K), 32 (Q5_K) or 33 million, go to columns of their own and the epilogue adds them to the accumulator, which then holds isum rounded once, like an int32 sum.
// A tile's other rows come out the same bits either way.  Measured against 64 bits (fp32 linears, K = 7168, 2-norm of 64 x 1024): activations 1 + 0.01 n on Q5_K
// 24.8e-7 with one accumulator, 7.0e-7 like this, 7.6e-7 in the row kernels (int32); all weights and activations at their largest Q4_K 2.5e-7, 0.3e-7, 0.4e-7, Q5_K 4.8e-7,
// 1.3e-7 (a stage's sum may pass 2^24 by one bit), 0.3e-7, Q6_K 7.7e-7, 0.3e-7, 0.3e-7.
//
// What bounds it: an expert's weights are read from HBM once per 64 of its tokens (1024 tokens of 256 experts: about once), so the routed
// experts are HBM-bound, and the work per weight has to stay under what an SM has per weight byte that arrives (24 B per cycle):
//   * the weights go registers -> tensor memory (tcgen05.st, a thread = a weight row = a lane) and never to shared memory as operands.  Through
//     shared memory, 2 B per weight written and 2 B read by the MMA would take 128 B per cycle to 21 weights per cycle, half of what HBM brings;
//     and an MMA of 128 x 64 x 16 runs in 32 cycles with A in tensor memory against 48 with A in shared memory (measured; N = 32: 17 and 40).
//   * nibbles become fp16 by or-ing them into the mantissa of 1024 and one fused multiply-add with (sc, -1024 sc), Q6_K's upper two bits into that of 4 or 16
//     (fewer shifts, and the offset is a product of 11 bits): 9 and 11 instructions for 8
//     weights.  The pairs come out as (0, 2), (1, 3) of four; the activations are stored in that order (kq_pos4).
//   * a scale per 256-block needs the accumulator drained per 256-block: two matrices of 128 rows per CTA (gate and up of the same experts, or
//     256 rows of one) take turns, one drained while the other multiplies, and share the activation tiles.
// CTA: 28 warps in 7 groups of 4.  Groups 0-3 producers: (matrix 0, first operand stage), (matrix 1, first), (0, second), (1, second), a warp = 32 rows, a stage in
//      two parts of 32 columns that are filled, multiplied and given back by themselves (whole stages: 129 us for the linear below, 2,640 for the experts):
//      raw blocks from a TMA ring -> registers -> TMEM; warp 16 TMA of activations, 17 / 18 MMA issuers of matrix 0 / 1, 19 TMA of weights;
//      groups 5 / 6 epilogue of matrix 0 / 1.  With many tokens (kTwoSets) an epilogue of two groups a matrix, half of the tokens each, beside two groups of producers: an
//      accumulator's drain is one thread's chain of loads and sums, and with 64 tokens the next product waits for it.  One warp of a group polls a barrier and the others wait in a hardware barrier behind it: polling
//      warps took a third of the issue slots, and the four roles' code is kept in rolled loops: unrolled it overran the instruction cache (10,000
//      cycles for a block of two matrices).  The warp's number and what the tiles say come through a shuffle, so that the compiler knows them to be the same in all
//      lanes and keeps a role's state, its branches and the MMAs' operands off the vector pipes (the other roles' share of the issue slots is what an issuer or
//      an epilogue warp waits for: 157 -> 129 us for the linear below, 2,782 -> 2,600 for the experts; 268 -> 69 branch instructions a block).
//      A block of two matrices takes 3,100 cycles at 64 tokens a tile (3,440 before), 1,890 at 16 (2,480; Q6_K 3,570, 4,120); HBM brings one every 1,550 (Q6_K 2,270).  Of the 3,100 the drain of an accumulator is
//      1,500 (producers issue beside it; 660 alone), the eight MMAs of either stage 600, the rest hand-overs.  Draining in two halves of the tokens, so that one is multiplied
//      while the other is drained, was slower (140 us, 2,770), and so were both matrices' drains in one thread (244) and other orders of the roles (165).
//      At 16 tokens the schedulers issue three instructions of four possible ones a cycle, nearly all of them the producers'; their share of polls and address arithmetic is small
//      (every producer warp polling for itself, barrier addresses in registers: within 1 %).
//      Measured, DeepSeek-V3 sizes: routed experts of 1024 tokens 2,910 -> 2,540 us (the operator's call); Q4_K linear 777 x 1536 -> 24576 180 -> 126 us, with two epilogue groups a matrix 112 (520 TFLOP/s).
//      Tried beside it: nibbles as e4m3 operands against two e4m3 digits of the activations, exact too and 3 instructions for 8 weights, but eight sums a block to be scaled instead of
//      one (207 us, experts 3,530); 8 epilogue threads' worth of registers so that all columns are loaded before they are scaled (125, 2,660); the headers in warps of their own (123, 2,630).
// TMEM: [accumulator | minima] x 2 matrices, then 64-column operand stages, 2 per matrix.
#include <algorithm>
#include <atomic>
#include <climits>

#include <cuda_fp16.h>

#include "act_quant.cuh"
#include "kq_gemm.cuh"
#include "umma.cuh"

namespace ktb {

using namespace umma;

template <int FMT>
struct KqCfg {
    static constexpr bool kQ6 = FMT == KQ_Q6K_T4 || FMT == KQ_Q6K_SOA8;
    static constexpr int kRow = FMT == KQ_Q4K ? 144 : FMT == KQ_Q5K ? 176 : 208;      // bytes of a row's block in a ring slot (Q6_K: without d)
    static constexpr int kStages = kQ6 ? 4 : 2;                                       // operand stages per block
    static constexpr float kScale = FMT == KQ_Q4K ? 1.f : FMT == KQ_Q5K ? 2.f : 4.f;  // what the fp16 integers were divided by
    // shared memory
    static constexpr int kRing = 3, kMat = 128 * kRow, kSlot = 2 * kMat;
    static constexpr int kB = kKqN * 512, kOffRing = 2 * kB, kOffMins = kOffRing + kRing * kSlot, kMins = kQ6 ? 0 : 128 * 32;        // minima: [matrix][2]
    static constexpr int kOffSums = kOffMins + 4 * kMins, kSums = kQ6 ? 0 : kKqN * 32, kOffMisc = kOffSums + 2 * kSums;
};
struct KqMisc {
    unsigned long long b_full[2], b_free[2], dx_full[4], dx_free[4], raw_full[3], raw_free[3], a_full[2][2][2], a_free[2][2][2], acc_full[2], acc_free[2], hdr_free[2][2];
    uint32_t tmem_base, marked[2], pad;      // marked: whether the matrix's block is summed stage by stage
    float dx[4][kKqN];
    uint32_t hdr[2][2][128];      // Q4_K, Q5_K: half2 (d, dmin) of a row's block
};
constexpr int kKqThreads = 896;
// How the 28 warps are dealt: SETS epilogue groups of four warps a matrix, each with its part of the tile's tokens, and 4 / SETS groups of producers
template <int SETS>
struct KqSplit {
    static constexpr int kProd = 16 / SETS, kEpi = kProd + 4;                 // first warps of the issuers and copies (four), and of the epilogue
    static constexpr int kHalves = 2 / SETS, kCols = kKqN / SETS;             // groups that share a matrix's operand stages; tokens of an epilogue thread at most
    // registers: producers, issuers, epilogue.  They draw on the launch's 7 x 72 per warp group
    static constexpr int kRegsP = SETS == 1 ? 48 : 56, kRegsI = SETS == 1 ? 72 : 40, kRegsE = SETS == 1 ? 120 : 88;
    static_assert(4 / SETS * kRegsP + kRegsI + 2 * SETS * kRegsE == 7 * 72, "register split");
};
template <int FMT>
constexpr int kq_smem() { return KqCfg<FMT>::kOffMisc + (int)sizeof(KqMisc) + 1024; }
static_assert(kq_smem<KQ_Q4K>() <= 232448 && kq_smem<KQ_Q5K>() <= 232448 && kq_smem<KQ_Q6K_T4>() <= 232448, "shared memory budget");

struct KqParams {
    const uint8_t* w[2];
    long expert_bytes, dpitch;
    int pair, R, nblk, T, rt, nt, splits, total, tiles_mul, hidden_type, t0;
    const float* dx;
    const uint8_t* marks;
    const unsigned long long* any;
    unsigned long long id;
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

template <int N>
__device__ __forceinline__ void regs_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void regs_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2, int c3, int c4) {
    asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];" ::"r"(dst), "l"(m), "r"(bar), "r"(c0), "r"(c1),
                 "r"(c2), "r"(c3), "r"(c4)
                 : "memory");
}
__device__ __forceinline__ void group_sync(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void kq_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// D[tmem] (+)= A[tmem] . B[smem], fp16: A's lane = row, a 32-bit column = two consecutive K; K = 16 per instruction.  Four of them on consecutive
// 8-column slices of A, against the four 32-byte steps of a 64-wide B tile.  One election.
__device__ __forceinline__ void mma_f16_ta4(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p, q, t;\n"
        ".reg .b32 r, a;\n"
        ".reg .b64 b;\n"
        "elect.sync r|q, 0xffffffff;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "setp.eq.b32 t, 0, 0;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "add.u32 a, %1, 8;\n"
        "add.u64 b, %2, 2;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, t;\n"
        "add.u32 a, %1, 16;\n"
        "add.u64 b, %2, 4;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, t;\n"
        "add.u32 a, %1, 24;\n"
        "add.u64 b, %2, 6;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, t;\n"
        "}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// the elected lane of a converged warp leaves `value` for those who wait for `bar`, and arrives there
__device__ __forceinline__ void kq_tell(uint32_t at, uint32_t value, uint32_t bar) {
    asm volatile(
        "{\n"
        ".reg .pred q;\n"
        ".reg .b32 r;\n"
        "elect.sync r|q, 0xffffffff;\n"
        "@q st.shared.b32 [%0], %1;\n"
        "@q mbarrier.arrive.shared::cta.b64 _, [%2];\n"
        "}\n" ::"r"(at), "r"(value), "r"(bar)
        : "memory");
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
template <uint32_t MASK, uint32_t BASE>
__device__ __forceinline__ __half2 bits_in(uint32_t a) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(MASK), "r"(BASE));
    return as_h2(d);
}
__device__ __forceinline__ __half2 bits_at8(uint32_t a) { return bits_in<0x03000300u, 0x44004400u>(a); }      // 4 + the two bits at 8
__device__ __forceinline__ __half2 bits_at6(uint32_t a) { return bits_in<0x00c000c0u, 0x4c004c00u>(a); }      // 16 + the two bits at 6
__device__ __forceinline__ float half_of(f32x2 v, int hi) { return __uint_as_float((uint32_t)(hi ? v >> 32 : v)); }
// byte I of w, 0 .. 255, in both halves as an fp16 integer less BIAS: one byte permutation puts it into the mantissa of 1024
template <int I, int BIAS = 0>
__device__ __forceinline__ __half2 h2_byte(uint32_t w) {
    return __hsub2(as_h2(__byte_perm(w, kMagic, 0x5050u | I * 0x0101u)), as_h2(kMagic + BIAS * 0x10001u));
}

// the 6-bit scales and minima of a Q4_K / Q5_K header (words 1-3 of the block) as bytes: sub-blocks 0-3 | 4-7 (get_scale_min_k4)
template <int H>      // four scales or minima as bytes: sub-blocks 0-3 (w: word 0 or 1) or 4-7 (top: word 2's low or high nibbles)
__device__ __forceinline__ uint32_t kq_six(uint32_t w, uint32_t top) {
    return H ? (top & 0x0f0f0f0fu) | ((w >> 2) & 0x30303030u) : w & 0x3f3f3f3fu;
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
    t.e = uniform(t.e); t.row0 = uniform(t.row0); t.p0 = uniform(t.p0); t.n = uniform(t.n);
    t.sb0 = uniform(t.sb0); t.nsb = uniform(t.nsb);
    return t;
}

// four rows a lane of the marks of block sb of rows p0 .. p0 + n: not 0 in some lane where the block has to be summed stage by stage
__device__ __forceinline__ uint32_t kq_mark(const KqParams& p, int sb, int p0, int n, int lane) {
    const int left = n - 4 * lane;
    if (left <= 0) return 0;
    const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(p.marks + (long)sb * p.dpitch + p0) + lane);
    return left < 4 ? w & ((1u << (8 * left)) - 1) : w;
}

// 16 columns (32 weights of a row) of an operand stage from 4 words of quants; sl / sh: scales of the low / high nibbles' values
__device__ __forceinline__ void kq_unpack4(const uint32_t* w, __half2 sl, __half2 sh, uint32_t (&o)[16]) {
    const __half2 cl = __hmul2(sl, __float2half2_rn(-1024.f)), s16 = __hmul2(sh, __float2half2_rn(1.f / 16.f)), ch = __hmul2(sh, __float2half2_rn(-64.f));
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const uint32_t a = w[j], b = a >> 8;
        o[4 * j] = as_u32(__hfma2(magic_and<0x000f000fu>(a), sl, cl));
        o[4 * j + 1] = as_u32(__hfma2(magic_and<0x000f000fu>(b), sl, cl));
        o[4 * j + 2] = as_u32(__hfma2(magic_and<0x00f000f0u>(a), s16, ch));
        o[4 * j + 3] = as_u32(__hfma2(magic_and<0x00f000f0u>(b), s16, ch));
    }
}
// Q5_K, halved: the fifth bits are bits 0 (low nibbles) and 1 (high nibbles) of the bytes of t
__device__ __forceinline__ void kq_unpack5(const uint32_t* w, const uint32_t* q, int shift, __half2 sl, __half2 sh, uint32_t (&o)[16]) {
    const __half2 s2 = __hmul2(sl, __float2half2_rn(0.5f)), cl = __hmul2(sl, __float2half2_rn(-512.f)), s32 = __hmul2(sh, __float2half2_rn(1.f / 32.f)), ch = __hmul2(sh, __float2half2_rn(-32.f));
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const uint32_t a = w[j], b = a >> 8, t = q[j] >> shift;
        o[4 * j] = as_u32(__hfma2(as_h2((a & 0x000f000fu) | ((t << 4) & 0x00100010u) | kMagic), s2, cl));
        o[4 * j + 1] = as_u32(__hfma2(as_h2((b & 0x000f000fu) | ((t >> 4) & 0x00100010u) | kMagic), s2, cl));
        o[4 * j + 2] = as_u32(__hfma2(as_h2((a & 0x00f000f0u) | ((t << 7) & 0x01000100u) | kMagic), s32, ch));
        o[4 * j + 3] = as_u32(__hfma2(as_h2((b & 0x00f000f0u) | ((t >> 1) & 0x01000100u) | kMagic), s32, ch));
    }
}
__device__ __forceinline__ void kq_words8(const uint8_t* a, const uint8_t* b, uint32_t (&w)[8]) {
    const uint4 x = *reinterpret_cast<const uint4*>(a), y = *reinterpret_cast<const uint4*>(b);
    w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w; w[4] = y.x; w[5] = y.y; w[6] = y.z; w[7] = y.w;
}
// where 16-byte word c (0-7 ql, 8-11 qh, 12 scales) of row r's Q6_K block sits in a matrix's part of a ring slot
template <int FMT>
__device__ __forceinline__ int kq_q6_word(int r, int c) {
    if (FMT == KQ_Q6K_T4) return (r >> 2) * 832 + c * 64 + (r & 3) * 16;                       // [4-row item][word][row], as it lies in memory
    if (c < 8) return r * 128 + ((c ^ (r & 7)) << 4);                                          // 128-byte swizzle
    if (c < 12) return 128 * 128 + r * 64 + (((c - 8) ^ ((r >> 1) & 3)) << 4);                 // 64-byte swizzle
    return 128 * 192 + r * 16;
}
struct KqMaps { CUtensorMap q, sums, w[2][3]; };      // activations, their sums; weights of matrix 0 / 1 (Q6_K in 8-row groups: ql, qh, scales)

template <int FMT, bool MARKS, int SETS>
__device__ __forceinline__ void kq_roles(const KqMaps& maps, const KqParams& p, uint8_t* smem, KqMisc& misc, uint32_t base, uint32_t tmem, int total) {
    using C = KqCfg<FMT>;
    using S = KqSplit<SETS>;
    constexpr bool Q6 = C::kQ6;
    constexpr int kAccCols = 2 * kKqN, kColA = 2 * kAccCols;      // per matrix: accumulator, minima or the sum of one stage; then the operand stages
    const int tid = threadIdx.x, lane = tid & 31, warp = uniform(tid >> 5);      // (known to be uniform: see above)
    if (warp < S::kProd) {
        // ========================================================================== producers
        regs_down<S::kRegsP>();
        const int mat = (warp >> 2) & 1, half = warp >> 3, r = tid & 127, grp = warp >> 2;      // row of the tile's matrix = TMEM lane; operand stages half, half + kHalves, ...
        const bool leader = (warp & 3) == 0;
        const uint32_t dst0 = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + kColA + mat * 128;
        int slot = 0, sphase = 0;
        unsigned it = 0;       // blocks so far
        for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
            const int nsb = kq_tile(p, tile).nsb;
            for (int s = 0; s < nsb; s++, it++) {
                const uint8_t* src = smem + C::kOffRing + slot * C::kSlot + mat * C::kMat;
                bar_wait(smem_u32(&misc.raw_full[slot]), sphase);
                const uint8_t* const row = src + r * C::kRow;
#pragma unroll 1
                for (int h = half; h < C::kStages; h += S::kHalves) {
                    const int buf = h & 1;
                    const unsigned uses = it * (C::kStages / 2) + (h >> 1);      // of the buffer so far
                    const uint32_t dst = dst0 + buf * 64;
                    // either part of an operand stage is free, is filled and goes to the issuer by itself: one is multiplied while the other is filled
                    auto open = [&](int part) {
                        if (leader) {
                            bar_wait(smem_u32(&misc.a_free[mat][buf][part]), (uses & 1) ^ 1);
                            if (!Q6 && !h && part) bar_wait(smem_u32(&misc.hdr_free[mat][it & 1]), ((it >> 1) & 1) ^ 1);
                        }
                        group_sync(1 + grp);
                        tc_fence_after();
                    };
                    auto close = [&](int part) {
                        tmem_wait_st();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) bar_arrive(smem_u32(&misc.a_full[mat][buf][part]));
                    };
                    uint32_t w[8], o[16];
                    if (!Q6) {
                        const uint4 head = *reinterpret_cast<const uint4*>(row);
                        const uint32_t sc = h ? kq_six<1>(head.y, head.w) : kq_six<0>(head.y, 0);
#pragma unroll
                        for (int part = 0; part < 2; part++) {      // chunk c = 2h + part: low nibbles are sub-block 2c, high nibbles sub-block 2c + 1
                            const __half2 sl = part ? h2_byte<2>(sc) : h2_byte<0>(sc), sh = part ? h2_byte<3>(sc) : h2_byte<1>(sc);
                            const uint8_t* q = row + C::kRow - 128 + 32 * (2 * h + part);
                            kq_words8(q, q + 16, w);
                            open(part);
                            if (FMT == KQ_Q4K) {
#pragma unroll
                                for (int i = 0; i < 2; i++) {
                                    kq_unpack4(w + 4 * i, sl, sh, o);
                                    tmem_st16(dst + 32 * part + 16 * i, o);
                                }
                            } else {
                                uint32_t qh[8];
                                kq_words8(row + 16, row + 32, qh);
#pragma unroll
                                for (int i = 0; i < 2; i++) {
                                    kq_unpack5(w + 4 * i, qh + 4 * i, 2 * (2 * h + part), sl, sh, o);
                                    tmem_st16(dst + 32 * part + 16 * i, o);
                                }
                            }
                            if (part && !h) {      // the group of a block's first stage also hands on (d, dmin) and the minima, each twice, against the sixteen 16-value activation sums
                                misc.hdr[mat][it & 1][r] = head.x;
                                uint8_t* m = smem + C::kOffMins + (mat * 2 + (it & 1)) * C::kMins + (r >> 3) * 256 + (r & 7) * 16;      // K-major core matrices of 8 rows x 16 bytes
#pragma unroll
                                for (int i = 0; i < 2; i++) {
                                    const uint32_t mn = i ? kq_six<1>(head.z, head.w >> 4) : kq_six<0>(head.z, 0);
                                    *reinterpret_cast<uint4*>(m + i * 128) = make_uint4(as_u32(h2_byte<0>(mn)), as_u32(h2_byte<1>(mn)), as_u32(h2_byte<2>(mn)), as_u32(h2_byte<3>(mn)));
                                }
                                fence_async_smem();
                            }
                            close(part);
                        }
                    } else {
                        // quarter (hh, pp) of the block: elements 128 hh + 32 pp + l (ql low nibbles, qh bits 2 pp) and + 64 (high nibbles, bits 4 + 2 pp), l < 32;
                        // first 32 columns sc * low four bits / 4, last 32 columns sc * (16 * high two bits - 32) / 4; a scale per 16 elements
                        const int hh = h >> 1, pp = h & 1;
                        const uint2 s8 = *reinterpret_cast<const uint2*>(src + kq_q6_word<FMT>(r, 12) + 8 * hh);
                        const uint32_t pair = __byte_perm(s8.x, s8.y, pp ? 0x7632 : 0x5410) ^ 0x80808080u;      // scales of (low, i = 0), (low, 1), (high, 0), (high, 1), plus 128
                        const __half2 sl[2] = {h2_byte<0, 128>(pair), h2_byte<1, 128>(pair)}, sh[2] = {h2_byte<2, 128>(pair), h2_byte<3, 128>(pair)};
                        const __half2 quarter = __float2half2_rn(0.25f);
                        kq_words8(src + kq_q6_word<FMT>(r, 2 * h), src + kq_q6_word<FMT>(r, 2 * h + 1), w);
                        open(0);
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            kq_unpack4(w + 4 * i, __hmul2(sl[i], quarter), __hmul2(sh[i], quarter), o);
                            tmem_st16(dst + 16 * i, o);
                        }
                        kq_words8(src + kq_q6_word<FMT>(r, 8 + 2 * hh), src + kq_q6_word<FMT>(r, 9 + 2 * hh), w);
                        close(0);
                        open(1);
                        // 4 sc (b - 2) for the two bits b: in the top mantissa bits of 4 they add b, two places lower in 16 too; 4 sc times that, less 24 sc or 72 sc (exact:
                        // 9 * 128 has 11 bits).  Bits 0-1 of the even bytes go up by 6, of the odd ones stay; 2-3: 4 up, 4 down; 4-5: 4 up, 4 down; 6-7 stay, 6 down
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            const __half2 l4 = __hmul2(sl[i], __float2half2_rn(4.f)), h4 = __hmul2(sh[i], __float2half2_rn(4.f));
                            const __half2 l24 = __hmul2(sl[i], __float2half2_rn(-24.f)), l72 = __hmul2(sl[i], __float2half2_rn(-72.f));
                            const __half2 h24 = __hmul2(sh[i], __float2half2_rn(-24.f)), h72 = __hmul2(sh[i], __float2half2_rn(-72.f));
                            if (pp == 0) {
#pragma unroll
                                for (int j = 0; j < 4; j++) {
                                    const uint32_t a = w[4 * i + j];
                                    o[4 * j] = as_u32(__hfma2(bits_at6(a << 6), l4, l72));
                                    o[4 * j + 1] = as_u32(__hfma2(bits_at8(a), l4, l24));
                                    o[4 * j + 2] = as_u32(__hfma2(bits_at8(a << 4), h4, h24));
                                    o[4 * j + 3] = as_u32(__hfma2(bits_at8(a >> 4), h4, h24));
                                }
                            } else {
#pragma unroll
                                for (int j = 0; j < 4; j++) {
                                    const uint32_t a = w[4 * i + j];
                                    o[4 * j] = as_u32(__hfma2(bits_at6(a << 4), l4, l72));
                                    o[4 * j + 1] = as_u32(__hfma2(bits_at6(a >> 4), l4, l72));
                                    o[4 * j + 2] = as_u32(__hfma2(bits_at6(a), h4, h72));
                                    o[4 * j + 3] = as_u32(__hfma2(bits_at8(a >> 6), h4, h24));
                                }
                            }
                            tmem_st16(dst + 32 + 16 * i, o);
                        }
                        close(1);
                    }
                }
                if (lane == 0) bar_arrive(smem_u32(&misc.raw_free[slot]));
                if (++slot == C::kRing) { slot = 0; sphase ^= 1; }
            }
        }
    } else if (warp < S::kEpi) {
        if (SETS > 1) regs_down<S::kRegsI>();
        if (warp == S::kProd) {
            // ====================================================================== activations
            const bool one = lane == 0;
            if (one) tma_prefetch_desc(&maps.q);
            {
                unsigned it = 0;
                for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
                    const KqTile t = kq_tile(p, tile);
                    const int groups = (t.n + 31) >> 5;
                    for (int s = 0; s < t.nsb; s++, it++) {
                        const int b = it & 1, sb = t.sb0 + s;
                        bar_wait(smem_u32(&misc.b_free[b]), ((it >> 1) & 1) ^ 1);
                        const int d = it & 3;
                        if (one) {
                            const uint32_t full = smem_u32(&misc.b_full[b]);
                            bar_expect_tx(full, groups * 32 * (Q6 ? 512 : 544));
                            for (int g = 0; g < groups; g++) {
#pragma unroll
                                for (int c = 0; c < 4; c++) tma_load_2d(base + b * C::kB + c * (kKqN * 128) + g * 4096, &maps.q, full, sb * 256 + c * 64, t.p0 + 32 * g);
                                if (!Q6) tma_load_2d(base + C::kOffSums + b * C::kSums + g * 1024, &maps.sums, full, sb * 16, t.p0 + 32 * g);
                            }
                        }
                        bar_wait(smem_u32(&misc.dx_free[d]), ((it >> 2) & 1) ^ 1);
                        if (one) {
                            bar_expect_tx(smem_u32(&misc.dx_full[d]), kKqN * 4);
                            kq_bulk(smem_u32(&misc.dx[d][0]), p.dx + (long)sb * p.dpitch + t.p0, kKqN * 4, smem_u32(&misc.dx_full[d]));
                        }
                        __syncwarp();
                    }
                }
            }
            __syncwarp();
        } else if (warp == S::kProd + 3) {
            // ====================================================================== weights: the blocks of 2 x 128 rows as they lie in memory
            const bool one = lane == 0;
            {
                int slot = 0, sphase = 1;
                for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
                    const KqTile t = kq_tile(p, tile);
                    const int row = t.e * p.R + t.row0;
                    for (int s = 0; s < t.nsb; s++) {
                        const int sb = t.sb0 + s;
                        bar_wait(smem_u32(&misc.raw_free[slot]), sphase);
                        if (one) {
                            const uint32_t full = smem_u32(&misc.raw_full[slot]);
                            bar_expect_tx(full, C::kSlot);
#pragma unroll
                            for (int mat = 0; mat < 2; mat++) {
                                const uint32_t dst = base + C::kOffRing + slot * C::kSlot + mat * C::kMat;
                                const CUtensorMap* m = maps.w[mat];
                                const int r0 = row + (p.pair ? 0 : 128 * mat);
                                if (!Q6) tma_load_2d(dst, m, full, sb * C::kRow, r0);
                                else if (FMT == KQ_Q6K_T4) tma_load_5d(dst, m, full, 0, sb, 0, 0, r0 >> 2);
                                else {
                                    tma_load_3d(dst, m, full, sb * 128, 0, r0 >> 3);
                                    tma_load_3d(dst + 128 * 128, m + 1, full, sb * 64, 0, r0 >> 3);
                                    tma_load_3d(dst + 128 * 192, m + 2, full, sb * 16, 0, r0 >> 3);
                                }
                            }
                        }
                        __syncwarp();
                        if (++slot == C::kRing) { slot = 0; sphase ^= 1; }
                    }
                }
            }
            __syncwarp();
        } else {
            // ====================================================================== tensor-core issuers (converged warps), one per matrix
            const int mat = warp - S::kProd - 1;
            const uint32_t acc = tmem + mat * kAccCols, a0 = tmem + kColA + mat * 128;
            unsigned it = 0, uses = 0, fills = 0;      // blocks, stages / 2, and accumulators handed to the epilogue so far
            for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
                const KqTile t = kq_tile(p, tile);
                const uint32_t idesc = instr_desc(1, 0, 0, 0, 0, 128, (t.n + 15) & ~15);      // f32 += f16 . f16
                for (int s = 0; s < t.nsb; s++, it++) {
                    const int b = it & 1;
                    const bool marked = MARKS && __any_sync(0xffffffffu, kq_mark(p, t.sb0 + s, t.p0, t.n, lane));
                    // the accumulator is the epilogue's until it gives it back
                    auto taken = [&] { bar_wait(smem_u32(&misc.acc_free[mat]), (fills & 1) ^ 1); };
                    auto give = [&] {
                        mma_commit(smem_u32(&misc.acc_full[mat]));
                        if (MARKS) kq_tell(smem_u32(&misc.marked[mat]), marked, smem_u32(&misc.acc_full[mat]));
                        fills++;
                    };
                    bar_wait(smem_u32(&misc.b_full[b]), (it >> 1) & 1);
                    taken();
                    uint64_t bd = smem_desc(base + b * C::kB, 16, 1024, kLayoutSw128);      // (the address field counts 16 bytes, and nothing carries out of it)
                    const uint64_t md = smem_desc(base + C::kOffMins + (mat * 2 + b) * C::kMins, 128, 256, kLayoutNone), sd = smem_desc(base + C::kOffSums + b * C::kSums, 16, 256, kLayoutSw32);
                    constexpr uint64_t kStep = kKqN * 128 >> 4;      // Q6_K: both terms of a quarter's 64 weights meet one tile of activations
                    // the two parts of stage h into d, from nothing or from what it holds
                    auto stage = [&](int h, uint32_t d, bool add) {
#pragma unroll 1
                        for (int part = 0; part < 2; part++) {
                            bar_wait(smem_u32(&misc.a_full[mat][h & 1][part]), uses & 1);
                            tc_fence_after();
                            mma_f16_ta4(d, a0 + (h & 1) * 64 + part * 32, bd, idesc, add || part);
                            if (!Q6 || part) bd += kStep;
                            mma_commit(smem_u32(&misc.a_free[mat][h & 1][part]));
                        }
                        if (h & 1) uses++;
                    };
                    if (!marked) {
#pragma unroll 1
                        for (int h = 0; h < C::kStages; h++) {
                            stage(h, acc, h);
                            if (!Q6 && h == 0) mma_f16(acc + kKqN, md, sd, idesc, 0);
                        }
                    } else {      // the first stage's sum in the accumulator, each other one behind it, where the epilogue adds it; the minima's product last
#pragma unroll 1
                        for (int h = 0; h < C::kStages; h++) {
                            if (h > 1) taken();
                            stage(h, acc + (h ? kKqN : 0), false);
                            if (h && h < C::kStages - Q6) give();
                        }
                        if (!Q6) {
                            taken();
                            tc_fence_after();
                            mma_f16(acc + kKqN, md, sd, idesc, 0);
                        }
                    }
                    give();
                    mma_commit(smem_u32(&misc.b_free[b]));
                }
            }
        }
    } else {
        // ========================================================================== epilogue: a thread owns one weight row and its group's part of the tile's tokens
        regs_up<S::kRegsE>();
        const int grp = (warp - S::kEpi) >> 2, mat = grp & 1, sp = warp & 3, r = 32 * sp + lane;
        const bool leader = sp == 0;
        unsigned it = 0, fills = 0;
        for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
            const KqTile t = kq_tile(p, tile);
            const int row = t.row0 + (p.pair ? 0 : 128 * mat) + r;
            const int most = SETS == 1 ? kKqN : t.n > 32 ? 32 : 16, col0 = most * (grp >> 1), cols = min(most, t.n - col0);      // (none where <= 0)
            const uint32_t tacc = tmem + ((uint32_t)(32 * sp) << 16) + mat * kAccCols + col0;
            // a Q6_K block's d comes straight from memory, a block ahead
            const uint16_t* dsrc = nullptr;
            uint16_t dnext = 0;
            if (Q6) {
                const int rc = min(row, p.R - 1);
                const uint8_t* w = p.w[p.pair ? mat : 0] + (long)t.e * p.expert_bytes;
                dsrc = reinterpret_cast<const uint16_t*>(FMT == KQ_Q6K_T4 ? w + (long)(rc >> 2) * 4 * p.nblk * SZ_Q6_K + 13L * 64 * p.nblk + (rc & 3) * p.nblk * 2
                                                                         : w + (long)(rc >> 3) * 8 * p.nblk * SZ_Q6_K + 1664L * p.nblk + (rc & 7) * p.nblk * 2) + t.sb0;
                dnext = __ldg(dsrc);
            }
            f32x2 acc[S::kCols / 2];
#pragma unroll
            for (int n = 0; n < S::kCols / 2; n++) acc[n] = 0;
            for (int s = 0; s < t.nsb; s++, it++) {
                const uint16_t dcur = dnext;
                if (Q6 && s + 1 < t.nsb) dnext = __ldg(dsrc + s + 1);
                if (leader) bar_wait(smem_u32(&misc.dx_full[it & 3]), (it >> 2) & 1);
                auto sums = [&] {
                    if (leader) bar_wait(smem_u32(&misc.acc_full[mat]), fills & 1);
                    fills++;
                    group_sync(5 + grp);
                    tc_fence_after();
                };
                sums();
                if (MARKS && misc.marked[mat]) {      // a stage's sum, in the columns behind the accumulator, joins it here
#pragma unroll 1
                    for (int h = 1;; h++) {
#pragma unroll 1
                        for (int c = 0; c < cols; c += 16) {
                            uint32_t v[16], m[16];
                            tmem_ld16(tacc + c, v);
                            tmem_ld16(tacc + kKqN + c, m);
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 16; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(m[i]));
                            tmem_st16(tacc + c, v);
                        }
                        tmem_wait_st();
                        if (Q6 && h + 1 == C::kStages) break;      // nothing follows the last stage
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) bar_arrive(smem_u32(&misc.acc_free[mat]));
                        sums();
                        if (!Q6) break;                            // that was the minima's product
                    }
                }
                const __half2 dm = as_h2(Q6 ? (uint32_t)dcur : misc.hdr[mat][it & 1][r]);
                const float dw = __low2float(dm) * C::kScale, dmin = -__high2float(dm);
                const f32x2 dw2 = pack2(dw, dw), dmin2 = pack2(dmin, dmin);
                const ulonglong2* dx = reinterpret_cast<const ulonglong2*>(misc.dx[it & 3] + col0);
                auto give = [&] {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) bar_arrive(smem_u32(&misc.acc_free[mat]));
                };
                if (SETS > 1 && cols <= 0) give();
#pragma unroll
                for (int c = 0; c < S::kCols / 16; c++) {
                    if (16 * c < cols) {
                        uint32_t v[16], m[16];
                        tmem_ld16(tacc + 16 * c, v);
                        if (!Q6) tmem_ld16(tacc + kKqN + 16 * c, m);
                        tmem_wait_ld();
                        if (16 * c + 16 >= cols) give();      // the last columns are out: the next block may be multiplied while these are scaled
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
                __syncwarp();
                if (lane == 0) {
                    bar_arrive(smem_u32(&misc.hdr_free[mat][it & 1]));
                    bar_arrive(smem_u32(&misc.dx_free[it & 3]));
                }
            }
            // eight tokens at a time in a rolled loop, the sums moving down to its registers, and no branch per value: with ggml's rounding in branches a tile's output took
            // 11,000 cycles, half of a tile of 6 blocks; now 5,500
            int left = cols;
            if (p.y && p.bsz) left = min(left, *p.bsz - p.t0 - t.p0 - col0);
            if (row >= p.R) left = 0;
            const float bias = p.y && p.bias && left > 0 ? p.bias[row] : 0.f;
            const int type = p.y ? p.hidden_type : KTB200_TYPE_F32;
            const long first = ((long)t.split * p.T + t.p0 + col0) * p.R;
            uint8_t* const out = reinterpret_cast<uint8_t*>(p.y ? p.y : p.out[mat]) + (type == KTB200_TYPE_F32 ? 4 : 2) * first;
            uint32_t at = (uint32_t)row;
#pragma unroll 1
            for (; left > 0; left -= 8) {
                if (type == KTB200_TYPE_F32) {
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        if (i < left) reinterpret_cast<float*>(out)[at + (uint32_t)(i * p.R)] = half_of(acc[i >> 1], i & 1) + bias;
                } else {
#pragma unroll
                    for (int i = 0; i < 8; i += 2) {
                        const uint32_t v = pack16(half_of(acc[i >> 1], 0) + bias, half_of(acc[i >> 1], 1) + bias, type == KTB200_TYPE_BF16);
                        if (i < left) reinterpret_cast<uint16_t*>(out)[at + (uint32_t)(i * p.R)] = (uint16_t)v;
                        if (i + 1 < left) reinterpret_cast<uint16_t*>(out)[at + (uint32_t)((i + 1) * p.R)] = (uint16_t)(v >> 16);
                    }
                }
                at += 8u * p.R;
#pragma unroll
                for (int n = 0; n + 4 < S::kCols / 2; n++) acc[n] = acc[n + 4];
            }
        }
    }
}

template <int FMT, bool MARKS, int SETS>
__device__ __forceinline__ void kq_body(const KqMaps& maps, const KqParams& p) {
    using C = KqCfg<FMT>;
    using S = KqSplit<SETS>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    KqMisc& misc = *reinterpret_cast<KqMisc*>(smem + C::kOffMisc);
    const int tid = threadIdx.x, warp = uniform(tid >> 5);
    const int total = p.n_tiles ? *p.n_tiles * p.tiles_mul : p.total;
    if (tid == 0) {
        for (int i = 0; i < 2; i++) {
            bar_init(smem_u32(&misc.b_full[i]), 1); bar_init(smem_u32(&misc.b_free[i]), 2);
            bar_init(smem_u32(&misc.acc_full[i]), MARKS ? 2 : 1); bar_init(smem_u32(&misc.acc_free[i]), 4 * SETS);
            for (int j = 0; j < 2; j++) {
                for (int k = 0; k < 2; k++) { bar_init(smem_u32(&misc.a_full[i][j][k]), 4); bar_init(smem_u32(&misc.a_free[i][j][k]), 1); }
                bar_init(smem_u32(&misc.hdr_free[i][j]), 4 * SETS);
            }
        }
        for (int i = 0; i < 4; i++) { bar_init(smem_u32(&misc.dx_full[i]), 1); bar_init(smem_u32(&misc.dx_free[i]), 8 * SETS); }
        for (int i = 0; i < C::kRing; i++) { bar_init(smem_u32(&misc.raw_full[i]), 1); bar_init(smem_u32(&misc.raw_free[i]), S::kProd); }
        bar_fence_init();
    }
    if (warp == S::kProd + 1) tmem_alloc(smem_u32(&misc.tmem_base), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = uniform(misc.tmem_base);

    kq_roles<FMT, MARKS, SETS>(maps, p, smem, misc, base, tmem, total);
    tc_fence_before();
    __syncthreads();
    if (warp == S::kProd + 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

template <int FMT, int SETS>
__device__ __noinline__ void kq_body_marked(const KqMaps& maps, const KqParams& p) { kq_body<FMT, true, SETS>(maps, p); }
// The form for activations with marked blocks is apart from the other, and the quantiser's word says which one a call needs: in one form the calls without marks took 6-10 %
// longer (777 x 1536 -> 24576 177 -> 194 us: a block's hand-overs wait for its mark, an MMA whose operand depends on it waits for that to be made uniform).
//   KQ_BOTH             one launch, the marked form as a function: costs the other one 3-4 % (registers), and nothing where launches bound a call (512 -> 512, 64 rows: 25 us)
//   KQ_PLAIN, KQ_MARKED two launches, of which one ends at once; the second starts beside the first.  6 us more for short calls, 1 % for long ones (1024 tokens through the
//                       routed experts 2920 us against 3013 with KQ_BOTH, 2893 without marks): experts, and from kPairBlocks blocks of a tile per CTA on
enum KqForms { KQ_PLAIN, KQ_MARKED, KQ_BOTH };
constexpr int kPairBlocks = 40;
template <int FMT, KqForms FORMS, int SETS>
__global__ void __launch_bounds__(kKqThreads, 1) kq_gemm_kernel(const __grid_constant__ KqMaps maps, const __grid_constant__ KqParams p) {
    const bool marks = *p.any == p.id;
    if (FORMS == KQ_BOTH) {
        if (marks) kq_body_marked<FMT, SETS>(maps, p);
        else kq_body<FMT, false, SETS>(maps, p);
    } else {
        if (FORMS == KQ_PLAIN) griddep_launch_dependents();
        if (marks == (FORMS == KQ_MARKED)) kq_body<FMT, FORMS == KQ_MARKED, SETS>(maps, p);
        if (FORMS == KQ_MARKED) griddep_wait();      // (what follows it in the stream follows both)
    }
}

// ---------------------------------------------------------------------------------------------------------------- activations
// whether a block is beyond its limit (kq_limit); s: the lane's sum of quants
__device__ __forceinline__ bool kq_beyond(uint32_t w0, uint32_t w1, int s, bool q6, int limit) {
    const int size = __reduce_add_sync(0xffffffffu, __dp4a((int)__vabs4(w0), 0x01010101, __dp4a((int)__vabs4(w1), 0x01010101, 0)));
    return (q6 ? 2 * size : size + abs(__reduce_add_sync(0xffffffffu, s))) > limit;
}
__device__ __forceinline__ void kq_store_block(const KqActs& a, long row, int b, int K, int lane, bool q6, uint32_t w0, uint32_t w1, float d, int s2, bool beyond) {
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
    if (lane == 0) {
        a.d[(long)b * a.pitch + row] = d;
        a.marks[(long)b * a.pitch + row] = beyond;
        if (beyond) *a.any = a.id;
    }
}
// one warp per (token, 256-block): quantised once, stored for every row the token has
__global__ void __launch_bounds__(256) kq_quant_kernel(const void* x, int hidden_type, int T, int K, const int* pos, int k, int q6, int limit, const KqActs a) {
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
    const bool beyond = kq_beyond(w0, w1, s, q6, limit);
    if (!pos) kq_store_block(a, t, b, K, lane, q6, w0, w1, d, s2, beyond);
    else
        for (int j = 0; j < k; j++) {
            const int row = pos[t * k + j];
            if (row >= 0) kq_store_block(a, row, b, K, lane, q6, w0, w1, d, s2, beyond);
        }
}
// (without pos: rows 0 .. n, each the sum of `splits` parts)
// kParts: loads of so many parts in flight (one where there are no parts: the registers of four halve the warps of an SM, 36 us -> 75 for 1024 tokens' 8 choices of 2048 columns)
template <int kParts>
__global__ void __launch_bounds__(256) kq_act_quant_kernel(const float* g, const float* u, const int* pos, int splits, int n, int K, int use_silu, int q6, int limit, const KqActs a) {
    const int lane = threadIdx.x & 31, nblk = K / QK_K;
    const long gw = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (gw >= (long)n * nblk) return;
    const int i = (int)(gw / nblk), b = (int)(gw - (long)i * nblk), row = pos ? pos[i] : i;
    if (row < 0) return;
    const long o = (long)row * K + (long)b * QK_K + lane * 8;
    float gv[8], uv[8];
    // the parts in their order, the loads of kParts of them in flight: one after the other, the 37 of a shared expert's 24 tokens took 19 us
    for (int p0 = 0; p0 < (kParts == 1 ? 1 : splits); p0 += kParts) {
        float4 x[kParts][4];
#pragma unroll
        for (int p = 0; p < kParts; p++)
            if (kParts == 1 || p0 + p < splits) {
                const long at = (long)(p0 + p) * n * K + o;
                x[p][0] = *reinterpret_cast<const float4*>(g + at); x[p][1] = *reinterpret_cast<const float4*>(g + at + 4);
                x[p][2] = *reinterpret_cast<const float4*>(u + at); x[p][3] = *reinterpret_cast<const float4*>(u + at + 4);
            }
#pragma unroll
        for (int p = 0; p < kParts; p++)
            if (kParts == 1 || p0 + p < splits) {
                const float gx[8] = {x[p][0].x, x[p][0].y, x[p][0].z, x[p][0].w, x[p][1].x, x[p][1].y, x[p][1].z, x[p][1].w};
                const float ux[8] = {x[p][2].x, x[p][2].y, x[p][2].z, x[p][2].w, x[p][3].x, x[p][3].y, x[p][3].z, x[p][3].w};
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    gv[j] = p0 + p ? gv[j] + gx[j] : gx[j];
                    uv[j] = p0 + p ? uv[j] + ux[j] : ux[j];
                }
            }
    }
    float v[8], d;
    uint32_t w0, w1;
    int s;
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = (use_silu ? act_silu(gv[j]) : act_relu(gv[j])) * uv[j];
    warp_q8k_words(v, w0, w1, d, s);
    const int s2 = s + __shfl_xor_sync(0xffffffffu, s, 1);
    const bool beyond = kq_beyond(w0, w1, s, q6, limit);
    kq_store_block(a, row, b, K, lane, q6, w0, w1, d, s2, beyond);
}
// y = sum of the K parts + bias, in the hidden type (accumulate: y + that sum, rounded first).  The parts are added in 64 bits: the launch is bound by their bytes, and
// a chain of 32 in fp32 was half of the error of a long row (K = 16384)
__global__ void __launch_bounds__(256) kq_finish_kernel(const float* part, int splits, int T, int R, void* y, int hidden_type, const float* bias, int accumulate, const int* bsz, int t0) {
    const long i = (long)blockIdx.x * 256 + threadIdx.x, n = (long)(bsz ? max(0, min(T, *bsz - t0)) : T) * R;
    if (i >= n) return;
    double sum = 0.0;
    for (int s0 = 0; s0 < splits; s0 += 8) {
        float x[8];
#pragma unroll
        for (int s = 0; s < 8; s++) x[s] = s0 + s < splits ? part[(long)(s0 + s) * T * R + i] : 0.f;
#pragma unroll
        for (int s = 0; s < 8; s++)
            if (s0 + s < splits) sum += x[s];
    }
    float v = (float)sum;
    if (bias) v += bias[i % R];
    if (accumulate) v = load_hidden(y, i, hidden_type) + round_hidden(v, hidden_type);
    store_hidden(y, i, hidden_type, v);
}

unsigned long long kq_next_id() {
    static std::atomic<unsigned long long> next{0x6b715f6964000001ull};
    return next.fetch_add(1, std::memory_order_relaxed);
}

int kq_quant(const void* x, int hidden_type, int T, int K, const int* pos, int k, bool q6, int limit, const KqActs& a, cudaStream_t s) {
    kq_quant_kernel<<<(unsigned)(((long)T * (K / QK_K) + 7) / 8), 256, 0, s>>>(x, hidden_type, T, K, pos, k, q6, limit, a);
    KTB_LAUNCH_CHECK();
    return KTB200_OK;
}
int kq_act_quant(const float* g, const float* u, const int* pos, int n, int K, int use_silu, bool q6, int limit, const KqActs& a, cudaStream_t s) {
    kq_act_quant_kernel<1><<<(unsigned)(((long)n * (K / QK_K) + 7) / 8), 256, 0, s>>>(g, u, pos, 1, n, K, use_silu, q6, limit, a);
    KTB_LAUNCH_CHECK();
    return KTB200_OK;
}

// ---------------------------------------------------------------------------------------------------------------- launch
// a tensor map of `rank` dimensions (innermost first) with the given byte strides of dimensions 1 .. rank - 1
static int kq_map(CUtensorMap* map, CUtensorMapDataType type, const void* ptr, int rank, const cuuint64_t* dim, const cuuint64_t* stride, const cuuint32_t* box, CUtensorMapSwizzle sw) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) { set_error("kq_gemm: cuTensorMapEncodeTiled is not available from this driver"); return KTB200_ECUDA; }
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    const CUresult cr = enc(map, type, rank, const_cast<void*>(ptr), dim, stride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) { set_error("kq_gemm: cuTensorMapEncodeTiled failed (%d)", (int)cr); return KTB200_ECUDA; }
    return KTB200_OK;
}
// boxes of 32 rows x `cols` fp16 of a row-major matrix
static int kq_map_acts(CUtensorMap* map, const void* ptr, long width, long rows, int cols, CUtensorMapSwizzle sw) {
    const cuuint64_t dim[2] = {(cuuint64_t)width, (cuuint64_t)rows}, stride[1] = {(cuuint64_t)width * 2};
    const cuuint32_t box[2] = {(cuuint32_t)cols, 32};
    return kq_map(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, ptr, 2, dim, stride, box, sw);
}
// one block of 128 rows of a matrix of `rows` rows (all experts') of nblk blocks
static int kq_map_weights(CUtensorMap* m, KqFmt f, const void* w, long rows, int nblk) {
    const CUtensorMapDataType u8 = CU_TENSOR_MAP_DATA_TYPE_UINT8;
    const cuuint64_t nb = (cuuint64_t)nblk;
    if (!kq_is_q6(f)) {
        const int bytes = f == KQ_Q4K ? SZ_Q4_K : SZ_Q5_K;
        const cuuint64_t dim[2] = {nb * bytes, (cuuint64_t)rows}, stride[1] = {nb * bytes};
        const cuuint32_t box[2] = {(cuuint32_t)bytes, 128};
        return kq_map(m, u8, w, 2, dim, stride, box, CU_TENSOR_MAP_SWIZZLE_NONE);
    }
    if (f == KQ_Q6K_T4) {      // [4-row item][word][row][block][16 bytes]
        const cuuint64_t dim[5] = {16, nb, 4, 13, (cuuint64_t)rows / 4}, stride[4] = {16, 16 * nb, 64 * nb, 4 * nb * SZ_Q6_K};
        const cuuint32_t box[5] = {16, 1, 4, 13, 32};
        return kq_map(m, u8, w, 5, dim, stride, box, CU_TENSOR_MAP_SWIZZLE_NONE);
    }
    const int bytes[3] = {128, 64, 16}, off[3] = {0, 1024, 1536};      // 8-row groups: [ql: row][block] | [qh: row][block] | [scales: row][block]
    const CUtensorMapSwizzle sw[3] = {CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_SWIZZLE_NONE};
    for (int i = 0; i < 3; i++) {
        const cuuint64_t dim[3] = {nb * bytes[i], 8, (cuuint64_t)rows / 8}, stride[2] = {nb * bytes[i], 8 * nb * SZ_Q6_K};
        const cuuint32_t box[3] = {(cuuint32_t)bytes[i], 8, 16};
        const int rc = kq_map(m + i, u8, reinterpret_cast<const uint8_t*>(w) + (size_t)off[i] * nblk, 3, dim, stride, box, sw[i]);
        if (rc) return rc;
    }
    return KTB200_OK;
}
template <int FMT, int SETS>
static int kq_launch_as(const KqMaps& maps, const KqParams& p, int grid, cudaStream_t s) {
    constexpr int smem = kq_smem<FMT>();
    if (!p.tinfo && (long)p.total * ((p.nblk + p.splits - 1) / p.splits) < (long)kPairBlocks * grid) {
        KTB_CUDA_CHECK(cudaFuncSetAttribute(kq_gemm_kernel<FMT, KQ_BOTH, SETS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        kq_gemm_kernel<FMT, KQ_BOTH, SETS><<<grid, kKqThreads, smem, s>>>(maps, p);
        KTB_LAUNCH_CHECK();
        return KTB200_OK;
    }
    KTB_CUDA_CHECK(cudaFuncSetAttribute(kq_gemm_kernel<FMT, KQ_PLAIN, SETS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    KTB_CUDA_CHECK(cudaFuncSetAttribute(kq_gemm_kernel<FMT, KQ_MARKED, SETS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kq_gemm_kernel<FMT, KQ_PLAIN, SETS><<<grid, kKqThreads, smem, s>>>(maps, p);
    KTB_LAUNCH_CHECK();
    KTB_CUDA_CHECK(launch_pdl(kq_gemm_kernel<FMT, KQ_MARKED, SETS>, dim3(grid), dim3(kKqThreads), (size_t)smem, s, maps, p));
    KTB_LAUNCH_CHECK();
    return KTB200_OK;
}

// Two epilogue groups a matrix for a Q4_K matrix against more than 48 tokens: measured against one group (us) 777 x 1536 -> 24576 126 -> 112, 333 of it 65.0 -> 60.9, 2048 -> 8192 64 tokens
// 27.5 -> 25.4, 333 44.5 -> 42.4, 512 -> 4096 64 tokens 18.4 -> 16.5, and the same time where K splits leave the launch to its copies (7168 -> 2048, 65-333 tokens).  With 12-48
// tokens 1-10 % slower (half as many producers; 1536 -> 24576, 17 tokens 20.8 -> 23.0), and in Q6_K and Q5_K, whose producers do more, at any number (Q6_K 333 tokens 80.7 -> 93.6)
constexpr int kTwoSets = 49;
template <int FMT>
static int kq_launch(const KqMaps& maps, const KqParams& p, int grid, cudaStream_t s) {
    if constexpr (FMT == KQ_Q4K)
        if (!p.tinfo && p.T >= kTwoSets) return kq_launch_as<FMT, 2>(maps, p, grid, s);
    return kq_launch_as<FMT, 1>(maps, p, grid, s);
}

int kq_gemm(const KqGemm& g, int device, cudaStream_t s) {
    KqParams p{};
    for (int i = 0; i < 2; i++) { p.w[i] = reinterpret_cast<const uint8_t*>(g.w[i]); p.out[i] = g.out[i]; }
    p.expert_bytes = g.expert_bytes; p.dpitch = g.acts->pitch; p.pair = g.pair; p.R = g.R; p.nblk = g.K / QK_K; p.dx = g.acts->d; p.marks = g.acts->marks; p.any = g.acts->any; p.id = g.acts->id;
    p.tinfo = g.tinfo; p.n_tiles = g.n_tiles_dev; p.tiles_mul = g.tiles_mul; p.y = g.y; p.hidden_type = g.hidden_type; p.bias = g.bias; p.bsz = g.bsz;
    p.t0 = g.t0; p.T = g.T; p.splits = g.splits; p.rt = (g.R + kKqRows - 1) / kKqRows; p.nt = (g.T + kKqN - 1) / kKqN; p.total = p.rt * p.nt * g.splits;
    KqMaps maps;
    int rc = kq_map_acts(&maps.q, g.acts->q, g.K, g.acts->rows, 64, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc == KTB200_OK) rc = kq_map_acts(&maps.sums, g.acts->sums, g.K / 16, g.acts->rows, 16, CU_TENSOR_MAP_SWIZZLE_32B);
    for (int i = 0; i < 2 && rc == KTB200_OK; i++) rc = kq_map_weights(maps.w[i], g.fmt, g.w[i], (long)g.experts * g.R, p.nblk);
    if (rc) return rc;
    const int sms = num_sms(device), grid = g.tinfo || p.total > sms ? sms : p.total;
    switch (g.fmt) {
        case KQ_Q4K: return kq_launch<KQ_Q4K>(maps, p, grid, s);
        case KQ_Q5K: return kq_launch<KQ_Q5K>(maps, p, grid, s);
        case KQ_Q6K_T4: return kq_launch<KQ_Q6K_T4>(maps, p, grid, s);
        case KQ_Q6K_SOA8: return kq_launch<KQ_Q6K_SOA8>(maps, p, grid, s);
        default: set_error("kq_gemm: unsupported weight type"); return KTB200_EINVAL;
    }
}

// K in parts when the tiles leave SMs idle, two blocks or more each
static int kq_splits(int tiles, int nblk, int sms) {
    const int n = sms / tiles < nblk / 2 ? sms / tiles : nblk / 2;
    return n < 1 ? 1 : n;
}

// fp32 results, where the order of a long fp32 chain shows: parts of at most kKqChain blocks
constexpr int kKqChain = 10;
static int kq_splits_of(int tiles, int nblk, int sms, int hidden_type) {
    const int n = kq_splits(tiles, nblk, sms);
    return hidden_type == KTB200_TYPE_F32 ? std::max(n, (nblk + kKqChain - 1) / kKqChain) : n;
}

int kq_linear(FmtId fmt, const void* w, int R, int K, const void* x, int hidden_type, int T, void* y, const float* bias, const int* bsz, int device, cudaStream_t s) {
    const KqFmt f = kq_fmt(fmt);
    if (f == KQ_NONE || (uintptr_t)w % 16) return 1;
    // rows per pass: bounds the scratch (fp32 results in parts: to 256 MB of those)
    const int nparts = kq_splits_of(INT_MAX, K / QK_K, 1, hidden_type);
    const int chunk = nparts == 1 ? 4096 : std::max(256L, std::min(4096L, (1L << 26) / ((long)nparts * R) / kKqN * kKqN));
    const size_t hb = type_size(hidden_type);
    for (int t0 = 0; t0 < T; t0 += chunk) {
        const int n = T - t0 < chunk ? T - t0 : chunk, sms = num_sms(device);
        const int tiles = ((R + kKqRows - 1) / kKqRows) * ((n + kKqN - 1) / kKqN), nblk = K / QK_K;
        const int splits = kq_splits_of(tiles, nblk, sms, hidden_type);
        ScratchBlock mem(s);
        const size_t act = (KqActs::bytes(n, K) + 255) / 256 * 256;
        const size_t scratch = act + (splits > 1 ? (size_t)splits * n * R * 4 : 0);
        if (T <= 8) {      // (so few rows need none: without it the row kernels take them, and the call has no error to tell of)
            if (mem.take(device, scratch) != cudaSuccess) return 1;
        } else if (!mem.taken(device, scratch)) {
            return KTB200_ECUDA;
        }
        const KqActs a(mem.ptr, n, K);
        int rc = kq_quant(reinterpret_cast<const uint8_t*>(x) + (size_t)t0 * K * hb, hidden_type, n, K, nullptr, 1, kq_is_q6(f), kq_limit(f), a, s);
        if (rc) return rc;
        KqGemm g{};
        g.fmt = f; g.w[0] = g.w[1] = w; g.experts = 1; g.R = R; g.K = K; g.acts = &a; g.T = n; g.splits = splits; g.hidden_type = hidden_type; g.bias = bias; g.t0 = t0;
        void* yc = reinterpret_cast<uint8_t*>(y) + (size_t)t0 * R * hb;
        float* part = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(mem.ptr) + act);
        if (splits == 1) { g.y = yc; g.bsz = bsz; }
        else g.out[0] = g.out[1] = part;
        rc = kq_gemm(g, device, s);
        if (rc) return rc;
        if (splits > 1) {
            kq_finish_kernel<<<(unsigned)(((long)n * R + 255) / 256), 256, 0, s>>>(part, splits, n, R, yc, hidden_type, bias, 0, bsz, t0);
            KTB_LAUNCH_CHECK();
        }
    }
    return KTB200_OK;
}

int kq_mlp(const ktb200_mlp* m, const void* x, int T, void* y, int accumulate, const int* bsz, cudaStream_t s) {
    const KqFmt f[3] = {kq_fmt(pick_fmt(m->gate_type, m->gu_soa)), kq_fmt(pick_fmt(m->up_type, m->gu_soa)), kq_fmt(pick_fmt(m->down_type, m->down_layout))};
    const void* w[3] = {m->gate, m->up, m->down};
    for (int i = 0; i < 3; i++)
        if (f[i] == KQ_NONE || (uintptr_t)w[i] % 16) return 1;
    if (kq_is_q6(f[0]) != kq_is_q6(f[1])) return 1;      // (gate and up read the same activations)
    constexpr int kChunk = 1024;      // rows per pass: bounds the scratch
    const int H = m->H, I = m->I, dev = m->device, sms = num_sms(dev);
    const size_t hb = type_size(m->hidden_type);
    for (int t0 = 0; t0 < T; t0 += kChunk) {
        const int n = T - t0 < kChunk ? T - t0 : kChunk, nt = (n + kKqN - 1) / kKqN;
        const int su = kq_splits((I + kKqRows - 1) / kKqRows * nt, H / QK_K, sms), sd = kq_splits_of((H + kKqRows - 1) / kKqRows * nt, I / QK_K, sms, m->hidden_type);
        auto up = [](size_t b) { return (b + 255) / 256 * 256; };
        const size_t n_x = up(KqActs::bytes(n, H)), n_a = up(KqActs::bytes(n, I)), n_g = up((size_t)su * n * I * 4), n_d = up((size_t)sd * n * H * 4);
        ScratchBlock mem(s);
        if (!mem.taken(dev, n_x + n_a + 2 * n_g + n_d)) return kNoScratch;
        uint8_t* at = reinterpret_cast<uint8_t*>(mem.ptr);
        const KqActs xa(at, n, H), aa(at + n_x, n, I);
        float *gu[2] = {reinterpret_cast<float*>(at + n_x + n_a), reinterpret_cast<float*>(at + n_x + n_a + n_g)}, *part = reinterpret_cast<float*>(at + n_x + n_a + 2 * n_g);
        int rc = kq_quant(reinterpret_cast<const uint8_t*>(x) + (size_t)t0 * H * hb, m->hidden_type, n, H, nullptr, 1, kq_is_q6(f[0]), std::min(kq_limit(f[0]), kq_limit(f[1])), xa, s);
        if (rc) return rc;
        KqGemm g{};
        g.experts = 1; g.R = I; g.K = H; g.acts = &xa; g.T = n; g.splits = su;
        for (int i = 0; i < 2; i++) {
            g.fmt = f[i]; g.w[0] = g.w[1] = w[i]; g.out[0] = g.out[1] = gu[i];
            rc = kq_gemm(g, dev, s);
            if (rc) return rc;
        }
        (su > 1 ? kq_act_quant_kernel<4> : kq_act_quant_kernel<1>)<<<(unsigned)(((long)n * (I / QK_K) + 7) / 8), 256, 0, s>>>(gu[0], gu[1], nullptr, su, n, I, 1, kq_is_q6(f[2]), kq_limit(f[2]), aa);
        KTB_LAUNCH_CHECK();
        g.fmt = f[2]; g.w[0] = g.w[1] = w[2]; g.R = H; g.K = I; g.acts = &aa; g.splits = sd; g.out[0] = g.out[1] = part;
        rc = kq_gemm(g, dev, s);
        if (rc) return rc;
        kq_finish_kernel<<<(unsigned)(((long)n * H + 255) / 256), 256, 0, s>>>(part, sd, n, H, reinterpret_cast<uint8_t*>(y) + (size_t)t0 * H * hb, m->hidden_type, nullptr, accumulate, bsz, t0);
        KTB_LAUNCH_CHECK();
    }
    return KTB200_OK;
}

}  // namespace ktb
