// Prompt-sized products against GGUF K-quant matrices on the tensor cores (kq_gemm.cu): what the routed experts (grouped.cu) and the dense
// linears (moe.cu) hand to it.
#pragma once
#include "common.cuh"
#include "handles.cuh"

namespace ktb {

enum KqFmt { KQ_Q4K, KQ_Q5K, KQ_Q6K_T4, KQ_Q6K_SOA8, KQ_NONE };
static inline KqFmt kq_fmt(FmtId f) {
    return f == FMT_Q4K ? KQ_Q4K : f == FMT_Q5K ? KQ_Q5K : f == FMT_Q6K4T ? KQ_Q6K_T4 : f == FMT_Q6K8 ? KQ_Q6K_SOA8 : KQ_NONE;
}
static inline bool kq_is_q6(KqFmt f) { return f == KQ_Q6K_T4 || f == KQ_Q6K_SOA8; }

// Which 256-blocks of activations might take a partial sum of the product past 2^24, where an fp32 accumulator stops to be exact, as a bound on twice ...
//   Q4_K, Q5_K (weights 0 .. 63 * 15, 0 .. 63 * 31): the larger of the sums of the block's positive and negative quants.  At or below it every sum is exact.
//   Q6_K (weights of either sign, at most 128 * 32): the sum of the quants' magnitudes.  Flatter than 14000 (a normal block has 9300, all quants equal 32512);
//   below it only weights of more than 2^24 / 14000 = 1198 on average that all lie along the activations' signs get there.
// Blocks beyond it are marked and summed stage by stage (kq_gemm.cu).
static inline int kq_limit(KqFmt f) { return 2 * (f == KQ_Q4K ? 17753 : f == KQ_Q5K ? 8590 : 14000); }

constexpr int kKqN = 64;       // tokens of a tile
constexpr int kKqRows = 256;   // weight rows of a tile: 128 of each of two matrices, or 256 of one

unsigned long long kq_next_id();

// Q8_K activations as the product reads them: the int8 quants as fp16 (exact) in the order in which the weights come out of their blocks,
// the block scales with the row fastest, and (Q4_K, Q5_K) the sixteen 16-value sums of a block as fp16 (|sum| <= 2032: exact).
struct KqActs {
    __half* q;        // [rows][K]
    __half* sums;     // [rows][K / 16]
    float* d;         // [K / 256][pitch], pitch a multiple of 4 and at least rows + kKqN
    uint8_t* marks;   // [K / 256][pitch]: 1 where a block is beyond kq_limit
    unsigned long long *any, id;      // *any == id: there is such a block.  The number is this batch's alone, so the word needs no clearing (a replayed graph may find its own)
    long rows, pitch;
    static size_t bytes(long rows, int K) { return (size_t)rows * K * 2 + (size_t)rows * (K / 16) * 2 + (size_t)(K / QK_K) * pitch_of(rows) * 5 + 1280; }
    static long pitch_of(long rows) { return (rows + kKqN + 3) / 4 * 4; }
    KqActs(void* mem, long n, int K) : any(reinterpret_cast<unsigned long long*>(mem)), id(kq_next_id()), rows(n), pitch(pitch_of(n)) {
        uint8_t* p = reinterpret_cast<uint8_t*>(mem) + 256;
        d = reinterpret_cast<float*>(p);
        p += ((size_t)(K / QK_K) * pitch * 4 + 255) / 256 * 256;
        marks = p;
        p += ((size_t)(K / QK_K) * pitch + 255) / 256 * 256;
        q = reinterpret_cast<__half*>(p);
        p += (size_t)rows * K * 2;
        sums = reinterpret_cast<__half*>(p);
    }
};

struct KqGemm {
    KqFmt fmt;
    const void* w[2];          // pair: one matrix each; else both are the same matrix, a tile's second 128 rows following its first
    bool pair;
    long expert_bytes;         // bytes between two experts' matrices
    int experts;
    int R, K;
    const KqActs* acts;
    // experts: device tables made by the caller; a tile is {expert, first row, first activation row (a multiple of 4), tokens}
    const int4* tinfo;
    const int* n_tiles_dev;    // their number / tiles_mul on the device
    int tiles_mul;
    // one matrix against `T` rows (tinfo null): K is cut into `splits` parts when there are few tiles
    int T, splits;
    float* out[2];             // fp32 [rows][R] (splits: [splits][T][R])
    void* y;                   // or, splits == 1: the hidden type, + bias, rows at or beyond *bsz - t0 untouched
    int hidden_type;
    const float* bias;
    const int* bsz;
    int t0;
};
int kq_gemm(const KqGemm& g, int device, cudaStream_t s);

// x [T][K] (hidden type) -> Q8_K activations; row t goes to rows pos[t * k .. + k) that are not negative, or to row t when pos is null
int kq_quant(const void* x, int hidden_type, int T, int K, const int* pos, int k, bool q6, int limit, const KqActs& a, cudaStream_t s);
// act(g) * u of rows pos[0 .. n) (fp32 [rows][K]) -> Q8_K activations of the same rows
int kq_act_quant(const float* g, const float* u, const int* pos, int n, int K, int use_silu, bool q6, int limit, const KqActs& a, cudaStream_t s);

// y = x . W^T for a batch of T rows of one matrix.  Returns 1 when the shape does not suit it.
int kq_linear(FmtId fmt, const void* w, int R, int K, const void* x, int hidden_type, int T, void* y, const float* bias, const int* bsz, int device, cudaStream_t s);
// y (+)= W_down (silu(W_gate x) * W_up x) for a batch of T rows.  Returns 1 when the matrices' layouts do not suit it.
int kq_mlp(const ktb200_mlp* m, const void* x, int T, void* y, int accumulate, const int* bsz, cudaStream_t s);

}  // namespace ktb
