// Internal layout shared by the kernels of the link-prediction training step (ge2_lp_step).
//
// Data flow of one step (S = corruption sides, Bp = C * ceil(B/C) padded batch rows, ld = padded row length):
//   prep     : gather src/dst/relation rows, apply the relation operator        -> Q[S][Bp][ld], pos[S][Bp]
//              gather negative rows                                              -> K[S][C*N][ld]
//   scores   : per (side, chunk): S = Q K^T, mask, row logsumexp with the positive score,
//              P = exp(S - lse), dQ = P K, dK = P^T Q  (score tiles never leave the SM)   -> lse, dQ, dK
//   finish   : relation-operator backward, d pos terms, duplicate-reducing scatter into node_grad / rel_grad, loss
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>

#include "common.cuh"

namespace ge2 {

constexpr float kLpF16GradUnscale = 1.0f / 16384.0f;  // the tensor path leaves dQ and dK scaled by 2^14 (its W tiles are)

struct LpLayout {
    int S;        // sides
    int npc;      // rows per chunk = ceil(B / C)
    int Bp;       // C * npc
    int ld;       // padded row length of Q / K / dQ / dK (floats)
    int64_t CN;   // C * N
    // workspace sections
    float* dQ;        // [S][Bp][ld]
    float* dK;        // [S][CN][ld]   cleared by the logsumexp pass, added to by the gradient pass
    float* pos;       // [S][Bp]
    float* lse;       // [S][Bp]
    int32_t* mask;    // [S][CN]  batch row whose score in this (chunk, column) is masked, or -1
    // operands of the scores kernels.  f16: one fp16 copy of Q [S][Bp][ld] and of K [S][CN][ld].  fp32: three bf16 planes of each
    // ([3][S][Bp][ld], [3][S][CN][ld]) whose sum is the fp32 value.
    __half* Qh;
    __half* Kh;
    __nv_bfloat16* Qs;
    __nv_bfloat16* Ks;
    double* loss_acc; // [1] sum over rows of (lse - pos): zeroed by the prepare kernel, added to by the scores kernels
    float* part;      // [S][Bp][8][2] per-row partial (max, sum) of the logsumexp pass when a row block's tiles are split over CTAs
    float* lse2s;     // [S*C][row_blocks*128] row logsumexp in base-2 units minus the probability scale exponent; 1e30 for rows past the chunk
    float* o_part;    // f16: [CTAs][2][128][ld] parts of dQ of the (at most two) row blocks a CTA of the query launch shares with others
    int n_items;        // S * C * row_blocks
    float grad_unscale; // factor the finish kernel applies to what it reads from dQ / dK: 1, or 2^-14 on the tensor path
    size_t bytes;
};

struct LpKernelArgs {
    ge2_lp_desc d;
    LpLayout L;
};

inline size_t lp_align(size_t x) { return (x + 255) & ~(size_t)255; }

__host__ __device__ inline int lp_row_ld(int D) { return D <= 64 ? 64 : 128; }

// Which of the two fp16 forms a step takes.  The two-pass form adds every row block's part into dK, which is the faster way while dK stays in
// the L2 beside the operands.  The streaming form writes every row once and spends less on a tile (2.3 ... 2.6 us for both its launches on one
// CTA, 2.6 ... 2.8), but each of its blocks costs a fill and a drain of the pipeline, more where a block is cut between CTAs, and its
// launches some 8 us more: of its two launches the one over the negatives has T blocks a chunk (T tiles of 128 negatives) with
// only as many tiles each as the chunk has row blocks.  So the line in bytes of dK rises with T and falls with the row blocks, less steeply
// for rows of 64 columns, whose tiles are half the traffic; without cuts it stays at 64 MB.  And where T is small and the last tile
// mostly padding, the line is twice as high: the two-pass form skips the columns that do not exist.  Whatever the size of dK, the streaming form
// is taken where every CTA has enough tiles and a chunk is neither a few row blocks high nor many tiles wide: from 12 tiles a CTA on for rows
// of 64 columns, whose tiles spend less on contractions, from 40 on for wider ones.
// Both forms at 4 020 shapes (chunks of 50 ... 2 000 rows, 100 ... 20 000 negatives, dK of 2 ... 290 MB, one and two sides), us, two-pass : streaming
//   D = 64, two sides: 100 x 997 rows, 246 negatives 86 : 69; 100 x 743, 1 111 negatives 203 : 165; 2 x 1 605, 15 438 negatives (D = 50) 67 : 118
//   D = 128, two sides: 18 x 1 941 rows, 2 031 negatives 203 : 165; 53 x 902, 587 negatives 111 : 117; 39 x 515, 936 negatives 84 : 88
//   dK above 64 MB, D = 128: 100 x 571 rows, 1 661 negatives 475 : 265; 50 x 629, 6 746 negatives (D = 50) 520 : 378; 15 x 613, 19 777 254 : 310
// The form that is taken is 0.9 % slower than the better one on average, and 25 % at most (by the bytes of dK alone: 2.1 and 28 %).
inline bool lp_uses_flash(const ge2_lp_desc& d, int S, int64_t CN, int ld) {
    if (d.precision != GE2_PRECISION_F16) return false;
    const int64_t T = ceil_div<int64_t>(d.N, 128), blocks = ceil_div(rows_per_chunk(d.B, d.C), 128), units = S * d.C * T * blocks;
    if (T <= 16 && (ld == 64 ? blocks > 2 && units > 12 * kNumSMs : blocks > 3 && units > 40 * kNumSMs)) return true;
    const double row_blocks = (double)blocks, mb = (double)S * CN * ld * 4 / (1 << 20);
    if (S * d.C * T % kNumSMs == 0) return mb > 64;
    const double over = ld == 128 ? 4.0 * (T - 1) : T > 8 ? 2.0 * (T - 8) : 0.0;
    const bool padded = ld == 128 && T >= 3 && T <= 6 && 128 * T * 8 > 9 * (int64_t)d.N;
    return mb > (64 + over / (row_blocks * sqrt(row_blocks))) * (padded ? 2 : 1);
}

// streaming: false = the two-pass form whatever lp_uses_flash says (its layout is the other's without the last section)
inline LpLayout lp_make_layout(const ge2_lp_desc& d, void* base, bool streaming = true) {
    LpLayout L;
    L.S = (d.has_relations && d.use_inverse) ? 2 : 1;
    L.npc = rows_per_chunk(d.B, d.C);
    L.Bp = d.C * L.npc;
    L.ld = lp_row_ld(d.D);
    L.CN = (int64_t)d.C * d.N;
    char* p = (char*)base;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        size_t o = off;
        off += lp_align(bytes);
        return o;
    };
    size_t odQ = take((size_t)L.S * L.Bp * L.ld * 4);
    size_t odK = take((size_t)L.S * L.CN * L.ld * 4);
    size_t opos = take((size_t)L.S * L.Bp * 4);
    size_t olse = take((size_t)L.S * L.Bp * 4);
    size_t omask = take((size_t)L.S * L.CN * 4);
    size_t oloss = take(8);
    const bool half_copies = d.precision == GE2_PRECISION_F16;
    const size_t planes = half_copies ? 1 : 3;
    size_t oQ = take(planes * L.S * L.Bp * L.ld * 2);
    size_t oK = take(planes * L.S * L.CN * L.ld * 2);
    size_t opart = take((size_t)L.S * L.Bp * 16 * 4);
    const int row_blocks = (L.npc + 127) / 128;
    L.n_items = L.S * d.C * row_blocks;
    size_t olse2 = take((size_t)L.n_items * 128 * 4);
    streaming = streaming && lp_uses_flash(d, L.S, L.CN, L.ld);
    size_t oopart = take(streaming ? (size_t)kNumSMs * 2 * 128 * L.ld * 4 : 0);
    L.o_part = streaming ? (float*)(p + oopart) : nullptr;
    L.dQ = (float*)(p + odQ);
    L.dK = (float*)(p + odK);
    L.pos = (float*)(p + opos);
    L.lse = (float*)(p + olse);
    L.mask = (int32_t*)(p + omask);
    L.loss_acc = (double*)(p + oloss);
    L.Qh = half_copies ? (__half*)(p + oQ) : nullptr;
    L.Kh = half_copies ? (__half*)(p + oK) : nullptr;
    L.Qs = half_copies ? nullptr : (__nv_bfloat16*)(p + oQ);
    L.Ks = half_copies ? nullptr : (__nv_bfloat16*)(p + oK);
    L.part = (float*)(p + opart);
    L.grad_unscale = half_copies ? kLpF16GradUnscale : 1.0f;
    L.lse2s = (float*)(p + olse2);
    L.bytes = off;
    return L;
}

// CTAs of a persistent scores launch over `units` tiles, one a CTA at a time and one CTA an SM: no more than it takes for the longest share to be
// as short as it is with one on every SM, but at most eight SMs are left to others (what runs on them meanwhile: the next batch's sampler and
// unique-map in a pipelined step).
inline int scores_ctas(long long units) {
    if (units <= kNumSMs) return (int)(units < 1 ? 1 : units);
    const long long share = ceil_div<long long>(units, kNumSMs), ctas = ceil_div(units, share);
    return (int)(ctas < kNumSMs - 8 ? kNumSMs - 8 : ctas);
}
constexpr int kLp32Rows = 128, kLp32Cols = 64;  // a tile of the fp32 path
inline long long scores_units(const ge2_lp_desc& d, int S) {
    const int cols = d.precision == GE2_PRECISION_F16 ? 128 : kLp32Cols;
    return (long long)S * d.C * ceil_div(rows_per_chunk(d.B, d.C), 128) * ceil_div(d.N, cols);
}

// scores kernels (one per precision); both fill lse, dQ, dK (+ optional score dumps) from Q, K, pos, mask
int lp_scores_fp32(const LpKernelArgs& a, cudaStream_t stream);
int lp_scores_f16(const LpKernelArgs& a, cudaStream_t stream);
int lp_flash_f16(const LpKernelArgs& a, cudaStream_t stream);


}  // namespace ge2
