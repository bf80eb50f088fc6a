// Selected-negative scoring for the DNS / GAN / tournament samplers: a query row is scored against the few negatives chosen
// for it instead of against its whole chunk.
//
// Follows, in the reference project:
//   scores of chosen pairs, forward     gege/src/cuda/src/nn/decoders/edge/distmult_selected_neg_cuda.cu:15-85
//                                       (one thread per (row, chosen negative) walking D; dot product, or
//                                       sqrt(max(|q - n|^2, 1e-8)) for the L2 comparator)
//   ... backward                        same file :88-202 (query gradient: a thread per (row, d) looping the chosen negatives;
//                                       negative gradient: an atomic add per (row, chosen, d); L2: one thread per pair)
//   tournament selection                gege/src/cpp/src/nn/decoders/edge/distmult_selected_neg_cuda.cpp:46-121 (per tile of
//                                       groups: bmm -> view [.., groups, T] -> max(3) -> gather; the negatives of a chunk form
//                                       `selected` groups of T = N / selected consecutive ones, a row keeps the best of each)
//
// Here a warp owns a query row: the row sits in registers (D <= 128, four values a lane), every chosen negative row is read
// once with coalesced (16-byte, where the rows allow it) loads and serves the score, the query gradient and the negative gradient of its pair in one pass
// (the reference's backward reads every pair twice, in two launches).  The tournament never stores the [rows x N] scores: they are
// contracted tile by tile on the tensor cores, with fp32 operands split exactly, and the group winners are read off the tiles.
#include <math_constants.h>

#include <algorithm>

#include "tc_pipe.cuh"

namespace ge2 {
namespace {

constexpr int kMaxD = 128;
constexpr int kPairThreads = 256, kPairWarps = kPairThreads / 32;
constexpr float kL2Floor = 1e-8f;  // the reference's kSelectedNegL2Tol, compared in float

struct PairArgs {
    const float* chunked;     // [chunks * R, D]
    const float* negatives;   // [chunks, N, D]
    const int64_t* selected;  // [chunks * R, K] columns of the row's chunk
    int64_t rows, R, N, K;
    int D, kind;
    int32_t* status;
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// A row of D <= 128 floats over the 32 lanes, four values a lane.  VEC (D a multiple of 4, 16-byte aligned rows): lane l holds
// elements 4l .. 4l+3, one 16-byte access; else lane l holds elements l, l+32, l+64, l+96.  Values past D are 0.
template <bool VEC>
__device__ __forceinline__ void load_row(float (&v)[4], const float* __restrict__ p, int lane, int D) {
    if (VEC) {
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (lane * 4 < D) t = __ldg(reinterpret_cast<const float4*>(p) + lane);
        v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = lane + 32 * j < D ? __ldg(p + lane + 32 * j) : 0.f;
    }
}

template <bool VEC>
__device__ __forceinline__ void store_row(float* __restrict__ p, const float (&v)[4], int lane, int D) {
    if (VEC) {
        if (lane * 4 < D) reinterpret_cast<float4*>(p)[lane] = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (lane + 32 * j < D) p[lane + 32 * j] = v[j];
    }
}

template <bool VEC>
__device__ __forceinline__ void add_row(float* __restrict__ p, const float (&v)[4], int lane, int D) {
    if (VEC) {
        if (lane * 4 < D) atomicAdd(reinterpret_cast<float4*>(p) + lane, make_float4(v[0], v[1], v[2], v[3]));  // four element-wise adds, one request
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (lane + 32 * j < D) atomicAdd(p + lane + 32 * j, v[j]);
    }
}

// this lane's share of q . n (DOT) or |q - n|^2 (L2); lanes past D hold zeros in both
template <int KIND>
__device__ __forceinline__ float pair_partial(const float (&q)[4], const float (&n)[4]) {
    float part = 0.f;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if (KIND == GE2_SELECTED_DOT) {
            part = __fmaf_rn(q[j], n[j], part);
        } else {
            const float diff = q[j] - n[j];
            part = __fmaf_rn(diff, diff, part);
        }
    }
    return part;
}

template <int KIND>
__device__ __forceinline__ float finish_score(float sum) {
    return KIND == GE2_SELECTED_DOT ? sum : sqrtf(fmaxf(sum, kL2Floor));
}

// out[row, k] = score(chunked[row], negatives[chunk(row), selected[row, k]]); an index outside [0, N) scores 0 and sets BAD_INDEX.
// Four pairs a turn: their partial sums are folded across the warp together (6 shuffles for 4 sums instead of 20), lanes 0, 8,
// 16 and 24 end up with the totals of pairs 0, 1, 2 and 3.
template <bool VEC, int KIND>
__global__ void __launch_bounds__(kPairThreads) selected_scores_kernel(PairArgs a, float* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * kPairWarps;
    const bool hi = (lane & 16) != 0, mid = (lane & 8) != 0;
    const int my_pair = (hi ? 2 : 0) + (mid ? 1 : 0);
    for (int64_t row = (int64_t)blockIdx.x * kPairWarps + (threadIdx.x >> 5); row < a.rows; row += warps) {
        const int64_t c = row / a.R;
        float qv[4];
        load_row<VEC>(qv, a.chunked + row * a.D, lane, a.D);
        const int64_t* sel = a.selected + row * a.K;
        const float* negs = a.negatives + c * a.N * a.D;
        float* out_row = out + row * a.K;
        int64_t k = 0;
        for (; k + 4 <= a.K; k += 4) {
            float v[4];
            unsigned ok = 0u;  // one address per load for the warp: the columns and everything decided by them are warp-uniform
#pragma unroll
            for (int p = 0; p < 4; p++) {
                int64_t idx = __ldg(sel + k + p);
                if (idx >= 0 && idx < a.N) ok |= 1u << p;
                else idx = 0;  // a stand-in row for the loads; its score is dropped below
                float nv[4];
                load_row<VEC>(nv, negs + idx * a.D, lane, a.D);
                v[p] = pair_partial<KIND>(qv, nv);
            }
            const float r0 = (hi ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], 16);
            const float r1 = (hi ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], 16);
            float sum = (mid ? r1 : r0) + __shfl_xor_sync(0xffffffffu, mid ? r0 : r1, 8);
            sum += __shfl_xor_sync(0xffffffffu, sum, 4);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            if ((lane & 7) == 0) out_row[k + my_pair] = ((ok >> my_pair) & 1u) ? finish_score<KIND>(sum) : 0.f;
            if (ok != 0xFu && lane == 0) or_status(a.status, GE2_STATUS_BAD_INDEX);
        }
        for (; k < a.K; k++) {
            const int64_t idx = __ldg(sel + k);
            const bool ok = idx >= 0 && idx < a.N;
            float nv[4];
            load_row<VEC>(nv, negs + (ok ? idx : 0) * a.D, lane, a.D);
            const float sum = warp_sum(pair_partial<KIND>(qv, nv));
            if (lane == 0) {
                if (!ok) or_status(a.status, GE2_STATUS_BAD_INDEX);
                out_row[k] = ok ? finish_score<KIND>(sum) : 0.f;
            }
        }
    }
}

// grad_chunked[row] = sum_k d score / d q; grad_negatives (zeroed by the caller of the kernel) += d score / d n per pair.
// dot: dq = g n, dn = g q.  L2: dq = g (q - n) / |q - n|, dn = -dq, nothing when |q - n|^2 <= 1e-8.
template <bool VEC, int KIND>
__global__ void __launch_bounds__(kPairThreads) selected_scores_backward_kernel(PairArgs a, const float* __restrict__ grad_out,
                                                                                float* __restrict__ grad_chunked,
                                                                                float* __restrict__ grad_negatives) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * kPairWarps;
    for (int64_t row = (int64_t)blockIdx.x * kPairWarps + (threadIdx.x >> 5); row < a.rows; row += warps) {
        const int64_t c = row / a.R;
        float qv[4], acc[4] = {0.f, 0.f, 0.f, 0.f};
        load_row<VEC>(qv, a.chunked + row * a.D, lane, a.D);
        const int64_t* sel = a.selected + row * a.K;
        const float* g_row = grad_out + row * a.K;
        for (int64_t k = 0; k < a.K; k++) {
            const int64_t idx = __ldg(sel + k);
            if (idx < 0 || idx >= a.N) {  // warp-uniform
                if (lane == 0) or_status(a.status, GE2_STATUS_BAD_INDEX);
                continue;
            }
            const float g = __ldg(g_row + k);
            const int64_t n_off = (c * a.N + idx) * a.D;
            float nv[4], dn[4];
            load_row<VEC>(nv, a.negatives + n_off, lane, a.D);
            if (KIND == GE2_SELECTED_DOT) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    acc[j] = __fmaf_rn(g, nv[j], acc[j]);
                    dn[j] = g * qv[j];
                }
            } else {
                const float sq = warp_sum(pair_partial<KIND>(qv, nv));
                if (sq <= kL2Floor) continue;  // warp-uniform: every lane holds the same sum
                const float coeff = g / sqrtf(sq);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float v = coeff * (qv[j] - nv[j]);
                    acc[j] += v;
                    dn[j] = -v;
                }
            }
            add_row<VEC>(grad_negatives + n_off, dn, lane, a.D);
        }
        store_row<VEC>(grad_chunked + row * a.D, acc, lane, a.D);
    }
}

// ---------------------------------------------------------------------------------------------------------------------------
// the same with the rows that are gathered in shared memory
// ---------------------------------------------------------------------------------------------------------------------------
// A pair moves 4 D bytes; from L2 that is what bounds the kernels above (2 GB at 50 000 rows x 100 pairs, D = 100: 282 us forward, and 495 us
// backward, where every pair also sends 4 D bytes of reductions).  Here a CTA keeps what its pairs gather in shared memory:
//   scores, query gradient (pair_rows_kernel): the negatives of a chunk, in as many slices of the columns as they need to fit; the CTA's
//     rows are gone through once a slice
//   negative gradient (pair_columns_kernel): a block of query rows; its pairs are sorted by negative first (counting sort), so that a
//     negative's sum stays in registers and reaches L2 once a block instead of once a pair
// Eight lanes take a pair, 16 bytes a lane and load, four pairs a warp side by side: conflict-free whatever the pairs, and the sums of 32
// pairs fold in 7 shuffles.  Bound by shared memory (4 cycles a pair at D = 100) and the issue slots beside it (70 - 78 % of
// its cycles in use): 50 000 rows x 100 pairs, D = 100: 146 us forward, 127 + 180 us backward.
constexpr int kRowsThreads = 1024, kRowsWarps = kRowsThreads / 32;
constexpr int kPairSmem = 208 * 1024;
enum PairMode { kPairScores = 0, kPairCoeffs = 1, kPairQueryGrad = 2 };

// four columns from column c of a row of D floats, zeros past it
__device__ __forceinline__ float4 row_piece(const float* __restrict__ row, int c, int D, bool vec) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec) {
        if (c < D) v = __ldg(reinterpret_cast<const float4*>(row + c));
    } else {
        if (c < D) v.x = __ldg(row + c);
        if (c + 1 < D) v.y = __ldg(row + c + 1);
        if (c + 2 < D) v.z = __ldg(row + c + 2);
        if (c + 3 < D) v.w = __ldg(row + c + 3);
    }
    return v;
}

// mode scores: out = score of every pair.  coeffs (L2): out = grad / |q - n| (0 where the reference's gradient is).  query gradient:
// out[row] = sum_k w n (dot) or w (q - n) (L2), w = the pairs' weights (grad, or the coefficients).
// L: 16-byte pieces a lane has of a slice (W4 pieces wide, ns slices)
template <int L, int KIND, int MODE>
__global__ void __launch_bounds__(kRowsThreads, 1) pair_rows_kernel(PairArgs a, int ns, int W4, int cpc, int vec, const float* __restrict__ weights,
                                                                    float* __restrict__ out) {
    extern __shared__ __align__(16) float4 pr_tile[];  // [N][W4], then a row of zeros for pairs that do not exist
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, jl = lane & 7, g = lane >> 3;
    const int64_t c = blockIdx.x / cpc;
    const int part = (int)(blockIdx.x - c * cpc), N = (int)a.N, D = a.D, K = (int)a.K;
    const int64_t r_begin = a.R * part / cpc, r_end = a.R * (part + 1) / cpc;
    const float* negs = a.negatives + c * a.N * D;
    const uint32_t tile = (uint32_t)__cvta_generic_to_shared(pr_tile) + jl * 16;
    for (int s = 0; s < ns; s++) {
        __syncthreads();
#pragma unroll 4
        for (int i = threadIdx.x; i < N * W4; i += kRowsThreads) {
            const int j = (int)((uint32_t)i / (uint32_t)W4);
            pr_tile[i] = row_piece(negs + (int64_t)j * D, (s * W4 + i - j * W4) * 4, D, vec);
        }
        for (int i = threadIdx.x; i < W4; i += kRowsThreads) pr_tile[N * W4 + i] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
        for (int64_t r = r_begin + warp; r < r_end; r += kRowsWarps) {
            const int64_t row = c * a.R + r;
            const int64_t* sel = a.selected + row * a.K;
            float4 q[L], acc[L];
#pragma unroll
            for (int l = 0; l < L; l++) {
                acc[l] = make_float4(0.f, 0.f, 0.f, 0.f);
                q[l] = jl + 8 * l < W4 && (KIND == GE2_SELECTED_L2 || MODE != kPairQueryGrad) ? row_piece(a.chunked + row * D, (s * W4 + jl + 8 * l) * 4, D, vec) : acc[l];
            }
            // column and weight of pair k0 + lane; those of the next 32 pairs are on their way meanwhile
            int64_t next = -2;
            float next_w = 0.f;
            auto fetch = [&](int k) {
                next = -2;
                next_w = 0.f;
                if (k + lane < K) {
                    next = __ldg(sel + k + lane);
                    if (MODE == kPairQueryGrad) next_w = __ldg(weights + row * a.K + k + lane);
                }
            };
            fetch(0);
#pragma unroll 1
            for (int k0 = 0; k0 < K; k0 += 32) {
                int idx = N;
                const float w = next_w;
                if (next >= 0 && next < N) idx = (int)next;
                else if (next != -2 && s == 0) or_status(a.status, GE2_STATUS_BAD_INDEX);
                const int at0 = idx * (W4 * 16);
                fetch(k0 + 32);
                float val[8];
                auto turn = [&](int i) {
                    const uint32_t n = tile + __shfl_sync(0xffffffffu, at0, 4 * i + g);
                    const float wp = MODE == kPairQueryGrad ? __shfl_sync(0xffffffffu, w, 4 * i + g) : 0.f;
                    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int l = 0; l < L; l++) {
                        float4 x = q[l];  // (past the slice: a difference of zero, or zero)
                        if (l + 1 < L || jl + 8 * l < W4) asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(n + l * 128));
                        if (MODE == kPairQueryGrad) {
                            if (KIND == GE2_SELECTED_L2) x = make_float4(q[l].x - x.x, q[l].y - x.y, q[l].z - x.z, q[l].w - x.w);
                            acc[l].x = fmaf(wp, x.x, acc[l].x), acc[l].y = fmaf(wp, x.y, acc[l].y);
                            acc[l].z = fmaf(wp, x.z, acc[l].z), acc[l].w = fmaf(wp, x.w, acc[l].w);
                        } else if (KIND == GE2_SELECTED_DOT) {
                            sum.x = fmaf(q[l].x, x.x, sum.x), sum.y = fmaf(q[l].y, x.y, sum.y), sum.z = fmaf(q[l].z, x.z, sum.z), sum.w = fmaf(q[l].w, x.w, sum.w);
                        } else {
                            const float dx = q[l].x - x.x, dy = q[l].y - x.y, dz = q[l].z - x.z, dw = q[l].w - x.w;
                            sum.x = fmaf(dx, dx, sum.x), sum.y = fmaf(dy, dy, sum.y), sum.z = fmaf(dz, dz, sum.z), sum.w = fmaf(dw, dw, sum.w);
                        }
                    }
                    val[i] = (sum.x + sum.y) + (sum.z + sum.w);
                };
                if (K - k0 > 28) {
#pragma unroll
                    for (int i = 0; i < 8; i++) turn(i);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        val[i] = 0.f;
                        if (k0 + 4 * i < K) turn(i);  // warp-uniform
                    }
                }
                if (MODE != kPairQueryGrad) {
                    // lane jl of a group ends up with the sum of the group's pair of turn jl
#pragma unroll
                    for (int h = 4; h > 0; h >>= 1) {
#pragma unroll
                        for (int i = 0; i < h; i++) {
                            const bool up = (jl & h) != 0;
                            const float keep = up ? val[i + h] : val[i], send = up ? val[i] : val[i + h];
                            val[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
                        }
                    }
                    const int p = 4 * jl + g;
                    const bool there = __shfl_sync(0xffffffffu, idx, p) < N;
                    if (k0 + p < K) {
                        float* at = out + row * a.K + k0 + p;
                        float sum = val[0];
                        if (s > 0) sum += *at;
                        if (s == ns - 1) {
                            if (MODE == kPairScores) sum = there ? finish_score<KIND>(sum) : 0.f;
                            else sum = there && sum > kL2Floor ? __ldg(weights + row * a.K + k0 + p) / sqrtf(sum) : 0.f;
                        }
                        *at = sum;
                    }
                }
            }
            if (MODE == kPairQueryGrad) {
#pragma unroll
                for (int l = 0; l < L; l++) {
#pragma unroll
                    for (int o = 8; o < 32; o <<= 1) {
                        acc[l].x += __shfl_xor_sync(0xffffffffu, acc[l].x, o), acc[l].y += __shfl_xor_sync(0xffffffffu, acc[l].y, o);
                        acc[l].z += __shfl_xor_sync(0xffffffffu, acc[l].z, o), acc[l].w += __shfl_xor_sync(0xffffffffu, acc[l].w, o);
                    }
                    const int col = (s * W4 + jl + 8 * l) * 4;
                    if (g == 0 && jl + 8 * l < W4 && col < D) {
                        float* at = out + row * D + col;
                        if (vec) {
                            *reinterpret_cast<float4*>(at) = acc[l];
                        } else {
                            at[0] = acc[l].x;
                            if (col + 1 < D) at[1] = acc[l].y;
                            if (col + 2 < D) at[2] = acc[l].z;
                            if (col + 3 < D) at[3] = acc[l].w;
                        }
                    }
                }
            }
        }
    }
}

// out[n] += sum over the block's pairs of negative n of w q (dot) or -w (q - n) (L2)
template <int L, int KIND>
__global__ void __launch_bounds__(kRowsThreads, 1) pair_columns_kernel(PairArgs a, int cpc, int vec, const float* __restrict__ weights, float2* __restrict__ sorted,
                                                                       float* __restrict__ out) {
    extern __shared__ __align__(16) float4 pc_rows[];  // [rows of the block and a row of zeros][D4], then the counters [N]
    __shared__ int s_warp[kRowsWarps], s_base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, jl = lane & 7, g = lane >> 3;
    const int64_t c = blockIdx.x / cpc;
    const int part = (int)(blockIdx.x - c * cpc), N = (int)a.N, D = a.D, D4 = (D + 3) >> 2;
    const int64_t r_begin = a.R * part / cpc;
    const int rows = (int)(a.R * (part + 1) / cpc - r_begin);
    const int64_t row0 = c * a.R + r_begin;
    int* count = reinterpret_cast<int*>(pc_rows + (a.R / cpc + 2) * D4);
    for (int j = tid; j < N; j += kRowsThreads) count[j] = 0;
    if (tid == 0) s_base = 0;
#pragma unroll 4
    for (int i = tid; i < rows * D4; i += kRowsThreads) {
        const int r = (int)((uint32_t)i / (uint32_t)D4);
        pc_rows[i] = row_piece(a.chunked + (row0 + r) * D, (i - r * D4) * 4, D, vec);
    }
    for (int i = tid; i < D4; i += kRowsThreads) pc_rows[rows * D4 + i] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    // counting sort of the block's pairs by negative
    const int64_t p0 = row0 * a.K;
    const int pairs = rows * (int)a.K;
#pragma unroll 4
    for (int i = tid; i < pairs; i += kRowsThreads) {
        const int64_t j = __ldg(a.selected + p0 + i);
        if (j >= 0 && j < a.N) atomicAdd(&count[j], 1);
    }
    __syncthreads();
    for (int b = 0; b < N; b += kRowsThreads) {  // exclusive scan of the counters, in place
        const int own = b + tid < N ? count[b + tid] : 0;
        int incl = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        int before = s_base;
        for (int w = 0; w < warp; w++) before += s_warp[w];
        if (b + tid < N) count[b + tid] = before + incl - own;
        __syncthreads();
        if (tid == kRowsThreads - 1) s_base = before + incl;
        __syncthreads();
    }
    float2* mine = sorted + p0;  // (weight, row of the block)
#pragma unroll 4
    for (int i = tid; i < pairs; i += kRowsThreads) {
        const int64_t j = __ldg(a.selected + p0 + i);
        if (j >= 0 && j < a.N) mine[atomicAdd(&count[j], 1)] = make_float2(__ldg(weights + p0 + i), __int_as_float((int)((uint32_t)i / (uint32_t)a.K) * D4));
    }
    __syncthreads();  // (also orders the block's own global writes before the reads below)
    // count[j] is now the end of negative j's pairs, count[j - 1] their begin
    for (int j = warp; j < N; j += kRowsWarps) {
        const int begin = j == 0 ? 0 : count[j - 1], end = count[j];
        if (begin == end) continue;
        float4 acc[L], nv[L];
#pragma unroll
        for (int l = 0; l < L; l++) {
            acc[l] = make_float4(0.f, 0.f, 0.f, 0.f);
            nv[l] = KIND == GE2_SELECTED_L2 && jl + 8 * l < D4 ? row_piece(a.negatives + (c * a.N + j) * D, (jl + 8 * l) * 4, D, vec) : acc[l];
        }
#pragma unroll 1
        for (int k0 = begin; k0 < end; k0 += 32) {
            float2 e = make_float2(0.f, __int_as_float(rows * D4));
            if (k0 + lane < end) e = __ldcg(mine + k0 + lane);
            auto turn = [&](int i) {
                const float w = __shfl_sync(0xffffffffu, e.x, 4 * i + g);
                const float4* q = pc_rows + __float_as_int(__shfl_sync(0xffffffffu, e.y, 4 * i + g)) + jl;
#pragma unroll
                for (int l = 0; l < L; l++) {
                    float4 x = nv[l];  // (past the row: a difference of zero, or zero)
                    if (l + 1 < L || jl + 8 * l < D4) x = q[8 * l];
                    if (KIND == GE2_SELECTED_L2) x = make_float4(nv[l].x - x.x, nv[l].y - x.y, nv[l].z - x.z, nv[l].w - x.w);
                    acc[l].x = fmaf(w, x.x, acc[l].x), acc[l].y = fmaf(w, x.y, acc[l].y);
                    acc[l].z = fmaf(w, x.z, acc[l].z), acc[l].w = fmaf(w, x.w, acc[l].w);
                }
            };
            if (end - k0 > 28) {
#pragma unroll 4
                for (int i = 0; i < 8; i++) turn(i);
            } else {
#pragma unroll 1
                for (int i = 0; k0 + 4 * i < end; i++) turn(i);
            }
        }
        // the four groups' sums; group l then sends piece jl + 8 l
        float4 send = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int l = 0; l < L; l++) {
#pragma unroll
            for (int o = 8; o < 32; o <<= 1) {
                acc[l].x += __shfl_xor_sync(0xffffffffu, acc[l].x, o), acc[l].y += __shfl_xor_sync(0xffffffffu, acc[l].y, o);
                acc[l].z += __shfl_xor_sync(0xffffffffu, acc[l].z, o), acc[l].w += __shfl_xor_sync(0xffffffffu, acc[l].w, o);
            }
            if (g == l) send = acc[l];
        }
        const int col = (jl + 8 * g) * 4;
        if (g < L && col < D) {
            float* at = out + (c * a.N + j) * D + col;
            if (vec) {
                atomicAdd(reinterpret_cast<float4*>(at), send);
            } else {
                atomicAdd(at, send.x);
                if (col + 1 < D) atomicAdd(at + 1, send.y);
                if (col + 2 < D) atomicAdd(at + 2, send.z);
                if (col + 3 < D) atomicAdd(at + 3, send.w);
            }
        }
    }
}

// How a problem is cut for the kernels above.  possible: they can take it; taken: they do, otherwise the rows are gathered from L2.
struct PairCut {
    bool possible, taken;
    int ns, W4, L;      // slices of the negatives
    int cpc, cpc_rows;  // CTAs a chunk: negatives resident, query rows resident
    int L_rows;
};
enum PairOp { kOpScores = 0, kOpBackwardDot = 1, kOpBackwardL2 = 2 };
inline PairOp backward_op(int kind) { return kind == GE2_SELECTED_L2 ? kOpBackwardL2 : kOpBackwardDot; }

// Which form is the faster one, as an estimate of both in us: sums of what either spends its time on, fitted to both forms' times at 1 400
// shapes (1 ... 320 chunks of 20 ... 5 000 rows, 50 ... 2 500 negatives, 1 ... 500 chosen, D = 16 ... 128; 10 to 15 % off a time on average).
//   gather    a pair, and its columns; the longest warp's pairs one after the other; a row; a pair read element by element
//   resident  a wave of CTAs (chunks beyond one an SM, or that do not divide the SMs, leave some of them idle); filling shared memory once
//             a slice; a turn of the CTA's warps over a row, over 32 of its pairs, over their columns; for the negatives' gradient also a
//             block's rows and pairs (sorted, then summed) and the negatives that it goes through
// Backward, dot, gathered : resident: 7 chunks of 1 428 rows x 4 pairs, 2 310 negatives, D = 128: 11 : 84 us; 5 x 2 192 x 31, 1 980, 50: 34 : 81;
// 14 x 353 x 179, 461, 128: 107 : 74; 128 x 613 x 60, 966, 16: 322 : 159.  At 900 further shapes the form taken is 0.5 - 0.7 % behind the better
// one on average (with a line at four pairs a negative and CTA: 19 - 34 %, up to 11 times).
inline bool resident_pays(const PairArgs& a, const PairCut& p, PairOp op) {
    static constexpr double kGather[3][6] = {
        {2.7, 3.0e-5, 1.8e-7, 0.15, 1.9e-4, 4.0e-6}, {4.1, 1.94e-5, 1.83e-6, 0.20, 1.7e-4, 1.42e-5}, {4.25, 6.44e-5, 7.5e-7, 0.36, 1.9e-4, 1.97e-5}};
    static constexpr double kRows[3][5] = {{2.6, 3.7e-4, 0.99, 0.40, 0.0127}, {0.0, 7.5e-4, 0.61, 0.42, 0.0038}, {0.0, 1.34e-3, 1.48, 1.26, 0.0079}};
    static constexpr double kColumns[3][5] = {{0.0, 0.0, 0.0, 0.0, 0.0}, {9.8, 9.9e-4, 6.9e-3, 1.12e-3, 1.05e-3}, {12.5, 1.63e-3, 7.6e-3, 1.13e-3, 1.53e-3}};
    const int64_t chunks = a.rows / a.R, warps = (int64_t)kNumSMs * 8 * kPairWarps;
    const double pairs = (double)a.rows * a.K, D4 = (a.D + 3) / 4;
    const double* g = kGather[op];
    const double gather = g[0] + pairs * (g[1] + g[2] * D4 + (a.D % 4 != 0 ? g[5] : 0.0)) + g[3] * ceil_div<int64_t>(a.rows, warps) * a.K + g[4] * a.rows;
    const double turns = (double)p.ns * ceil_div<int64_t>(ceil_div<int64_t>(a.R, p.cpc), kRowsWarps);
    const double* r = kRows[op];
    double resident = ceil_div<int64_t>(chunks * p.cpc, kNumSMs) *
                      (r[0] + r[1] * p.ns * a.N * p.W4 + turns * (r[2] + r[3] * ceil_div<int64_t>(a.K, 32) + r[4] * a.K * p.L));
    const double block = (double)ceil_div<int64_t>(a.R, p.cpc_rows);
    const double* c = kColumns[op];
    resident += ceil_div<int64_t>(chunks * p.cpc_rows, kNumSMs) * (c[0] + c[2] * a.N + block * (c[1] * D4 + a.K * (c[3] + c[4] * p.L_rows)));
    return resident < gather;
}

inline PairCut pair_cut(const PairArgs& a, PairOp op) {
    PairCut p = {};
    const int64_t chunks = a.R > 0 ? a.rows / a.R : 0;
    const int D4 = (a.D + 3) / 4;
    const int64_t w4 = a.N > 0 ? kPairSmem / (16 * (a.N + 1)) : 0;
    // A slice narrower than four pieces would leave most lanes idle, and a block's pairs are counted in 31 bits.
    if (chunks < 1 || a.K < 1 || w4 < 4 || chunks > 65535 || a.K > (1 << 20) || a.R > (1 << 24)) return p;
    p.ns = (int)ceil_div<int64_t>(D4, w4);
    p.W4 = ceil_div(D4, p.ns);
    p.L = ceil_div(p.W4, 8);
    p.cpc = (int)std::max<int64_t>(1, std::min<int64_t>(kNumSMs / chunks, a.R));
    const int64_t most_rows = (kPairSmem - 4 * a.N) / (16 * D4) - 2;
    p.cpc_rows = (int)std::max<int64_t>(p.cpc, ceil_div<int64_t>(a.R, most_rows));
    p.L_rows = ceil_div(D4, 8);
    p.possible = ceil_div<int64_t>(a.R, p.cpc) * a.K < (1 << 30);
    p.taken = p.possible && resident_pays(a, p, op);
    return p;
}

// Scratch of the backward pass.  None where the rows are gathered, so that a small call costs its caller no allocation -- but where a CTA has four
// pairs a negative it is asked for all the same, as it was when that was the line: a caller may have sized its scratch once.
inline size_t pair_scratch_bytes(const PairArgs& a, const PairCut& p) {
    if (!p.possible || !(p.taken || ceil_div<int64_t>(a.R, p.cpc) * a.K >= 4 * a.N)) return 0;
    return (size_t)(a.rows * a.K) * (a.kind == GE2_SELECTED_L2 ? 12 : 8);  // sorted (weight, row) pairs; L2: the weights themselves too
}

template <int KIND, int MODE>
int launch_pair_rows(const PairArgs& a, const PairCut& p, bool vec, const float* weights, float* out, cudaStream_t stream) {
    const size_t smem = (size_t)(a.N + 1) * p.W4 * 16;
    const dim3 grid((unsigned)(a.rows / a.R * p.cpc));
    auto go = [&](auto kernel) {
        GE2_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem));
        kernel<<<grid, kRowsThreads, smem, stream>>>(a, p.ns, p.W4, p.cpc, vec ? 1 : 0, weights, out);
        GE2_LAUNCH_CHECK();
        return GE2_OK;
    };
    switch (p.L) {
        case 1: return go(pair_rows_kernel<1, KIND, MODE>);
        case 2: return go(pair_rows_kernel<2, KIND, MODE>);
        case 3: return go(pair_rows_kernel<3, KIND, MODE>);
        default: return go(pair_rows_kernel<4, KIND, MODE>);
    }
}

template <int KIND>
int launch_pair_columns(const PairArgs& a, const PairCut& p, bool vec, const float* weights, float2* sorted, float* out, cudaStream_t stream) {
    const size_t smem = (size_t)(a.R / p.cpc_rows + 2) * ((a.D + 3) / 4) * 16 + (size_t)a.N * 4;
    const dim3 grid((unsigned)(a.rows / a.R * p.cpc_rows));
    auto go = [&](auto kernel) {
        GE2_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem));
        kernel<<<grid, kRowsThreads, smem, stream>>>(a, p.cpc_rows, vec ? 1 : 0, weights, sorted, out);
        GE2_LAUNCH_CHECK();
        return GE2_OK;
    };
    switch (p.L_rows) {
        case 1: return go(pair_columns_kernel<1, KIND>);
        case 2: return go(pair_columns_kernel<2, KIND>);
        case 3: return go(pair_columns_kernel<3, KIND>);
        default: return go(pair_columns_kernel<4, KIND>);
    }
}

// ---------------------------------------------------------------------------------------------------------------------------
// tournament selection
// ---------------------------------------------------------------------------------------------------------------------------
// Scores are contracted on the tensor cores: both operands are split exactly into three bf16 terms in shared memory (x = xh + xm + xl) and
// a tile of 128 query rows x 64 negatives is xl yh + xh yl + xm ym + xm yh + xh ym + xh yh, the small products first; what is left
// out is below 2^-24 of |x y|, the sums are fp32 in tensor memory.  Two negatives with equal rows get equal scores, so ties stay ties.
//
// A CTA keeps a tile of query rows and takes a contiguous share of all (chunk, row tile, group) triples, so every SM is busy to the end and a
// share begins and ends on a group boundary.  Warps by role: 8 warps convert rows (fp32, read along the row) into one of two tile
// buffers, one issues the contractions, 8 epilogue warps in two sets walk the scores: a thread owns a row, keeps the running winner of a
// group in registers and writes it where the group ends.  The sets take the groups in turns and read a part of one at a time, at most 16 columns
// from wherever it begins, so that a column costs a compare, a select and a maximum (50 000 rows x 1 000 negatives, D = 100: groups of 10 in 102 us, of
// 1 000 in 86; 118 and
// 121 with one set that walked all columns and asked at each whether a group ends there; one set taking all groups by parts: 110 for groups of 10).
// Groups of less than five end so often that a part each, and a write of each winner to a sector of its own, costs more than that walk:
// there one set asks at every column, winners are put aside, and 17 ... 32 of the warp's 32 rows leave together, a row at a time (us, this way
// and by parts: groups of two 205 and 448, of three 176 and 299, of four 162 and 199, of five 152 and 141, of seven 136 and 117).
// Groups need not fit tiles.
// Bound by the contractions (6 ceil(D / 16) steps of 48 cycles a tile at best, 78 beside the conversion's shared-memory stores) and, with short groups, the
// writes of the winners.  As fp32 multiply-adds: 405 us.
using namespace tc;
constexpr int kTourRows = 128, kTourCols = 64, kTourPlanes = 3;
constexpr int kTourEpiWarps = 8, kTourMma = kTourEpiWarps, kTourConv0 = kTourMma + 1, kTourConvWarps = 8, kTourThreads = (kTourConv0 + kTourConvWarps) * 32;

struct TourArgs {
    const float* chunked;    // [chunks, R, D]
    const float* negatives;  // [chunks, N, D]
    int64_t R, N, K, T;      // T = N / K negatives in a group
    int64_t row_tiles, shares_total;  // shares_total = chunks * row_tiles * K groups to deal out
    int D;
    float* out_scores;       // [chunks * R, K]
    int64_t* out_idx;        // [chunks * R, K] column of the winner in its chunk
    int32_t* status;
};

template <int NB>
struct TourSmem {
    static constexpr int kQBlock = kTourRows * 128, kYBlock = kTourCols * 128;
    static constexpr int kQPlane = NB * kQBlock, kYPlane = NB * kYBlock;
    static constexpr int kQ = 0, kY = kTourPlanes * kQPlane, kStage = kY + 2 * kTourPlanes * kYPlane;
    static constexpr int kMisc = kStage + 4 * 32 * 33 * 8;  // winners put aside: per epilogue warp [32 rows][33] scores, then columns
    static constexpr int kBytes = (kMisc + 256 + 1024) > 120 * 1024 ? (kMisc + 256 + 1024) : 120 * 1024;  // one CTA an SM
};
enum TourBar { kTQFull = 0, kTQEmpty, kTYFull, kTYEmpty = kTYFull + 2, kTSFull = kTYEmpty + 2, kTSEmpty = kTSFull + 2, kTourBars = kTSEmpty + 2 };

// four consecutive columns of a row (zeros past D), read with the widest access its alignment allows
template <int VEC>
__device__ __forceinline__ float4 tour_load(const float* __restrict__ row, int c, int D, bool there) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (VEC == 4) {
        if (there && c < D) v = __ldg(reinterpret_cast<const float4*>(row + c));
    } else if (VEC == 2) {
        float2 x = make_float2(0.f, 0.f), y = x;
        if (there && c < D) x = __ldg(reinterpret_cast<const float2*>(row + c));
        if (there && c + 2 < D) y = __ldg(reinterpret_cast<const float2*>(row + c + 2));
        v = make_float4(x.x, x.y, y.x, y.y);
    } else {
        if (there && c < D) v.x = __ldg(row + c);
        if (there && c + 1 < D) v.y = __ldg(row + c + 1);
        if (there && c + 2 < D) v.z = __ldg(row + c + 2);
        if (there && c + 3 < D) v.w = __ldg(row + c + 3);
    }
    return v;
}

// one CTA's walk over its share: segments of (chunk, row tile) with a run of groups each
struct TourSegment {
    int64_t chunk, row0, col, col_end, group;  // columns [col, col_end) of the chunk, the first of them the first of `group`
};
__device__ __forceinline__ bool tour_segment(const TourArgs& a, int64_t at, int64_t end, TourSegment& s, int64_t& next) {
    if (at >= end) return false;
    const int64_t item = at / a.K, g = at - item * a.K;
    int64_t g_end = g + (end - at) < a.K ? g + (end - at) : a.K;
    const int64_t most = a.T < (1 << 29) ? (1 << 29) / a.T : 1;  // columns of a segment are counted in 32 bits
    if (g_end - g > most) g_end = g + most;
    s.chunk = item / a.row_tiles;
    s.row0 = (item - s.chunk * a.row_tiles) * kTourRows;
    s.group = g;
    s.col = g * a.T;
    s.col_end = g_end * a.T;
    next = at + (g_end - g);
    return true;
}

template <int NB, int VEC, bool STAGED>
__global__ void __launch_bounds__(kTourThreads, 1) tournament_kernel(const __grid_constant__ TourArgs a) {
    using SM = TourSmem<NB>;
    extern __shared__ unsigned char tour_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)tour_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + SM::kMisc);
    uint32_t* s_tmem = (uint32_t*)(smem + SM::kMisc + kTourBars * 8);
    volatile int* s_abort = (volatile int*)(smem + SM::kMisc + kTourBars * 8 + 4);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t begin = a.shares_total * blockIdx.x / gridDim.x, end = a.shares_total * (blockIdx.x + 1) / gridDim.x;
    auto spin_wait = [&](int bar, uint32_t parity) { return warp_spin_wait(&bars[bar], parity, s_abort, a.status); };
    auto warp_wait = [&](int bar, uint32_t parity) { return warp_pipe_wait(&bars[bar], parity, s_abort, a.status); };
    if (tid == 0) {
        mbar_init(&bars[kTQFull], kTourConvWarps);
        mbar_init(&bars[kTQEmpty], 1);
        for (int k = 0; k < 2; k++) {
            mbar_init(&bars[kTYFull + k], kTourConvWarps);
            mbar_init(&bars[kTYEmpty + k], 1);
            mbar_init(&bars[kTSFull + k], 1);
            mbar_init(&bars[kTSEmpty + k], STAGED ? 4 : kTourEpiWarps);
        }
        *s_abort = 0;
        mbar_init_fence();
    }
    if (warp == kTourMma) {
        tmem_alloc(s_tmem, 128);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;

    if (warp >= kTourConv0) {
        // ---- rows -> three bf16 planes, 128-byte-swizzled; a warp takes eight consecutive rows at a time ----
        const int cw = warp - kTourConv0, D = a.D, c = lane * 4;
        auto convert8 = [&](const float* base, int64_t valid, unsigned char* tile, int plane_bytes, int block_bytes, int r0) {
            float4 v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = tour_load<VEC>(base + (int64_t)(r0 + k) * D, c, D, r0 + k < valid);
            if (NB == 1 && lane >= 16) return;
            unsigned char* at0 = tile + (lane >> 4) * block_bytes + r0 * 128 + (lane & 1) * 8;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                unsigned char* at = at0 + k * 128 + ((((lane & 15) >> 1) ^ k) << 4);  // r0 is a multiple of 8: k = row % 8
#pragma unroll
                for (int p = 0; p < kTourPlanes; p++) {
                    const __nv_bfloat162 lo = __floats2bfloat162_rn(v[k].x, v[k].y), hi = __floats2bfloat162_rn(v[k].z, v[k].w);
                    const uint2 pk = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
                    *reinterpret_cast<uint2*>(at + p * plane_bytes) = pk;
                    v[k].x -= __uint_as_float(pk.x << 16), v[k].y -= __uint_as_float(pk.x & 0xffff0000u);
                    v[k].z -= __uint_as_float(pk.y << 16), v[k].w -= __uint_as_float(pk.y & 0xffff0000u);
                }
            }
        };
        uint32_t items = 0, tiles = 0;
        TourSegment sg;
        bool ok = true;
        for (int64_t at = begin, next = 0; ok && tour_segment(a, at, end, sg, next); at = next, items++) {
            ok = warp_wait(kTQEmpty, (items & 1) ^ 1);
            if (!ok) break;
#pragma unroll 1
            for (int r = 0; r < 2; r++)
                convert8(a.chunked + (sg.chunk * a.R + sg.row0) * D, a.R - sg.row0, smem + SM::kQ, SM::kQPlane, SM::kQBlock, cw * 16 + r * 8);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[kTQFull]);
            for (int64_t n0 = sg.col; n0 < sg.col_end; n0 += kTourCols, tiles++) {
                const int b = tiles & 1;
                ok = warp_wait(kTYEmpty + b, ((tiles >> 1) & 1) ^ 1);
                if (!ok) break;
                convert8(a.negatives + (sg.chunk * a.N + n0) * D, sg.col_end - n0, smem + SM::kY + b * kTourPlanes * SM::kYPlane, SM::kYPlane, SM::kYBlock, cw * 8);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars[kTYFull + b]);
            }
        }
    } else if (warp == kTourMma) {
        constexpr uint32_t kIdesc = idesc_bf16(kTourRows, kTourCols, 0, 0);
        constexpr uint32_t kFirst = 2 | 0 << 2 | 1 << 4 | 1 << 6 | 0 << 8 | 0 << 10, kSecond = 0 | 2 << 2 | 1 << 4 | 0 << 6 | 1 << 8 | 0 << 10;
        const uint32_t dQ = desc_lo_sw128(smem_u32(smem + SM::kQ), 16), dY0 = desc_lo_sw128(smem_u32(smem + SM::kY), 16);
        const int KS = (a.D + kMmaK - 1) / kMmaK;
        uint32_t items = 0, tiles = 0;
        TourSegment sg;
        bool ok = true;
        with_steps<NB>(KS, [&](auto steps) {
            for (int64_t at = begin, next = 0; ok && tour_segment(a, at, end, sg, next); at = next, items++) {
                ok = spin_wait(kTQFull, items & 1);
                if (!ok) break;
                for (int64_t n0 = sg.col; n0 < sg.col_end; n0 += kTourCols, tiles++) {
                    const int b = tiles & 1;
                    const uint32_t use = (tiles >> 1) & 1;
                    ok = spin_wait(kTYFull + b, use) && spin_wait(kTSEmpty + b, use ^ 1);
                    if (!ok) break;
                    tc_fence_after();
    #pragma unroll 1
                    for (int p = 0; p < 6; p++) {
                        const uint32_t da = dQ + ((kFirst >> (2 * p)) & 3) * (SM::kQPlane >> 4),
                                       db = dY0 + (b * kTourPlanes + ((kSecond >> (2 * p)) & 3)) * (SM::kYPlane >> 4);
                        mma_kmajor<steps, SM::kQBlock, SM::kYBlock>(tmem + b * kTourCols, da, db, kIdesc, p > 0 ? 1u : 0u);
                    }
                    mma_commit_warp(&bars[kTYEmpty + b]);
                    if (n0 + kTourCols >= sg.col_end) mma_commit_warp(&bars[kTQEmpty]);
                    mma_commit_warp(&bars[kTSFull + b]);  // last: whoever waits for it has seen the others' arrivals land before the CTA exits
                }
            }
        });
    } else if (warp < (STAGED ? 4 : kTourEpiWarps)) {
        // ---- winners: thread = row; columns in order, the running winner of the group in registers ----
        const int quarter = warp & 3, set = warp >> 2;
        const uint32_t lane_sel = (uint32_t)(quarter * 32) << 16;
        uint32_t tiles = 0;
        TourSegment sg;
        bool ok = true;
        for (int64_t at = begin, next = 0; ok && tour_segment(a, at, end, sg, next); at = next) {
            const int rows = (int)(a.R - sg.row0 - quarter * 32 < 32 ? a.R - sg.row0 - quarter * 32 : 32);  // of this warp
            const int64_t first = (sg.chunk * a.R + sg.row0 + quarter * 32) * a.K + sg.group;
            const int T = (int)a.T;
            int todo = (int)((sg.col_end - sg.col) / a.T);  // groups of this segment still to be written; columns are counted from its first
            float best = -CUDART_INF_F;
            int best_c = 0;
            if (!STAGED) {
                // Two sets of four warps take the groups in turns, a part of one at a time, 16 columns at most; a part that ends the tile is read
                // with the columns before it, which lie in the tile.
                float* out_s = a.out_scores + first + lane * a.K + set;
                int64_t* out_i = a.out_idx + first + lane * a.K + set;
                int g_begin = set < todo ? set * T : INT_MAX, g_end = set < todo ? g_begin + T : INT_MAX;
                best_c = g_begin;
                todo -= set;
                for (int64_t n0 = sg.col; n0 < sg.col_end; n0 += kTourCols, tiles++) {
                    const int b = tiles & 1, rel = (int)(n0 - sg.col), cols = (int)(sg.col_end - n0 < kTourCols ? sg.col_end - n0 : kTourCols);
                    ok = warp_wait(kTSFull + b, (tiles >> 1) & 1);
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll 1
                    for (int c = max(g_begin - rel, 0); c < cols;) {
                        const int c0 = min(c, kTourCols - 16), stop = min(min(cols, g_end - rel), c0 + 16);
                        float v[16];
                        tmem_ld_32x16(tmem + b * kTourCols + c0 + lane_sel, v);
                        if (stop - c < 16) {
#pragma unroll
                            for (int j = 0; j < 16; j++) v[j] = j >= c - c0 && j < stop - c0 ? v[j] : -CUDART_INF_F;
                        }
#pragma unroll
                        for (int j = 0; j < 16; j++) {
                            best_c = v[j] > best ? rel + c0 + j : best_c;  // the first of equal scores wins, a NaN never
                            best = fmaxf(best, v[j]);
                        }
                        c = stop;
                        if (rel + c == g_end) {
                            if (lane < rows) {
                                *out_s = best;
                                *out_i = sg.col + best_c;
                            }
                            out_s += 2;
                            out_i += 2;
                            todo -= 2;
                            g_begin = todo > 0 ? g_end + T : INT_MAX;
                            g_end = todo > 0 ? g_begin + T : INT_MAX;
                            best = -CUDART_INF_F;
                            best_c = g_begin;
                            c = g_begin - rel;
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars[kTSEmpty + b]);
                }
                continue;
            }
            // groups of a few columns: straight-line and predicated, since with one warp a scheduler a branch per column leaves it waiting for
            // latencies (81 cycles a column)
            float* const st_s = reinterpret_cast<float*>(smem + SM::kStage) + warp * (32 * 33 * 2);
            int* const st_c = reinterpret_cast<int*>(st_s) + 32 * 33;
            int cnt = 0, done = 0;  // winners put aside, and written
            auto flush = [&]() {
                __syncwarp();
#pragma unroll 4
                for (int r = 0; r < rows; r++) {
                    if (lane < cnt) {
                        a.out_scores[first + r * a.K + done + lane] = st_s[r * 33 + lane];
                        a.out_idx[first + r * a.K + done + lane] = sg.col + st_c[r * 33 + lane];
                    }
                }
                __syncwarp();
                done += cnt;
                cnt = 0;
            };
            int left = T;  // columns from the current position to the end of the group
            for (int64_t n0 = sg.col; n0 < sg.col_end; n0 += kTourCols, tiles++) {
                const int b = tiles & 1;
                ok = warp_wait(kTSFull + b, (tiles >> 1) & 1);
                if (!ok) break;
                tc_fence_after();
#pragma unroll 1
                for (int k = 0; k < kTourCols; k += 16) {
                    float v[16];
                    tmem_ld_32x16(tmem + b * kTourCols + k + lane_sel, v);
                    if (k == kTourCols - 16) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&bars[kTSEmpty + b]);
                    }
                    const int col0 = (int)(n0 - sg.col) + k;
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        best_c = v[j] > best ? col0 + j : best_c;
                        best = fmaxf(best, v[j]);
                        const bool end = left == j + 1;  // the same for all threads
                        const bool put = end && todo > 0;
                        if (put) {
                            st_s[lane * 33 + cnt] = best;
                            st_c[lane * 33 + cnt] = best_c;
                        }
                        cnt += put ? 1 : 0;
                        todo -= end ? 1 : 0;
                        best = end ? -CUDART_INF_F : best;
                        best_c = end ? col0 + j + 1 : best_c;
                        left += end ? T : 0;
                    }
                    left -= 16;
                    if (cnt > 16) flush();
                }
            }
            if (ok) flush();
        }
    }
    // ---- common exit ----
    tc_fence_before();
    __syncthreads();
    if (warp == kTourMma) {
        tc_fence_after();
        tmem_dealloc(tmem, 128);
    }
}

template <int NB, int VEC>
int launch_tournament(const TourArgs& a, cudaStream_t stream) {
    // per-device function attribute; setting it on every call keeps multi-device processes correct and is not a stream operation
    auto kernel = a.T < 5 ? tournament_kernel<NB, VEC, true> : tournament_kernel<NB, VEC, false>;
    GE2_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TourSmem<NB>::kBytes));
    kernel<<<(unsigned)std::min<int64_t>(kNumSMs, a.shares_total), kTourThreads, TourSmem<NB>::kBytes, stream>>>(a);
    GE2_LAUNCH_CHECK();
    return GE2_OK;
}

int check_pairs(int kind, const void* chunked, const void* negatives, const void* selected, int64_t chunks, int64_t rows_per_chunk,
                int64_t num_negs, int64_t num_selected, int D) {
    if (kind != GE2_SELECTED_DOT && kind != GE2_SELECTED_L2) return GE2_ERR_INVALID_ARGUMENT;
    if (chunks < 0 || rows_per_chunk < 0 || num_negs <= 0 || num_selected < 0 || D <= 0) return GE2_ERR_INVALID_ARGUMENT;
    if (D > kMaxD) return GE2_ERR_UNSUPPORTED;
    if (chunks * rows_per_chunk * num_selected > 0 && (chunked == nullptr || negatives == nullptr || selected == nullptr)) return GE2_ERR_INVALID_ARGUMENT;
    return GE2_OK;
}

// 16-byte accesses to rows: D a multiple of 4 and every table that is touched 16-byte aligned
bool rows_are_vectors(int D, const void* p0, const void* p1, const void* p2, const void* p3) {
    return (D & 3) == 0 && (((uintptr_t)p0 | (uintptr_t)p1 | (uintptr_t)p2 | (uintptr_t)p3) & 15) == 0;
}

PairArgs pair_args(int kind, const float* chunked, const float* negatives, const int64_t* selected, int64_t chunks, int64_t rows_per_chunk,
                   int64_t num_negs, int64_t num_selected, int D, int32_t* status) {
    PairArgs a;
    a.chunked = chunked;
    a.negatives = negatives;
    a.selected = selected;
    a.rows = chunks * rows_per_chunk;
    a.R = rows_per_chunk;
    a.N = num_negs;
    a.K = num_selected;
    a.D = D;
    a.kind = kind;
    a.status = status;
    return a;
}

}  // namespace
}  // namespace ge2

using namespace ge2;

extern "C" int ge2_selected_neg_scores(int kind, const float* chunked, const float* negatives, const int64_t* selected, int64_t chunks,
                                       int64_t rows_per_chunk, int64_t num_negs, int64_t num_selected, int D, float* out_scores,
                                       int32_t* status, ge2_stream_t stream_) {
    const int rc = check_pairs(kind, chunked, negatives, selected, chunks, rows_per_chunk, num_negs, num_selected, D);
    if (rc != GE2_OK) return rc;
    const int64_t rows = chunks * rows_per_chunk;
    if (rows * num_selected == 0) return GE2_OK;
    if (out_scores == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    const PairArgs a = pair_args(kind, chunked, negatives, selected, chunks, rows_per_chunk, num_negs, num_selected, D, status);
    const bool vec = rows_are_vectors(D, chunked, negatives, nullptr, nullptr);
    const PairCut cut = pair_cut(a, kOpScores);
    if (cut.taken)
        return kind == GE2_SELECTED_DOT ? launch_pair_rows<GE2_SELECTED_DOT, kPairScores>(a, cut, vec, nullptr, out_scores, as_stream(stream_))
                                        : launch_pair_rows<GE2_SELECTED_L2, kPairScores>(a, cut, vec, nullptr, out_scores, as_stream(stream_));
    const dim3 grid((unsigned)stream_grid(rows, kPairWarps));
    cudaStream_t stream = as_stream(stream_);
    if (kind == GE2_SELECTED_DOT) {
        if (vec) selected_scores_kernel<true, GE2_SELECTED_DOT><<<grid, kPairThreads, 0, stream>>>(a, out_scores);
        else selected_scores_kernel<false, GE2_SELECTED_DOT><<<grid, kPairThreads, 0, stream>>>(a, out_scores);
    } else {
        if (vec) selected_scores_kernel<true, GE2_SELECTED_L2><<<grid, kPairThreads, 0, stream>>>(a, out_scores);
        else selected_scores_kernel<false, GE2_SELECTED_L2><<<grid, kPairThreads, 0, stream>>>(a, out_scores);
    }
    GE2_LAUNCH_CHECK();
    return GE2_OK;
}

extern "C" int ge2_selected_neg_scores_backward(int kind, const float* grad_out, const float* chunked, const float* negatives,
                                                const int64_t* selected, int64_t chunks, int64_t rows_per_chunk, int64_t num_negs,
                                                int64_t num_selected, int D, float* grad_chunked, float* grad_negatives, int32_t* status,
                                                ge2_stream_t stream) {
    return ge2_selected_neg_scores_backward_ws(kind, grad_out, chunked, negatives, selected, chunks, rows_per_chunk, num_negs, num_selected, D,
                                               grad_chunked, grad_negatives, status, nullptr, 0, stream);
}

extern "C" size_t ge2_selected_neg_backward_workspace_bytes(int kind, int64_t chunks, int64_t rows_per_chunk, int64_t num_negs, int64_t num_selected, int D) {
    if (chunks <= 0 || rows_per_chunk <= 0 || num_negs <= 0 || num_selected <= 0 || D <= 0 || D > kMaxD) return 0;
    const PairArgs a = pair_args(kind, nullptr, nullptr, nullptr, chunks, rows_per_chunk, num_negs, num_selected, D, nullptr);
    return pair_scratch_bytes(a, pair_cut(a, backward_op(kind)));
}

extern "C" int ge2_selected_neg_scores_backward_ws(int kind, const float* grad_out, const float* chunked, const float* negatives,
                                                   const int64_t* selected, int64_t chunks, int64_t rows_per_chunk, int64_t num_negs,
                                                   int64_t num_selected, int D, float* grad_chunked, float* grad_negatives, int32_t* status,
                                                   void* workspace, size_t workspace_bytes, ge2_stream_t stream_) {
    const int rc = check_pairs(kind, chunked, negatives, selected, chunks, rows_per_chunk, num_negs, num_selected, D);
    if (rc != GE2_OK) return rc;
    const int64_t rows = chunks * rows_per_chunk;
    cudaStream_t stream = as_stream(stream_);
    if (chunks > 0) {
        if (grad_negatives == nullptr) return GE2_ERR_INVALID_ARGUMENT;
        GE2_CUDA_TRY(cudaMemsetAsync(grad_negatives, 0, (size_t)(chunks * num_negs * D) * sizeof(float), stream));
    }
    if (rows == 0) return GE2_OK;
    if (grad_chunked == nullptr || (num_selected > 0 && grad_out == nullptr)) return GE2_ERR_INVALID_ARGUMENT;
    // with nothing selected the kernel still writes the zero query gradient
    const PairArgs a = pair_args(kind, chunked, negatives, selected, chunks, rows_per_chunk, num_negs, num_selected, D, status);
    const bool vec = rows_are_vectors(D, chunked, negatives, grad_chunked, grad_negatives);
    const PairCut cut = pair_cut(a, backward_op(kind));
    if (cut.taken && workspace != nullptr && workspace_bytes >= pair_scratch_bytes(a, cut) && ((uintptr_t)workspace & 7) == 0) {
        float2* sorted = reinterpret_cast<float2*>(workspace);
        float* coeffs = reinterpret_cast<float*>(sorted + rows * num_selected);
        if (kind == GE2_SELECTED_DOT) {
            const int rc2 = launch_pair_rows<GE2_SELECTED_DOT, kPairQueryGrad>(a, cut, vec, grad_out, grad_chunked, stream);
            return rc2 != GE2_OK ? rc2 : launch_pair_columns<GE2_SELECTED_DOT>(a, cut, vec, grad_out, sorted, grad_negatives, stream);
        }
        int rc2 = launch_pair_rows<GE2_SELECTED_L2, kPairCoeffs>(a, cut, vec, grad_out, coeffs, stream);
        if (rc2 == GE2_OK) rc2 = launch_pair_rows<GE2_SELECTED_L2, kPairQueryGrad>(a, cut, vec, coeffs, grad_chunked, stream);
        return rc2 != GE2_OK ? rc2 : launch_pair_columns<GE2_SELECTED_L2>(a, cut, vec, coeffs, sorted, grad_negatives, stream);
    }
    const dim3 grid((unsigned)stream_grid(rows, kPairWarps));
    if (kind == GE2_SELECTED_DOT) {
        if (vec) selected_scores_backward_kernel<true, GE2_SELECTED_DOT><<<grid, kPairThreads, 0, stream>>>(a, grad_out, grad_chunked, grad_negatives);
        else selected_scores_backward_kernel<false, GE2_SELECTED_DOT><<<grid, kPairThreads, 0, stream>>>(a, grad_out, grad_chunked, grad_negatives);
    } else {
        if (vec) selected_scores_backward_kernel<true, GE2_SELECTED_L2><<<grid, kPairThreads, 0, stream>>>(a, grad_out, grad_chunked, grad_negatives);
        else selected_scores_backward_kernel<false, GE2_SELECTED_L2><<<grid, kPairThreads, 0, stream>>>(a, grad_out, grad_chunked, grad_negatives);
    }
    GE2_LAUNCH_CHECK();
    return GE2_OK;
}

extern "C" int ge2_tournament_select(const float* selector_chunked, const float* selector_negatives, const float* score_chunked,
                                     const float* score_negatives, int64_t chunks, int64_t rows_per_chunk, int64_t num_negs,
                                     int64_t num_selected, int D, float* out_scores, int64_t* out_idx, ge2_stream_t stream_) {
    if (chunks < 0 || rows_per_chunk < 0 || num_negs <= 0 || num_selected <= 0 || D <= 0) return GE2_ERR_INVALID_ARGUMENT;
    if (num_negs % num_selected != 0) return GE2_ERR_INVALID_ARGUMENT;  // the reference's TORCH_CHECK
    if (D > kMaxD || chunks > 65535) return GE2_ERR_UNSUPPORTED;
    if (chunks * rows_per_chunk == 0) return GE2_OK;
    if (selector_chunked == nullptr || selector_negatives == nullptr || out_scores == nullptr || out_idx == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    if (score_chunked == nullptr) score_chunked = selector_chunked;
    if (score_negatives == nullptr) score_negatives = selector_negatives;
    cudaStream_t stream = as_stream(stream_);

    if (num_negs / num_selected > (1 << 30)) return GE2_ERR_UNSUPPORTED;
    TourArgs a;
    a.chunked = selector_chunked;
    a.negatives = selector_negatives;
    a.R = rows_per_chunk;
    a.N = num_negs;
    a.K = num_selected;
    a.T = num_negs / num_selected;
    a.D = D;
    a.row_tiles = ceil_div<int64_t>(rows_per_chunk, kTourRows);
    a.shares_total = chunks * a.row_tiles * num_selected;
    a.out_scores = out_scores;
    a.out_idx = out_idx;
    a.status = nullptr;
    const uintptr_t mis = (uintptr_t)(D * 4) | (uintptr_t)selector_chunked | (uintptr_t)selector_negatives;
    const int vec = (mis & 15) == 0 ? 4 : (mis & 7) == 0 ? 2 : 1;
    const int rc = D <= 64 ? (vec == 4 ? launch_tournament<1, 4>(a, stream) : vec == 2 ? launch_tournament<1, 2>(a, stream) : launch_tournament<1, 1>(a, stream))
                           : (vec == 4 ? launch_tournament<2, 4>(a, stream) : vec == 2 ? launch_tournament<2, 2>(a, stream) : launch_tournament<2, 1>(a, stream));
    if (rc != GE2_OK) return rc;
    if (score_chunked != selector_chunked || score_negatives != selector_negatives) {
        // a selector separate from the scorer: the winners are scored again with the scorer's rows
        return ge2_selected_neg_scores(GE2_SELECTED_DOT, score_chunked, score_negatives, out_idx, chunks, rows_per_chunk, num_negs, num_selected,
                                       D, out_scores, nullptr, stream_);
    }
    return GE2_OK;
}
