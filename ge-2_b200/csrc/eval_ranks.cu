// Link-prediction evaluation: the rank of every test edge among ALL candidate nodes, both corruption sides, with the
// reference's filter semantics (a filtered score is replaced by -1e9 before the comparison).
//
// Follows, in the reference project (paths relative to gege/src/cpp/src):
//   scores   nn/decoders/edge/decoder_methods.cpp:597-659 (node_corrupt_forward: relation-adjusted source against the
//            destination and against every negative; the inverse relation applied to the destination against the sources),
//            relation operators nn/decoders/edge/relation_operators.cpp:3-31
//   filter   data/samplers/negative.cpp:421-575 (pairs (edge row, negative column) whose score becomes -1e9);
//            filtered evaluation uses one chunk holding every node (negative.cpp:585-589)
//   ranks    reporting/reporting.cpp:52-54: rank = #(negative score >= positive score) + 1
//
// A score is DEFINED as the chain acc = fma(q[d], e[d], acc), d ascending, in fp32 -- the positive's, a candidate's, a filter
// pair's -- so that "the candidate is the positive's own node" compares equal and the correction for a filter pair undoes exactly
// what the counting pass counted.  Counting by evaluating two thousand million such chains took 18.5 ms for 1 000 edges of a
// 1 M-node graph (D = 100), 0.29 of the fp32 rate; but almost every comparison is decided long before its last bit.  So the
// counting pass computes every score on the tensor cores, together with a bound on how far it can be from the chain's value, counts
// what is decided, and evaluates the chain itself only for candidates within the bound of the positive's score (a few in ten
// thousand): the same ranks, bit for bit.  The [B x nodes] score matrix is never stored.
#include <algorithm>

#include <cuda_fp16.h>

#include "tc_pipe.cuh"

namespace ge2 {
namespace {

using namespace tc;

constexpr int kMaxD = 128;
constexpr int kTileQ = 128;       // query rows of a score tile
constexpr int kTileN = 256;       // candidates of a score tile
constexpr int kGroupTiles = 16;   // most query tiles of a group
constexpr int kAccs = 2;          // score accumulators in tensor memory
constexpr int kCountThreads = 896, kTmaWarp = 0, kMmaWarp = 1, kCopyWarp = 2, kEpiWarp0 = 4, kEpiWarps = 16, kConvWarp0 = 20, kConvWarps = 8;
constexpr int kConvRows = kTileN / kConvWarps, kConvBatch = 8;
constexpr int kListCap = 64;      // undecided candidates a warp collects before it hands 32 of them on
constexpr int kPrepRows = 32, kPrepThreads = 256;
constexpr int kSettleThreads = 128;

struct EvalArgs {
    ge2_eval_desc d;
    float* Q;                     // [S][Bp][D] relation-adjusted query rows
    __half* Qsplit;               // [2][S * Bp][ld] the same, divided by qinv, as a sum of two fp16 terms (the second holds what the first leaves)
    float* qinv;                  // [S][Bp] a power of two: the row's largest element divided by it is near 2^8
    float* pos;                   // [S][Bp] positive scores; +inf for rows without a rank
    float* qnorm;                 // [S][Bp] 2-norm of the query rows, rounded up (infinity: decide nothing); -1 for rows without a rank (padding, bad ids)
    unsigned long long* hash;     // open-addressing set of filter pairs already applied (keys are pair + 1, 0 = empty)
    int64_t hash_slots;           // power of two
    uint2* open_list;             // (query row, candidate column) of comparisons the counting pass left open
    unsigned long long* open_count;  // how many were put there (may exceed open_cap: the rest was evaluated in place)
    int64_t open_cap;
    unsigned char* stage;         // D > 64: [kNumSMs] split candidate tiles on their way into shared memory; null: no room for them
    int64_t Bp;
    int S, ld;
    int vec;                      // floats per access to a candidate row: 4 or 2 (rows aligned and whole), else 1
};

__device__ __forceinline__ const float* node_row(const ge2_eval_desc& d, int64_t col) {
    const int64_t id = d.neg_ids != nullptr ? __ldg(d.neg_ids + col) : col;
    if (id < 0 || id >= d.num_nodes) return nullptr;
    return d.node_emb + id * d.emb_stride;
}

// the score as it is defined: one fma after the other, d ascending
__device__ __forceinline__ float score_chain(const float* __restrict__ q, const float* __restrict__ e, int D, int vec) {
    float acc = 0.f;
    if (vec == 4) {
#pragma unroll 5
        for (int k = 0; k < D / 4; k++) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(q) + k), b = __ldg(reinterpret_cast<const float4*>(e) + k);
            acc = __fmaf_rn(a.x, b.x, acc);
            acc = __fmaf_rn(a.y, b.y, acc);
            acc = __fmaf_rn(a.z, b.z, acc);
            acc = __fmaf_rn(a.w, b.w, acc);
        }
    } else if (vec == 2) {
#pragma unroll 5
        for (int k = 0; k < D / 2; k++) {
            const float2 a = __ldg(reinterpret_cast<const float2*>(q) + k), b = __ldg(reinterpret_cast<const float2*>(e) + k);
            acc = __fmaf_rn(a.x, b.x, acc);
            acc = __fmaf_rn(a.y, b.y, acc);
        }
    } else {
#pragma unroll 8
        for (int k = 0; k < D; k++) acc = __fmaf_rn(__ldg(q + k), __ldg(e + k), acc);
    }
    return acc;
}

// the same with more loads on their way (and more registers than a call out of the counting pass can have)
__device__ __forceinline__ float score_chain_ahead(const float* __restrict__ q, const float* __restrict__ e, int D, int vec) {
    float acc = 0.f;
    if (vec == 4) {
        constexpr int kAhead = 7;
        const int n = D / 4;
#pragma unroll 1
        for (int k0 = 0; k0 < n; k0 += kAhead) {  // loads of a round are on their way together, those of the last one too
            float4 x[kAhead], y[kAhead];
#pragma unroll
            for (int k = 0; k < kAhead; k++)
                if (k0 + k < n) x[k] = __ldg(reinterpret_cast<const float4*>(q) + k0 + k), y[k] = __ldg(reinterpret_cast<const float4*>(e) + k0 + k);
#pragma unroll
            for (int k = 0; k < kAhead; k++)
                if (k0 + k < n) {
                    acc = __fmaf_rn(x[k].x, y[k].x, acc);
                    acc = __fmaf_rn(x[k].y, y[k].y, acc);
                    acc = __fmaf_rn(x[k].z, y[k].z, acc);
                    acc = __fmaf_rn(x[k].w, y[k].w, acc);
                }
        }
    } else if (vec == 2) {
        constexpr int kAhead = 9;
        const int n = D / 2;
#pragma unroll 1
        for (int k0 = 0; k0 < n; k0 += kAhead) {
            float2 x[kAhead], y[kAhead];
#pragma unroll
            for (int k = 0; k < kAhead; k++)
                if (k0 + k < n) x[k] = __ldg(reinterpret_cast<const float2*>(q) + k0 + k), y[k] = __ldg(reinterpret_cast<const float2*>(e) + k0 + k);
#pragma unroll
            for (int k = 0; k < kAhead; k++)
                if (k0 + k < n) {
                    acc = __fmaf_rn(x[k].x, y[k].x, acc);
                    acc = __fmaf_rn(x[k].y, y[k].y, acc);
                }
        }
    } else {
#pragma unroll 8
        for (int k = 0; k < D; k++) acc = __fmaf_rn(__ldg(q + k), __ldg(e + k), acc);
    }
    return acc;
}

// a power of two p with p * x in [2^8, 2^9) (1 for x = 0 and where none is a normal number; inf and NaN leave everything undecided anyway)
__device__ __forceinline__ float pow2_near_256(float x) {
    const int e = 127 + 8 + 127 - (int)((__float_as_uint(x) >> 23) & 255u);
    return x > 0.f && e >= 1 && e <= 254 ? __uint_as_float((uint32_t)e << 23) : 1.f;
}

// Query rows, positive scores, rank = 1.  32 rows per CTA: the threads share out the (row, column) pairs, so that a row is read along
// its columns and all loads of a CTA are in flight together; the rows meet in shared memory, and one lane per row walks the positive
// score's chain there.  (A thread per row reading global memory on its own took 45 us for 2 000 rows of D = 100.)
__global__ void __launch_bounds__(kPrepThreads) eval_prep_kernel(EvalArgs a) {
    __shared__ float sq[kPrepRows][kMaxD + 1], se[kPrepRows][kMaxD + 1];
    __shared__ float s_scale[kPrepRows];
    __shared__ int64_t s_a[kPrepRows], s_b[kPrepRows], s_r[kPrepRows];  // rows of the two endpoints and the relation; s_a < 0: no rank
    const ge2_eval_desc& d = a.d;
    const int tid = threadIdx.x;
    const int D = d.D, h = D / 2;
    const int64_t w0 = (int64_t)blockIdx.x * kPrepRows, rows = (int64_t)a.S * a.Bp;
    const int s = w0 >= a.Bp ? 1 : 0;  // Bp is a multiple of kPrepRows: a CTA's rows are of one side
    const int64_t i0 = w0 - (s ? a.Bp : 0);
    if (tid < kPrepRows) {
        const int64_t i = i0 + tid;
        bool ok = i < d.B;
        int64_t sid = 0, did = 0, rid = 0;
        if (ok) {
            sid = d.src_ids[i * d.edge_stride];
            did = d.dst_ids[i * d.edge_stride];
            if (d.has_relations) rid = d.rel_ids[i * d.rel_stride];
            ok = sid >= 0 && sid < d.num_nodes && did >= 0 && did < d.num_nodes && (!d.has_relations || (rid >= 0 && rid < d.R));
            if (!ok) or_status(d.status, GE2_STATUS_BAD_INDEX);
        }
        s_a[tid] = ok ? (s == 0 ? sid : did) : -1;  // the endpoint the relation is applied to
        s_b[tid] = s == 0 ? did : sid;              // the endpoint it is compared with
        s_r[tid] = rid;
    }
    __syncthreads();
    const float* rel = d.has_relations ? (s == 0 ? d.rel : d.inv_rel) : nullptr;
    const int col = tid & (a.ld - 1), step = kPrepThreads / a.ld;  // ld is 64 or 128: a thread keeps its column
#pragma unroll 4
    for (int lr = tid / a.ld; lr < kPrepRows; lr += step) {
        float v = 0.f;
        const int64_t ra = s_a[lr];
        if (ra >= 0 && col < D) {
            const float* ea = d.node_emb + ra * d.emb_stride;
            const float x = __ldg(ea + col);
            if (rel == nullptr) {
                v = x;
            } else {
                const float* r = rel + s_r[lr] * D;
                const float y = __ldg(r + col);
                if (d.decoder == GE2_DECODER_DISTMULT) {
                    v = __fmul_rn(x, y);
                } else {  // complex product, columns [0, h) real and [h, D) imaginary; separate roundings as the reference's tensor ops
                    const int cp = col < h ? col + h : col - h;
                    const float xp = __ldg(ea + cp), yp = __ldg(r + cp);
                    v = col < h ? __fsub_rn(__fmul_rn(x, y), __fmul_rn(xp, yp)) : __fadd_rn(__fmul_rn(xp, y), __fmul_rn(x, yp));
                }
            }
            se[lr][col] = __ldg(d.node_emb + s_b[lr] * d.emb_stride + col);
        }
        sq[lr][col] = v;
        if (col < D) a.Q[(w0 + lr) * D + col] = v;
    }
    __syncthreads();
    if (tid >= 64 && tid < 64 + kPrepRows) {
        const int lr = tid - 64;
        float most = 0.f;
        for (int k = 0; k < D; k++) most = fmaxf(most, fabsf(sq[lr][k]));
        s_scale[lr] = pow2_near_256(most);
        a.qinv[w0 + lr] = 1.f / s_scale[lr];
    }
    __syncthreads();
#pragma unroll 4
    for (int lr = tid / a.ld; lr < kPrepRows; lr += step) {
        const int64_t w = w0 + lr;
        const float v = sq[lr][col] * s_scale[lr];
        const __half hi = __float2half_rn(v);
        a.Qsplit[w * a.ld + col] = hi;
        a.Qsplit[(rows + w) * a.ld + col] = __float2half_rn(v - __half2float(hi));
    }
    if (tid < kPrepRows) {
        const bool ok = s_a[tid] >= 0;
        float acc = 0.f;
        if (ok)
            for (int k = 0; k < D; k++) acc = __fmaf_rn(sq[tid][k], se[tid][k], acc);
        a.pos[w0 + tid] = ok ? acc : INFINITY;
        const int64_t i = i0 + tid;
        if (i < d.B) {
            (s == 0 ? d.dst_ranks : d.src_ranks)[i] = ok ? 1 : 0;  // no rank for a row with bad ids
            float* out = s == 0 ? d.pos_scores : d.inv_pos_scores;
            if (out != nullptr && ok) out[i] = acc;
        }
    } else if (tid < 2 * kPrepRows) {
        const int lr = tid - kPrepRows;
        float sumsq = 0.f;
        // of the scaled row, whose largest element is 2^8 or more: squares of the row itself vanish below 2.6e-23.  A row that has no such
        // scale (zeros, elements at the end of the range, infinities and NaN) leaves everything undecided.
        for (int k = 0; k < D; k++) sumsq = fmaf(sq[lr][k] * s_scale[lr], sq[lr][k] * s_scale[lr], sumsq);
        a.qnorm[w0 + lr] = s_a[lr] < 0 ? -1.f : sumsq >= 65536.f ? sqrtf(sumsq) * 1.001f / s_scale[lr] : INFINITY;
    }
}

__device__ __forceinline__ void add_to_rank(const EvalArgs& a, int64_t w, int64_t n) {
    if (__ldg(a.qnorm + w) < 0.f) return;  // a row without a rank
    const int s = w >= a.Bp ? 1 : 0;
    const int64_t i = w - (s ? a.Bp : 0);
    atomicAdd(reinterpret_cast<unsigned long long*>((s == 0 ? a.d.dst_ranks : a.d.src_ranks) + i), (unsigned long long)n);
}

// an undecided comparison, by the score's definition
template <bool kAhead>
__device__ __forceinline__ void settle(const EvalArgs& a, uint2 what) {
    const float* e = node_row(a.d, what.y);
    // a candidate id outside the table scores 0
    const float* q = a.Q + (int64_t)what.x * a.d.D;
    const float s = e == nullptr ? 0.f : kAhead ? score_chain_ahead(q, e, a.d.D, a.vec) : score_chain(q, e, a.d.D, a.vec);
    if (s >= a.pos[what.x]) add_to_rank(a, what.x, 1);
}
__device__ __noinline__ void settle_in_place(const EvalArgs& a, uint2 what) { settle<false>(a, what); }

// fma(v, scale, shift) clamped to [0, 1]
__device__ __forceinline__ float saturated(float v, float scale, float shift) {
    float t;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(t) : "f"(v), "f"(scale), "f"(shift));
    return t;
}
// pairs of fp32 in one register pair
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float sum2(uint64_t a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
    return x + y;
}

// How the counting pass is dealt out: blockIdx.y = query group (an even share of the query tiles), blockIdx.x of gridDim.x = an even
// share of the candidate tiles.
struct CountSched {
    int q_tiles, groups;
    int64_t cand_tiles, num_cols;
    int staged;   // do CTAs convert the next candidate tile into EvalArgs::stage while one is contracted? (one CTA an SM)
    float bound;  // |score on the tensor cores - score chain| <= bound * |q| * |e| (+ underflow terms)
};

template <int NB>
struct CountSmem {
    static constexpr int kSlots = 5;                                  // ring of query blocks (128 rows x 64 columns of one term)
    static constexpr int kCandBufs = NB == 2 ? 1 : 2;                 // a candidate tile of D > 64 leaves no room for a second: it waits in global memory
    static constexpr int kCandBlock = kTileN * 128;                   // 64 columns of one term
    static constexpr int kCandBytes = 2 * NB * kCandBlock;            // one candidate tile, both terms
    static constexpr int kCand = 0;
    static constexpr int kRing = kCandBufs * kCandBytes;
    static constexpr int kCnt = kRing + kSlots * kBlockBytes;         // [query row of the group]
    static constexpr int kList = kCnt + kGroupTiles * kTileQ * 4;     // per epilogue warp: kListCap (row, column)
    static constexpr int kMisc = kList + kEpiWarps * kListCap * 8;
    static constexpr int kEnd = kMisc + 512;
    static constexpr int kBytes = kEnd + 1024;                        // 1024 bytes of slack to align the base
    static_assert(kBytes <= 227 * 1024, "counting pass exceeds the shared memory of an SM");
};
enum CountBar { kQFull = 0, kQEmpty = 8, kCFull = 16, kCEmpty = 18, kAccFull = 20, kAccEmpty = 24, kStaged = 28, kCountBars = 29 };

// #(candidates whose score is >= the positive's) for every query row.
//
// Rows are scaled by a power of two (a query by its own, candidates by one for 32 of them) and every value x is taken as h + l,
// h = fp16(x), l = fp16(x - h): |x - h - l| <= 2^-22 |x| + 2^-25, |l| <= 2^-11 |x| (the second term of the first is 2^-33 of the largest element
// and below).
// A tile of 128 queries x 256 candidates is lq he + hq le + hq he, three products on the tensor cores, the small ones first as far
// as the ring of query blocks allows.  What separates the result from the chain's value is (a) the dropped lq le and the
// remainders, 3 * 2^-22 of sum |q||e|, (b) the tensor cores' additions, at most one ulp (2^-23) of the accumulator for each of the
// 16 products and the accumulator itself in each step that meets a full-sized accumulator (ceil(D / 16) of hq he, and those of the
// second 64 columns' hq le), (c) the chain's own rounding, D * 2^-24; and sum |q||e| <= |q|_2 |e|_2.  A score further than that from
// the positive's is decided; the others go to a list, and the chain is evaluated for them afterwards.  Values that make the bound or
// the score infinite or NaN leave everything undecided.
//
// One CTA per SM, warps by role: TMA producer of query blocks, MMA issuer, 16 epilogue warps (a thread owns one query row and a
// quarter of the tile's columns: its threshold is a register), 8 warps that read candidate rows (fp32, each once per query group),
// split them and write them swizzled, and one that copies.  The candidates stay while the group's query tiles stream past: 64 KB of query
// blocks for 21 contractions of 128 x 256 x 16 (128 candidates instead of 256 left the contractions waiting for query blocks).  D <= 64:
// two candidate tiles fit.  Wider: the next one is split into global memory (128 KB a CTA, which stay in the L2) while this one is
// contracted, and comes in as four bulk copies: 6 800 cycles without a tile instead of the 15 400 of splitting it there and then, of 67 000 a tile.
// 2 000 queries x 1 M nodes, D = 100: 1.11 ms (1.17 without the staging, 18.5 as chains of fp32 multiply-adds); 600 x 200 000, D = 128: 188 us in
// all instead of 226; 2 000 queries x 14 951 nodes, D = 50: 28 us (142).  Of the first, 0.64 ms are the contractions at the clock that
// power leaves; the rest is waiting for query blocks (13 %), candidate tiles (10 %) and accumulators (9 %).
template <int NB, int VEC>
__global__ void __launch_bounds__(kCountThreads, 1)
    eval_count_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ EvalArgs a, CountSched sc) {
    using SM = CountSmem<NB>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + SM::kMisc);
    uint32_t* s_tmem = (uint32_t*)(smem + SM::kMisc + kCountBars * 8);
    volatile int* s_abort = (volatile int*)(smem + SM::kMisc + kCountBars * 8 + 4);
    // [2][kConvWarps] of the 32 candidates of a converting warp: a bound of their scaled norms, and the scale
    float2* s_cand = (float2*)(smem + SM::kMisc + kCountBars * 8 + 16);
    int* cnt = (int*)(smem + SM::kCnt);
    const ge2_eval_desc& d = a.d;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t tb = sc.cand_tiles * blockIdx.x / gridDim.x, te = sc.cand_tiles * (blockIdx.x + 1) / gridDim.x;
    const int q0 = (int)((int64_t)blockIdx.y * sc.q_tiles / sc.groups), q1 = (int)((int64_t)(blockIdx.y + 1) * sc.q_tiles / sc.groups);
    auto warp_wait = [&](int bar, uint32_t parity) { return warp_pipe_wait(&bars[bar], parity, s_abort, d.status); };
    auto spin_wait = [&](int bar, uint32_t parity) { return warp_spin_wait(&bars[bar], parity, s_abort, d.status); };

    if (warp == kTmaWarp && lane == 0) {
        for (int k = 0; k < SM::kSlots; k++) {
            mbar_init(&bars[kQFull + k], 1);
            mbar_init(&bars[kQEmpty + k], 1);
        }
        for (int k = 0; k < SM::kCandBufs; k++) {
            mbar_init(&bars[kCFull + k], kConvWarps);
            mbar_init(&bars[kCEmpty + k], 1 + kEpiWarps);  // the tile's contractions and everybody who reads its norms are done
        }
        for (int k = 0; k < kAccs; k++) {
            mbar_init(&bars[kAccFull + k], 1);
            mbar_init(&bars[kAccEmpty + k], kEpiWarps);
        }
        mbar_init(&bars[kStaged], kConvWarps);
        *s_abort = 0;
        mbar_init_fence();
        prefetch_tensormap(&tmQ);
    }
    if (warp == kMmaWarp) {
        tmem_alloc(s_tmem, 512);
        tmem_relinquish();
    }
    for (int k = tid; k < kGroupTiles * kTileQ; k += kCountThreads) cnt[k] = 0;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    griddep_wait();  // the query rows come from the kernel before this one
    const uint32_t tmem = *s_tmem;

    if (warp == kTmaWarp) {
        int slot = 0;
        uint32_t phase = 1;
        bool ok = true;
        for (int64_t t = tb; ok && t < te; t++) {
            for (int qt = q0; ok && qt < q1; qt++) {
#pragma unroll
                for (int k = 0; k < 2 * NB; k++) {  // second terms first
                    ok = ok && spin_wait(kQEmpty + slot, phase);
                    if (!ok) break;
                    mbar_expect_tx_warp(&bars[kQFull + slot], kBlockBytes);
                    tma_load_3d_warp(smem + SM::kRing + slot * kBlockBytes, &tmQ, (k % NB) * 64, qt * kTileQ, k < NB ? 1 : 0, &bars[kQFull + slot]);
                    if (++slot == SM::kSlots) slot = 0, phase ^= 1;
                }
            }
        }
    } else if (warp == kMmaWarp) {
        constexpr uint32_t kIdesc = idesc_f16(kTileQ, kTileN, 0, 0);
        const uint32_t ring = desc_lo_sw128(smem_u32(smem + SM::kRing), 16), cand = desc_lo_sw128(smem_u32(smem + SM::kCand), 16);
        constexpr uint32_t kSlotStep = kBlockBytes >> 4, kCandStep = SM::kCandBlock >> 4;
        const int KS = (d.D + kMmaK - 1) / kMmaK;
        int slot = 0;
        uint32_t phase = 0, ac = 0, cc = 0;
        bool ok = true;
        with_steps<NB>(KS, [&](auto steps) {
            for (int64_t t = tb; ok && t < te; t++, cc++) {
                const int cb = cc % SM::kCandBufs;
                if (!spin_wait(kCFull + cb, (cc / SM::kCandBufs) & 1)) break;
                const uint32_t ch = cand + cb * (2 * NB * kCandStep), cl = ch + NB * kCandStep;
                for (int qt = q0; ok && qt < q1; qt++, ac++) {
                    const int ab = ac % kAccs;
                    ok = spin_wait(kAccEmpty + ab, ((ac / kAccs) & 1) ^ 1);
                    if (!ok) break;
                    const uint32_t acc = tmem + ab * kTileN;
                    auto product = [&](uint32_t da, uint32_t db, int b, bool first) {  // one 64-column block
                        if (b < NB - 1) mma_kmajor<4, kBlockBytes, SM::kCandBlock>(acc, da, db + b * kCandStep, kIdesc, first ? 0u : 1u);
                        else mma_kmajor<steps - 4 * (NB - 1), kBlockBytes, SM::kCandBlock>(acc, da, db + b * kCandStep, kIdesc, first ? 0u : 1u);
                    };
    #pragma unroll
                    for (int k = 0; k < 2 * NB; k++) {
                        ok = ok && spin_wait(kQFull + slot, phase);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t da = ring + slot * kSlotStep;
                        if (k < NB) {
                            product(da, ch, k, k == 0);
                        } else {
                            product(da, cl, k - NB, false);
                            product(da, ch, k - NB, false);
                        }
                        mma_commit_warp(&bars[kQEmpty + slot]);
                        if (k == 2 * NB - 1) mma_commit_warp(&bars[kAccFull + ab]);
                        if (++slot == SM::kSlots) slot = 0, phase ^= 1;
                    }
                }
                if (ok) mma_commit_warp(&bars[kCEmpty + cb]);
            }
        });
        // the last arrivals that the tensor pipe makes on barriers of this CTA have landed before it can exit
        if (ok && cc > 0) spin_wait(kCEmpty + (cc - 1) % SM::kCandBufs, ((cc - 1) / SM::kCandBufs) & 1);
    } else if (warp == kCopyWarp) {
        // ---- staged candidate tiles: into shared memory as soon as it is free; the arrivals stand for those of the converting warps ----
        if (NB == 2 && sc.staged) {
            const unsigned char* stage = a.stage + (int64_t)(blockIdx.y * gridDim.x + blockIdx.x) * SM::kCandBytes;
            uint32_t cc = 1;
            for (int64_t t = tb + 1; t < te; t++, cc++) {
                if (!spin_wait(kStaged, (cc - 1) & 1) || !spin_wait(kCEmpty, (cc & 1) ^ 1)) break;
                if (lane == 0) mbar_expect_tx(&bars[kCFull], SM::kCandBytes);
                __syncwarp();
                if (lane > 0 && lane < kConvWarps) mbar_arrive(&bars[kCFull]);
                if (lane < 2 * NB) bulk_load_1d(smem + SM::kCand + lane * SM::kCandBlock, stage + lane * SM::kCandBlock, SM::kCandBlock, &bars[kCFull]);
                __syncwarp();
            }
        }
    } else if (warp >= kConvWarp0) {
        // ---- candidate rows: kConvRows per warp and tile, kConvBatch in flight ----
        // Kept small: this code runs once in tens of microseconds and comes out of a cold instruction cache every time; written out
        // three times over, with a sum across the warp for every row's norm, it took 40 000 cycles a tile.  (The access width is a
        // template parameter: chosen per load at run time it made every load wait for the one before.)
        const int cw = warp - kConvWarp0, D = d.D, c = lane * 4;
        const float* mine = nullptr;  // lane l: row l of this warp's share
        auto locate = [&](int64_t t) {
            const int64_t col = t * kTileN + cw * kConvRows + lane;
            mine = t < te && col < sc.num_cols ? node_row(d, col) : nullptr;
        };
        float4 v[kConvBatch];
        auto fetch = [&](int r0) {
#pragma unroll
            for (int k = 0; k < kConvBatch; k++) {
                const float* row = (const float*)__shfl_sync(0xffffffffu, (unsigned long long)mine, r0 + k);
                const bool there = row != nullptr;
                if (VEC == 4) {
                    v[k] = there && c < D ? __ldg(reinterpret_cast<const float4*>(row) + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
                } else if (VEC == 2) {
                    const float2 x = there && c < D ? __ldg(reinterpret_cast<const float2*>(row) + 2 * lane) : make_float2(0.f, 0.f);
                    const float2 y = there && c + 2 < D ? __ldg(reinterpret_cast<const float2*>(row) + 2 * lane + 1) : make_float2(0.f, 0.f);
                    v[k] = make_float4(x.x, x.y, y.x, y.y);
                } else {
                    v[k].x = there && c < D ? __ldg(row + c) : 0.f;
                    v[k].y = there && c + 1 < D ? __ldg(row + c + 1) : 0.f;
                    v[k].z = there && c + 2 < D ? __ldg(row + c + 2) : 0.f;
                    v[k].w = there && c + 3 < D ? __ldg(row + c + 3) : 0.f;
                }
            }
        };
        uint32_t cc = 0;
        int64_t t = tb;
        float scale = 1.f, norm2 = 0.f;
        int r0 = -kConvBatch;
        while (true) {  // one turn: the batch in registers (none in the first) goes to shared memory, the next one is fetched
            if (r0 >= 0) {
                const int cb = cc % SM::kCandBufs;
                const bool staged = NB == 2 && sc.staged && cc > 0;  // (the first tile goes straight to shared memory)
                if (r0 == 0) {
                    // the place it goes to is free: the copy before has been taken, or the tile before has been contracted
                    if (staged ? !warp_wait(kCFull, (cc & 1) ^ 1) : !warp_wait(kCEmpty + cb, ((cc / SM::kCandBufs) & 1) ^ 1)) break;
                    // a power of two for these 32 rows, from the first eight: the others may be 2^6 times larger before fp16 ends
                    float most = 0.f;
#pragma unroll
                    for (int k = 0; k < kConvBatch; k++) most = fmaxf(most, fmaxf(fmaxf(fabsf(v[k].x), fabsf(v[k].y)), fmaxf(fabsf(v[k].z), fabsf(v[k].w))));
                    scale = pow2_near_256(__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(most))));
                    norm2 = 0.f;  // largest squared norm that this lane's four columns contribute to a row
                }
                unsigned char* at0 = (staged ? a.stage + (int64_t)(blockIdx.y * gridDim.x + blockIdx.x) * SM::kCandBytes : smem + SM::kCand + cb * SM::kCandBytes) +
                                     (lane >> 4) * SM::kCandBlock + (lane & 1) * 8 + (cw * kConvRows + r0) * 128;
#pragma unroll
                for (int k = 0; k < kConvBatch; k++) {
                    const float4 x = make_float4(v[k].x * scale, v[k].y * scale, v[k].z * scale, v[k].w * scale);
                    const __half2 h0 = __floats2half2_rn(x.x, x.y), h1 = __floats2half2_rn(x.z, x.w);
                    const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
                    const __half2 l0 = __floats2half2_rn(x.x - f0.x, x.y - f0.y), l1 = __floats2half2_rn(x.z - f1.x, x.w - f1.y);
                    if (NB == 2 || lane < 16) {
                        unsigned char* at = at0 + k * 128 + ((((lane & 15) >> 1) ^ k) << 4);  // k = row % 8
                        *reinterpret_cast<uint2*>(at) = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
                        *reinterpret_cast<uint2*>(at + NB * SM::kCandBlock) =
                            make_uint2(*reinterpret_cast<const uint32_t*>(&l0), *reinterpret_cast<const uint32_t*>(&l1));
                    }
                    const float part = x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
                    norm2 = part > norm2 || !(part < INFINITY) ? part : norm2;  // (inf and NaN stay)
                }
                if (r0 == kConvRows - kConvBatch) {
                    // |e| of no row exceeds the root of the sum over lanes (tighter by a third with a sum per row, and not worth it)
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) norm2 += __shfl_xor_sync(0xffffffffu, norm2, o);
                    if (lane == 0) s_cand[(cc & 1) * kConvWarps + cw] = make_float2(sqrtf(norm2) * 1.001f, scale);
                    fence_proxy_async();  // written with ordinary stores; the MMA, or the copy, reads through the async proxy
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars[staged ? kStaged : kCFull + cb]);
                    t++;
                    cc++;
                    if (t >= te) break;
                }
            }
            r0 = (r0 + kConvBatch) & (kConvRows - 1);
            if (r0 == 0) {
                locate(t);
                if (mine != nullptr)  // all of the tile's rows on their way into L2
                    for (int k = 0; k < D * 4; k += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"((const char*)mine + k));
                __syncwarp();
            }
            fetch(r0);
        }
    } else if (warp >= kEpiWarp0) {
        const int ew = warp - kEpiWarp0, quarter = ew >> 2, lrow = (warp & 3) * 32 + lane;
        const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
        uint2* list = (uint2*)(smem + SM::kList) + ew * kListCap;
        int listed = 0;
        auto hand_on = [&](int n) {  // list entries [0, n), n <= 32: to the global list, or evaluated here when that is full
            __syncwarp();
            unsigned long long at = 0;
            if (lane == 0 && n > 0) at = atomicAdd(a.open_count, (unsigned long long)n);
            at = __shfl_sync(0xffffffffu, at, 0) + lane;
            if (lane < n) {
                if ((int64_t)at < a.open_cap) a.open_list[at] = list[lane];
                else settle_in_place(a, list[lane]);
            }
            __syncwarp();
        };
        uint32_t ac = 0, cc = 0;
        bool ok = true;
        for (int64_t t = tb; ok && t < te; t++, cc++) {
            const int cb = cc % SM::kCandBufs;
            const int64_t n0 = t * kTileN + quarter * 64;
            float pos = __ldg(a.pos + q0 * kTileQ + lrow), qn = __ldg(a.qnorm + q0 * kTileQ + lrow), qinv = __ldg(a.qinv + q0 * kTileQ + lrow);
            ok = warp_wait(kCFull + cb, (cc / SM::kCandBufs) & 1);
            if (!ok) break;
            float slope[2], cscale[2];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const float2 cand = s_cand[(cc & 1) * kConvWarps + quarter * 2 + k];
                cscale[k] = cand.y;
                slope[k] = cand.x < 60000.f ? 1.05f * (sc.bound * cand.x + 4e-7f) : INFINITY;  // (at the end of fp16 nothing is decided)
            }
            for (int qt = q0; qt < q1; qt++, ac++) {
                const int ab = ac % kAccs;
                // The accumulator v holds score * cscale / qinv.  It is turned into t = saturate(1/2 + (score - pos) / 2b): 1 when the
                // score is above by the bound or more, 0 when below, in between when it is open.  (Products below the smallest normal
                // number may vanish on either side: the constants cover them; the factor 1.05 in slope covers the roundings of t.)
                float scale[2], shift[2];
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const float b = fmaf(qn, slope[k], (8e-37f * qn + 2e-35f) * cscale[k]);  // times cscale, as pos below
                    const float r = __fdividef(0.5f, b), p = pos * cscale[k];
                    scale[k] = r * qinv;
                    shift[k] = fmaf(-p, r, 0.5f);
                    if (!(r < 1e30f) || !(scale[k] < 1e30f) || !(fabsf(p) < 1e30f)) scale[k] = 0.f, shift[k] = 0.5f;  // values without use: nothing is decided
                    if (qn < 0.f) scale[k] = shift[k] = 0.f;  // no rank: nothing counts
                }
                if (qt + 1 < q1) {
                    const int64_t w = (int64_t)(qt + 1) * kTileQ + lrow;
                    pos = __ldg(a.pos + w), qn = __ldg(a.qnorm + w), qinv = __ldg(a.qinv + w);
                }
                ok = warp_wait(kAccFull + ab, (ac / kAccs) & 1);
                if (!ok) break;
                tc_fence_after();
                int sure = 0;
#pragma unroll 1
                for (int k = 0; k < 2; k++) {
                    const int64_t left = sc.num_cols - n0 - k * 32;
                    const int nv = left < 32 ? (left < 0 ? 0 : (int)left) : 32;  // candidates among these 32 columns
                    float v[32];
                    tmem_ld_32x32(tmem + ab * kTileN + quarter * 64 + k * 32 + lane_sel, v);
                    if (k == 1) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&bars[kAccEmpty + ab]);
                    }
                    // The sum of the t is what counts when no t is fractional, which is when it equals the sum of their squares: two
                    // instructions a score (a saturating multiply-add and two halves of packed ones) instead of two compares and two
                    // conditional additions.
                    const float sc_k = k == 0 ? scale[0] : scale[1], sh_k = k == 0 ? shift[0] : shift[1];
                    float above;
                    bool clear;
                    if (nv == 32) {
                        uint64_t s1 = 0, s2 = 0;
#pragma unroll
                        for (int j = 0; j < 32; j += 2) {
                            const uint64_t t = pack2(saturated(v[j], sc_k, sh_k), saturated(v[j + 1], sc_k, sh_k));
                            s1 = add2(s1, t);
                            s2 = fma2(t, t, s2);
                        }
                        above = sum2(s1);
                        clear = above == sum2(s2);
                    } else {
                        above = 0.f;
                        clear = nv == 0;
                    }
                    if (!__all_sync(0xffffffffu, clear)) {
                        uint32_t open = 0;  // this row's undecided columns
                        float frac = 0.f;
                        above = 0.f;
#pragma unroll
                        for (int j = 0; j < 32; j++) {  // straight-line: a branch a column cost more than the rest of the tile
                            const float t = j < nv ? saturated(v[j], sc_k, sh_k) : 0.f;
                            const bool between = fmaf(-t, t, t) > 0.f;
                            open |= between ? 1u << j : 0u;
                            frac += between ? t : 0.f;
                            above += t;
                        }
                        above = rintf(above - frac);
                        unsigned who;
#pragma unroll 1
                        while ((who = __ballot_sync(0xffffffffu, open != 0u)) != 0u) {
                            if (open != 0u) {
                                list[listed + __popc(who & ((1u << lane) - 1u))] = make_uint2(qt * kTileQ + lrow, (uint32_t)(n0 + k * 32 + (__ffs(open) - 1)));
                                open &= open - 1u;
                            }
                            listed += __popc(who);
                            if (listed >= 32) {
                                hand_on(32);
                                listed -= 32;
                                if (lane < listed) list[lane] = list[32 + lane];  // the rest moves to the front (fewer than 32)
                                __syncwarp();
                            }
                        }
                    }
                    sure += (int)above;
                }
                if (sure != 0) atomicAdd(&cnt[(qt - q0) * kTileQ + lrow], sure);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[kCEmpty + cb]);
        }
        if (ok) hand_on(listed);
    }
    // ---- common exit: every role ends here, normally or after an abort; then tensor memory is released ----------
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        if (*s_abort && lane == 0)  // copies still in flight get a bounded chance to land
            for (int k = 0; k < SM::kSlots + SM::kCandBufs; k++) settle_bar(&bars[k < SM::kSlots ? kQFull + k : kCFull + k - SM::kSlots]);
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    for (int k = tid; k < (q1 - q0) * kTileQ; k += kCountThreads)
        if (cnt[k] != 0) add_to_rank(a, (int64_t)q0 * kTileQ + k, cnt[k]);
}

// A filter pair (edge row, candidate column): the first thread to enter the pair into the set undoes what the count pass did for it and
// counts the replacement score -1e9 instead (duplicates of a pair change nothing, like index_put_).
__device__ __forceinline__ void apply_filter_pair(const EvalArgs& a, int s, int64_t p, int64_t num_cols) {
    const ge2_eval_desc& d = a.d;
    const longlong2* __restrict__ pairs = reinterpret_cast<const longlong2*>(s == 0 ? d.dst_filter : d.src_filter);
    int64_t i, col;
    if ((((uintptr_t)pairs) & 15) == 0) {
        const longlong2 pr = __ldg(pairs + p);
        i = pr.x, col = pr.y;
    } else {
        i = reinterpret_cast<const int64_t*>(pairs)[2 * p], col = reinterpret_cast<const int64_t*>(pairs)[2 * p + 1];
    }
    if (i < 0 || i >= d.B || col < 0 || col >= num_cols) {
        or_status(d.status, GE2_STATUS_BAD_INDEX);
        return;
    }
    const int64_t w = (int64_t)s * a.Bp + i;
    const unsigned long long key = ((unsigned long long)s << 62) + (unsigned long long)i * (unsigned long long)num_cols + (unsigned long long)col + 1ull;
    unsigned long long slot = (key * 0x9E3779B97F4A7C15ull) >> 20 & (unsigned long long)(a.hash_slots - 1);
    // (the chain is walked while the answer is on its way: few pairs occur again)
    unsigned long long old = atomicCAS(&a.hash[slot], 0ull, key);
    const float* e = node_row(d, col);
    const float pos = a.pos[w];
    const float acc = e != nullptr ? score_chain_ahead(a.Q + w * d.D, e, d.D, a.vec) : 0.f;
    for (int64_t probe = 1; old != 0ull && old != key && probe < a.hash_slots; probe++) {
        slot = (slot + 1) & (unsigned long long)(a.hash_slots - 1);
        old = atomicCAS(&a.hash[slot], 0ull, key);
    }
    if (old != 0ull) {
        if (old != key) or_status(d.status, GE2_STATUS_FILTER_COLLISION);  // cannot happen: the set has twice as many slots as pairs
        return;
    }
    int64_t delta = 0;
    if (acc >= pos) delta -= 1;
    if (-1e9f >= pos) delta += 1;
    if (delta != 0) add_to_rank(a, w, delta);
}

// What the counting pass left open, and the filter: a thread each, blockIdx.x < filter_blocks the filter pairs (both sides), the others
// the open comparisons.  All of it adds to the ranks, in any order.
// Bound by the latency of scattered rows; 56 loads of a chain are on their way at a time (10: 98 us at 1 M nodes and 19.8 at 14 951, now 91 and 14.7).
__global__ void __launch_bounds__(kSettleThreads) eval_settle_kernel(const __grid_constant__ EvalArgs a, int64_t num_cols, int filter_blocks) {
    griddep_wait();
    if ((int)blockIdx.x < filter_blocks) {
        const int64_t p = (int64_t)blockIdx.x * kSettleThreads + threadIdx.x, n0 = a.d.dst_filter_n;
        if (p < n0) apply_filter_pair(a, 0, p, num_cols);
        else if (p - n0 < a.d.src_filter_n) apply_filter_pair(a, 1, p - n0, num_cols);
        return;
    }
    const int64_t n = min((int64_t)*a.open_count, a.open_cap), stride = (int64_t)(gridDim.x - filter_blocks) * kSettleThreads;
    for (int64_t k = (int64_t)(blockIdx.x - filter_blocks) * kSettleThreads + threadIdx.x; k < n; k += stride) settle<true>(a, a.open_list[k]);
}

int64_t hash_slots_for(int64_t pairs) {
    int64_t s = 64;
    while (s < 2 * pairs) s <<= 1;
    return s;
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

int split_ld(int D) { return D <= 64 ? 64 : 128; }

int sides_of(const ge2_eval_desc* d) { return (d->has_relations && d->use_inverse) ? 2 : 1; }

}  // namespace
}  // namespace ge2

using namespace ge2;

namespace {
// workspace sections of a call, in order
struct EvalSections {
    int64_t Bp;
    size_t q, split, pos, norm, qinv, hash, open_count, open, stage, bytes;
    int64_t open_cap;
    explicit EvalSections(const ge2_eval_desc* d) {
        const int S = sides_of(d);
        Bp = round_up<int64_t>(d->B, kTileQ);
        const int64_t pairs = (d->dst_filter_n > 0 ? d->dst_filter_n : 0) + (d->src_filter_n > 0 ? d->src_filter_n : 0);
        size_t off = 0;
        auto take = [&](size_t b) {
            const size_t o = off;
            off += align256(b);
            return o;
        };
        q = take((size_t)S * Bp * d->D * 4);
        split = take((size_t)2 * S * Bp * split_ld(d->D) * 2);
        pos = take((size_t)S * Bp * 4);
        norm = take((size_t)S * Bp * 4);
        qinv = take((size_t)S * Bp * 4);
        hash = take((size_t)hash_slots_for(pairs) * 8);
        open_count = take(8);
        // one comparison in a few thousand is left open on trained tables; what does not fit is evaluated on the spot
        const int64_t num_cols = d->neg_ids != nullptr ? d->num_negs : d->num_nodes;
        open_cap = std::min<int64_t>(std::max<int64_t>(S * Bp * std::max<int64_t>(num_cols, 0) / 1024, 4096), 4 << 20);
        open = take((size_t)open_cap * 8);
        stage = take(d->D > 64 && num_cols > (int64_t)kTileN ? (size_t)kNumSMs * CountSmem<2>::kCandBytes : 0);
        bytes = off;
    }
};

template <int NB>
int launch_count(const EvalArgs& a, CountSched sc, const CUtensorMap& tmQ, cudaStream_t stream) {
    // per-device function attribute; setting it on every call keeps multi-device processes correct and is not a stream operation
    auto kernel = a.vec == 4 ? eval_count_kernel<NB, 4> : a.vec == 2 ? eval_count_kernel<NB, 2> : eval_count_kernel<NB, 1>;
    GE2_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CountSmem<NB>::kBytes));
    // the number of query groups with the shortest longest CTA: query tiles of its group x candidate tiles of its share, a candidate
    // tile's conversion counted as two query tiles; groups run side by side as long as there are SMs for them
    int64_t best = INT64_MAX;
    for (int g = ceil_div(sc.q_tiles, kGroupTiles); g <= sc.q_tiles && g <= std::max(kNumSMs, ceil_div(sc.q_tiles, kGroupTiles)); g++) {
        const int64_t shares = std::min<int64_t>(std::max(1, kNumSMs / g), sc.cand_tiles);
        const int64_t waves = ceil_div<int64_t>(g, kNumSMs);
        const int64_t cost = waves * ceil_div<int64_t>(sc.cand_tiles, shares) * (ceil_div(sc.q_tiles, g) + 2);
        if (cost < best) best = cost, sc.groups = g;
    }
    if (sc.groups > 65535) return GE2_ERR_UNSUPPORTED;
    const dim3 grid((unsigned)std::min<int64_t>(std::max(1, kNumSMs / sc.groups), sc.cand_tiles), (unsigned)sc.groups);
    sc.staged = NB == 2 && a.stage != nullptr && sc.cand_tiles > grid.x && (int64_t)grid.x * grid.y <= kNumSMs;
    GE2_CUDA_TRY(launch_after(kernel, grid, dim3(kCountThreads), CountSmem<NB>::kBytes, stream, tmQ, a, sc));
    return GE2_OK;
}
}  // namespace

extern "C" size_t ge2_eval_workspace_bytes(const ge2_eval_desc* d) {
    if (d == nullptr || d->B <= 0 || d->D <= 0) return 0;
    return EvalSections(d).bytes;
}

extern "C" int ge2_eval_ranks(const ge2_eval_desc* d, ge2_stream_t stream_) {
    if (d == nullptr || d->B <= 0 || d->num_nodes <= 0 || d->D <= 0) return GE2_ERR_INVALID_ARGUMENT;
    if (d->D > kMaxD) return GE2_ERR_UNSUPPORTED;
    if (d->decoder != GE2_DECODER_DISTMULT && d->decoder != GE2_DECODER_COMPLEX) return GE2_ERR_INVALID_ARGUMENT;
    if (d->decoder == GE2_DECODER_COMPLEX && d->has_relations && (d->D & 1)) return GE2_ERR_INVALID_ARGUMENT;
    if (d->node_emb == nullptr || d->src_ids == nullptr || d->dst_ids == nullptr || d->dst_ranks == nullptr || d->edge_stride <= 0 ||
        d->emb_stride < d->D)
        return GE2_ERR_INVALID_ARGUMENT;
    if (d->has_relations && (d->rel_ids == nullptr || d->rel == nullptr || d->R <= 0 || d->rel_stride <= 0)) return GE2_ERR_INVALID_ARGUMENT;
    if (d->use_inverse && !d->has_relations) return GE2_ERR_INVALID_ARGUMENT;
    const int S = sides_of(d);
    if (S == 2 && (d->inv_rel == nullptr || d->src_ranks == nullptr)) return GE2_ERR_INVALID_ARGUMENT;
    if (d->dst_filter_n < 0 || d->src_filter_n < 0 || (d->dst_filter_n > 0 && d->dst_filter == nullptr) ||
        (d->src_filter_n > 0 && (d->src_filter == nullptr || S != 2)))
        return GE2_ERR_INVALID_ARGUMENT;
    const int64_t num_cols = d->neg_ids != nullptr ? d->num_negs : d->num_nodes;
    if (num_cols <= 0) return GE2_ERR_INVALID_ARGUMENT;
    const EvalSections at(d);
    // the last section can be missing: a candidate tile then is split only when the one before it is done with
    if (d->workspace == nullptr || ((uintptr_t)d->workspace & 255) != 0 || d->workspace_bytes < at.stage) return GE2_ERR_WORKSPACE;

    cudaStream_t stream = as_stream(stream_);
    char* p = (char*)d->workspace;
    EvalArgs a;
    a.d = *d;
    a.S = S;
    a.Bp = at.Bp;
    a.ld = split_ld(d->D);
    a.Q = (float*)(p + at.q);
    a.Qsplit = (__half*)(p + at.split);
    a.pos = (float*)(p + at.pos);
    a.qnorm = (float*)(p + at.norm);
    a.qinv = (float*)(p + at.qinv);
    a.hash = (unsigned long long*)(p + at.hash);
    a.hash_slots = hash_slots_for(d->dst_filter_n + d->src_filter_n);
    const uintptr_t mis = (uintptr_t)(d->D * 4) | (uintptr_t)(d->emb_stride * 4) | (uintptr_t)d->node_emb;
    a.vec = (mis & 15) == 0 ? 4 : (mis & 7) == 0 ? 2 : 1;
    a.open_list = (uint2*)(p + at.open);
    a.open_count = (unsigned long long*)(p + at.open_count);
    a.open_cap = at.open_cap;
    a.stage = d->workspace_bytes < at.bytes ? nullptr : (unsigned char*)(p + at.stage);
    const int64_t rows = (int64_t)S * a.Bp;
    if (rows > 0x7fffffffLL) return GE2_ERR_UNSUPPORTED;
    // the set of filter pairs and the counter behind it
    GE2_CUDA_TRY(cudaMemsetAsync(a.hash, 0, at.open_count + 8 - at.hash, stream));
    eval_prep_kernel<<<(unsigned)(rows / kPrepRows), kPrepThreads, 0, stream>>>(a);
    GE2_LAUNCH_CHECK();

    CUtensorMap tmQ;
    int rc = make_operand_map(&tmQ, a.Qsplit, false, a.ld, rows, 2);
    if (rc != GE2_OK) return rc;
    CountSched sc;
    sc.q_tiles = (int)(rows / kTileQ);
    const int steps = ceil_div(d->D, kMmaK), big_steps = steps + std::max(0, steps - 4);
    sc.bound = 1.02f * (big_steps * 17 * 1.1920929e-7f + d->D * 5.9604645e-8f + 3 * 2.3841858e-7f);
    constexpr int64_t kSegment = 1ll << 31;  // the list of open comparisons names a candidate by 32 bits
    for (int64_t c0 = 0; c0 < num_cols; c0 += kSegment) {
        EvalArgs seg = a;
        if (c0 > 0) {
            GE2_CUDA_TRY(cudaMemsetAsync(a.open_count, 0, 8, stream));
            if (d->neg_ids != nullptr) seg.d.neg_ids += c0;
            else seg.d.node_emb += c0 * d->emb_stride, seg.d.num_nodes -= c0;
        }
        sc.num_cols = std::min(num_cols - c0, kSegment);
        sc.cand_tiles = ceil_div<int64_t>(sc.num_cols, kTileN);
        rc = a.ld == 64 ? launch_count<1>(seg, sc, tmQ, stream) : launch_count<2>(seg, sc, tmQ, stream);
        if (rc != GE2_OK) return rc;
        // the filter goes with the first segment
        const int open_blocks = (int)std::min<int64_t>(ceil_div<int64_t>(a.open_cap, kSettleThreads), kNumSMs * 8);
        const int64_t filter_blocks = c0 == 0 ? ceil_div<int64_t>(d->dst_filter_n + d->src_filter_n, kSettleThreads) : 0;
        if (filter_blocks + open_blocks > 0x7fffffffLL) return GE2_ERR_UNSUPPORTED;
        GE2_CUDA_TRY(launch_after(eval_settle_kernel, dim3((unsigned)(filter_blocks + open_blocks)), dim3(kSettleThreads), 0, stream, seg, num_cols,
                                  (int)filter_blocks));
    }
    return GE2_OK;
}
