// Scores kernels of the link-prediction step's tensor path (kind::f16) for batches whose dK does not stay in the L2: the streaming
// softmax, in which every gradient row is written once.  The other kernels of this path (lp_scores_f16.cu) contract a logsumexp pass
// first and then make dQ and dK from one P; every row block of a chunk adds its part into global dK there, which is the faster way
// while those reductions hit the L2 and 1.6 GB of HBM traffic when they do not.
//
// Per (side, chunk) the work is Q [rows x D] against K [negatives x D]: S = Q K^T, row logsumexp (with the positive score),
// P = exp(S - lse), dQ = P K, dK = P^T Q.  The [rows x negatives] matrices never leave the SM.  Two launches of one kernel, each with
// a stationary block X of 128 rows, a stream of tiles Y of 128 rows past it, and for every tile
//     S = X Y^T  ->  P in fp16, written back over S in tensor memory  ->  O += P Y  (A from tensor memory, the same Y tile as B):
//
//   queries    X = rows of Q, Y = K: P = exp2(S log2 e - m) with a running row reference m, so that dQ needs no lse beforehand;
//              O / its row sum is dQ                                                                             -> dQ, lse, loss
//   negatives  X = rows of K, Y = Q: P = exp2(S log2 e - lse of the column)                                      -> dK
//
// Both launches are persistent: the (block, tile) units of the whole step are numbered consecutively and dealt to the
// CTAs (one per SM) as contiguous ranges of equal length, so every SM is busy to the end whatever the number of blocks.
// A block whose units straddle a CTA boundary is finished by two (rarely more) CTAs.  Queries: each leaves its part of O and the
// rows' (m, sum); the second launch weighs the parts and adds them up before its own drain begins.  Negatives: each adds its part to the
// output rows with TMA reduce-adds (those rows are cleared by the first launch).
//
// Shared memory holds two X blocks and a ring of Y tiles [128 x DP], fp16 in the 128-byte-swizzled layout TMA writes (64-element
// column blocks of 128 rows at a 128-byte pitch); a tile read along its rows is the K-major operand of S, read along its columns the
// MN-major operand of O.
// Tensor memory (512 columns): two score accumulators at 0 and 128, two O accumulators at 256 and 384.  Two groups of eight softmax
// warps take alternate tiles, each with its own score accumulator (and, for the queries, its own m and O), so one group
// exponentiates while the other's contractions run.
// Bound by the chain scores -> exponentials -> O -> scores of a group, 4900 ... 5800 cycles for its tile (the exp unit alone would take
// 1024 a tile): B = 100 000, N = 2000, D = 128, two sides: 282 + 235 us, with the other kernels 213 + 687 us.
// P carries a factor 2^14, so that probabilities down to 2^-38 keep their full significand instead of falling into fp16's subnormal
// range; dQ and dK leave this kernel with that factor still on them and the scatter kernel, their only reader, takes it off
// (LpLayout::grad_unscale).
//
// Warp roles, connected by mbarrier pipelines (no block-wide barrier inside the loops):
//   warps 0-15  softmax: warp w takes rows 32 (w & 3) ... + 31 (its quarter of the tensor-memory lanes) and columns 64 ((w >> 2) & 1)
//               ... + 63 of its group's (w >> 3) tiles
//   warps 16-19 drain: O -> registers (-> weighted sum of the two groups) -> staging slab -> TMA store / reduce-add
//   warp  20    TMA producer
//   warp  21    issues the contractions; also allocates and frees tensor memory
//   warps 22-23 what the softmax warps need to know about coming tiles (each for its group): which entries are masked and, for the
//               negatives, the columns' lse.  Queries: they first clear the dK rows the second launch reduces into
// Every mbarrier wait is bounded; a wait that runs out raises GE2_STATUS_PIPE_TIMEOUT and sets a block-wide abort flag
// that every other wait polls, so all roles fall through to the common exit where tensor memory is released.
#include <algorithm>

#include "lp_sched.cuh"
#include "tc_pipe.cuh"

namespace ge2 {
namespace {

using namespace tc;

constexpr int BM = 128;                 // rows of the stationary block (MMA M)
constexpr int BN = 128;                 // rows of a streamed tile
constexpr int kSoftmaxWarps = 16;
constexpr int kThreads = 768;
constexpr int kDrainWarp0 = kSoftmaxWarps, kDrainWarps = 4, kTmaWarp = 20, kMmaWarp = 21, kHelpWarp = 22;
constexpr int kStages = 4;              // Y ring: two tiles wait for their O contraction, two are on their way
constexpr int kInfoStages = 4;          // ring of what warps 22-23 find out about tiles
constexpr uint32_t kTmemCols = 512;
constexpr float kMasked = -1e9f;
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
constexpr int kWShift = 14;             // P is scaled by 2^14; undone by the reader of dQ / dK (kLpF16GradUnscale)
constexpr float kHeadStart = 3.f;       // queries: log2 of how far the reference is set above the maximum it is taken from
constexpr float kDeadRow = 1e30f;       // "lse" of a row past the end of its chunk: exp2(anything - 1e30) = 0

enum Bar { kBarXFull = 0, kBarXEmpty = 2, kBarYFull = 4, kBarYEmpty = kBarYFull + kStages, kBarSFull = kBarYEmpty + kStages, kBarPFull = kBarSFull + 2,
           kBarOFull = kBarPFull + 2, kBarOEmpty, kBarStat, kBarStatFree = kBarStat + 2, kBarMax = kBarStatFree + 2, kBarInfoFull = kBarMax + 8,
           kBarInfoEmpty = kBarInfoFull + kInfoStages, kNumBars = kBarInfoEmpty + kInfoStages };

template <int DP>
struct Layout {
    static constexpr int NB = DP / 64;               // column blocks of X / Y
    static constexpr int kTileBytes = NB * kBlockBytes;
    static constexpr int kX = 0;
    static constexpr int kY = kX + 2 * kTileBytes;
    static constexpr int kDrain = kY + kStages * kTileBytes;   // 4 drain warps x one slab (32 rows x 128 bytes), 128-byte swizzled
    static constexpr int kMisc = kDrain + kDrainWarps * 4096;  // barriers, tensor-memory address, abort flag
    static constexpr int kMax = kMisc + 1024;                  // row maxima of the column halves: [group][buffer][half][128]
    static constexpr int kStat = kMax + 2 * 2 * 2 * 128 * 4;   // (m, sum) at the end of a block: [buffer][group * 2 + half][128]
    static constexpr int kLse = kStat + 2 * 4 * 128 * 8;       // [kInfoStages][128]
    static constexpr int kMask = kLse + kInfoStages * 128 * 4; // [kInfoStages][128]
    static constexpr int kRange = kMask + kInfoStages * 128 * 4;  // first unit of every CTA of the query launch, and the end
    static constexpr int kEnd = kRange + (kNumSMs + 4) * 4;
    // at least 120 KB so that one CTA owns the SM and its tensor memory
    static constexpr int kDynamic = (kEnd + 1024) > 120 * 1024 ? (kEnd + 1024) : 120 * 1024;
    static_assert(kNumBars * 8 + 32 <= 1024, "barrier block overflows its slot");
    static_assert(kDynamic <= 227 * 1024, "exceeds the shared memory of an SM");
};

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ float exp2f_fast(float x) {  // one MUFU.EX2; 2^-inf = 0
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// base-2 logsumexp of a row from its positive score and the parts its sharers left
__device__ __noinline__ float combine_parts(const float2* part, int nparts, float pos2) {
    float m = pos2, l = 1.f;
#pragma unroll 1
    for (int k = 0; k < nparts && k < kMaxParts; k++) {
        const float2 pk = __ldg(&part[k]);
        const float nm = fmaxf(m, pk.x);
        l = l * exp2f_fast(m - nm) + pk.y * exp2f_fast(pk.x - nm);
        m = nm;
    }
    return m + __log2f(l);
}

struct FlashSched {
    Sched q, n;  // T, RB of each launch; units and grid of the launch in unitsA / gridA
};

template <int DP, bool NEG>
__global__ void __launch_bounds__(kThreads, 1)
    lp_flash_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmY, const __grid_constant__ CUtensorMap tmO,
                    const __grid_constant__ CUtensorMap tmOt, const __grid_constant__ LpKernelArgs a, const __grid_constant__ FlashSched fs) {
    using LY = Layout<DP>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sX = smem + LY::kX;
    unsigned char* sY = smem + LY::kY;
    uint64_t* bars = (uint64_t*)(smem + LY::kMisc);
    uint32_t* s_tmem = (uint32_t*)(smem + LY::kMisc + kNumBars * 8);
    volatile int* s_abort = (volatile int*)(smem + LY::kMisc + kNumBars * 8 + 4);
    float* s_max = reinterpret_cast<float*>(smem + LY::kMax);
    float2* s_stat = reinterpret_cast<float2*>(smem + LY::kStat);
    float* s_lse = reinterpret_cast<float*>(smem + LY::kLse);
    int* s_mask = reinterpret_cast<int*>(smem + LY::kMask);    // partner of the entry that is masked: queries: a column's row, negatives: a row's column; -1
    volatile int* s_any = (volatile int*)(smem + LY::kMisc + kNumBars * 8 + 16);  // [kInfoStages] does the tile hold a masked entry?
    int* s_range = reinterpret_cast<int*>(smem + LY::kRange);

    const ge2_lp_desc& d = a.d;
    const LpLayout& L = a.L;
    const Sched& sc = NEG ? fs.n : fs.q;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ub = range_begin(blockIdx.x, sc.unitsA, gridDim.x), ue = range_begin(blockIdx.x + 1, sc.unitsA, gridDim.x);
    const int n_iter = ue - ub;
    const int x_rows = NEG ? d.N : L.npc, y_rows = NEG ? L.npc : d.N;  // rows a chunk has on either side
    constexpr int NB = LY::NB;
    auto spin_wait = [&](int bar, uint32_t parity) { return warp_spin_wait(&bars[bar], parity, s_abort, d.status); };
    auto warp_wait = [&](int bar, uint32_t parity) { return warp_pipe_wait(&bars[bar], parity, s_abort, d.status); };

    if (warp == kTmaWarp && lane == 0) {
        for (int k = 0; k < 2; k++) {
            mbar_init(&bars[kBarXFull + k], 1);
            mbar_init(&bars[kBarXEmpty + k], 1);
            mbar_init(&bars[kBarSFull + k], 1);
            mbar_init(&bars[kBarPFull + k], kSoftmaxWarps / 2);  // one arrival per warp of the group that owns the tile
            mbar_init(&bars[kBarStat + k], kSoftmaxWarps);
            mbar_init(&bars[kBarStatFree + k], kDrainWarps);
        }
        for (int k = 0; k < kStages; k++) {
            mbar_init(&bars[kBarYFull + k], 1);
            mbar_init(&bars[kBarYEmpty + k], 1);
        }
        for (int k = 0; k < 8; k++) mbar_init(&bars[kBarMax + k], 2);  // the two column halves of 32 rows
        for (int k = 0; k < kInfoStages; k++) {
            mbar_init(&bars[kBarInfoFull + k], 1);
            mbar_init(&bars[kBarInfoEmpty + k], kSoftmaxWarps / 2);
        }
        mbar_init(&bars[kBarOFull], 1);
        mbar_init(&bars[kBarOEmpty], kDrainWarps);
        *s_abort = 0;
        mbar_init_fence();
        prefetch_tensormap(&tmX);
        prefetch_tensormap(&tmY);
    }
    if (NEG && tid <= fs.q.gridA) s_range[tid] = range_begin(tid, fs.q.unitsA, fs.q.gridA);
    if (warp == kMmaWarp) {
        tmem_alloc(s_tmem, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    griddep_wait();  // set-up done; from here on global memory written by the preceding kernel is read and its buffers rewritten
    const uint32_t tmem = *s_tmem;
    const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;  // this warp's quarter of the 128 tensor-memory lanes

    if (warp == kTmaWarp) {
        int sg = -1;
        IterA un(ub, sc);
        for (int it = 0; it < n_iter; it++, un.next(sc)) {
            if (it == 0 || un.tile == 0) {  // a new block
                sg++;
                const int xs = sg & 1;
                if (!spin_wait(kBarXEmpty + xs, ((sg >> 1) & 1) ^ 1)) break;
                mbar_expect_tx_warp(&bars[kBarXFull + xs], LY::kTileBytes);
#pragma unroll
                for (int b = 0; b < NB; b++) tma_load_3d_warp(sX + xs * LY::kTileBytes + b * kBlockBytes, &tmX, b * 64, un.rb * BM, un.zc, &bars[kBarXFull + xs]);
            }
            const int st = it % kStages;
            if (!spin_wait(kBarYEmpty + st, ((it / kStages) & 1) ^ 1)) break;
            mbar_expect_tx_warp(&bars[kBarYFull + st], LY::kTileBytes);
#pragma unroll
            for (int b = 0; b < NB; b++)
                tma_load_3d_warp(sY + st * LY::kTileBytes + b * kBlockBytes, &tmY, b * 64, un.tile * BN, un.zc, &bars[kBarYFull + st]);
        }
    } else if (warp == kMmaWarp) {
        // ================================ contractions ================================
        // S of the tile after next follows O of this one, so a score accumulator is overwritten only behind the contraction that reads
        // the P in it, and "S complete" also says that the group's previous O contraction is.
        const int D16 = ((d.D + kMmaK - 1) / kMmaK) * kMmaK;  // the embedding dimension rounded up to the MMA k step
        constexpr uint32_t kIdescS = idesc_f16(BM, BN, 0, 0);
        const uint32_t idesc_o = idesc_f16(BM, D16, 0, 1);
        const uint32_t dXk = desc_lo_sw128(smem_u32(sX), 16), dYk = desc_lo_sw128(smem_u32(sY), 16), dYm = desc_lo_sw128(smem_u32(sY), kBlockBytes);
        const int T = sc.T;
        int ts = decode_a(ub, sc).tile, tp = ts, sg = -1, so = -1, st_s = 0, st_p = 0, use = 0;  // tile within the block, block and stage of the next S and O
        uint32_t used = 0;  // accumulators that hold something of the current block
#pragma unroll 1
        for (int k = 0; k < n_iter + 2; k++) {
            const bool do_s = k < n_iter, do_p = k >= 2, last = k == n_iter - 1, first_s = k == 0 || ts == 0, first_p = k == 2 || tp == 0;
            if (do_s) {
                sg += first_s ? 1 : 0;
                if (first_s && !spin_wait(kBarXFull + (sg & 1), (sg >> 1) & 1)) break;
                if (!spin_wait(kBarYFull + st_s, use & 1)) break;
            }
            if (do_p) {
                if (first_p) {
                    used = 0;
                    so++;
                    if (!spin_wait(kBarOEmpty, (so & 1) ^ 1)) break;  // the drain has read the previous block's O
                }
                if (!spin_wait(kBarPFull + (k & 1), ((k - 2) >> 1) & 1)) break;
            }
            tc_fence_after();
            const uint32_t s = tmem + (k & 1) * 128;
            if (do_p) {
                const uint32_t o = tmem + 256 + (NEG ? 0 : (k & 1) * 128), p0 = s + 32, b0 = dYm + st_p * (LY::kTileBytes >> 4);
                const uint32_t more = (used >> (NEG ? 0 : k & 1)) & 1u;
#pragma unroll
                for (int ks = 0; ks < BN / kMmaK; ks++)  // P sits in columns 32 ... 63 and 96 ... 127 of the score accumulator
                    mma_f16_ts_warp(o, p0 + (ks >> 2) * 64 + (ks & 3) * 8, b0 + (uint32_t)koff_mnmajor(ks), idesc_o, ks > 0 ? 1u : more);
                used |= 1u << (NEG ? 0 : k & 1);
                mma_commit_warp(&bars[kBarYEmpty + st_p]);
                if (k == n_iter + 1 || tp == T - 1) mma_commit_warp(&bars[kBarOFull]);
                tp = tp == T - 1 ? 0 : tp + 1;
                st_p = st_p == kStages - 1 ? 0 : st_p + 1;
            }
            if (do_s) {
                const uint32_t x0 = dXk + (sg & 1) * (LY::kTileBytes >> 4), y0 = dYk + st_s * (LY::kTileBytes >> 4);
#pragma unroll
                for (int ks = 0; ks < DP / kMmaK; ks++) mma_f16_ss_warp(s, x0 + (uint32_t)koff_kmajor(ks), y0 + (uint32_t)koff_kmajor(ks), kIdescS, ks > 0);
                mma_commit_warp(&bars[kBarSFull + (k & 1)]);
                if (last || ts == T - 1) mma_commit_warp(&bars[kBarXEmpty + (sg & 1)]);
                ts = ts == T - 1 ? 0 : ts + 1;
                if (++st_s == kStages) st_s = 0, use++;
            }
        }
    } else if (warp < kSoftmaxWarps) {
        // ================================ softmax warps (0-15) ================================
        const int grp = warp >> 3, ch = (warp >> 2) & 1, wq = warp & 3;
        const int my_row = tid & 127;   // accumulator row / tensor-memory lane
        const uint32_t tS = tmem + grp * 128 + ch * 64 + lane_sel;  // this warp's 64 score columns
        IterA un(ub, sc);
        float m = -INFINITY, l = 0.f;  // queries: reference and sum (scaled by 2^14) of this group's tiles of the block; the reference is shared by the halves
        int sg = -1;
#pragma unroll 1
        for (int it = 0; it < n_iter; it++, un.next(sc)) {
            if (it == 0 || un.tile == 0) {
                sg++;
                m = -INFINITY;
                l = 0.f;
            }
            if ((it & 1) == grp) {
                const int nth = it >> 1, stage = it & (kInfoStages - 1);
                const int nv = y_rows - un.tile * BN - ch * 64;  // columns of this warp's 64 that exist
                if (!warp_wait(kBarInfoFull + stage, (it / kInfoStages) & 1)) break;
                uint32_t mb[2] = {0u, 0u};  // bits of those masked for my row
                if (s_any[stage]) {
                    const int* msk = s_mask + stage * 128;
                    if (NEG) {
                        const int col = msk[my_row] - ch * 64;
                        if ((unsigned)col < 64u) (col < 32 ? mb[0] : mb[1]) = 1u << (col & 31);
                    } else {
#pragma unroll
                        for (int k = 0; k < 2; k++) {
                            const int row = msk[ch * 64 + k * 32 + lane];
                            unsigned ballot = __ballot_sync(0xffffffffu, row >= 0 && (row >> 5) == wq);
                            while (ballot != 0) {
                                const int src = __ffs(ballot) - 1;
                                ballot &= ballot - 1;
                                if (__shfl_sync(0xffffffffu, row, src) == my_row) mb[k] |= 1u << src;
                            }
                        }
                    }
                }
                const bool odd = __any_sync(0xffffffffu, (mb[0] | mb[1]) != 0u) || nv < 64;
                if (!warp_wait(kBarSFull + grp, nth & 1)) break;
                tc_fence_after();
                // 32 scores: masked and absent ones replaced
                auto load = [&](int k, float (&v)[32]) {
                    tmem_ld_32x32(tS + k * 32, v);
                    if (odd) {
                        const float masked = NEG ? -INFINITY : kMasked;
                        const uint32_t bits = k == 0 ? mb[0] : mb[1];
                        const int live = nv - k * 32;
#pragma unroll
                        for (int j = 0; j < 32; j++) v[j] = j >= live ? -INFINITY : ((bits >> j) & 1u) ? masked : v[j];
                    }
                };
                float v[32];
                float shift = 0.f;
                if (!NEG) {
                    float tmax = -INFINITY;
                    float* dump = un.zc < d.C ? d.neg_scores : d.inv_neg_scores;
#pragma unroll 1
                    for (int k = 0; k < 2; k++) {
                        load(k, v);
                        float mx[4];
#pragma unroll
                        for (int q = 0; q < 4; q++) mx[q] = v[q];
#pragma unroll
                        for (int j = 4; j < 32; j++) mx[j & 3] = fmaxf(mx[j & 3], v[j]);
                        tmax = fmaxf(tmax, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
                        if (dump != nullptr && my_row < x_rows - un.rb * BM) {  // the score dump of the tests
                            float* drow = dump + ((int64_t)(un.zc >= d.C ? un.zc - d.C : un.zc) * L.npc + un.rb * BM + my_row) * d.N + un.tile * BN + ch * 64 + k * 32;
#pragma unroll
                            for (int j = 0; j < 32; j++)
                                if (k * 32 + j < nv) drow[j] = v[j];
                        }
                    }
                    // the row's maximum over both halves of the tile
                    float* mine = s_max + ((grp * 2 + (nth & 1)) * 2 + ch) * 128 + my_row;
                    *mine = tmax;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars[kBarMax + grp * 4 + wq]);
                    if (!warp_wait(kBarMax + grp * 4 + wq, nth & 1)) break;
                    tmax = fmaxf(tmax, mine[ch == 0 ? 128 : -128]) * kLog2e;
                    // The reference starts 2^3 above the first tile's maximum and follows only when it would be left more than a factor 2
                    // behind (P <= 2^15 fits fp16): O and the sum have to be rescaled when that happens, for 32 rows at a time, so it
                    // should be rare (without the head start some row of a warp did in nearly every tile).
                    const bool first = m == -INFINITY, up = tmax > m + 1.f;
                    tmax += kHeadStart;
                    if (__any_sync(0xffffffffu, up && !first)) {
                        const float f = up ? exp2f_fast(m - tmax) : 1.f;
                        l *= f;
#pragma unroll 1
                        for (int q = ch; q * 16 < d.D; q += 2) {
                            float o[16];
                            uint32_t w[16];
                            const uint32_t at = tmem + 256 + grp * 128 + lane_sel + q * 16;
                            tmem_ld_32x16(at, o);
#pragma unroll
                            for (int j = 0; j < 16; j++) w[j] = __float_as_uint(o[j] * f);
                            tmem_st_32x16(at, w);
                        }
                    }
                    if (up) m = tmax;
                    shift = m - (float)kWShift;
                }
                // P over the upper half of this warp's score columns, whose scores (the second 32) are in registers or used up by then
                float add[4] = {0.f, 0.f, 0.f, 0.f};
                const float* lse = s_lse + stage * 128 + ch * 64;
#pragma unroll 1
                for (int k = 1; k >= 0; k--) {
                    if (NEG || k == 0) load(k, v);  // (queries: the second half is still there)
                    uint32_t w[16];
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        float4 sh = make_float4(shift, shift, shift, shift);
                        if (NEG) sh = *reinterpret_cast<const float4*>(lse + k * 32 + 4 * q);
                        const float e0 = exp2f_fast(fmaf(v[4 * q], kLog2e, -sh.x)), e1 = exp2f_fast(fmaf(v[4 * q + 1], kLog2e, -sh.y));
                        const float e2 = exp2f_fast(fmaf(v[4 * q + 2], kLog2e, -sh.z)), e3 = exp2f_fast(fmaf(v[4 * q + 3], kLog2e, -sh.w));
                        if (!NEG) add[0] += e0, add[1] += e1, add[2] += e2, add[3] += e3;
                        w[2 * q] = pack_half2(e0, e1);
                        w[2 * q + 1] = pack_half2(e2, e3);
                    }
                    tmem_st_32x16(tS + 32 + k * 16, w);
                }
                l += (add[0] + add[1]) + (add[2] + add[3]);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&bars[kBarPFull + grp]);
                    mbar_arrive(&bars[kBarInfoEmpty + stage]);
                }
            }
            if (!NEG && (it == n_iter - 1 || un.tile == sc.T - 1)) {  // end of the block (or of this CTA's share of it)
                const int h = sg & 1;
                if (!warp_wait(kBarStatFree + h, ((sg >> 1) & 1) ^ 1)) break;
                s_stat[(h * 4 + grp * 2 + ch) * 128 + my_row] = make_float2(m, l);
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars[kBarStat + h]);
            }
        }
    } else if (warp < kTmaWarp) {
        // ================================ drain warps (16-19) ================================
        const int wq = warp & 3;
        if (NEG) {
            // dQ of the blocks the first launch split between CTAs, from the parts they left: boundary j of that launch is looked after
            // by CTA (j - 1) % gridDim.x of this one (a block with several boundaries by that of its first)
#pragma unroll 1
            for (int j = 1 + (int)blockIdx.x; j < fs.q.gridA; j += (int)gridDim.x) {
                const int u = range_begin(j, fs.q.unitsA, fs.q.gridA);
                const UnitA un = decode_a(u, fs.q);
                const int u0 = un.item * fs.q.T;
                if (un.tile == 0 || range_begin(j - 1, fs.q.unitsA, fs.q.gridA) > u0) continue;
                const int p_first = cta_of_unit(u0, fs.q.unitsA, fs.q.gridA);
                const int nparts = min(kMaxParts, cta_of_unit(u0 + fs.q.T - 1, fs.q.unitsA, fs.q.gridA) - p_first + 1);
                const int r0 = un.rb * BM + wq * 32, rows = min(32, L.npc - r0);
                if (rows <= 0) continue;
                const int64_t grow0 = (int64_t)un.zc * L.npc + r0;  // ([S][Bp] = [zc][npc])
                float lse2 = 0.f, loss = 0.f;
                if (lane < rows) {
                    const float pos2 = __ldg(&L.pos[grow0 + lane]) * kLog2e;
                    lse2 = combine_parts(reinterpret_cast<const float2*>(L.part) + (grow0 + lane) * kMaxParts, nparts, pos2);
                    L.lse[grow0 + lane] = lse2 * kLn2;
                    loss = (lse2 - pos2) * kLn2;
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
                if (lane == 0) atomicAdd(L.loss_acc, (double)loss);
                constexpr int kLanes = DP / 4, kSide = 32 / kLanes;  // lanes a row, rows side by side
                const int cl = (lane & (kLanes - 1)) * 4;
                // part p of a block is the first block of its CTA, except that of the CTA the block begins in (its last one)
                const float* o0 = L.o_part + (((int64_t)p_first * 2 + 1) * BM + wq * 32) * DP + cl;
                const float* o1 = L.o_part + (((int64_t)(p_first + 1) * 2) * BM + wq * 32) * DP + cl;
                const float2* part = reinterpret_cast<const float2*>(L.part) + grow0 * kMaxParts;
#pragma unroll 4
                for (int r = lane / kLanes; r < 32; r += kSide) {
                    const float lr = __shfl_sync(0xffffffffu, lse2, r);
                    if (r < rows) {
                        float4 s = *reinterpret_cast<const float4*>(o0 + r * DP), o = *reinterpret_cast<const float4*>(o1 + r * DP);
                        const float4 pw = __ldg(reinterpret_cast<const float4*>(part + r * kMaxParts));  // (m, sum) of the first two parts
                        const float w0 = exp2f_fast(pw.x - lr), w1 = exp2f_fast(pw.z - lr);
                        s.x = fmaf(w1, o.x, w0 * s.x), s.y = fmaf(w1, o.y, w0 * s.y), s.z = fmaf(w1, o.z, w0 * s.z), s.w = fmaf(w1, o.w, w0 * s.w);
#pragma unroll 1
                        for (int p = 2; p < nparts; p++) {
                            o = *reinterpret_cast<const float4*>(o1 + ((int64_t)(p - 1) * 2 * BM + r) * DP);
                            const float w = exp2f_fast(__ldg(&part[r * kMaxParts + p]).x - lr);
                            s.x = fmaf(w, o.x, s.x), s.y = fmaf(w, o.y, s.y), s.z = fmaf(w, o.z, s.z), s.w = fmaf(w, o.w, s.w);
                        }
                        *reinterpret_cast<float4*>(L.dQ + (grow0 + r) * DP + cl) = s;
                    }
                }
            }
        }
        // Only real columns leave the SM: D / 32 full slabs of 32 columns, then one narrow slab (its own tensor map, dense rows of `tail`
        // floats) for the remainder rounded up to 4, through a staging slab (128-byte rows, 16-byte chunks XOR-swizzled by row:
        // conflict-free stores, and the layout a SWIZZLE_128B tensor map expects).
        int full_slabs = d.D / 32, tail = ((d.D % 32) + 3) & ~3;
        if (tail == 32) {
            full_slabs++;
            tail = 0;
        }
        const int drain_slabs = full_slabs + (tail > 0 ? 1 : 0);
        unsigned char* scr = smem + LY::kDrain + wq * 4096;
        int sg = 0;
#pragma unroll 1
        for (int u = ub; u < ue; sg++) {
            const UnitA un = decode_a(u, sc);
            const int seg_end = min(ue, (un.item + 1) * sc.T);
            const bool whole = un.tile == 0 && seg_end == (un.item + 1) * sc.T;
            const int row0 = un.rb * BM + wq * 32;
            const bool live = row0 + lane < x_rows;
            float w0 = 1.f, w1 = 0.f;
            if (!NEG) {
                const int h = sg & 1, r = wq * 32 + lane;
                const int64_t grow = (int64_t)un.zc * L.npc + row0 + lane;
                const float pos2 = live ? __ldg(&L.pos[grow]) * kLog2e : 0.f;
                if (!warp_wait(kBarStat + h, (sg >> 1) & 1)) break;
                const float2 a0 = s_stat[(h * 4 + 0) * 128 + r], a1 = s_stat[(h * 4 + 1) * 128 + r];
                const float2 b0 = s_stat[(h * 4 + 2) * 128 + r], b1 = s_stat[(h * 4 + 3) * 128 + r];
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars[kBarStatFree + h]);
                const float m = fmaxf(a0.x, b0.x);  // (a group without a tile in this share: -inf, weight 0)
                w0 = exp2f_fast(a0.x - m), w1 = exp2f_fast(b0.x - m);
                const float l = ((a0.y + a1.y) * w0 + (b0.y + b1.y) * w1) * (1.f / (1 << kWShift));
                if (whole) {
                    const float nm = fmaxf(m, pos2);
                    const float lse2 = nm + __log2f(l * exp2f_fast(m - nm) + exp2f_fast(pos2 - nm));
                    const float f = exp2f_fast(m - lse2);
                    w0 *= f, w1 *= f;
                    float loss = 0.f;
                    if (live) {
                        L.lse[grow] = lse2 * kLn2;
                        loss = (lse2 - pos2) * kLn2;
                    }
                    L.lse2s[(int64_t)un.item * BM + r] = live ? lse2 - (float)kWShift : kDeadRow;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
                    if (lane == 0) atomicAdd(L.loss_acc, (double)loss);
                } else if (live) {
                    const int part = (int)blockIdx.x - cta_of_unit(un.item * sc.T, sc.unitsA, (int)gridDim.x);
                    if (part < kMaxParts) reinterpret_cast<float2*>(L.part)[grow * kMaxParts + part] = make_float2(m, l);
                }
            }
            // which groups had a tile: iterations u - ub ... seg_end - ub - 1 alternate between them
            const bool two = !NEG && seg_end - u > 1;
            const int only = !NEG && !two ? (u - ub) & 1 : 0;
            if (only == 1) w0 = w1;
            if (!warp_wait(kBarOFull, sg & 1)) break;
            tc_fence_after();
            float* part_rows = L.o_part + (((int64_t)blockIdx.x * 2 + (un.tile == 0 ? 1 : 0)) * BM + wq * 32 + lane) * DP;
            int y = row0, z = un.zc;
            // The coordinates are pinned in ordinary registers here, where the whole warp is active: taken straight from the
            // index arithmetic into the one-lane section below, the third coordinate was seen to reach the store as 0.
            asm volatile("" : "+r"(y), "+r"(z));
#pragma unroll 1
            for (int cb = 0; cb < drain_slabs; cb++) {
                float v[32];
                tmem_ld_32x32(tmem + 256 + only * 128 + lane_sel + cb * 32, v);
                if (!NEG) {
#pragma unroll
                    for (int j = 0; j < 32; j++) v[j] *= w0;
                    if (two) {
#pragma unroll
                        for (int q = 0; q < 2; q++) {
                            float o[16];
                            tmem_ld_32x16(tmem + 384 + lane_sel + cb * 32 + q * 16, o);
#pragma unroll
                            for (int j = 0; j < 16; j++) v[q * 16 + j] = fmaf(o[j], w1, v[q * 16 + j]);
                        }
                    }
                }
                if (cb == drain_slabs - 1) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars[kBarOEmpty]);
                }
                if (!NEG && !whole) {
#pragma unroll
                    for (int q = 0; q < 8; q++) *reinterpret_cast<float4*>(part_rows + cb * 32 + 4 * q) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                    continue;
                }
                if (lane == 0) bulk_wait_group_read<0>();  // the operation that last used the slab has read it
                __syncwarp();
                const bool narrow = cb == full_slabs;
                if (!narrow) {
#pragma unroll
                    for (int q = 0; q < 8; q++)
                        *reinterpret_cast<float4*>(scr + lane * 128 + ((q ^ (lane & 7)) << 4)) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                } else {
#pragma unroll
                    for (int q = 0; q < 8; q++)
                        if (q * 4 < tail)
                            *reinterpret_cast<float4*>(scr + lane * (tail * 4) + q * 16) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    const CUtensorMap* map = narrow ? &tmOt : &tmO;
                    if (NEG && !whole) tma_reduce_add_3d(map, cb * 32, y, z, scr);
                    else tma_store_3d(map, cb * 32, y, z, scr);
                    bulk_commit_group();
                }
            }
            u = seg_end;
        }
        if (lane == 0) bulk_wait_group<0>();  // all of this warp's stores have landed before the CTA can exit
        __syncwarp();
    } else {
        // ================================ warps 22-23 ================================
        const int grp = warp - kHelpWarp;
        if (!NEG) {
            // clear the dK rows the second launch reduces into: those of every block whose stream it cuts at a CTA boundary (boundary j
            // is looked after by CTA (j - 1) % gridDim.x)
#pragma unroll 1
            for (int j = 1 + (int)blockIdx.x; j < fs.n.gridA; j += (int)gridDim.x) {
                const UnitA un = decode_a(range_begin(j, fs.n.unitsA, fs.n.gridA), fs.n);
                if (un.tile == 0) continue;  // the boundary falls between two blocks: nothing is split
                float4* p4 = reinterpret_cast<float4*>(L.dK + ((int64_t)un.zc * d.N + (int64_t)un.rb * BM) * DP);
                const int n4 = min(BM, d.N - un.rb * BM) * (DP / 4);
#pragma unroll 4
                for (int k = grp * 32 + lane; k < n4; k += 64) p4[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        const float per_unit = NEG ? (float)fs.q.gridA / (float)fs.q.unitsA : 0.f;
        IterA un(ub, sc);
        if (grp == 1) un.next(sc);
#pragma unroll 1
        for (int it = grp; it < n_iter; it += 2, un.next(sc), un.next(sc)) {
            const int stage = it & (kInfoStages - 1);
            // filter words: one per negative, naming a batch row in the padded numbering
            int w[4];
            const int n0 = (NEG ? un.rb : un.tile) * 128;
            const int r0 = (un.zc >= d.C ? un.zc - d.C : un.zc) * L.npc + (NEG ? un.tile : un.rb) * 128;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int j = n0 + q * 32 + lane;
                w[q] = j < d.N ? __ldg(&L.mask[(int64_t)un.zc * d.N + j]) : -1;
            }
            float v[4];
            if (NEG) {
                const int item = un.zc * fs.q.RB + un.tile;  // the query block these columns are
                const int u0 = item * fs.q.T, u1 = u0 + fs.q.T;
                int p = min((int)((float)u0 * per_unit), fs.q.gridA - 1), nparts = 1;
                while (s_range[p] > u0) p--;
                while (s_range[p + 1] <= u0) p++;
                while (s_range[p + nparts] < u1) nparts++;
                const int64_t grow0 = (int64_t)un.zc * L.npc + un.tile * BN;
                if (nparts == 1) {
#pragma unroll
                    for (int q = 0; q < 4; q++) v[q] = __ldg(&L.lse2s[(int64_t)item * BM + q * 32 + lane]);
                } else {
                    float4 pk[4];  // (m, sum) of the first two parts
                    float pos2[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int r = min(q * 32 + lane, L.npc - 1 - un.tile * BN);
                        pk[q] = __ldg(reinterpret_cast<const float4*>(L.part + (grow0 + r) * kMaxParts * 2));
                        pos2[q] = __ldg(&L.pos[grow0 + r]) * kLog2e;
                    }
#pragma unroll 1
                    for (int q = 0; q < 4; q++) {
                        const float4 a4 = q == 0 ? pk[0] : q == 1 ? pk[1] : q == 2 ? pk[2] : pk[3];
                        const float ps = q == 0 ? pos2[0] : q == 1 ? pos2[1] : q == 2 ? pos2[2] : pos2[3];
                        float x;
                        if (nparts == 2) {
                            const float mm = fmaxf(ps, fmaxf(a4.x, a4.z));
                            x = mm + __log2f(exp2f_fast(ps - mm) + a4.y * exp2f_fast(a4.x - mm) + a4.w * exp2f_fast(a4.z - mm));
                        } else {
                            x = combine_parts(reinterpret_cast<const float2*>(L.part) + (grow0 + min(q * 32 + lane, L.npc - 1 - un.tile * BN)) * kMaxParts, nparts, ps);
                        }
                        x = un.tile * BN + q * 32 + lane < L.npc ? x - (float)kWShift : kDeadRow;
                        v[0] = q == 0 ? x : v[0], v[1] = q == 1 ? x : v[1], v[2] = q == 2 ? x : v[2], v[3] = q == 3 ? x : v[3];
                    }
                }
            }
            bool any = false;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                w[q] = w[q] >= r0 && w[q] < r0 + 128 ? w[q] - r0 : -1;
                any |= w[q] >= 0;
            }
            any = __any_sync(0xffffffffu, any);
            if (!warp_wait(kBarInfoEmpty + stage, ((it / kInfoStages) & 1) ^ 1)) break;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (any) s_mask[stage * 128 + q * 32 + lane] = w[q];
                if (NEG) s_lse[stage * 128 + q * 32 + lane] = v[q];
            }
            if (lane == 0) s_any[stage] = any;
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[kBarInfoFull + stage]);
        }
    }
    // ---- common exit: every role ends here, normally or after an abort; then tensor memory is released ----------
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        if (*s_abort && lane == 0) {
            // a wait ran out somewhere: give copies and contractions still in flight a bounded chance to land before the SM's shared and
            // tensor memory are handed to the next CTA
            for (int k = 0; k < kStages; k++) settle_bar(&bars[kBarYFull + k]);
            for (int k = 0; k < 2; k++) settle_bar(&bars[kBarSFull + k]);
            settle_bar(&bars[kBarOFull]);
        }
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

template <int DP>
int launch(const LpKernelArgs& a, cudaStream_t stream) {
    if (a.L.Qh == nullptr || a.L.Kh == nullptr || a.L.lse2s == nullptr || a.L.o_part == nullptr) return GE2_ERR_WORKSPACE;
    const int ZC = a.L.S * a.d.C;
    const int tail_cols = ((a.d.D % 32) + 3) & ~3;
    CUtensorMap tmQ, tmK, tmO[2], tmOt[2];
    int rc = make_operand_map(&tmQ, a.L.Qh, false, DP, a.L.npc, ZC);
    if (rc == GE2_OK) rc = make_operand_map(&tmK, a.L.Kh, false, DP, a.d.N, ZC);
    for (int k = 0; k < 2 && rc == GE2_OK; k++) {
        float* out = k == 0 ? a.L.dQ : a.L.dK;
        const int rows = k == 0 ? a.L.npc : a.d.N;
        rc = make_slab_map(&tmO[k], out, DP, rows, ZC);
        tmOt[k] = tmO[k];  // narrow slab for the last D % 32 columns (rounded up to 4), when there are any
        if (rc == GE2_OK && tail_cols > 0 && tail_cols < 32) rc = make_slab_map(&tmOt[k], out, DP, rows, ZC, tail_cols);
    }
    if (rc != GE2_OK) return rc;
    FlashSched fs;
    const int qb = ceil_div(a.L.npc, BM), nb = ceil_div(a.d.N, BN);
    const long long units = (long long)ZC * qb * nb;
    if (2 * units > 0x3fffffff) return GE2_ERR_UNSUPPORTED;
    fs.q.RB = qb, fs.q.T = nb, fs.n.RB = nb, fs.n.T = qb;
    fs.q.ZC = fs.n.ZC = ZC;
    fs.q.unitsA = fs.n.unitsA = fs.q.unitsB = fs.n.unitsB = (int)units;
    // every CTA's range is at least ceil(T / 7) units long, so a row block is shared by at most kMaxParts CTAs
    fs.q.gridA = fs.q.gridB = std::max(1, std::min(kNumSMs, (int)units / ceil_div(nb, kMaxParts - 1)));
    fs.n.gridA = fs.n.gridB = std::max(1, std::min(kNumSMs, (int)units));
    GE2_CUDA_TRY(cudaFuncSetAttribute(lp_flash_kernel<DP, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Layout<DP>::kDynamic));
    GE2_CUDA_TRY(cudaFuncSetAttribute(lp_flash_kernel<DP, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Layout<DP>::kDynamic));
    GE2_CUDA_TRY(launch_after(lp_flash_kernel<DP, false>, dim3((unsigned)fs.q.gridA), dim3(kThreads), Layout<DP>::kDynamic, stream, tmQ, tmK, tmO[0], tmOt[0], a, fs));
    GE2_CUDA_TRY(launch_after(lp_flash_kernel<DP, true>, dim3((unsigned)fs.n.gridA), dim3(kThreads), Layout<DP>::kDynamic, stream, tmK, tmQ, tmO[1], tmOt[1], a, fs));
    return GE2_OK;
}

}  // namespace

int lp_flash_f16(const LpKernelArgs& a, cudaStream_t stream) {
    if (a.L.ld == 64) return launch<64>(a, stream);
    if (a.L.ld == 128) return launch<128>(a, stream);
    return GE2_ERR_UNSUPPORTED;
}

}  // namespace ge2
