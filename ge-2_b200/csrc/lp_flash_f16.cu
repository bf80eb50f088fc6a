// Scores kernels of the link-prediction step's tensor path (kind::f16) for large batches (lp_uses_flash): the streaming
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
// Tensor memory (512 columns): two score accumulators at 0 and 128, two O accumulators at 256 and 384.  Two groups of four softmax
// warps, a thread a row, take alternate tiles, each with its own score accumulator, its own O and (queries) its own m, so one group
// exponentiates while the other's contractions run.  P goes to the contraction in two halves of 64 columns, the first while the second is
// exponentiated.
// Bound by the chain scores -> exponentials -> O -> scores of a group, about 4200 cycles for its tile: 2300 ... 2800 of exponentials (2048 if
// the unit for them were never idle, for both groups' tiles), 768 of contractions behind the last of them, the hand-overs.  The tensor pipe,
// 1024 cycles a tile, is half busy.  B = 100 000, N = 2000, D = 128, two sides: 226 + 212 us (two warps a row, with a pass over the
// scores for the maximum and an exchange of it: 259 + 231).
// Measured on the way there, in turn with a form that took 229 + 227: one issuing warp for both groups, 261 + 235; an issuing warp a
// group without turns, 246 + 244; with turns at the second half of O only, 229 + 227; halves of a tile as score tiles of their own (the
// tensor pipe then has 1280 cycles a tile, and every hand-over twice), 264 + 278; an L2 prefetch of tiles to come, 227 + 224; five stages and
// one X, 221 + 230; three stages, 325 + 287; the maximum of every 64 scores before their exponentials instead of sums of those, 253 + 209 (226 + 212).
// P carries a factor 2^14, for fp16's subnormal range: against its reference a P of the queries keeps its full significand down to 2^-28
// and its last bit down to 2^-38; the same holds for a probability in the negatives' launch, whose reference is the row's lse (a row whose
// positive leads by 2^38 and more adds nothing to dK).  dQ and dK leave this kernel with that factor still on them and the finish
// kernel, their only reader, takes it off (LpLayout::grad_unscale).
//
// A row's reference starts at its positive score, but from 2^6 to 2^14 above the maximum of the group's first tile: a P of 1 or more then belongs
// to that maximum, 14 octaves above the subnormal numbers, and later tiles have 2^8 to 2^16 of room, less what a sum of 16 takes, before the
// reference has to follow.  The positive alone, as a reference, takes P's bits where it leads by more: dQ of a row was off by 1 % at
// 20 nats and zero at 28.  It starts no lower than that because following costs: B = 100 000, N = 2000, tables trained for 400 steps (positives
// ahead by up to 2^11), Dot 64 and 128, both launches: 200 and 248 us; with at most 2^10 above the maximum 213 and 259, with 2^8 220
// and 269.  Where one batch of DistMult 128 is trained 650 times over, positives are ahead by 2^10 to 2^50 and later tiles' maxima
// ahead of the first's by as much: 271 us for the queries' launch, 227 with the positive alone.  (Moving as far towards the positive again, and all
// rows of the warp at once: 257 there, 1 to 2 us more on the tables before.)
//
// Warp roles, connected by mbarrier pipelines (no block-wide barrier inside the loops):
//   warps 0-7   softmax: warp w takes rows 32 (w & 3) ... + 31 (its quarter of the tensor-memory lanes) of its group's (w >> 2) tiles
//   warps 8-11  drain: O -> registers (-> weighted sum of the two groups) -> staging slab -> TMA store / reduce-add
//   warp  12    TMA producer
//   warps 13-14 issue the contractions of a group each; warp 13 also allocates and frees tensor memory
//   warp  15    what the softmax warps need to know about coming tiles: which entries are masked and, for the negatives, the columns'
//               lse.  Queries: it first clears the dK rows the second launch reduces into
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
constexpr int kGroupWarps = 4;          // softmax warps of a group: one a quarter of the tensor-memory lanes
constexpr int kSoftmaxWarps = 2 * kGroupWarps;
constexpr int kThreads = 512;           // 128 registers each at the launch; the drain warps take some of warps 12-15 (setmaxnreg)
constexpr int kLaunchRegs = 128, kDrainRegs = 184, kServiceRegs = 2 * kLaunchRegs - kDrainRegs;
constexpr int kDrainWarps = 4, kTmaWarp = 12, kMmaWarp = 13, kHelpWarp = 15;  // (an issuing warp a group)
constexpr int kStages = 4;              // Y ring: two tiles wait for their O contraction, two are on their way
constexpr int kInfoStages = 4;          // ring of what warp 15 finds out about tiles
constexpr uint32_t kTmemCols = 512;
constexpr float kMasked = -1e9f;
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
constexpr int kWShift = 14;             // P is scaled by 2^14; undone by the reader of dQ / dK (kLpF16GradUnscale)
constexpr float kHeadStart = 6.f;       // queries: log2 of how far the reference is set above the maximum it is taken from ...
constexpr float kFarthest = 14.f;       // ... and, for a positive that leads it, at most (the largest P of the tile then is 1)
constexpr float kNothing = 128.f;       // log2 of how much smaller than the positive's a term of the row's sum is nothing, in fp32 too
constexpr float kNoReference = -1e30f;  // queries: of a group without a tile of the block
constexpr float kDeadRow = 1e30f;       // "lse" of a row past the end of its chunk: exp2(anything - 1e30) = 0

enum Bar { kBarXFull = 0, kBarXEmpty = 2, kBarYFull = 6, kBarYEmpty = kBarYFull + kStages, kBarSFull = kBarYEmpty + kStages, kBarPFull = kBarSFull + 2,
           kBarHalf = kBarPFull + 4, kBarTurn = kBarHalf + 2, kBarOFull = kBarTurn + 2, kBarOEmpty = kBarOFull + 2, kBarStat = kBarOEmpty + 2, kBarStatFree = kBarStat + 2,
           kBarInfoFull = kBarStatFree + 2, kBarInfoEmpty = kBarInfoFull + kInfoStages, kNumBars = kBarInfoEmpty + kInfoStages };

template <int DP>
struct Layout {
    static constexpr int NB = DP / 64;               // column blocks of X / Y
    static constexpr int kTileBytes = NB * kBlockBytes;
    static constexpr int kX = 0;
    static constexpr int kY = kX + 2 * kTileBytes;
    static constexpr int kDrain = kY + kStages * kTileBytes;       // 4 drain warps x one slab (32 rows x 128 bytes), 128-byte swizzled
    static constexpr int kMisc = kDrain + kDrainWarps * 4096;  // barriers, tensor-memory address, abort flag
    static constexpr int kStat = kMisc + 1024;                     // (m, sum) at the end of a block: [buffer][group][128]
    static constexpr int kLse = kStat + 2 * 2 * 128 * 8;           // [kInfoStages][128]: minus the columns' lse
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

__device__ __forceinline__ float max3(float a, float b, float c) {  // one instruction
    float y;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}
// Registers of a warpgroup (four warps, all of which run this): given back to the CTA, taken from what others gave back.  The CTA is launched
// with kThreads x kLaunchRegs of them, and the shares add up to that, so the wait of the second form ends.
template <int N>
__device__ __forceinline__ void regs_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void regs_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}

// base-2 logsumexp of a row from its positive score and the parts its sharers left
__device__ __forceinline__ float combine_parts(const float2* part, int nparts, float pos2) {
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
    int masks;   // are any scores masked in this step?
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
    auto warp_wait = [&](int bar, uint32_t parity) { return warp_wait_inline(&bars[bar], parity, s_abort, d.status); };

    if (warp == kTmaWarp && lane == 0) {
        for (int k = 0; k < 2; k++) {
            mbar_init(&bars[kBarXFull + k], 1);
            mbar_init(&bars[kBarXEmpty + 2 * k], 1), mbar_init(&bars[kBarXEmpty + 2 * k + 1], 1);  // [buffer][group]
            mbar_init(&bars[kBarSFull + k], 1);
            mbar_init(&bars[kBarHalf + k], 1);
            mbar_init(&bars[kBarTurn + k], 1);
            mbar_init(&bars[kBarOFull + k], 1);
            mbar_init(&bars[kBarOEmpty + k], kDrainWarps);
            mbar_init(&bars[kBarStat + k], kSoftmaxWarps);
            mbar_init(&bars[kBarStatFree + k], kDrainWarps);
        }
        for (int k = 0; k < 4; k++) mbar_init(&bars[kBarPFull + k], kGroupWarps);  // [group][half of the tile's columns]: one arrival a warp
        for (int k = 0; k < kStages; k++) {
            mbar_init(&bars[kBarYFull + k], 1);
            mbar_init(&bars[kBarYEmpty + k], 1);
        }
        for (int k = 0; k < kInfoStages; k++) {
            mbar_init(&bars[kBarInfoFull + k], 1);
            mbar_init(&bars[kBarInfoEmpty + k], kGroupWarps);
        }
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

    if (warp < kSoftmaxWarps) {
        // ================================ softmax warps (0-7) ================================
        const int grp = warp >> 2, wq = warp & 3;
        const int my_row = tid & 127;   // accumulator row / tensor-memory lane
        const uint32_t tS = tmem + grp * 128 + lane_sel;
        IterA un(ub, sc);
        float m = kNoReference, l = 0.f;  // queries: reference and sum (scaled by 2^14) of this group's tiles of the block
        if (grp == 1) un.next(sc);
        int item = decode_a(ub, sc).item, sg = 0;  // the block at hand, and how many came before it
        bool begun = false;  // has this group made a P of the block at hand?
        auto leave = [&](int next) -> bool {  // queries: what this group knows about the blocks before `next`
            for (; item < next; item++, sg++) {
                const int h = sg & 1;
                if (!warp_wait(kBarStatFree + h, ((sg >> 1) & 1) ^ 1)) return false;
                s_stat[(h * 2 + grp) * 128 + my_row] = make_float2(m, l);
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars[kBarStat + h]);
                m = kNoReference;
                l = 0.f;
            }
            return true;
        };
        bool ok = true;
#pragma unroll 1
        for (int it = grp; it < n_iter; it += 2, un.next(sc), un.next(sc)) {
            if (!NEG && !(ok = leave(un.item))) break;
            if (!NEG && (it == grp || un.tile < 2)) {  // (a block's first tile for this group)
                const int r = un.rb * BM + my_row;
                m = r < x_rows ? fmaxf(__ldg(&L.pos[(int64_t)un.zc * L.npc + r]) * kLog2e, kNoReference) : 0.f;
                begun = false;
            }
            const int nth = it >> 1, stage = it & (kInfoStages - 1);
            const int nv = y_rows - un.tile * BN;  // columns of the tile that exist (negatives: the others' lse leaves nothing of them)
            if ((NEG || fs.masks) && !warp_wait(kBarInfoFull + stage, (it / kInfoStages) & 1)) break;
            const bool masked = fs.masks && s_any[stage];
            if (!warp_wait(kBarSFull + grp, nth & 1)) break;
            tc_fence_after();
            if (masked || (!NEG && nv < BN)) {
                // scores of masked entries, and of columns that do not exist, are replaced in tensor memory: few tiles have any
                const float value = NEG ? -INFINITY : kMasked;
                const int* msk = s_mask + stage * 128;
#pragma unroll 1
                for (int k = masked ? 0 : 4; k < 4; k++) {
                    const int w = msk[NEG ? my_row : k * 32 + lane];  // negatives: the column of my row, queries: the row of a column
                    unsigned left = __ballot_sync(0xffffffffu, NEG ? (w >> 5) == k : (w >> 5) == wq);
                    while (left != 0) {
                        const int src = __ffs(left) - 1;
                        left &= left - 1;
                        const int of = __shfl_sync(0xffffffffu, w, src);
                        const uint32_t at = tS + (NEG ? of : k * 32 + src);
                        const float x = tmem_ld_32x1(at);
                        tmem_st_32x1(at, (NEG ? lane == src : my_row == of) ? value : x);
                        tmem_st_wait();
                    }
                }
                if (!NEG) {
#pragma unroll 1
                    for (int c = nv; c < BN; c++) tmem_st_32x1(tS + c, -INFINITY);
                }
                tmem_st_wait();
            }
            if (!NEG) {
                float* dump = un.zc < d.C ? d.neg_scores : d.inv_neg_scores;
                if (__builtin_expect(dump != nullptr, 0)) {  // the score dump of the tests
                    float* drow = dump + ((int64_t)(un.zc >= d.C ? un.zc - d.C : un.zc) * L.npc + un.rb * BM + my_row) * d.N + un.tile * BN;
#pragma unroll 1
                    for (int c = 0; c < min(nv, BN); c++) {
                        const float x = tmem_ld_32x1(tS + c);
                        if (my_row < x_rows - un.rb * BM) drow[c] = x;
                    }
                }
            }
            // P over the lower half of the 64 score columns it is made from, with the next 64 on their way
            const float* neg_lse = s_lse + stage * 128;
            float va[32], vb[32];
            tmem_ld_32x32_start(tS + 64, va);
            tmem_ld_32x32_start(tS + 96, vb);
#pragma unroll 1
            for (int h = 1; h >= 0; h--) {
                uint32_t wa[16], wb[16];
                float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
                tmem_ld_wait(va, vb);
                auto largest = [&](const float (&a)[32]) {
                    float mx[4] = {max3(a[0], a[1], a[2]), max3(a[3], a[4], a[5]), max3(a[6], a[7], a[8]), max3(a[9], a[10], a[11])};
#pragma unroll
                    for (int j = 12; j < 28; j += 2) mx[(j >> 1) & 3] = max3(mx[(j >> 1) & 3], a[j], a[j + 1]);
                    return max3(max3(mx[0], a[28], a[29]), max3(mx[1], a[30], a[31]), fmaxf(mx[2], mx[3])) * kLog2e;
                };
                // Queries: the first reference (see above).  It follows only when a P might leave fp16's range: O and the sum have to be rescaled then, for
                // 32 rows at a time.  That is looked for in sums of the exponentials (of 16 of them: none is larger), not in a pass over
                // the scores, which was a tenth of the launch.  A first tile that is masked for the row as a whole says nothing about its scores:
                // the reference is 2^-128 of the positive then.
                if (!NEG && !begun && h == 1) {
                    float tmax = fmaxf(largest(va), largest(vb));
#pragma unroll 1
                    for (int k = 0; k < 2; k++) {
                        float x[32];
                        tmem_ld_32x32(tS + k * 32, x);
                        tmax = fmaxf(tmax, largest(x));
                    }
                    m = fmaxf(fmaxf(tmax + kHeadStart, m - kNothing), fminf(m, tmax + kFarthest));
                }
#pragma unroll 1
                for (bool settled = false;; settled = true) {
                    const float neg_shift = (float)kWShift - m;
                    sum[0] = sum[1] = make_float2(0.f, 0.f);
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        float (&v)[32] = k == 0 ? va : vb;
                        uint32_t (&w)[16] = k == 0 ? wa : wb;
#pragma unroll
                        for (int q = 0; q < 8; q++) {
                            float4 sh = make_float4(neg_shift, neg_shift, neg_shift, neg_shift);
                            if (NEG) sh = *reinterpret_cast<const float4*>(neg_lse + h * 64 + k * 32 + 4 * q);
                            float2 a = fma2(make_float2(v[4 * q], v[4 * q + 1]), make_float2(kLog2e, kLog2e), make_float2(sh.x, sh.y));
                            float2 b = fma2(make_float2(v[4 * q + 2], v[4 * q + 3]), make_float2(kLog2e, kLog2e), make_float2(sh.z, sh.w));
                            a.x = exp2f_fast(a.x), a.y = exp2f_fast(a.y), b.x = exp2f_fast(b.x), b.y = exp2f_fast(b.y);
                            if (!NEG) sum[0] = add2(sum[0], a), sum[1] = add2(sum[1], b);
                            w[2 * q] = pack_half2(a.x, a.y);
                            w[2 * q + 1] = pack_half2(b.x, b.y);
                            asm volatile("" : "+r"(w[2 * q]), "+r"(w[2 * q + 1]));  // (packed before anything else is looked at)
                        }
                    }
                    if (NEG || settled) break;
                    if (__builtin_expect(!__any_sync(0xffffffffu, fmaxf(fmaxf(sum[0].x, sum[0].y), fmaxf(sum[1].x, sum[1].y)) > 65504.f), 1)) break;
                    const float tmax = fmaxf(largest(va), largest(vb));
                    const bool up = tmax > m + 1.f - kHeadStart;  // (by at least a factor 2)
                    if (begun && __any_sync(0xffffffffu, up)) {
                        // (the contraction of this tile's first half may be adding to O)
                        if (h == 0 && !(ok = warp_wait(kBarHalf + grp, nth & 1))) break;
                        tc_fence_after();
                        const float f = up ? exp2f_fast(m - tmax - kHeadStart) : 1.f;
                        l *= f;
#pragma unroll 1
                        for (int q = 0; q * 32 < d.D; q++) {
                            const uint32_t at = tmem + 256 + grp * 128 + lane_sel + q * 32;
                            float o[32];
                            tmem_ld_32x32(at, o);
#pragma unroll
                            for (int k = 0; k < 2; k++) {
                                uint32_t x[16];
#pragma unroll
                                for (int j = 0; j < 16; j++) x[j] = __float_as_uint(o[k * 16 + j] * f);
                                tmem_st_32x16_start(at + k * 16, x);
                            }
                        }
                        tmem_st_wait();
                    }
                    if (up) m = tmax + kHeadStart;
                }
                if (!ok) break;
                if (!NEG) {
                    const float2 x = add2(sum[0], sum[1]);
                    l += x.x + x.y;
                }
                if (h == 1) {
                    tmem_ld_32x32_start(tS, va);
                    tmem_ld_32x32_start(tS + 32, vb);
                }
                tmem_st_32x16_start(tS + h * 64, wa);
                tmem_st_32x16_start(tS + h * 64 + 16, wb);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars[kBarPFull + grp * 2 + h]);
                begun = true;
            }
            if (!ok) break;
            if ((NEG || fs.masks) && lane == 0) mbar_arrive(&bars[kBarInfoEmpty + stage]);
        }
        if (!NEG && ok && n_iter > 0) leave(decode_a(ue - 1, sc).item + 1);
    } else if (warp < kTmaWarp) {
        regs_inc<kDrainRegs>();
        // ================================ drain warps (8-11) ================================
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
                float lse2 = 0.f, loss = 0.f, w0 = 0.f, w1 = 0.f;  // (the last two: weights of the first two parts of row `lane`)
                if (lane < rows) {
                    const float pos2 = __ldg(&L.pos[grow0 + lane]) * kLog2e;
                    lse2 = combine_parts(reinterpret_cast<const float2*>(L.part) + (grow0 + lane) * kMaxParts, nparts, pos2);
                    L.lse[grow0 + lane] = lse2 * kLn2;
                    loss = (lse2 - pos2) * kLn2;
                    const float4 pw = __ldg(reinterpret_cast<const float4*>(L.part) + (grow0 + lane) * (kMaxParts / 2));  // their (m, sum)
                    w0 = exp2f_fast(pw.x - lse2), w1 = exp2f_fast(pw.z - lse2);
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
#pragma unroll 1
                for (int r0 = lane / kLanes; r0 < 32; r0 += 8 * kSide) {  // eight rows' loads on their way at a time
                    float4 s[8], o[8];
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const int r = min(r0 + k * kSide, rows - 1);
                        s[k] = *reinterpret_cast<const float4*>(o0 + r * DP), o[k] = *reinterpret_cast<const float4*>(o1 + r * DP);
                    }
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const int r = r0 + k * kSide;
                        const float a0 = __shfl_sync(0xffffffffu, w0, r & 31), a1 = __shfl_sync(0xffffffffu, w1, r & 31), lr = __shfl_sync(0xffffffffu, lse2, r & 31);
                        s[k].x = fmaf(a1, o[k].x, a0 * s[k].x), s[k].y = fmaf(a1, o[k].y, a0 * s[k].y);
                        s[k].z = fmaf(a1, o[k].z, a0 * s[k].z), s[k].w = fmaf(a1, o[k].w, a0 * s[k].w);
                        if (r < rows) {
#pragma unroll 1
                            for (int p = 2; p < nparts; p++) {
                                const float4 x = *reinterpret_cast<const float4*>(o1 + ((int64_t)(p - 1) * 2 * BM + r) * DP);
                                const float w = exp2f_fast(__ldg(&part[r * kMaxParts + p]).x - lr);
                                s[k].x = fmaf(w, x.x, s[k].x), s[k].y = fmaf(w, x.y, s[k].y), s[k].z = fmaf(w, x.z, s[k].z), s[k].w = fmaf(w, x.w, s[k].w);
                            }
                            *reinterpret_cast<float4*>(L.dQ + (grow0 + r) * DP + cl) = s[k];
                        }
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
        int sg = 0, filled[2] = {0, 0};  // blocks so far, of them with a tile of either group
#pragma unroll 1
        for (int u = ub; u < ue; sg++) {
            const UnitA un = decode_a(u, sc);
            const int seg_end = min(ue, (un.item + 1) * sc.T);
            const bool whole = un.tile == 0 && seg_end == (un.item + 1) * sc.T;
            const int row0 = un.rb * BM + wq * 32;
            const bool live = row0 + lane < x_rows;
            // Iterations u - ub ... seg_end - ub - 1 alternate between the groups and their accumulators; the one that the next block's first tile
            // wants is read first.
            const int acc0 = (seg_end - ub) & 1;
            const bool two = seg_end - u > 1, have0 = two || ((u - ub) & 1) == acc0, have1 = two || !have0;
            int& n0 = acc0 == 0 ? filled[0] : filled[1];
            int& n1 = acc0 == 0 ? filled[1] : filled[0];
            float pos2 = 0.f;
            if (!NEG && live) pos2 = __ldg(&L.pos[(int64_t)un.zc * L.npc + row0 + lane]) * kLog2e;
            // the whole of O into registers, so that the accumulators are free before anything is stored; the first of them as it is, before the
            // other group is done
            float v[DP];
            if (have0) {
                if (!warp_wait(kBarOFull + acc0, n0++ & 1)) break;
                tc_fence_after();
            }
#pragma unroll
            for (int q = 0; q < DP / 32; q++) {
                float o[32];
                if (have0) tmem_ld_32x32(tmem + 256 + acc0 * 128 + lane_sel + q * 32, o);
#pragma unroll
                for (int j = 0; j < 32; j++) v[q * 32 + j] = have0 ? o[j] : 0.f;
            }
            tc_fence_before();
            __syncwarp();
            if (have0 && lane == 0) mbar_arrive(&bars[kBarOEmpty + acc0]);
            float w1 = 1.f, m = 0.f, l = 0.f, lse2 = 0.f;
            if (!NEG) {
                const int h = sg & 1, r = wq * 32 + lane;
                if (!warp_wait(kBarStat + h, (sg >> 1) & 1)) break;
                const float2 a0 = s_stat[(h * 2 + acc0) * 128 + r], b0 = s_stat[(h * 2 + (acc0 ^ 1)) * 128 + r];
                m = fmaxf(a0.x, b0.x);  // (a group without a tile in this share: weight 0)
                float w0 = exp2f_fast(a0.x - m);
                w1 = exp2f_fast(b0.x - m);
                l = (a0.y * w0 + b0.y * w1) * (1.f / (1 << kWShift));
                if (whole) {
                    const float nm = fmaxf(m, pos2);
                    lse2 = nm + __log2f(l * exp2f_fast(m - nm) + exp2f_fast(pos2 - nm));
                    const float f = exp2f_fast(m - lse2);
                    w0 *= f, w1 *= f;
                }
#pragma unroll
                for (int j = 0; j < DP; j++) v[j] *= w0;
            }
            if (have1) {
                if (!warp_wait(kBarOFull + (acc0 ^ 1), n1++ & 1)) break;
                tc_fence_after();
#pragma unroll
                for (int q = 0; q < DP / 32; q++) {
                    float o[32];
                    tmem_ld_32x32(tmem + 256 + (acc0 ^ 1) * 128 + lane_sel + q * 32, o);
#pragma unroll
                    for (int j = 0; j < 32; j++) v[q * 32 + j] = NEG ? v[q * 32 + j] + o[j] : fmaf(o[j], w1, v[q * 32 + j]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (have1 && lane == 0) mbar_arrive(&bars[kBarOEmpty + (acc0 ^ 1)]);
            if (!NEG) {
                if (lane == 0) mbar_arrive(&bars[kBarStatFree + (sg & 1)]);
                const int64_t grow = (int64_t)un.zc * L.npc + row0 + lane;
                if (whole) {
                    float loss = 0.f;
                    if (live) {
                        L.lse[grow] = lse2 * kLn2;
                        loss = (lse2 - pos2) * kLn2;
                    }
                    L.lse2s[(int64_t)un.item * BM + wq * 32 + lane] = live ? lse2 - (float)kWShift : kDeadRow;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
                    if (lane == 0) atomicAdd(L.loss_acc, (double)loss);
                } else if (live) {
                    const int part = (int)blockIdx.x - cta_of_unit(un.item * sc.T, sc.unitsA, (int)gridDim.x);
                    if (part < kMaxParts) reinterpret_cast<float2*>(L.part)[grow * kMaxParts + part] = make_float2(m, l);
                }
            }
            float* part_rows = L.o_part + (((int64_t)blockIdx.x * 2 + (un.tile == 0 ? 1 : 0)) * BM + wq * 32 + lane) * DP;
            int y = row0, z = un.zc;
            // The coordinates are pinned in ordinary registers here, where the whole warp is active: taken straight from the
            // index arithmetic into the one-lane section below, the third coordinate was seen to reach the store as 0.
            asm volatile("" : "+r"(y), "+r"(z));
#pragma unroll
            for (int cb = 0; cb < DP / 32; cb++) {
                if (cb >= drain_slabs) break;
                if (!NEG && !whole) {
#pragma unroll
                    for (int q = 0; q < 8; q++)
                        *reinterpret_cast<float4*>(part_rows + cb * 32 + 4 * q) =
                            make_float4(v[cb * 32 + 4 * q], v[cb * 32 + 4 * q + 1], v[cb * 32 + 4 * q + 2], v[cb * 32 + 4 * q + 3]);
                    continue;
                }
                if (lane == 0) bulk_wait_group_read<0>();  // the operation that last used the slab has read it
                __syncwarp();
                const bool narrow = cb == full_slabs;
                if (!narrow) {
#pragma unroll
                    for (int q = 0; q < 8; q++)
                        *reinterpret_cast<float4*>(scr + lane * 128 + ((q ^ (lane & 7)) << 4)) =
                            make_float4(v[cb * 32 + 4 * q], v[cb * 32 + 4 * q + 1], v[cb * 32 + 4 * q + 2], v[cb * 32 + 4 * q + 3]);
                } else {
#pragma unroll
                    for (int q = 0; q < 8; q++)
                        if (q * 4 < tail)
                            *reinterpret_cast<float4*>(scr + lane * (tail * 4) + q * 16) =
                                make_float4(v[cb * 32 + 4 * q], v[cb * 32 + 4 * q + 1], v[cb * 32 + 4 * q + 2], v[cb * 32 + 4 * q + 3]);
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
        regs_dec<kServiceRegs>();
        if (warp == kTmaWarp) {
            int sg = -1, users[2] = {0, 0}, uses[4] = {0, 0, 0, 0};  // of the X buffers: groups with a tile of the block there, uses so far [buffer][group]
            bool ok = true;
            IterA un(ub, sc);
            for (int it = 0; it < n_iter; it++, un.next(sc)) {
                if (it == 0 || un.tile == 0) {  // a new block
                    sg++;
                    const int xs = sg & 1;
#pragma unroll
                    for (int g = 0; g < 2; g++) {
                        int& n = xs == 0 ? uses[g] : uses[2 + g];
                        if (((xs == 0 ? users[0] : users[1]) >> g) & 1) ok = ok && warp_wait(kBarXEmpty + 2 * xs + g, n & 1), n++;
                    }
                    if (!ok) break;
                    (xs == 0 ? users[0] : users[1]) = min(sc.T - un.tile, n_iter - it) > 1 ? 3 : 1 << (it & 1);
                    mbar_expect_tx_warp(&bars[kBarXFull + xs], LY::kTileBytes);
#pragma unroll
                    for (int b = 0; b < NB; b++) tma_load_3d_warp(sX + xs * LY::kTileBytes + b * kBlockBytes, &tmX, b * 64, un.rb * BM, un.zc, &bars[kBarXFull + xs]);
                }
                const int st = it % kStages;
                if (!warp_wait(kBarYEmpty + st, ((it / kStages) & 1) ^ 1)) break;
                mbar_expect_tx_warp(&bars[kBarYFull + st], LY::kTileBytes);
#pragma unroll
                for (int b = 0; b < NB; b++)
                    tma_load_3d_warp(sY + st * LY::kTileBytes + b * kBlockBytes, &tmY, b * 64, un.tile * BN, un.zc, &bars[kBarYFull + st]);
            }
        } else if (warp < kHelpWarp) {
            // ================================ contractions ================================
            // One warp a group, so that one's waits do not keep the tensor pipe from the other's contractions.  S of the group's next tile follows O
            // of this one, so the score accumulator is overwritten only behind the contraction that reads the P in it, and "S complete"
            // also says that the O contraction is.
            const int g = warp - kMmaWarp;
            const int D16 = ((d.D + kMmaK - 1) / kMmaK) * kMmaK;  // the embedding dimension rounded up to the MMA k step
            constexpr uint32_t kIdescS = idesc_f16(BM, BN, 0, 0);
            const uint32_t idesc_o = idesc_f16(BM, D16, 0, 1);
            const uint32_t dXk = desc_lo_sw128(smem_u32(sX), 16), dYk = desc_lo_sw128(smem_u32(sY), 16), dYm = desc_lo_sw128(smem_u32(sY), kBlockBytes);
            const uint32_t s = tmem + g * 128, o = tmem + 256 + g * 128;
            const int T = sc.T;
            int ts = decode_a(ub, sc).tile + g, bs = 0;  // the tile whose S is next: number within its block, block within this share
            while (ts >= T) ts -= T, bs++;
            int to = 0, bo = -1, used = -1, filled = 0;  // the one whose O is next; the block o holds something of; blocks it has held
            uint32_t par = 0;                            // of this group's tiles
            // The groups take turns at O of a tile and S of the next one: if both were given to the pipe at once, both would be done
            // late, and the groups would wait and exponentiate at the same time ever after.
#pragma unroll 1
            for (int k = g; k < n_iter + 2; k += 2) {
                const bool do_s = k < n_iter, do_o = k >= 2;
                const int xs = bs & 1, st = k % kStages, ko = k - 2;
                // whatever S needs besides its place is there before O is issued: nothing comes between the two in the pipe
                if (do_s) {
                    if (bs != bo && !warp_wait(kBarXFull + xs, (bs >> 1) & 1)) break;
                    if (!warp_wait(kBarYFull + st, (k / kStages) & 1)) break;
                }
                bool ok = true;
                if (do_o) {
                    uint32_t more = 1u;
                    if (used != bo) {  // a new block: the drain has read what is there
                        if (!warp_wait(kBarOEmpty + g, (filled & 1) ^ 1)) break;
                        filled++;
                        used = bo;
                        more = 0u;
                    }
                    const uint32_t y0 = dYm + (ko % kStages) * (LY::kTileBytes >> 4);
#pragma unroll
                    for (int h = 1; h >= 0; h--) {  // P of columns 64 h ... + 63 of the tile sits in columns 64 h ... + 31 of the score accumulator
                        if (!(ok = warp_wait(kBarPFull + g * 2 + h, par) && (h == 0 || warp_wait(kBarTurn + g, g == 0 ? par : par ^ 1u)))) break;
                        tc_fence_after();
#pragma unroll
                        for (int ks = 4 * h; ks < 4 * h + 4; ks++) {
                            mma_f16_ts_warp(o, s + h * 64 + (ks & 3) * 8, y0 + (uint32_t)koff_mnmajor(ks), idesc_o, more);
                            more = 1u;
                        }
                        if (!NEG && h == 1) mma_commit_warp(&bars[kBarHalf + g]);
                    }
                } else if (g == 1) {
                    ok = warp_wait(kBarTurn + 1, 0);
                }
                if (!ok) break;
                if (do_s) {
                    const uint32_t x0 = dXk + xs * (LY::kTileBytes >> 4), y0 = dYk + st * (LY::kTileBytes >> 4);
                    if (!do_o) tc_fence_after();
#pragma unroll
                    for (int ks = 0; ks < DP / kMmaK; ks++) mma_f16_ss_warp(s, x0 + (uint32_t)koff_kmajor(ks), y0 + (uint32_t)koff_kmajor(ks), kIdescS, ks > 0);
                    mma_commit_warp(&bars[kBarSFull + g]);
                    if (ts + 2 >= T || k + 2 >= n_iter) mma_commit_warp(&bars[kBarXEmpty + 2 * xs + g]);
                }
                if (lane == 0) mbar_arrive(&bars[kBarTurn + (g ^ 1)]);
                __syncwarp();
                if (do_o) {
                    mma_commit_warp(&bars[kBarYEmpty + ko % kStages]);
                    if (to + 2 >= T || !do_s) mma_commit_warp(&bars[kBarOFull + g]);  // the group's last tile of the block
                    par ^= 1u;
                }
                to = ts, bo = bs;
                ts += 2;
                while (ts >= T) ts -= T, bs++;
            }
        } else {
            // ================================ warp 15 ================================
            if (!NEG) {
                // clear the dK rows the second launch reduces into: those of every block whose stream it cuts at a CTA boundary (boundary j
                // is looked after by CTA (j - 1) % gridDim.x)
#pragma unroll 1
                for (int j = 1 + (int)blockIdx.x; j < fs.n.gridA; j += (int)gridDim.x) {
                    const UnitA un = decode_a(range_begin(j, fs.n.unitsA, fs.n.gridA), fs.n);
                    if (un.tile == 0) continue;  // the boundary falls between two blocks: nothing is split
                    float4* p4 = reinterpret_cast<float4*>(L.dK + ((int64_t)un.zc * d.N + (int64_t)un.rb * BM) * DP);
                    const int n4 = min(BM, d.N - un.rb * BM) * (DP / 4);
#pragma unroll 8
                    for (int k = lane; k < n4; k += 32) p4[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
            const int n_info = NEG || fs.masks ? n_iter : 0;
            const float per_unit = NEG ? (float)fs.q.gridA / (float)fs.q.unitsA : 0.f;
            int w[4] = {-1, -1, -1, -1};  // of a tile: filter words (one per negative, naming a batch row in the padded numbering)
            float v[4];                   // ... negatives: the columns' lse
            auto read = [&](const IterA& un) {
                if (fs.masks) {
                    const int n0 = (NEG ? un.rb : un.tile) * 128;
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int j = n0 + q * 32 + lane;
                        w[q] = j < d.N ? __ldg(&L.mask[(int64_t)un.zc * d.N + j]) : -1;
                    }
                }
                if (NEG) {
                    const int item = un.zc * fs.q.RB + un.tile;  // the query block these columns are
                    const int u0 = item * fs.q.T, u1 = u0 + fs.q.T;
                    int p = min((int)((float)u0 * per_unit), fs.q.gridA - 1), nparts = 1;
                    while (s_range[p] > u0) p--;
                    while (s_range[p + 1] <= u0) p++;
                    while (s_range[p + nparts] < u1) nparts++;
                    if (nparts == 1) {
#pragma unroll
                        for (int q = 0; q < 4; q++) v[q] = __ldg(&L.lse2s[(int64_t)item * BM + q * 32 + lane]);
                    } else {  // a block that the first launch split between CTAs
                        const int64_t grow0 = (int64_t)un.zc * L.npc + un.tile * BN;
                        float4 pk[4];  // (m, sum) of the first two parts
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const int64_t r = grow0 + min(q * 32 + lane, L.npc - 1 - un.tile * BN);
                            pk[q] = __ldg(reinterpret_cast<const float4*>(L.part + r * kMaxParts * 2));
                            v[q] = __ldg(&L.pos[r]) * kLog2e;
                        }
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const int r = min(q * 32 + lane, L.npc - 1 - un.tile * BN);
                            const float mm = fmaxf(v[q], fmaxf(pk[q].x, pk[q].z));
                            float x = mm + __log2f(exp2f_fast(v[q] - mm) + pk[q].y * exp2f_fast(pk[q].x - mm) + pk[q].w * exp2f_fast(pk[q].z - mm));
                            if (nparts > 2) x = combine_parts(reinterpret_cast<const float2*>(L.part) + (grow0 + r) * kMaxParts, nparts, v[q]);
                            v[q] = r == q * 32 + lane ? x - (float)kWShift : kDeadRow;
                        }
                    }
                }
            };
            IterA un(ub, sc);
            if (n_info > 0) read(un);
#pragma unroll 1
            for (int it = 0; it < n_info; it++) {
                const int stage = it & (kInfoStages - 1);
                const int r0 = (un.zc >= d.C ? un.zc - d.C : un.zc) * L.npc + (NEG ? un.tile : un.rb) * 128;
                int cw[4];
                float cv[4];
                bool any = false;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    cw[q] = w[q] >= r0 && w[q] < r0 + 128 ? w[q] - r0 : -1;
                    any |= cw[q] >= 0;
                    if (NEG) cv[q] = v[q];
                }
                un.next(sc);
                if (it + 1 < n_info) read(un);  // (on their way while this tile's are written)
                any = __any_sync(0xffffffffu, any);
                if (!warp_wait(kBarInfoEmpty + stage, ((it / kInfoStages) & 1) ^ 1)) break;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (any) s_mask[stage * 128 + q * 32 + lane] = cw[q];
                    if (NEG) s_lse[stage * 128 + q * 32 + lane] = -cv[q];
                }
                if (lane == 0) s_any[stage] = any;
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars[kBarInfoFull + stage]);
            }
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
            for (int k = 0; k < 2; k++) settle_bar(&bars[kBarOFull + k]);
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
    fs.masks = a.d.deg_sample_rows != nullptr || a.d.dst_filter_n > 0 || a.d.src_filter_n > 0;
    fs.q.unitsA = fs.n.unitsA = fs.q.unitsB = fs.n.unitsB = (int)units;
    // every CTA's range is at least ceil(T / 7) units long, so a row block is shared by at most kMaxParts CTAs
    fs.q.gridA = fs.q.gridB = std::max(1, std::min(scores_ctas(units), (int)units / ceil_div(nb, kMaxParts - 1)));
    fs.n.gridA = fs.n.gridB = scores_ctas(units);
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
