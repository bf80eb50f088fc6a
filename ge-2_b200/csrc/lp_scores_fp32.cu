// fp32 scores kernels of the link-prediction step (the 1e-4-parity path) on the tensor cores.
// Stand in for the reference's bmm + logsumexp + cross_entropy + autograd chain
// (cpp/src/nn/decoders/edge/comparators.cpp:128-138, cpp/src/nn/loss.cpp:46-63 of the reference project).
//
// Every fp32 operand is the exact sum of three bf16 values, x = xh + xm + xl (24 bits as 8 + 8 + 8, any exponent), and a product is
// taken as xl yh + xh yl + xm ym + xm yh + xh ym + xh yh: what is left out is below 2^-24 of |x y|, the size of one fp32 rounding.
// tcgen05.mma kind::f16 sums such products in fp32, but it truncates every addend and every sum (measured: products aligned to 25
// fraction bits of the largest addend, the sum cut to 24 bits), where the CUDA cores round.  So no long sum is left to it:
//   * the small products come first, when the accumulator is small; only the ceil(k / 16) steps of xh yh add to a full one;
//   * dQ, a sum over all negatives, is summed per tile of 64 negatives only; the tiles are added in registers, rounded to nearest;
//   * dK, a sum over all rows of a chunk, leaves every tile of 128 rows by fp32 atomic adds.
// Exponentials and logarithms are CUDA's expf / logf.  Errors against float64 are about those of a kernel of fp32 multiply-adds: gradients a
// quarter above, scores a little below (figures further down).
//
// Two persistent launches, as on the f16 path (lp_scores_f16.cu): a block X of 128 query rows stays on the SM and tiles Y of 64
// negatives stream past it,
//   lp_lse32_kernel    S = X Y^T tile by tile, running (max, sum) per row                                             -> lse, loss
//   lp_grad32_kernel   S again, P = exp(S - lse) split into W (three planes in shared memory), dQ += W Y, dK^T = X^T W
// Operands sit in shared memory (X of the logsumexp pass: in tensor memory) as planes of 64-column blocks in the 128-byte-swizzled layout that TMA writes; read along rows a
// block is a K-major operand, along columns an MN-major one, so each serves both of its contractions.
//
// Bound by the contractions: 6 products a multiply-add, 4 contractions' worth of them (S twice, dQ, dK) = 24 x S B N D x 2 flops of bf16, at
// N = 64 with both operands in shared memory limited by its bandwidth (48 cycles a k-step; A in tensor memory: 32).
// B = 10 000, 1 000 negatives, D = 100, two sides: 31 + 86 us (one kernel of fp32 multiply-adds: 776 us); 1 000 edges, D = 50: 9.7 + 17.5 us
// (202 us).  Relative 2-norm error against float64 at B = 4 000, N = 1 000, D = 100 (and that of the multiply-adds): node gradient 5.3e-7
// (4.2e-7), scores 1.5e-7 (1.6e-7).
// The logsumexp pass keeps X in tensor memory, and two warps issue a tile in turns: 31.0 us instead of 35.4 with X in shared memory and one warp (2950
// cycles a tile, 2470 of them contractions, the rest that warp's waits and commits).  X straight from global memory into tensor memory: 38.3 us, a
// row a lane reads 32 lines an instruction.
// The gradient pass takes 7200 cycles a tile, 5760 of them contractions: S, softmax and W of the next tile wait for the last plane of Y, for which
// the ring has no room before dQ.  Tried: one issuing warp and planes of Y loaded twice, so that S runs two tiles ahead (108 us); two warps and two
// rings for the same (98 ... 100 us); W split before the wait for its buffer (90 us).
#include <math.h>

#include <algorithm>

#include "lp_sched.cuh"
#include "tc_pipe.cuh"

namespace ge2 {
namespace {

using namespace tc;

constexpr int BM = 128, BN = 64;
constexpr int kPlanes = 3;
constexpr float kMasked = -1e9f;
constexpr float kDeadRow = 1e30f;  // "lse" of a row past the end of its chunk: exp(anything - 1e30) = 0
constexpr int kLseStages = 3;      // logsumexp pass: tiles of Y under way (its two issuing warps rely on there being no more)
constexpr int kYSlots = 5;         // gradient pass: ring of Y planes; three belong to a tile, two are ahead

// the six products, small ones first: plane of the first / second operand, two bits each
constexpr uint32_t codes(int a, int b, int c, int d, int e, int f) { return (uint32_t)(a | b << 2 | c << 4 | d << 6 | e << 8 | f << 10); }
constexpr uint32_t kFirst = codes(2, 0, 1, 1, 0, 0), kSecond = codes(0, 2, 1, 0, 1, 0);  // (l,h) (h,l) (m,m) (m,h) (h,m) (h,h)
// the gradient pass takes Y planes in the order m, h, l of their arrival, and gives them back in the same order
constexpr uint32_t kFirstS = codes(0, 1, 2, 1, 0, 0), kSecondS = codes(1, 1, 0, 0, 2, 0);   // S:  (h,m) (m,m) (l,h) (m,h) (h,l) (h,h)
constexpr uint32_t kFirstDq = codes(0, 1, 0, 2, 1, 0), kSecondDq = codes(1, 1, 2, 0, 0, 0); // dQ: (h,m) (m,m) | (h,l) | (l,h) (m,h) (h,h)
__device__ __forceinline__ int slot_of_plane(int plane) { return plane == 1 ? 0 : plane == 0 ? 1 : 2; }

template <int DP>
struct Layout32 {
    static constexpr int NB = DP / 64;
    static constexpr int kXBlock = BM * 128, kYBlock = BN * 128;
    static constexpr int kXPlane = NB * kXBlock, kYPlane = NB * kYBlock, kWPlane = BM * 128;
    static constexpr int kX = 0, kY = kPlanes * kXPlane;
    // logsumexp pass: X is in tensor memory
    static constexpr int kXCols = NB * 32;                            // tensor-memory columns of a plane of X
    static constexpr int kXHalves = NB == 1 ? 2 : 1;                  // buffers for the halves of X on their way there, each like a tile of Y
    static constexpr int kXHalf = kLseStages * kPlanes * kYPlane;
    static constexpr int kXch = kXHalf + kXHalves * kPlanes * kYPlane;  // [2][128] (max, sum) of the right half of the columns
    static constexpr int kMiscA = kXch + 2 * BM * 8;
    static constexpr int kBytesA = (kMiscA + 512 + 1024) > 120 * 1024 ? (kMiscA + 512 + 1024) : 120 * 1024;  // one CTA an SM
    // gradient pass
    static constexpr int kW = kY + kYSlots * kYPlane;
    static constexpr int kMiscB = kW + kPlanes * kWPlane;
    static constexpr int kBytesB = (kMiscB + 512 + 1024) > 120 * 1024 ? (kMiscB + 512 + 1024) : 120 * 1024;
    static_assert(kBytesA <= 227 * 1024 && kBytesB <= 227 * 1024, "exceeds the shared memory of an SM");
};

// the filter words of 32 columns starting at n0 + base: lane l holds column l's; bit j of the result = column j is masked for row `brow`
__device__ __forceinline__ uint32_t mask_bits(int32_t word, int wrow0, int brow) {
    uint32_t mb = 0u;
    unsigned ballot = __ballot_sync(0xffffffffu, (unsigned)(word - wrow0) < 32u);
    while (ballot != 0) {
        const int src = __ffs(ballot) - 1;
        ballot &= ballot - 1;
        if (__shfl_sync(0xffffffffu, word, src) == brow) mb |= 1u << src;
    }
    return mb;
}

// Three planes of 64 rows of X, staged like a tile of Y -> tensor memory, for one warp: lane = row, two consecutive elements a column
template <int DP>
__device__ __forceinline__ void x_to_tmem(uint32_t taddr, const unsigned char* stage, int row) {
    using LY = Layout32<DP>;
#pragma unroll 1
    for (int p = 0; p < kPlanes; p++) {
#pragma unroll
        for (int c = 0; c < LY::kXCols; c += 16) {
            const unsigned char* src = stage + p * LY::kYPlane + (c / 32) * LY::kYBlock + row * 128;
            uint32_t r[16];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint4 q = *reinterpret_cast<const uint4*>(src + ((((c % 32) / 4 + k) ^ (row & 7)) << 4));
                r[4 * k] = q.x, r[4 * k + 1] = q.y, r[4 * k + 2] = q.z, r[4 * k + 3] = q.w;
            }
            tmem_st_32x16_start(taddr + p * LY::kXCols + c, r);
        }
    }
    tmem_st_wait();
}

// =====================================================================================================================
// launch 1: row logsumexp
// =====================================================================================================================
constexpr int kSoftWarps = 8;                                    // 4 row quarters x 2 halves of 32 columns
constexpr int kTmaWarpA = 8, kMmaWarpA = 9, kLoadWarpA = 11, kLoadWarps = 4, kThreadsA = 480;  // two MMA warps
enum BarA { kAXIn = 0, kAXOut = kAXIn + 2, kAXFull = kAXOut + 2, kAXEmpty = kAXFull + 2, kAYFull = kAXEmpty + 2, kAYEmpty = kAYFull + kLseStages, kASFull = kAYEmpty + kLseStages, kASEmpty = kASFull + 2, kAXch = kASEmpty + 2,
            kAXchFree = kAXch + 2, kNumBarsA = kAXchFree + 2 };
// tensor memory: scores at 0 and 64, X of two blocks
constexpr uint32_t kTmXa = 128;

template <int DP>
__global__ void __launch_bounds__(kThreadsA, 1)
    lp_lse32_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, LpKernelArgs a, Sched sc) {
    using LY = Layout32<DP>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    float2* s_xch = reinterpret_cast<float2*>(smem + LY::kXch);
    uint64_t* bars = (uint64_t*)(smem + LY::kMiscA);
    uint32_t* s_tmem = (uint32_t*)(smem + LY::kMiscA + kNumBarsA * 8);
    volatile int* s_abort = (volatile int*)(smem + LY::kMiscA + kNumBarsA * 8 + 4);
    const ge2_lp_desc& d = a.d;
    const LpLayout& L = a.L;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ub = range_begin(blockIdx.x, sc.unitsA, gridDim.x), ue = range_begin(blockIdx.x + 1, sc.unitsA, gridDim.x);
    const int n_iter = ue - ub;
    auto spin_wait = [&](int bar, uint32_t parity) { return warp_spin_wait(&bars[bar], parity, s_abort, d.status); };
    auto warp_wait = [&](int bar, uint32_t parity) { return warp_pipe_wait(&bars[bar], parity, s_abort, d.status); };

    if (warp == kTmaWarpA && lane == 0) {
        for (int k = 0; k < kLseStages; k++) {
            mbar_init(&bars[kAYFull + k], 1);
            mbar_init(&bars[kAYEmpty + k], 1);
        }
        for (int k = 0; k < 2; k++) {
            mbar_init(&bars[kAXIn + k], 1);
            mbar_init(&bars[kAXOut + k], kLoadWarps / 2);
            mbar_init(&bars[kAXFull + k], kLoadWarps);
            mbar_init(&bars[kAXEmpty + k], 2);
            mbar_init(&bars[kASFull + k], 1);
            mbar_init(&bars[kASEmpty + k], kSoftWarps);
            mbar_init(&bars[kAXch + k], kSoftWarps / 2);
            mbar_init(&bars[kAXchFree + k], kSoftWarps / 2);
        }
        *s_abort = 0;
        mbar_init_fence();
        prefetch_tensormap(&tmQ);
        prefetch_tensormap(&tmK);
    }
    if (warp == kMmaWarpA) {
        tmem_alloc(s_tmem, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    griddep_wait();  // set-up done; from here on global memory written by the preceding kernel is read and its buffers rewritten
    const uint32_t tmem = *s_tmem;

    if (warp == kTmaWarpA) {
        bool ok = true;
        int sg = -1;
        auto load = [&](const CUtensorMap& map, int row, int zc, int at, int full) {
            mbar_expect_tx_warp(&bars[full], kPlanes * LY::kYPlane);
            for (int p = 0; p < kPlanes; p++)
                for (int b = 0; b < LY::NB; b++) tma_load_3d_warp(smem + at + p * LY::kYPlane + b * LY::kYBlock, &map, b * 64, row, p * sc.ZC + zc, &bars[full]);
        };
        IterA un(ub, sc);
        for (int it = 0; ok && it < n_iter; it++, un.next(sc)) {
            const bool fresh = it == 0 || un.tile == 0;
            auto second_half = [&] { load(tmQ, un.rb * BM + BM / 2, un.zc, LY::kXHalf + (LY::kXHalves - 1) * kPlanes * LY::kYPlane, kAXIn + 1); };
            if (fresh) {
                sg++;
                ok = spin_wait(kAXOut, (sg & 1) ^ 1) && spin_wait(kAXOut + 1, (sg & 1) ^ 1);
                if (!ok) break;
                load(tmQ, un.rb * BM, un.zc, LY::kXHalf, kAXIn);
                if (LY::kXHalves == 2) second_half();
            }
            const int st = it % kLseStages;
            ok = spin_wait(kAYEmpty + st, ((it / kLseStages) & 1) ^ 1);
            if (!ok) break;
            load(tmK, un.tile * BN, un.zc, st * kPlanes * LY::kYPlane, kAYFull + st);
            if (fresh && LY::kXHalves == 1) {
                ok = spin_wait(kAXOut, sg & 1);
                if (!ok) break;
                second_half();
            }
        }
    } else if (warp < kLoadWarpA && warp >= kMmaWarpA) {
        // two warps, a tile in turns: the pipe has the other's contractions while one waits
        constexpr uint32_t kIdesc = idesc_bf16(BM, BN, 0, 0);
        const uint32_t dY0 = desc_lo_sw128(smem_u32(smem), 16);
        const int KS = (d.D + kMmaK - 1) / kMmaK, sb = warp - kMmaWarpA;
        int sg = -1;
        IterA un(ub, sc);
        with_steps<LY::NB>(KS, [&](auto steps) {
            for (int it = 0; it < n_iter; it++, un.next(sc)) {
                if (it == 0 || un.tile == 0) {
                    if (sg >= 0) mma_commit_warp(&bars[kAXEmpty + (sg & 1)]);
                    sg++;
                    // by both warps, also by one that has no tile in the block: it then gives back no X that has not come
                    if (!spin_wait(kAXFull + (sg & 1), (sg >> 1) & 1)) break;
                }
                if ((it & 1) != sb) continue;
                const int st = it % kLseStages, xb = sg & 1;
                // The scores first: with those of tile it - 2 read, those of it - 3 are, so that the last use of this stage, the other warp's, lies
                // behind, and the phase waited for is the next one of its barrier.
                if (!spin_wait(kASEmpty + sb, ((it >> 1) & 1) ^ 1)) break;
                if (!spin_wait(kAYFull + st, (it / kLseStages) & 1)) break;
                tc_fence_after();
                const uint32_t dY = dY0 + st * (kPlanes * LY::kYPlane >> 4), tX = tmem + kTmXa + xb * (kPlanes * LY::kXCols);
#pragma unroll 1
                for (int p = 0; p < 6; p++)
                    mma_ts_kmajor<steps, LY::kYBlock>(tmem + sb * BN, tX + ((kFirst >> (2 * p)) & 3) * LY::kXCols,
                                                      dY + ((kSecond >> (2 * p)) & 3) * (LY::kYPlane >> 4), kIdesc, p > 0 ? 1u : 0u);
                mma_commit_warp(&bars[kAYEmpty + st]);
                mma_commit_warp(&bars[kASFull + sb]);
            }
        });
        // the last arrivals of the pipe on a block's barrier land before the CTA exits; those on the others come before scores that are waited for
        if (sg > 0) spin_wait(kAXEmpty + ((sg - 1) & 1), ((sg - 1) >> 1) & 1);
    } else if (warp >= kLoadWarpA) {
        // X of every block, a block ahead of the contractions: each pair of warps moves the half that holds its quarters of the lanes
        const int quarter = warp & 3, half = quarter >> 1;
        const uint32_t lane_sel = (uint32_t)(quarter * 32) << 16;
        for (int sg = 0, at = ub; at < ue; sg++) {
            const int xb = sg & 1;
            if (!warp_wait(kAXEmpty + xb, ((sg >> 1) & 1) ^ 1)) break;
            if (!warp_wait(kAXIn + half, sg & 1)) break;
            tc_fence_after();
            x_to_tmem<DP>(tmem + kTmXa + xb * (kPlanes * LY::kXCols) + lane_sel, smem + LY::kXHalf + half * (LY::kXHalves - 1) * kPlanes * LY::kYPlane, (quarter & 1) * 32 + lane);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&bars[kAXFull + xb]);
                mbar_arrive(&bars[kAXOut + half]);
            }
            at += sc.T - at % sc.T;
            if (sg > 0) continue;
            // clear what the gradient pass will add to: dK, and the dQ rows of every block whose stream that pass cuts at a CTA boundary
            const int wz = (warp - kLoadWarpA) * 32 + lane;
            const int64_t n4 = (int64_t)sc.ZC * d.N * (DP / 4);
            const int64_t z0 = n4 * blockIdx.x / gridDim.x, z1 = n4 * (blockIdx.x + 1) / gridDim.x;
            float4* p4 = reinterpret_cast<float4*>(L.dK);
            for (int64_t k = z0 + wz; k < z1; k += kLoadWarps * 32) p4[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int j = 1 + (int)blockIdx.x; j < sc.gridB; j += (int)gridDim.x) {
                const int u = range_begin(j, sc.unitsB, sc.gridB);
                if (u <= 0 || u >= sc.unitsB) continue;
                const UnitA un = decode_a(u, sc);
                if (un.tile == 0) continue;  // the boundary falls between two blocks: nothing is split
                float4* q4 = reinterpret_cast<float4*>(L.dQ + ((int64_t)un.zc * L.npc + (int64_t)un.rb * BM) * DP);
                const int n = min(BM, L.npc - un.rb * BM) * (DP / 4);
                for (int k = wz; k < n; k += kLoadWarps * 32) q4[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    } else {
        // ---- softmax warps: warp w takes rows 32 (w & 3) ... + 31 and columns 32 (w >> 2) ... + 31 of every tile ----
        const int half = warp >> 2, my_row = tid & 127;
        const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
        float run_m = -INFINITY, run_l = 0.f;
        int sg = -1;
        IterA un(ub, sc), ahead(ub, sc);
        auto mask_word = [&](const IterA& u) {
            const int n0 = u.tile * BN + half * 32;
            return lane < d.N - n0 ? __ldg(&L.mask[(int64_t)u.zc * d.N + n0 + lane]) : -1;
        };
        int32_t word = n_iter > 0 ? mask_word(ahead) : -1;
        for (int it = 0; it < n_iter; it++, un.next(sc)) {
            const int s = un.zc / d.C, c = un.zc - s * d.C, row0 = un.rb * BM, valid_rows = min(BM, L.npc - row0);
            if (it == 0 || un.tile == 0) {
                sg++;
                run_m = -INFINITY;
                run_l = 0.f;
            }
            const int n0 = un.tile * BN + half * 32, nv = min(32, d.N - n0);  // live columns among this warp's (may be <= 0)
            const int brow = c * L.npc + row0 + my_row;  // batch row in the padded numbering the filter uses
            const uint32_t mb = mask_bits(word, brow - lane, brow);
            ahead.next(sc);
            word = it + 1 < n_iter ? mask_word(ahead) : -1;  // the next tile's, a trip to memory ahead of its use
            const int sb = it & 1;
            if (!warp_wait(kASFull + sb, (it >> 1) & 1)) break;
            tc_fence_after();
            float v[32];
            tmem_ld_32x32(tmem + sb * BN + half * 32 + lane_sel, v);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[kASEmpty + sb]);
            if (nv > 0) {
                float* dump = s == 0 ? d.neg_scores : d.inv_neg_scores;
                if (__any_sync(0xffffffffu, mb != 0u)) {
#pragma unroll
                    for (int j = 0; j < 32; j++) v[j] = ((mb >> j) & 1u) ? kMasked : v[j];
                }
                if (dump != nullptr && my_row < valid_rows) {
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (j < nv) dump[(int64_t)brow * d.N + n0 + j] = v[j];
                }
                if (nv < 32) {
#pragma unroll
                    for (int j = 0; j < 32; j++) v[j] = j < nv ? v[j] : -INFINITY;
                }
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int j = 0; j < 32; j++) mx[j & 3] = fmaxf(mx[j & 3], v[j]);
                const float nm = fmaxf(run_m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
                float add[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int j = 0; j < 32; j++) add[j & 3] += expf(v[j] - nm);  // exp(-inf) = 0 for absent columns
                run_l = fmaf(run_l, expf(run_m - nm), (add[0] + add[1]) + (add[2] + add[3]));
                run_m = nm;
            }
            if (it == n_iter - 1 || un.tile == sc.T - 1) {
                // end of the block, or of this CTA's share of it: the halves of a row meet
                const int h = sg & 1;
                if (half == 1) {
                    if (!warp_wait(kAXchFree + h, ((sg >> 1) & 1) ^ 1)) break;
                    s_xch[h * BM + my_row] = make_float2(run_m, run_l);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars[kAXch + h]);
                } else {
                    if (!warp_wait(kAXch + h, (sg >> 1) & 1)) break;
                    const float2 o = s_xch[h * BM + my_row];
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars[kAXchFree + h]);
                    float m = fmaxf(run_m, o.x), l = 0.f;
                    if (m > -INFINITY) l = run_l * expf(run_m - m) + o.y * expf(o.x - m);
                    const int first = cta_of_unit(un.item * sc.T, sc.unitsA, (int)gridDim.x);
                    const bool whole = first == (int)blockIdx.x && un.tile == sc.T - 1;
                    const int64_t grow = (int64_t)s * L.Bp + c * L.npc + row0 + my_row;
                    if (!whole) {  // shared with a neighbouring CTA: the gradient pass combines the partials
                        const int part = (int)blockIdx.x - first;
                        if (my_row < valid_rows && part < kMaxParts) reinterpret_cast<float2*>(L.part)[grow * kMaxParts + part] = make_float2(m, l);
                    } else {
                        float lse = kDeadRow, loss = 0.f;
                        if (my_row < valid_rows) {
                            const float pos = __ldg(&L.pos[grow]), nm = fmaxf(m, pos);
                            lse = nm + logf(l * expf(m - nm) + expf(pos - nm));
                            L.lse[grow] = lse;
                            loss = lse - pos;
                        }
                        L.lse2s[(int64_t)un.item * BM + my_row] = lse;
#pragma unroll
                        for (int k = 16; k > 0; k >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, k);
                        if (lane == 0) atomicAdd(L.loss_acc, (double)loss);
                    }
                }
            }
        }
    }
    // ---- common exit: every role ends here, normally or after an abort; then tensor memory is released ----------
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarpA) {
        if (*s_abort && lane == 0) {  // copies still in flight get a bounded chance to land
            for (int k = 0; k < 2; k++) settle_bar(&bars[kAXIn + k]);
            for (int k = 0; k < kLseStages; k++) settle_bar(&bars[kAYFull + k]);
        }
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// =====================================================================================================================
// launch 2: both gradients
// =====================================================================================================================
constexpr int kDrainWarps = 8, kDrainWarp0 = kSoftWarps, kTmaWarpB = 16, kMmaWarpB = 17, kGradWarpB = 18, kThreadsB = 608;
enum BarB { kBXFull = 0, kBXEmpty, kBYFull, kBYEmpty = kBYFull + kYSlots, kBSFull = kBYEmpty + kYSlots, kBSEmpty = kBSFull + 2, kBWFull = kBSEmpty + 2,
            kBWEmpty, kBGFull, kBGEmpty = kBGFull + 2, kNumBarsB = kBGEmpty + 2 };
// tensor memory: scores at 0 and 64, dK^T of a tile at 128 and 192, dQ of a tile at 256 and 384
constexpr uint32_t kTmS = 0, kTmDk = 128, kTmDq = 256;

template <int DP>
__global__ void __launch_bounds__(kThreadsB, 1)
    lp_grad32_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, LpKernelArgs a, Sched sc) {
    using LY = Layout32<DP>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + LY::kMiscB);
    uint32_t* s_tmem = (uint32_t*)(smem + LY::kMiscB + kNumBarsB * 8);
    volatile int* s_abort = (volatile int*)(smem + LY::kMiscB + kNumBarsB * 8 + 4);
    const ge2_lp_desc& d = a.d;
    const LpLayout& L = a.L;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ub = range_begin(blockIdx.x, sc.unitsB, gridDim.x), ue = range_begin(blockIdx.x + 1, sc.unitsB, gridDim.x);
    const int n_iter = ue - ub;
    auto spin_wait = [&](int bar, uint32_t parity) { return warp_spin_wait(&bars[bar], parity, s_abort, d.status); };
    auto warp_wait = [&](int bar, uint32_t parity) { return warp_pipe_wait(&bars[bar], parity, s_abort, d.status); };

    if (warp == kTmaWarpB && lane == 0) {
        mbar_init(&bars[kBXFull], 1);
        mbar_init(&bars[kBXEmpty], 1);
        for (int k = 0; k < kYSlots; k++) {
            mbar_init(&bars[kBYFull + k], 1);
            mbar_init(&bars[kBYEmpty + k], 1);
        }
        for (int k = 0; k < 2; k++) {
            mbar_init(&bars[kBSFull + k], 1);
            mbar_init(&bars[kBSEmpty + k], kSoftWarps);
            mbar_init(&bars[kBGFull + k], 1);
            mbar_init(&bars[kBGEmpty + k], kDrainWarps);
        }
        mbar_init(&bars[kBWFull], kSoftWarps);
        mbar_init(&bars[kBWEmpty], 1);
        *s_abort = 0;
        mbar_init_fence();
        prefetch_tensormap(&tmQ);
        prefetch_tensormap(&tmK);
    }
    if (warp == kMmaWarpB) {
        tmem_alloc(s_tmem, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    griddep_wait();  // set-up done; from here on global memory written by the preceding kernel is read and its buffers rewritten
    const uint32_t tmem = *s_tmem;
    const int KS = (d.D + kMmaK - 1) / kMmaK;

    if (warp == kTmaWarpB) {
        int sg = -1, slot = 0;
        uint32_t phase = 1;
        bool ok = true;
        IterA un(ub, sc);
        for (int it = 0; ok && it < n_iter; it++, un.next(sc)) {
            if (it == 0 || un.tile == 0) {
                sg++;
                if (!spin_wait(kBXEmpty, (sg & 1) ^ 1)) break;
                mbar_expect_tx_warp(&bars[kBXFull], kPlanes * LY::kXPlane);
                for (int p = 0; p < kPlanes; p++)
                    for (int b = 0; b < LY::NB; b++)
                        tma_load_3d_warp(smem + LY::kX + p * LY::kXPlane + b * LY::kXBlock, &tmQ, b * 64, un.rb * BM, p * sc.ZC + un.zc, &bars[kBXFull]);
            }
            for (int k = 0; k < kPlanes; k++) {
                ok = spin_wait(kBYEmpty + slot, phase);
                if (!ok) break;
                const int p = k == 0 ? 1 : k == 1 ? 0 : 2;  // m, h, l
                mbar_expect_tx_warp(&bars[kBYFull + slot], LY::kYPlane);
                for (int b = 0; b < LY::NB; b++)
                    tma_load_3d_warp(smem + LY::kY + slot * LY::kYPlane + b * LY::kYBlock, &tmK, b * 64, un.tile * BN, p * sc.ZC + un.zc, &bars[kBYFull + slot]);
                if (++slot == kYSlots) slot = 0, phase ^= 1;
            }
        }
    } else if (warp == kMmaWarpB) {
        // ---- S = X Y^T ----
        constexpr uint32_t kIdesc = idesc_bf16(BM, BN, 0, 0);
        const uint32_t dX = desc_lo_sw128(smem_u32(smem + LY::kX), 16), dY0 = desc_lo_sw128(smem_u32(smem + LY::kY), 16);
        int sg = -1, slot0 = 0;
        uint32_t ph0 = 0;
        bool ok = true;
        IterA un(ub, sc);
        with_steps<LY::NB>(KS, [&](auto steps) {
            for (int it = 0; ok && it < n_iter; it++, un.next(sc)) {
                if (it == 0 || un.tile == 0) {
                    sg++;
                    if (!spin_wait(kBXFull, sg & 1)) break;
                }
                const int sb = it & 1, su = it >> 1;
                if (!spin_wait(kBSEmpty + sb, (su & 1) ^ 1)) break;
                int seen = 0;  // planes of this tile known to have arrived, in the order m, h, l
    #pragma unroll 1
                for (int p = 0; p < 6; p++) {
                    const int k = slot_of_plane((kSecondS >> (2 * p)) & 3);
                    const int slot = slot0 + k >= kYSlots ? slot0 + k - kYSlots : slot0 + k;
                    if (k >= seen) {
                        ok = spin_wait(kBYFull + slot, slot0 + k >= kYSlots ? ph0 ^ 1 : ph0);
                        if (!ok) break;
                        seen = k + 1;
                        tc_fence_after();
                    }
                    const uint32_t da = dX + ((kFirstS >> (2 * p)) & 3) * (LY::kXPlane >> 4), db = dY0 + slot * (LY::kYPlane >> 4);
                    mma_kmajor<steps, LY::kXBlock, LY::kYBlock>(tmem + kTmS + sb * BN, da, db, kIdesc, p > 0 ? 1u : 0u);
                }
                if (!ok) break;
                mma_commit_warp(&bars[kBSFull + sb]);
                slot0 += kPlanes;
                if (slot0 >= kYSlots) slot0 -= kYSlots, ph0 ^= 1;
            }
        });
    } else if (warp == kGradWarpB) {
        // ---- dQ [128 x D] of the tile = W Y, then dK^T [d x 64] = X^T W ----
        // dQ first: it gives the planes of Y back, and the one of the next tile that had no room in the ring arrives while dK^T is summed
        const uint32_t kIdescDk = idesc_bf16(128, BN, 1, 1), kIdescDq = idesc_bf16(BM, KS * kMmaK, 0, 1);
        // X along its columns: the second 64 of them lie a block further (for D <= 64 there are none, and what is read there ends up in
        // accumulator rows that nobody reads)
        const uint32_t dXm = desc_lo_sw128(smem_u32(smem + LY::kX), LY::kXBlock), dWm = desc_lo_sw128(smem_u32(smem + LY::kW), 16 * 1024),
                       dWk = desc_lo_sw128(smem_u32(smem + LY::kW), 16), dYm0 = desc_lo_sw128(smem_u32(smem + LY::kY), LY::kYBlock);
        int slot0 = 0;
        IterA un(ub, sc);
        for (int it = 0; it < n_iter; it++, un.next(sc)) {
            const int pb = it & 1;
            if (!spin_wait(kBGEmpty + pb, ((it >> 1) & 1) ^ 1)) break;
            // (no wait on X or Y: W was made from scores that were made from them)
            if (!spin_wait(kBWFull, it & 1)) break;
            tc_fence_after();
#pragma unroll 1
            for (int p = 0; p < 6; p++) {
                const int k = slot_of_plane((kSecondDq >> (2 * p)) & 3);
                const int slot = slot0 + k >= kYSlots ? slot0 + k - kYSlots : slot0 + k;
                const uint32_t da = dWk + ((kFirstDq >> (2 * p)) & 3) * (LY::kWPlane >> 4), db = dYm0 + slot * (LY::kYPlane >> 4);
#pragma unroll
                for (int ks = 0; ks < BN / kMmaK; ks++)
                    mma_f16_ss_warp(tmem + kTmDq + pb * 128, da + ks * (32 >> 4), db + ks * (2048 >> 4), kIdescDq, (p > 0 || ks > 0) ? 1u : 0u);
                if (p == 1 || p == 2 || p == 5) mma_commit_warp(&bars[kBYEmpty + slot]);  // the last product with this plane of Y
            }
#pragma unroll 1
            for (int p = 0; p < 6; p++) {
                const uint32_t da = dXm + ((kFirst >> (2 * p)) & 3) * (LY::kXPlane >> 4), db = dWm + ((kSecond >> (2 * p)) & 3) * (LY::kWPlane >> 4);
#pragma unroll
                for (int ks = 0; ks < BM / kMmaK; ks++)
                    mma_f16_ss_warp(tmem + kTmDk + pb * BN, da + ks * (2048 >> 4), db + ks * (2048 >> 4), kIdescDk, (p > 0 || ks > 0) ? 1u : 0u);
            }
            mma_commit_warp(&bars[kBWEmpty]);
            if (it == n_iter - 1 || un.tile == sc.T - 1) mma_commit_warp(&bars[kBXEmpty]);
            mma_commit_warp(&bars[kBGFull + pb]);  // last: whoever waits for it has seen the others' arrivals land before the CTA exits
            slot0 += kPlanes;
            if (slot0 >= kYSlots) slot0 -= kYSlots;
        }
    } else if (warp < kSoftWarps) {
        // ---- softmax warps: warp w takes rows 32 (w & 3) ... + 31 and columns 32 (w >> 2) ... + 31 of every tile ----
        const int half = warp >> 2, my_row = tid & 127;
        const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
        float lrow = kDeadRow;
        IterA un(ub, sc), ahead(ub, sc);
        auto mask_word = [&](const IterA& u) {
            const int n0 = u.tile * BN + half * 32;
            return lane < d.N - n0 ? __ldg(&L.mask[(int64_t)u.zc * d.N + n0 + lane]) : -1;
        };
        int32_t word = n_iter > 0 ? mask_word(ahead) : -1;
        for (int it = 0; it < n_iter; it++, un.next(sc)) {
            const int s = un.zc / d.C, c = un.zc - s * d.C, row0 = un.rb * BM;
            const int brow = c * L.npc + row0 + my_row;
            if (it == 0 || un.tile == 0) {
                // was the block run by one CTA of the logsumexp pass (that launch's grid and ranges are known here)?
                const int first = cta_of_unit(un.item * sc.T, sc.unitsA, sc.gridA);
                const int nparts = cta_of_unit(un.item * sc.T + sc.T - 1, sc.unitsA, sc.gridA) - first + 1;
                if (nparts == 1) {
                    lrow = __ldg(&L.lse2s[(int64_t)un.item * BM + my_row]);
                } else {
                    // combine the partial (max, sum) pairs its sharers left; the CTA that starts the block here also writes the lse for
                    // the finish kernel and adds the rows' loss terms
                    const int64_t grow = (int64_t)s * L.Bp + brow;
                    const bool writer = un.tile == 0 && half == 0;
                    float loss = 0.f;
                    lrow = kDeadRow;
                    if (my_row < min(BM, L.npc - row0)) {
                        const float2* part = reinterpret_cast<const float2*>(L.part) + grow * kMaxParts;
                        float m = -INFINITY, l = 0.f;
                        for (int k = 0; k < nparts && k < kMaxParts; k++) {
                            const float2 pk = __ldg(&part[k]);
                            const float nm = fmaxf(m, pk.x);
                            if (nm > -INFINITY) {
                                l = l * expf(m - nm) + pk.y * expf(pk.x - nm);
                                m = nm;
                            }
                        }
                        const float pos = __ldg(&L.pos[grow]), nm = fmaxf(m, pos);
                        lrow = nm + logf(l * expf(m - nm) + expf(pos - nm));
                        if (writer) {
                            L.lse[grow] = lrow;
                            loss = lrow - pos;
                        }
                    }
                    if (writer) {
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
                        if (lane == 0) atomicAdd(L.loss_acc, (double)loss);
                    }
                }
            }
            const int nv = min(32, d.N - un.tile * BN - half * 32);  // live columns among this warp's (may be <= 0)
            const uint32_t mb = mask_bits(word, brow - lane, brow);
            ahead.next(sc);
            word = it + 1 < n_iter ? mask_word(ahead) : -1;
            const int sb = it & 1;
            if (!warp_wait(kBSFull + sb, (it >> 1) & 1)) break;
            tc_fence_after();
            float v[32];
            tmem_ld_32x32(tmem + kTmS + sb * BN + half * 32 + lane_sel, v);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[kBSEmpty + sb]);
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] = expf(v[j] - lrow);
            // masked entries were overwritten in place by the reference: no gradient reaches them; columns past the chunk have none
            if (nv < 32 || __any_sync(0xffffffffu, mb != 0u)) {
#pragma unroll
                for (int j = 0; j < 32; j++) v[j] = j < nv && !((mb >> j) & 1u) ? v[j] : 0.f;
            }
            if (!warp_wait(kBWEmpty, (it & 1) ^ 1)) break;
            unsigned char* w0 = smem + LY::kW + my_row * 128;
#pragma unroll 1
            for (int p = 0; p < kPlanes; p++) {
#pragma unroll
                for (int q = 0; q < 4; q++) {  // 8 values = one 16-byte chunk; what is left of them stays for the next plane
                    uint32_t pk[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const __nv_bfloat162 h = __floats2bfloat162_rn(v[8 * q + 2 * e], v[8 * q + 2 * e + 1]);
                        pk[e] = *reinterpret_cast<const uint32_t*>(&h);
                        v[8 * q + 2 * e] -= __uint_as_float(pk[e] << 16);
                        v[8 * q + 2 * e + 1] -= __uint_as_float(pk[e] & 0xffff0000u);
                    }
                    *reinterpret_cast<uint4*>(w0 + p * LY::kWPlane + (((half * 4 + q) ^ (my_row & 7)) << 4)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                }
            }
            fence_proxy_async_smem();  // W was written with ordinary stores; the MMA reads it through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[kBWFull]);
        }
    } else {
        // ---- drain warps: dK^T leaves by atomics (lanes run along a row of dK), dQ is summed in registers over the block's tiles ----
        constexpr int kCols = DP / 2;  // columns of dQ a thread sums: its row, half of them
        const int w = warp - kDrainWarp0, quarter = warp & 3, half = w >> 2;
        const uint32_t lane_sel = (uint32_t)(quarter * 32) << 16;
        const int dcol = quarter * 32 + lane;  // dK^T: this lane's embedding column
        float acc[kCols];
        bool whole = false;
        IterA un(ub, sc);
        for (int it = 0; it < n_iter; it++, un.next(sc)) {
            if (it == 0 || un.tile == 0) {
                whole = un.tile == 0 && (ub + it + sc.T <= ue);  // this CTA runs the block's whole stream
#pragma unroll
                for (int k = 0; k < kCols; k++) acc[k] = 0.f;
            }
            const int pb = it & 1;
            if (!warp_wait(kBGFull + pb, (it >> 1) & 1)) break;
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < kCols; k += 16) {
                float t[16];
                tmem_ld_32x16(tmem + kTmDq + pb * 128 + half * kCols + k + lane_sel, t);
#pragma unroll
                for (int j = 0; j < 16; j++) acc[k + j] += t[j];
            }
            const int n0 = un.tile * BN + half * 32;
            float* dk = L.dK + ((int64_t)un.zc * d.N + n0) * DP + dcol;
#pragma unroll 1
            for (int k = 0; k < 32; k += 16) {
                float t[16];
                tmem_ld_32x16(tmem + kTmDk + pb * BN + half * 32 + k + lane_sel, t);
                if (k == 16) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars[kBGEmpty + pb]);
                }
                if (dcol < d.D) {
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        if (n0 + k + j < d.N) atomicAdd(dk + (int64_t)(k + j) * DP, t[j]);
                }
            }
            if (it == n_iter - 1 || un.tile == sc.T - 1) {
                const int row = un.rb * BM + dcol;  // dQ: this lane's row
                if (row < L.npc) {
                    float4* q4 = reinterpret_cast<float4*>(L.dQ + ((int64_t)un.zc * L.npc + row) * DP + half * kCols);
#pragma unroll
                    for (int k = 0; k < kCols; k += 4) {
                        if (half * kCols + k >= d.D) continue;
                        const float4 x = make_float4(acc[k], acc[k + 1], acc[k + 2], acc[k + 3]);
                        if (whole) q4[k / 4] = x;
                        else atomicAdd(q4 + k / 4, x);
                    }
                }
            }
        }
    }
    // ---- common exit: every role ends here, normally or after an abort; then tensor memory is released ----------
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarpB) {
        if (*s_abort && lane == 0) {  // copies and contractions still in flight get a bounded chance to land
            for (int k = 0; k < kYSlots; k++) settle_bar(&bars[kBYFull + k]);
            for (int k = 0; k < 2; k++) settle_bar(&bars[kBGFull + k]);
        }
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

template <int DP>
int launch(const LpKernelArgs& a, cudaStream_t stream) {
    using LY = Layout32<DP>;
    const int ZC = a.L.S * a.d.C;
    CUtensorMap tmQ, tmQHalf, tmK;
    int rc = make_operand_map(&tmQ, a.L.Qs, true, DP, a.L.npc, (int64_t)kPlanes * ZC, BM);
    if (rc != GE2_OK) return rc;
    rc = make_operand_map(&tmQHalf, a.L.Qs, true, DP, a.L.npc, (int64_t)kPlanes * ZC, BM / 2);
    if (rc != GE2_OK) return rc;
    rc = make_operand_map(&tmK, a.L.Ks, true, DP, a.d.N, (int64_t)kPlanes * ZC, BN);
    if (rc != GE2_OK) return rc;
    Sched sc;
    sc.RB = ceil_div(a.L.npc, BM);
    sc.T = ceil_div(a.d.N, BN);
    sc.ZC = ZC;
    const long long units = (long long)ZC * sc.RB * sc.T;
    if (units > 0x3fffffff) return GE2_ERR_UNSUPPORTED;
    sc.unitsA = sc.unitsB = (int)units;
    // every CTA's range is at least ceil(T / 7) units long, so a row block is shared by at most kMaxParts CTAs
    sc.gridA = std::max(1, std::min(scores_ctas(units), sc.unitsA / ceil_div(sc.T, kMaxParts - 1)));
    sc.gridB = scores_ctas(units);
    // per-device function attributes; setting them on every launch keeps multi-device processes correct and is not a stream operation
    GE2_CUDA_TRY(cudaFuncSetAttribute(lp_lse32_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, LY::kBytesA));
    GE2_CUDA_TRY(cudaFuncSetAttribute(lp_grad32_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, LY::kBytesB));
    GE2_CUDA_TRY(launch_after(lp_lse32_kernel<DP>, dim3((unsigned)sc.gridA), dim3(kThreadsA), LY::kBytesA, stream, tmQHalf, tmK, a, sc));
    GE2_CUDA_TRY(launch_after(lp_grad32_kernel<DP>, dim3((unsigned)sc.gridB), dim3(kThreadsB), LY::kBytesB, stream, tmQ, tmK, a, sc));
    return GE2_OK;
}

}  // namespace

int lp_scores_fp32(const LpKernelArgs& a, cudaStream_t stream) {
    if (a.L.ld == 64) return launch<64>(a, stream);
    if (a.L.ld == 128) return launch<128>(a, stream);
    return GE2_ERR_UNSUPPORTED;
}

}  // namespace ge2
