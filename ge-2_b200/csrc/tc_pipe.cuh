// What the tensor-memory kernels share on top of tc_ptx.cuh: operand tiles in the 128-byte-swizzled layout (offsets and matrix
// descriptors), bounded pipeline waits with a block-wide abort flag, exact splitting of fp32 values into bf16 terms, and the
// host side of tensor maps.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include <type_traits>

#include "common.cuh"
#include "tc_ptx.cuh"

namespace ge2 {
namespace tc {

constexpr int kBlockBytes = 128 * 128;  // operand block: 128 rows of 64 16-bit elements
constexpr int kMmaK = 16;               // k extent of one kind::f16 MMA (32 bytes)

// ---- operand tiles --------------------------------------------------------------------------------------------------------
// Descriptors are built once per tile; a k-step only adds its byte offset (>> 4) to the start-address field, which cannot
// carry out of the field because shared-memory addresses stay below 256 KB.
// K-major operand: k-step `ks` (16 elements = 32 bytes) sits in column block ks/4 at byte (ks%4)*32; 8-row groups are 1024 bytes apart
__host__ __device__ constexpr uint64_t koff_kmajor(int ks) { return (uint64_t)(((ks >> 2) * kBlockBytes + (ks & 3) * 32) >> 4); }
// MN-major operand: k-step `ks` is rows [16 ks, 16 ks + 16) = two 8-row groups of 1024 bytes; the 64-element MN blocks are
// kBlockBytes apart
__host__ __device__ constexpr uint64_t koff_mnmajor(int ks) { return (uint64_t)((ks * 2048) >> 4); }

// byte offset of the 16-byte chunk holding elements [col, col + 8) of row `row` in the swizzled block layout (col % 8 == 0)
__device__ __forceinline__ uint32_t swz_chunk_offset(int row, int col) {
    const int chunk = (col & 63) >> 3;
    return (uint32_t)((col >> 6) * kBlockBytes + row * 128 + ((chunk ^ (row & 7)) << 4));
}

// ---- bounded waits --------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded waits that also give up as soon as another role has raised the abort flag.  Only the first poll is inlined: a kernel of
// several roles waits in a dozen places, and the loops in all of them were 45 of the 117 KB of code of one such kernel, in the way of
// what its warps run all the time.
static __device__ __noinline__ bool pipe_wait_slow(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int32_t* status) {
    for (uint32_t i = 0; i < (1u << 20); i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if (i > 64) __nanosleep(i > 4096 ? 256 : 32);  // long waits (a role idle for a whole block) must not eat issue slots
        if ((i & 255u) == 255u && *abort_flag) return false;
    }
    *abort_flag = 1;
    or_status(status, GE2_STATUS_PIPE_TIMEOUT);
    return false;
}
// For the warps that feed the tensor pipe and its copies: the whole warp polls, and nobody sleeps (a slot is refilled within a few
// hundred nanoseconds, about as long as a sleeping lane takes to come back)
static __device__ __noinline__ bool warp_spin_slow(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int32_t* status) {
    for (uint32_t i = 0; i < (1u << 24); i++) {
        if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity) ? 1 : 0)) return true;
        if ((i & 255u) == 255u && __any_sync(0xffffffffu, *abort_flag)) return false;
    }
    *abort_flag = 1;
    or_status(status, GE2_STATUS_PIPE_TIMEOUT);
    return false;
}
__device__ __forceinline__ bool warp_spin_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int32_t* status) {
    return __all_sync(0xffffffffu, mbar_try_wait(bar, parity) ? 1 : 0) || warp_spin_slow(bar, parity, abort_flag, status);
}
// The same for a whole warp: one lane polls; then every lane observes the completed phase itself
static __device__ __noinline__ bool warp_pipe_wait_slow(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int32_t* status) {
    int ok = 1;
    if ((threadIdx.x & 31) == 0) ok = pipe_wait_slow(bar, parity, abort_flag, status) ? 1 : 0;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (ok) ok = mbar_try_wait(bar, parity) ? 1 : 0;
    return __all_sync(0xffffffffu, ok) != 0;
}
__device__ __forceinline__ bool warp_pipe_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int32_t* status) {
    return __all_sync(0xffffffffu, mbar_try_wait(bar, parity) ? 1 : 0) || warp_pipe_wait_slow(bar, parity, abort_flag, status);
}

// The same without a call: a kernel that shares its registers out among its warps (setmaxnreg) cannot have any.
__device__ __forceinline__ bool warp_wait_inline(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int32_t* status) {
#pragma unroll 1
    for (uint32_t i = 0; i < (1u << 20); i++) {
        if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity) ? 1 : 0)) return true;
        if ((i & 15u) == 15u && __any_sync(0xffffffffu, *abort_flag)) return false;
    }
    *abort_flag = 1;
    or_status(status, GE2_STATUS_PIPE_TIMEOUT);
    return false;
}

// What may still be on its way when the roles of a kernel have left their loops after a wait that ran out -- a copy into shared memory, a
// contraction -- gets a bounded chance to land before that memory goes to the next CTA.  The barrier it arrives on is in either phase: one that
// has completed its phase 0 is in its phase 1.
__device__ __forceinline__ void settle_bar(uint64_t* bar) { mbar_wait(bar, mbar_try_wait(bar, 0) ? 1u : 0u, 1u << 14); }

// ---- contractions ---------------------------------------------------------------------------------------------------------
// D (+)= A B^T over the first STEPS k-steps (1 ... 4 NB) of operands of 64-column blocks, both K-major, in straight-line code.
template <int STEPS, int A_BLOCK, int B_BLOCK>
__device__ __forceinline__ void mma_kmajor(uint32_t acc, uint32_t da, uint32_t db, uint32_t idesc, uint32_t accumulate) {
#pragma unroll
    for (int ks = 0; ks < STEPS; ks++)
        mma_f16_ss_warp(acc, da + (((ks >> 2) * A_BLOCK + (ks & 3) * 32) >> 4), db + (((ks >> 2) * B_BLOCK + (ks & 3) * 32) >> 4), idesc,
                        ks > 0 ? 1u : accumulate);
}
// The same with A in tensor memory: two elements a column, 8 columns a k-step.  A is not read from shared memory then, which is what bounds a
// contraction of N = 64 (48 cycles a k-step with A there, 32 this way).
template <int STEPS, int B_BLOCK>
__device__ __forceinline__ void mma_ts_kmajor(uint32_t acc, uint32_t ta, uint32_t db, uint32_t idesc, uint32_t accumulate) {
#pragma unroll
    for (int ks = 0; ks < STEPS; ks++)
        mma_f16_ts_warp(acc, ta + ks * 8, db + (((ks >> 2) * B_BLOCK + (ks & 3) * 32) >> 4), idesc, ks > 0 ? 1u : accumulate);
}
// Makes the number of k-steps of rows of NB 64-column blocks, 4 NB - 3 ... 4 NB, a constant of the body given, which holds the issuing warp's
// whole loop.  The issue must not stop between contractions, for the tensor pipe has next to no queue: the six contractions of a three-plane
// product (7 steps of N = 64 each) take 2016 cycles this way, the rate of the pipe, 2829 with a branch on the number of steps before each,
// and 3600 where the other warps of the SM are busy too.
template <int NB, class Body>
__device__ __forceinline__ void with_steps(int steps, Body&& body) {
    constexpr int kFull = 4 * (NB - 1);
    switch (steps - kFull) {
        case 1: body(std::integral_constant<int, kFull + 1>()); break;
        case 2: body(std::integral_constant<int, kFull + 2>()); break;
        case 3: body(std::integral_constant<int, kFull + 3>()); break;
        default: body(std::integral_constant<int, kFull + 4>()); break;
    }
}

// ---- host: tensor maps ----------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime's driver entry point lookup: the library does not link libcuda, so it still
// loads on a machine without a driver
inline EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
        return (EncodeTiledFn)p;
    }();
    return fn;
}

inline int encode_3d(CUtensorMap* map, CUtensorMapDataType type, int elem_bytes, void* base, int64_t ld, int64_t rows, int64_t mats, int box_cols,
                     int box_rows, CUtensorMapSwizzle swizzle, CUtensorMapL2promotion promotion) {
    EncodeTiledFn fn = encode_fn();
    if (fn == nullptr) return GE2_ERR_CUDA;
    cuuint64_t dims[3] = {(cuuint64_t)ld, (cuuint64_t)rows, (cuuint64_t)mats};
    cuuint64_t strides[2] = {(cuuint64_t)ld * elem_bytes, (cuuint64_t)rows * ld * elem_bytes};
    cuuint32_t box[3] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, type, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, promotion, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        g_last_cuda_error = (int)r;
        return GE2_ERR_CUDA;
    }
    return GE2_OK;
}

// [mats][rows][ld 16-bit elements] as a 3-D tensor of operand blocks: box = 64 elements x box_rows rows of one matrix, 128-byte swizzle,
// rows past the matrix end read as zero
inline int make_operand_map(CUtensorMap* map, void* base, bool bf16, int64_t ld, int64_t rows, int64_t mats, int box_rows = 128) {
    return encode_3d(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, base, ld, rows, mats, 64, box_rows,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
}

// [mats][rows][ld floats] as a 3-D tensor for stores: box = 32 floats x 32 rows with the 128-byte swizzle, or (narrow slab)
// box_cols < 32 floats x 32 rows, dense
inline int make_slab_map(CUtensorMap* map, float* base, int64_t ld, int64_t rows, int64_t mats, int box_cols = 32) {
    return encode_3d(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, ld, rows, mats, box_cols, 32,
                     box_cols == 32 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE);
}

}  // namespace tc
}  // namespace ge2
