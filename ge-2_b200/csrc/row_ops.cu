// Row-wise bandwidth kernels: gather / scatter-add of embedding rows, sparse Adagrad (batch-local and fused with the
// scatter into the resident table), dense Adagrad for the relation tables, partition-slot remap of edge endpoints,
// slab copies and the on-device negative sampler.  All are HBM-bound: each touched float is read once and written
// once, rows are contiguous (D*4 bytes), accesses are 16-byte vectors when D % 4 == 0 (8-byte for even D).
//
// Floating-point updates use explicit round-to-nearest intrinsics so no multiply-add contraction happens: the result
// is bit-identical to evaluating the reference's chain of element-wise ATen ops (cpp/src/data/batch.cpp:264-266,
// cpp/src/nn/optim.cpp:130-137 of the reference project) one IEEE operation at a time.
#include <algorithm>

#include "adagrad.cuh"
#include "lp_internal.cuh"
#include "unique_map.cuh"

namespace ge2 {
namespace {

template <int V>
struct Vec;
template <>
struct Vec<4> {
    using type = float4;
};
template <>
struct Vec<2> {
    using type = float2;
};
template <>
struct Vec<1> {
    using type = float;
};

template <int V>
__device__ __forceinline__ void to_arr(const typename Vec<V>::type& v, float (&a)[V]);
template <>
__device__ __forceinline__ void to_arr<4>(const float4& v, float (&a)[4]) {
    a[0] = v.x; a[1] = v.y; a[2] = v.z; a[3] = v.w;
}
template <>
__device__ __forceinline__ void to_arr<2>(const float2& v, float (&a)[2]) {
    a[0] = v.x; a[1] = v.y;
}
template <>
__device__ __forceinline__ void to_arr<1>(const float& v, float (&a)[1]) {
    a[0] = v;
}
template <int V>
__device__ __forceinline__ typename Vec<V>::type from_arr(const float (&a)[V]);
template <>
__device__ __forceinline__ float4 from_arr<4>(const float (&a)[4]) {
    return make_float4(a[0], a[1], a[2], a[3]);
}
template <>
__device__ __forceinline__ float2 from_arr<2>(const float (&a)[2]) {
    return make_float2(a[0], a[1]);
}
template <>
__device__ __forceinline__ float from_arr<1>(const float (&a)[1]) {
    return a[0];
}

__device__ __forceinline__ int64_t live_rows(int64_t rows, const int32_t* rows_dev) {
    if (rows_dev == nullptr) return rows;
    int64_t r = (int64_t)__ldg(rows_dev);
    if (r < 0) r = 0;
    return r < rows ? r : rows;
}

template <int V>
__global__ void __launch_bounds__(256) sparse_adagrad_kernel(const float* __restrict__ grad, float* __restrict__ state, float* out_delta,
                                                             float* __restrict__ out_upd, int64_t rows, const int32_t* rows_dev, int vec_per_row,
                                                             float neg_lr) {
    using VT = typename Vec<V>::type;
    const int64_t total = live_rows(rows, rows_dev) * vec_per_row;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        float g[V], s[V], d[V], u[V];
        to_arr<V>(reinterpret_cast<const VT*>(grad)[i], g);
        to_arr<V>(reinterpret_cast<const VT*>(state)[i], s);
        adagrad_elems<V>(g, s, d, u, neg_lr);
        reinterpret_cast<VT*>(state)[i] = from_arr<V>(s);
        if (out_upd != nullptr) reinterpret_cast<VT*>(out_upd)[i] = from_arr<V>(u);
        reinterpret_cast<VT*>(out_delta)[i] = from_arr<V>(d);
    }
}

template <int V, bool kAdd>
__global__ void __launch_bounds__(256) index_rows_kernel(float* __restrict__ table, int64_t table_rows, const int64_t* __restrict__ ids,
                                                         int64_t n, const int32_t* n_dev, int vec_per_row, float* __restrict__ dense,
                                                         int32_t* status) {
    using VT = typename Vec<V>::type;
    const int64_t total = live_rows(n, n_dev) * vec_per_row;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const int64_t l = i / vec_per_row;
        const int c = (int)(i - l * vec_per_row);
        const int64_t row = __ldg(&ids[l]);
        if (row < 0 || row >= table_rows) {
            or_status(status, GE2_STATUS_BAD_INDEX);
            if (!kAdd) {  // a row outside the table reads as zeros
                float z[V];
#pragma unroll
                for (int k = 0; k < V; k++) z[k] = 0.f;
                reinterpret_cast<VT*>(dense)[i] = from_arr<V>(z);
            }
            continue;
        }
        VT* trow = reinterpret_cast<VT*>(table) + row * vec_per_row + c;
        if (kAdd) {
            float a[V], b[V];
            to_arr<V>(*trow, a);
            to_arr<V>(reinterpret_cast<const VT*>(dense)[i], b);
#pragma unroll
            for (int k = 0; k < V; k++) a[k] = __fadd_rn(a[k], b[k]);
            *trow = from_arr<V>(a);
        } else {
            reinterpret_cast<VT*>(dense)[i] = *trow;
        }
    }
}

// Fused accumulateGradients + indexAdd(embeddings) + indexAdd(state): one read-modify-write of the touched rows.
// A group of 2^lg lanes (enough for a row where 32 are) takes two consecutive rows at a time, so that their loads overlap; with
// row_shared only the rows it names are touched (the others were finished where their gradient arose), and those that
// are not cost one load.
template <int V>
__device__ __forceinline__ void adagrad_rows(int64_t block, int64_t blocks, float* __restrict__ table, float* __restrict__ state, int64_t table_rows,
                                             const int64_t* __restrict__ unique_ids, int64_t U, const int32_t* U_dev, float* __restrict__ node_grad,
                                             int vec_per_row, int lg, float neg_lr, int clear_grad, const uint8_t* __restrict__ row_shared,
                                             int32_t* status) {
    using VT = typename Vec<V>::type;
    constexpr int kRows = 2;
    const int64_t rows = live_rows(U, U_dev);
    const int64_t groups = (blocks * blockDim.x) >> lg;
    const int l = threadIdx.x & ((1 << lg) - 1);
    for (int64_t r0 = ((block * blockDim.x + threadIdx.x) >> lg) * kRows; r0 < rows; r0 += groups * kRows) {
        int64_t row[kRows];
        bool on[kRows];
#pragma unroll
        for (int k = 0; k < kRows; k++) {
            on[k] = r0 + k < rows && (row_shared == nullptr || row_shared[r0 + k] != 0);
            row[k] = r0 + k < rows ? __ldg(&unique_ids[r0 + k]) : 0;
        }
#pragma unroll
        for (int k = 0; k < kRows; k++) {
            if (on[k] && (row[k] < 0 || row[k] >= table_rows)) {
                or_status(status, GE2_STATUS_BAD_INDEX);
                on[k] = false;
            }
        }
        for (int c = l; c < vec_per_row; c += 1 << lg) {
            float g[kRows][V], s[kRows][V], e[kRows][V];
#pragma unroll
            for (int k = 0; k < kRows; k++) {
                if (!on[k]) continue;
                to_arr<V>(reinterpret_cast<const VT*>(node_grad)[(r0 + k) * vec_per_row + c], g[k]);
                to_arr<V>(reinterpret_cast<const VT*>(state)[row[k] * vec_per_row + c], s[k]);
                to_arr<V>(reinterpret_cast<const VT*>(table)[row[k] * vec_per_row + c], e[k]);
            }
#pragma unroll
            for (int k = 0; k < kRows; k++) {
                if (!on[k]) continue;
                float dl[V], up[V];
                adagrad_elems<V>(g[k], s[k], dl, up, neg_lr);
#pragma unroll
                for (int v = 0; v < V; v++) {
                    e[k][v] = __fadd_rn(e[k][v], dl[v]);
                    g[k][v] = 0.f;
                }
                reinterpret_cast<VT*>(state)[row[k] * vec_per_row + c] = from_arr<V>(s[k]);
                reinterpret_cast<VT*>(table)[row[k] * vec_per_row + c] = from_arr<V>(e[k]);
                if (clear_grad) reinterpret_cast<VT*>(node_grad)[(r0 + k) * vec_per_row + c] = from_arr<V>(g[k]);
            }
        }
    }
}

template <int V>
__global__ void __launch_bounds__(256) adagrad_scatter_kernel(float* __restrict__ table, float* __restrict__ state, int64_t table_rows,
                                                              const int64_t* __restrict__ unique_ids, int64_t U, const int32_t* U_dev,
                                                              float* __restrict__ node_grad, int vec_per_row, int lg, float neg_lr, int clear_grad,
                                                              const uint8_t* __restrict__ row_shared, int32_t* status) {
    griddep_wait();  // the gradient rows come from the kernel before this one
    adagrad_rows<V>(blockIdx.x, gridDim.x, table, state, table_rows, unique_ids, U, U_dev, node_grad, vec_per_row, lg, neg_lr, clear_grad, row_shared, status);
}

template <int V>
__device__ __forceinline__ void adagrad_dense(int64_t block, int64_t blocks, float* __restrict__ param, float* __restrict__ sum, float* __restrict__ grad,
                                              int64_t vecs, float neg_lr, float eps, float grad_scale, int clear_grad) {
    using VT = typename Vec<V>::type;
    const int64_t stride = blocks * blockDim.x;
#pragma unroll 1
    for (int64_t i = block * blockDim.x + threadIdx.x; i < vecs; i += stride) {
        float g[V], s[V], p[V];
        to_arr<V>(reinterpret_cast<const VT*>(grad)[i], g);
        to_arr<V>(reinterpret_cast<const VT*>(sum)[i], s);
        to_arr<V>(reinterpret_cast<const VT*>(param)[i], p);
#pragma unroll
        for (int v = 0; v < V; v++) {
            if (grad_scale != 1.0f) g[v] = __fmul_rn(g[v], grad_scale);
            s[v] = __fadd_rn(s[v], __fmul_rn(g[v], g[v]));
            const float den = __fadd_rn(__fsqrt_rn(s[v]), eps);
            p[v] = __fadd_rn(p[v], __fmul_rn(neg_lr, __fdiv_rn(g[v], den)));
            g[v] = 0.f;
        }
        reinterpret_cast<VT*>(sum)[i] = from_arr<V>(s);
        reinterpret_cast<VT*>(param)[i] = from_arr<V>(p);
        if (clear_grad) reinterpret_cast<VT*>(grad)[i] = from_arr<V>(g);
    }
}

template <int V>
__global__ void __launch_bounds__(256) dense_adagrad_kernel(float* __restrict__ param, float* __restrict__ sum, float* __restrict__ grad,
                                                            int64_t vecs, float neg_lr, float eps, float grad_scale, int clear_grad) {
    griddep_wait();
    adagrad_dense<V>(blockIdx.x, gridDim.x, param, sum, grad, vecs, neg_lr, eps, grad_scale, clear_grad);
}

// Both in one launch, for a step whose launches follow one another: the first blocks take the dense tables, the others the rows.  Two launches
// fewer of 3 us each, where the tables are two (steps of 1 000 and 7 919 edges issued launch by launch: 59.3 -> 57.7 and 68.9 -> 67.2 us; in a graph, without the fork
// that put them beside each other, 10 000 edges: 82.6 -> 81.9).
struct DenseTables {
    float *param[2], *sum[2], *grad[2];
};
template <int V, int VD>
__global__ void __launch_bounds__(256) adagrad_step_kernel(float* __restrict__ table, float* __restrict__ state, int64_t table_rows,
                                                           const int64_t* __restrict__ unique_ids, int64_t U, const int32_t* U_dev,
                                                           float* __restrict__ node_grad, int vec_per_row, int lg, float neg_lr,
                                                           const uint8_t* __restrict__ row_shared, int32_t* status, const DenseTables dense, int blocks_each,
                                                           int num_dense, int64_t vecs, float neg_dense_lr, float eps, float grad_scale) {
    griddep_wait();  // the gradients come from the kernel before this one
    const int first = blocks_each * num_dense, b = blockIdx.x;
    if (b < first) {
        const int k = b >= blocks_each ? 1 : 0;
        adagrad_dense<VD>(b - k * blocks_each, blocks_each, k ? dense.param[1] : dense.param[0], k ? dense.sum[1] : dense.sum[0], k ? dense.grad[1] : dense.grad[0],
                          vecs, neg_dense_lr, eps, grad_scale, 1);
    } else {
        adagrad_rows<V>(b - first, (int)gridDim.x - first, table, state, table_rows, unique_ids, U, U_dev, node_grad, vec_per_row, lg, neg_lr, 1, row_shared, status);
    }
}

// ---- dense Adagrad fused with the relation-gradient all-reduce over peer memory -------------------------------------
// Every rank keeps its relation gradients in a buffer its peers can read: two halves used by alternate steps, then one
// 8-byte arrival flag per rank, one 8-byte verdict word and one 8-byte wait-time counter.  Two launches per rank and step:
//   peer_arrive_kernel (one warp): announce "my gradients of step t are complete" by writing t + 1 into my slot of every
//     peer's flag row, then wait -- lane p polls peer p, bounded by a time budget -- until every peer has announced the
//     same, and publish ONE verdict for the step in this rank's verdict word (t + 1 = go, 0 = a peer never arrived);
//   dense_adagrad_peers_kernel: every block reads that verdict, so all of them either run the optimizer step on the sum
//     of the ranks' gradients (read straight from the peers over NVLink, 16 bytes at a time) and clear the half the step
//     after next will accumulate into, or all of them leave the tables and the buffer untouched.
// Why one barrier is enough: a rank announces step t + 1 only when its step-t launches are over, so whoever gets past
// the wait of step t + 1 knows that nobody reads the half of step t any more.
__device__ __forceinline__ void st_release_sys_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_acquire_sys_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long global_timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

constexpr int kMaxPeers = 16;
struct PeerBuffers {
    float* buf[kMaxPeers];  // this process's mapping of every rank's gradient buffer, own rank included
};

__global__ void __launch_bounds__(32) peer_arrive_kernel(PeerBuffers peers, int world, int rank, int64_t numel,
                                                         const unsigned long long* __restrict__ step_dev, unsigned long long budget_ns,
                                                         int32_t* status) {
    const unsigned long long epoch = *step_dev + 1ull;
    const int64_t flags_off = 2 * numel;  // in floats; numel is even, so the flags are 8-byte aligned
    const int lane = threadIdx.x;
    int ok = 1;
    const unsigned long long t_enter = global_timer_ns();
    if (lane < world) {
        st_release_sys_u64(reinterpret_cast<unsigned long long*>(peers.buf[lane] + flags_off) + rank, epoch);
        const unsigned long long* mine = reinterpret_cast<const unsigned long long*>(peers.buf[rank] + flags_off) + lane;
        const unsigned long long t0 = global_timer_ns();
        ok = 0;
        // bounded twice: by the time budget and by an iteration count (should the timer not advance)
        for (uint32_t i = 0; i < (1u << 26); i++) {
            if (ld_acquire_sys_u64(mine) >= epoch) {
                ok = 1;
                break;
            }
            if ((i & 15u) == 15u && global_timer_ns() - t0 > budget_ns) break;
            __nanosleep(i < 64 ? 20 : 400);
        }
    }
    const bool all_ok = __all_sync(0xffffffffu, ok);
    const unsigned waited = __reduce_max_sync(0xffffffffu, lane < world ? (unsigned)min(global_timer_ns() - t_enter, 0xffffffffull) : 0u);
    if (lane == 0) {
        unsigned long long* verdict = reinterpret_cast<unsigned long long*>(peers.buf[rank] + flags_off) + world;
        *verdict = all_ok ? epoch : 0ull;
        verdict[1] += waited;  // diagnostic: nanoseconds this rank has spent in this kernel waiting for the slowest rank
        if (!all_ok) or_status(status, GE2_STATUS_PEER_TIMEOUT);
    }
}

template <int V>
__global__ void __launch_bounds__(256) dense_adagrad_peers_kernel(float* __restrict__ param, float* __restrict__ sum, PeerBuffers peers, int world,
                                                                  int rank, int64_t numel, const unsigned long long* __restrict__ step_dev,
                                                                  float neg_lr, float eps, float grad_scale) {
    using VT = typename Vec<V>::type;
    const unsigned long long epoch = *step_dev + 1ull;
    const int64_t flags_off = 2 * numel;
    // the one verdict of this step, written by the launch before this one on the same stream
    if (*(reinterpret_cast<const unsigned long long*>(peers.buf[rank] + flags_off) + world) != epoch) return;
    const int64_t cur = (int64_t)((epoch - 1ull) & 1ull) * numel;  // half holding this step's gradients
    const int64_t other = numel - cur;                            // half to clear for the step after next
    const int64_t nv = numel / V;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += stride) {
        float g[V], t[V], sm[V], pr[V], z[V];
#pragma unroll
        for (int k = 0; k < V; k++) g[k] = 0.f, z[k] = 0.f;
        for (int p = 0; p < world; p++) {  // volatile-style load: never a stale cached copy of peer memory
            to_arr<V>(__ldcv(reinterpret_cast<const VT*>(peers.buf[p] + cur) + i), t);
#pragma unroll
            for (int k = 0; k < V; k++) g[k] += t[k];
        }
        to_arr<V>(reinterpret_cast<const VT*>(sum)[i], sm);
        to_arr<V>(reinterpret_cast<const VT*>(param)[i], pr);
#pragma unroll
        for (int k = 0; k < V; k++) {
            const float gk = __fmul_rn(g[k], grad_scale);
            sm[k] = __fadd_rn(sm[k], __fmul_rn(gk, gk));
            const float den = __fadd_rn(__fsqrt_rn(sm[k]), eps);
            pr[k] = __fadd_rn(pr[k], __fmul_rn(neg_lr, __fdiv_rn(gk, den)));
        }
        reinterpret_cast<VT*>(sum)[i] = from_arr<V>(sm);
        reinterpret_cast<VT*>(param)[i] = from_arr<V>(pr);
        reinterpret_cast<VT*>(peers.buf[rank] + other)[i] = from_arr<V>(z);
    }
}

__global__ void __launch_bounds__(256) remap_edges_kernel(const int64_t* __restrict__ edges, int64_t n, int cols,
                                                          const int64_t* __restrict__ part_to_slot, int num_partitions,
                                                          int64_t partition_size, int64_t* __restrict__ out, int32_t* status) {
    const int64_t total = n * cols;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const int c = (int)(i % cols);
        int64_t v = edges[i];
        if (c == 0 || c == cols - 1) {
            const int64_t part = v / partition_size;  // ids are non-negative: same as the reference's floor of a double division
            int64_t slot = -1;
            if (v >= 0 && part < num_partitions) slot = __ldg(&part_to_slot[part]);
            if (slot < 0) {
                or_status(status, GE2_STATUS_BAD_INDEX);
                v = -1;
            } else {
                v = slot * partition_size + (v - part * partition_size);
            }
        }
        out[i] = v;
    }
}

struct SlabMoves {
    int32_t src[16];
    int32_t dst[16];
    int32_t count;
};

__global__ void __launch_bounds__(256) copy_slabs_kernel(const float4* __restrict__ src, float4* __restrict__ dst, SlabMoves moves,
                                                         int64_t slab_vec4) {
    const int m = blockIdx.y;
    const float4* s = src + (int64_t)moves.src[m] * slab_vec4;
    float4* d = dst + (int64_t)moves.dst[m] * slab_vec4;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < slab_vec4; i += stride) d[i] = s[i];
}

__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// (out of line: a 64-bit division is 1 KB of code, and kernels this short are bound by fetching theirs)
__device__ __noinline__ uint64_t div_u64(uint64_t a, uint64_t b) { return a / b; }

// What the sampler marks in the unique-map's bitsets on the way (words == null: nothing).  A marking kernel of its own reads every id again, one
// launch later: steps issued launch by launch, 1 000 edges, 69.2 us with it, 65.4 without.
struct SampleMarks {
    unsigned long long *words, *dup;
    int64_t domain;  // ids below it get a local id
    int32_t* status;
};

__global__ void __launch_bounds__(256) sample_negatives_kernel(const int64_t* __restrict__ src_ids, const int64_t* __restrict__ dst_ids,
                                                               int64_t edge_stride, int B, int C, int N, int n_deg, int64_t domain,
                                                               int want_src, uint64_t key, int64_t* __restrict__ packed,
                                                               int64_t* __restrict__ deg_rows, const uint64_t* __restrict__ step_dev,
                                                               int64_t num_batches, const int64_t* __restrict__ rel_ids,
                                                               int64_t* __restrict__ out_rel, const int64_t* __restrict__ num_batches_dev,
                                                               SampleMarks mk) {
    bool bad = false;
    auto mark = [&](int64_t id) {
        if (mk.words == nullptr) return;
        if ((uint64_t)id < (uint64_t)mk.domain) mark_id(mk.words, mk.dup, id);
        else bad = true;
    };
    // graph-replay form: the batch index lives on the device, so the same launch serves every batch of the epoch
    if (step_dev != nullptr) {
        const uint64_t step = *step_dev;
        if (num_batches_dev != nullptr) {  // ... and so does the length of the resident edge list
            num_batches = *num_batches_dev;
            if (num_batches < 1) num_batches = 1;
        }
        const int64_t off = (int64_t)(step - div_u64(step, (uint64_t)num_batches) * (uint64_t)num_batches) * B * edge_stride;
        src_ids += off;
        dst_ids += off;
        if (rel_ids != nullptr) rel_ids += off;
        key += step * 0x9E3779B97F4A7C15ull;
    }
    const int64_t CN = (int64_t)C * N;
    const int64_t total = 2 * (int64_t)B + CN;
    int64_t* out_src_neg = packed + 2 * (int64_t)B;
    int64_t* out_dst_neg = out_src_neg + (want_src ? CN : 0);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
#pragma unroll 1
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        if (i < B) {
            const int64_t id = src_ids[i * edge_stride];
            packed[i] = id;
            mark(id);
            if (out_rel != nullptr) out_rel[i] = rel_ids[i * edge_stride];
        } else if (i < 2 * (int64_t)B) {
            const int64_t id = dst_ids[(i - B) * edge_stride];
            packed[i] = id;
            mark(id);
        } else {
            const int64_t e = i - 2 * (int64_t)B;
            const int c = e >> 32 ? (int)div_u64((uint64_t)e, (uint64_t)N) : (int)((uint32_t)e / (uint32_t)N);
            const int j = (int)(e - (int64_t)c * N);
            const uint64_t r = splitmix64(key ^ splitmix64((uint64_t)e));
            if (j < n_deg) {
                const int64_t row = (int64_t)__umul64hi(r, (uint64_t)B);
                if (deg_rows != nullptr) deg_rows[(int64_t)c * n_deg + j] = row;
                const int64_t id = dst_ids[row * edge_stride], other = want_src ? src_ids[row * edge_stride] : id;
                out_dst_neg[e] = id;
                if (want_src) out_src_neg[e] = other;
                mark(id);
                if (other != id) mark(other);  // (equal ones, a negative of both sides, count as one occurrence)
            } else {
                const int64_t id = (int64_t)__umul64hi(r, (uint64_t)domain);
                out_dst_neg[e] = id;
                if (want_src) out_src_neg[e] = id;
                mark(id);
            }
        }
    }
    if (bad) atomicOr(mk.status, GE2_STATUS_ID_OUT_OF_RANGE);
}

inline int vec_width(int D, const void* a, const void* b = nullptr, const void* c = nullptr, const void* d = nullptr) {
    uintptr_t bits = (uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d;
    if (D % 4 == 0 && (bits & 15) == 0) return 4;
    if (D % 2 == 0 && (bits & 7) == 0) return 2;
    return 1;
}

}  // namespace
}  // namespace ge2

using namespace ge2;

extern "C" int ge2_sparse_adagrad(const float* grad, float* state_local, float* out_delta, float* out_state_update, int64_t rows,
                                  const int32_t* rows_dev, int32_t D, float lr, ge2_stream_t stream_) {
    if (rows < 0 || D <= 0) return GE2_ERR_INVALID_ARGUMENT;
    if (rows == 0) return GE2_OK;
    if (grad == nullptr || state_local == nullptr || out_delta == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    cudaStream_t stream = as_stream(stream_);
    const int V = vec_width(D, grad, state_local, out_delta, out_state_update);
    const int grid = stream_grid(rows * (D / V), 256);
    if (V == 4) sparse_adagrad_kernel<4><<<grid, 256, 0, stream>>>(grad, state_local, out_delta, out_state_update, rows, rows_dev, D / 4, -lr);
    else if (V == 2) sparse_adagrad_kernel<2><<<grid, 256, 0, stream>>>(grad, state_local, out_delta, out_state_update, rows, rows_dev, D / 2, -lr);
    else sparse_adagrad_kernel<1><<<grid, 256, 0, stream>>>(grad, state_local, out_delta, out_state_update, rows, rows_dev, D, -lr);
    GE2_LAUNCH_CHECK();
    return GE2_OK;
}

template <bool kAdd>
static int index_rows(float* table, int64_t table_rows, const int64_t* ids, int64_t n, const int32_t* n_dev, int32_t D, float* dense,
                      int32_t* status, ge2_stream_t stream_) {
    if (n < 0 || D <= 0 || table_rows < 0) return GE2_ERR_INVALID_ARGUMENT;
    if (n == 0) return GE2_OK;
    if (table == nullptr || ids == nullptr || dense == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    cudaStream_t stream = as_stream(stream_);
    const int V = vec_width(D, table, dense);
    const int grid = stream_grid(n * (D / V), 256);
    if (V == 4) index_rows_kernel<4, kAdd><<<grid, 256, 0, stream>>>(table, table_rows, ids, n, n_dev, D / 4, dense, status);
    else if (V == 2) index_rows_kernel<2, kAdd><<<grid, 256, 0, stream>>>(table, table_rows, ids, n, n_dev, D / 2, dense, status);
    else index_rows_kernel<1, kAdd><<<grid, 256, 0, stream>>>(table, table_rows, ids, n, n_dev, D, dense, status);
    GE2_LAUNCH_CHECK();
    return GE2_OK;
}

extern "C" int ge2_index_read(const float* table, int64_t table_rows, const int64_t* ids, int64_t n, const int32_t* n_dev, int32_t D,
                              float* out, int32_t* status, ge2_stream_t stream) {
    return index_rows<false>(const_cast<float*>(table), table_rows, ids, n, n_dev, D, out, status, stream);
}

extern "C" int ge2_index_add(float* table, int64_t table_rows, const int64_t* ids, int64_t n, const int32_t* n_dev, int32_t D,
                             const float* values, int32_t* status, ge2_stream_t stream) {
    return index_rows<true>(table, table_rows, ids, n, n_dev, D, const_cast<float*>(values), status, stream);
}

extern "C" int ge2_adagrad_scatter(float* table, float* state, int64_t table_rows, const int64_t* unique_ids, int64_t U,
                                   const int32_t* U_dev, float* node_grad, int32_t D, float lr, int32_t clear_grad, int32_t* status,
                                   ge2_stream_t stream) {
    return ge2_adagrad_scatter_shared(table, state, table_rows, unique_ids, U, U_dev, node_grad, D, lr, clear_grad, nullptr, status, stream);
}

extern "C" int ge2_adagrad_scatter_shared(float* table, float* state, int64_t table_rows, const int64_t* unique_ids, int64_t U,
                                          const int32_t* U_dev, float* node_grad, int32_t D, float lr, int32_t clear_grad,
                                          const uint8_t* row_shared, int32_t* status, ge2_stream_t stream_) {
    if (U < 0 || D <= 0 || table_rows < 0) return GE2_ERR_INVALID_ARGUMENT;
    if (U == 0) return GE2_OK;
    if (table == nullptr || state == nullptr || unique_ids == nullptr || node_grad == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    cudaStream_t stream = as_stream(stream_);
    const int V = vec_width(D, table, state, node_grad), vpr = D / V;
    int lg = 0;
    while (lg < 5 && (1 << lg) < vpr) lg++;
    const dim3 g((unsigned)stream_grid(ceil_div<int64_t>(U, 2) << lg, 256)), b(256);
    if (V == 4) GE2_CUDA_TRY(launch_after(adagrad_scatter_kernel<4>, g, b, 0, stream, table, state, table_rows, unique_ids, U, U_dev, node_grad, vpr, lg, -lr, clear_grad, row_shared, status));
    else if (V == 2) GE2_CUDA_TRY(launch_after(adagrad_scatter_kernel<2>, g, b, 0, stream, table, state, table_rows, unique_ids, U, U_dev, node_grad, vpr, lg, -lr, clear_grad, row_shared, status));
    else GE2_CUDA_TRY(launch_after(adagrad_scatter_kernel<1>, g, b, 0, stream, table, state, table_rows, unique_ids, U, U_dev, node_grad, vpr, lg, -lr, clear_grad, row_shared, status));
    return GE2_OK;
}

extern "C" int ge2_dense_adagrad(float* param, float* sum_state, float* grad, int64_t numel, float lr, float eps, float grad_scale,
                                 int32_t clear_grad, ge2_stream_t stream_) {
    if (numel < 0) return GE2_ERR_INVALID_ARGUMENT;
    if (numel == 0) return GE2_OK;
    if (param == nullptr || sum_state == nullptr || grad == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    cudaStream_t stream = as_stream(stream_);
    if (numel % 4 == 0 && (((uintptr_t)param | (uintptr_t)sum_state | (uintptr_t)grad) & 15) == 0)
        GE2_CUDA_TRY(launch_after(dense_adagrad_kernel<4>, dim3((unsigned)stream_grid(numel / 4, 256)), dim3(256), 0, stream, param, sum_state, grad, numel / 4, -lr, eps, grad_scale, clear_grad));
    else
        GE2_CUDA_TRY(launch_after(dense_adagrad_kernel<1>, dim3((unsigned)stream_grid(numel, 256)), dim3(256), 0, stream, param, sum_state, grad, numel, -lr, eps, grad_scale, clear_grad));
    return GE2_OK;
}

extern "C" int ge2_dense_adagrad_peers(float* param, float* sum_state, float* const* peer_bufs, int32_t world, int32_t rank, int64_t numel,
                                       const uint64_t* step_dev, float lr, float eps, float grad_scale, uint32_t wait_budget_us, int32_t* status,
                                       ge2_stream_t stream_) {
    if (numel <= 0 || (numel & 1) || world < 1 || world > kMaxPeers || rank < 0 || rank >= world) return GE2_ERR_INVALID_ARGUMENT;
    if (param == nullptr || sum_state == nullptr || peer_bufs == nullptr || step_dev == nullptr || status == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    PeerBuffers pb;
    for (int p = 0; p < kMaxPeers; p++) pb.buf[p] = p < world ? peer_bufs[p] : nullptr;
    for (int p = 0; p < world; p++)
        if (pb.buf[p] == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    const unsigned long long budget_ns = (wait_budget_us == 0 ? 4000000ull : (unsigned long long)wait_budget_us) * 1000ull;
    cudaStream_t stream = as_stream(stream_);
    const unsigned long long* step = reinterpret_cast<const unsigned long long*>(step_dev);
    peer_arrive_kernel<<<1, 32, 0, stream>>>(pb, world, rank, numel, step, budget_ns, status);
    GE2_LAUNCH_CHECK();
    uintptr_t bits = (uintptr_t)param | (uintptr_t)sum_state;
    for (int p = 0; p < world; p++) bits |= (uintptr_t)pb.buf[p];
    if (numel % 4 == 0 && (bits & 15) == 0)
        dense_adagrad_peers_kernel<4><<<stream_grid(numel / 4, 256), 256, 0, stream>>>(param, sum_state, pb, world, rank, numel, step, -lr, eps, grad_scale);
    else
        dense_adagrad_peers_kernel<1><<<stream_grid(numel, 256), 256, 0, stream>>>(param, sum_state, pb, world, rank, numel, step, -lr, eps, grad_scale);
    GE2_LAUNCH_CHECK();
    return GE2_OK;
}

extern "C" int ge2_enable_peer_access(int32_t peer_device) {
    int dev = 0;
    GE2_CUDA_TRY(cudaGetDevice(&dev));
    if (peer_device == dev) return GE2_OK;
    int can = 0;
    GE2_CUDA_TRY(cudaDeviceCanAccessPeer(&can, dev, peer_device));
    if (!can) return GE2_ERR_INVALID_ARGUMENT;
    const cudaError_t e = cudaDeviceEnablePeerAccess(peer_device, 0);
    if (e == cudaErrorPeerAccessAlreadyEnabled) {
        (void)cudaGetLastError();
        return GE2_OK;
    }
    GE2_CUDA_TRY(e);
    return GE2_OK;
}

extern "C" int ge2_sample_negatives(const int64_t* src_ids, const int64_t* dst_ids, int64_t edge_stride, int32_t B, int32_t C, int32_t N,
                                    int32_t n_deg, int64_t domain, int32_t want_src_negs, uint64_t seed, uint64_t batch_index,
                                    int64_t* out_packed_ids, int64_t* out_deg_rows, ge2_stream_t stream_) {
    if (B <= 0 || C <= 0 || N <= 0 || n_deg < 0 || n_deg > N || domain <= 0 || edge_stride <= 0) return GE2_ERR_INVALID_ARGUMENT;
    if (src_ids == nullptr || dst_ids == nullptr || out_packed_ids == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    if (n_deg > 0 && out_deg_rows == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    const int64_t total = 2 * (int64_t)B + (int64_t)C * N;
    const uint64_t key = seed * 0xD1342543DE82EF95ull + batch_index * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull;
    sample_negatives_kernel<<<stream_grid(total, 256), 256, 0, as_stream(stream_)>>>(src_ids, dst_ids, edge_stride, B, C, N, n_deg, domain,
                                                                                   want_src_negs, key, out_packed_ids, out_deg_rows, nullptr, 1,
                                                                                   nullptr, nullptr, nullptr, SampleMarks{});
    GE2_LAUNCH_CHECK();
    return GE2_OK;
}

static int sample_batch_impl(const int64_t* edges, int32_t cols, int64_t num_batches, const int64_t* num_batches_dev, const uint64_t* step_dev,
                             int32_t B, int32_t C, int32_t N, int32_t n_deg, int64_t domain, int32_t want_src_negs, uint64_t seed,
                             int64_t* out_packed_ids, int64_t* out_deg_rows, int64_t* out_rel_ids, ge2_stream_t stream_) {
    if (B <= 0 || C <= 0 || N <= 0 || n_deg < 0 || n_deg > N || domain <= 0 || num_batches <= 0 || (cols != 2 && cols != 3))
        return GE2_ERR_INVALID_ARGUMENT;
    if (edges == nullptr || step_dev == nullptr || out_packed_ids == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    if ((n_deg > 0 && out_deg_rows == nullptr) || (cols == 3 && out_rel_ids == nullptr)) return GE2_ERR_INVALID_ARGUMENT;
    const int64_t total = 2 * (int64_t)B + (int64_t)C * N;
    const uint64_t key = seed * 0xD1342543DE82EF95ull + 0x632BE59BD9B4E019ull;
    sample_negatives_kernel<<<stream_grid(total, 256), 256, 0, as_stream(stream_)>>>(
        edges, edges + cols - 1, cols, B, C, N, n_deg, domain, want_src_negs, key, out_packed_ids, out_deg_rows, step_dev, num_batches,
        cols == 3 ? edges + 1 : nullptr, cols == 3 ? out_rel_ids : nullptr, num_batches_dev, SampleMarks{});
    GE2_LAUNCH_CHECK();
    return GE2_OK;
}

extern "C" int ge2_sample_batch(const int64_t* edges, int32_t cols, int64_t num_batches, const uint64_t* step_dev, int32_t B, int32_t C,
                                int32_t N, int32_t n_deg, int64_t domain, int32_t want_src_negs, uint64_t seed, int64_t* out_packed_ids,
                                int64_t* out_deg_rows, int64_t* out_rel_ids, ge2_stream_t stream) {
    return sample_batch_impl(edges, cols, num_batches, nullptr, step_dev, B, C, N, n_deg, domain, want_src_negs, seed, out_packed_ids,
                             out_deg_rows, out_rel_ids, stream);
}

extern "C" int ge2_sample_batch_dev(const int64_t* edges, int32_t cols, const int64_t* num_batches_dev, const uint64_t* step_dev, int32_t B,
                                    int32_t C, int32_t N, int32_t n_deg, int64_t domain, int32_t want_src_negs, uint64_t seed,
                                    int64_t* out_packed_ids, int64_t* out_deg_rows, int64_t* out_rel_ids, ge2_stream_t stream) {
    if (num_batches_dev == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    return sample_batch_impl(edges, cols, 1, num_batches_dev, step_dev, B, C, N, n_deg, domain, want_src_negs, seed, out_packed_ids,
                             out_deg_rows, out_rel_ids, stream);
}

__global__ void advance_step_kernel(uint64_t* step, int n) {
    if ((int)threadIdx.x < n) step[threadIdx.x] += 1;
}

extern "C" int ge2_advance_step(uint64_t* step_dev, int32_t n, ge2_stream_t stream_) {
    if (step_dev == nullptr || n < 1 || n > 32) return GE2_ERR_INVALID_ARGUMENT;
    advance_step_kernel<<<1, 32, 0, as_stream(stream_)>>>(step_dev, n);
    GE2_LAUNCH_CHECK();
    return GE2_OK;
}

static int front_check(const ge2_front_desc* f) {
    if (f == nullptr || f->B <= 0 || f->C <= 0 || f->N <= 0 || f->n_deg < 0 || f->n_deg > f->N || f->domain <= 0 || f->mapped <= 0 ||
        (f->cols != 2 && f->cols != 3))
        return GE2_ERR_INVALID_ARGUMENT;
    if (f->step_dev != nullptr && f->num_batches <= 0 && f->num_batches_dev == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    if (f->edges == nullptr || f->packed == nullptr || f->unique == nullptr || f->inverse == nullptr || f->count == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    if (f->n_deg > 0 && f->deg_rows == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    if (f->sms < 0 || f->sms > kNumSMs) return GE2_ERR_INVALID_ARGUMENT;
    if (f->num_counters < 0 || f->num_counters > 32 || (f->num_counters > 0 && f->counters == nullptr)) return GE2_ERR_INVALID_ARGUMENT;
    const int64_t n = 2 * (int64_t)f->B + (f->want_src_negs ? 2 : 1) * (int64_t)f->C * f->N;
    if (n > kUniqueMaxIds || num_words_of(f->mapped) > kUniqueMaxIds) return GE2_ERR_UNSUPPORTED;
    if (f->unique_ws == nullptr || ((uintptr_t)f->unique_ws & 255) != 0 || f->unique_ws_bytes < unique_ws_bytes(f->mapped, f->shared != nullptr ? 2 : 1))
        return GE2_ERR_WORKSPACE;
    return GE2_OK;
}

extern "C" int ge2_sample_unique(const ge2_front_desc* f, ge2_stream_t stream_) {
    const int rc = front_check(f);
    if (rc != GE2_OK) return rc;
    cudaStream_t stream = as_stream(stream_);
    const int sms = f->sms == 0 ? kNumSMs : f->sms;
    const UniqueWorkspace ws = unique_carve(f->unique_ws, f->mapped, f->shared != nullptr);
    const int64_t CN = (int64_t)f->C * f->N, total = 2 * (int64_t)f->B + CN;
    GE2_CUDA_TRY(cudaMemsetAsync(ws.tile_state, 0, ws.clear_bytes, stream));
    uint64_t key = f->seed * 0xD1342543DE82EF95ull + 0x632BE59BD9B4E019ull;
    if (f->step_dev == nullptr) key += f->batch_index * 0x9E3779B97F4A7C15ull;
    const bool rel = f->cols == 3 && f->rel_ids != nullptr;
    sample_negatives_kernel<<<std::min(stream_grid(total, 256), sms * 6), 256, 0, stream>>>(
        f->edges, f->edges + f->cols - 1, f->cols, f->B, f->C, f->N, f->n_deg, f->domain, f->want_src_negs, key, f->packed, f->deg_rows, f->step_dev,
        f->num_batches, rel ? f->edges + 1 : nullptr, rel ? f->rel_ids : nullptr, f->num_batches_dev,
        SampleMarks{ws.words, ws.dup, f->mapped, ws.status});
    GE2_LAUNCH_CHECK();
    return unique_emit(ws, f->packed, total + (f->want_src_negs ? CN : 0), f->mapped, f->unique, f->inverse, f->count, f->shared, f->counters,
                           f->num_counters, sms, stream);
}

extern "C" int ge2_remap_edges_to_slots(const int64_t* edges, int64_t n, int32_t cols, const int64_t* partition_to_slot,
                                        int32_t num_partitions, int64_t partition_size, int64_t* out, int32_t* status,
                                        ge2_stream_t stream_) {
    if (n < 0 || (cols != 2 && cols != 3) || num_partitions <= 0 || partition_size <= 0) return GE2_ERR_INVALID_ARGUMENT;
    if (n == 0) return GE2_OK;
    if (edges == nullptr || partition_to_slot == nullptr || out == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    remap_edges_kernel<<<stream_grid(n * cols, 256), 256, 0, as_stream(stream_)>>>(edges, n, cols, partition_to_slot, num_partitions,
                                                                                 partition_size, out, status);
    GE2_LAUNCH_CHECK();
    return GE2_OK;
}

extern "C" int ge2_copy_slabs(const float* src, float* dst, const int32_t* moves_host, int32_t num_moves, int64_t slab_floats,
                              ge2_stream_t stream_) {
    if (num_moves < 0 || num_moves > 16 || slab_floats < 0) return GE2_ERR_INVALID_ARGUMENT;
    if (num_moves == 0 || slab_floats == 0) return GE2_OK;
    if (src == nullptr || dst == nullptr || moves_host == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    if ((slab_floats & 3) != 0 || (((uintptr_t)src | (uintptr_t)dst) & 15) != 0) return GE2_ERR_UNSUPPORTED;
    SlabMoves mv;
    mv.count = num_moves;
    for (int k = 0; k < num_moves; k++) {
        mv.src[k] = moves_host[2 * k];
        mv.dst[k] = moves_host[2 * k + 1];
        if (mv.src[k] < 0 || mv.dst[k] < 0) return GE2_ERR_INVALID_ARGUMENT;
    }
    const int64_t v4 = slab_floats / 4;
    dim3 grid((unsigned)stream_grid(v4, 256 * 4, 8), (unsigned)num_moves);
    copy_slabs_kernel<<<grid, 256, 0, as_stream(stream_)>>>(reinterpret_cast<const float4*>(src), reinterpret_cast<float4*>(dst), mv, v4);
    GE2_LAUNCH_CHECK();
    return GE2_OK;
}

namespace {
struct RowUpdate {
    float *table, *state;
    int64_t table_rows;
    const int64_t* unique;
    int64_t U;
    const int32_t* U_dev;
    float* grad;
    int D;
    float lr;
    const uint8_t* shared;
    int32_t* status;
};
template <int V, int VD>
int launch_adagrad_step(const RowUpdate& r, const DenseTables& dense, int num_dense, int64_t numel, float dense_lr, float eps, float grad_scale, cudaStream_t stream) {
    const int vpr = r.D / V;
    int lg = 0;
    while (lg < 5 && (1 << lg) < vpr) lg++;
    const int64_t vecs = numel / VD;
    const int each = stream_grid(vecs, 256), rows = stream_grid(ceil_div<int64_t>(r.U, 2) << lg, 256);
    GE2_CUDA_TRY(launch_after(adagrad_step_kernel<V, VD>, dim3((unsigned)(each * num_dense + rows)), dim3(256), 0, stream, r.table, r.state, r.table_rows, r.unique, r.U,
                              r.U_dev, r.grad, vpr, lg, -r.lr, r.shared, r.status, dense, each, num_dense, vecs, -dense_lr, eps, grad_scale));
    return GE2_OK;
}
}  // namespace

extern "C" int ge2_adagrad_step(float* table, float* state, int64_t table_rows, const int64_t* unique_ids, int64_t U, const int32_t* U_dev, float* node_grad,
                                int32_t D, float lr, const uint8_t* row_shared, int32_t* status, int32_t num_dense, float* const* dense_param,
                                float* const* dense_state, float* const* dense_grad, int64_t dense_numel, float dense_lr, float eps, float grad_scale,
                                ge2_stream_t stream) {
    if (U < 0 || D <= 0 || table_rows < 0 || num_dense < 0 || num_dense > 2 || dense_numel < 0) return GE2_ERR_INVALID_ARGUMENT;
    if (U > 0 && (table == nullptr || state == nullptr || unique_ids == nullptr || node_grad == nullptr)) return GE2_ERR_INVALID_ARGUMENT;
    if (dense_numel == 0) num_dense = 0;
    DenseTables dense = {};
    uintptr_t bits = (uintptr_t)(dense_numel % 4) * 4;
    for (int k = 0; k < num_dense; k++) {
        if (dense_param == nullptr || dense_state == nullptr || dense_grad == nullptr) return GE2_ERR_INVALID_ARGUMENT;
        dense.param[k] = dense_param[k], dense.sum[k] = dense_state[k], dense.grad[k] = dense_grad[k];
        if (dense.param[k] == nullptr || dense.sum[k] == nullptr || dense.grad[k] == nullptr) return GE2_ERR_INVALID_ARGUMENT;
        bits |= (uintptr_t)dense_param[k] | (uintptr_t)dense_state[k] | (uintptr_t)dense_grad[k];
    }
    if (num_dense > 0 && U > 0) {
        const RowUpdate r = {table, state, table_rows, unique_ids, U, U_dev, node_grad, D, lr, row_shared, status};
        const int V = vec_width(D, table, state, node_grad);
        auto go = [&](auto kernel) { return kernel(r, dense, num_dense, dense_numel, dense_lr, eps, grad_scale, as_stream(stream)); };
        if ((bits & 15) == 0) return V == 4 ? go(launch_adagrad_step<4, 4>) : V == 2 ? go(launch_adagrad_step<2, 4>) : go(launch_adagrad_step<1, 4>);
        return V == 4 ? go(launch_adagrad_step<4, 1>) : V == 2 ? go(launch_adagrad_step<2, 1>) : go(launch_adagrad_step<1, 1>);
    }
    int rc = ge2_adagrad_scatter_shared(table, state, table_rows, unique_ids, U, U_dev, node_grad, D, lr, 1, row_shared, status, stream);
    for (int k = 0; rc == GE2_OK && k < num_dense; k++)
        rc = ge2_dense_adagrad(dense.param[k], dense.sum[k], dense.grad[k], dense_numel, dense_lr, eps, grad_scale, 1, stream);
    return rc;
}

extern "C" int ge2_train_step(const ge2_train_desc* t, ge2_stream_t stream) {
    // everything is looked at before the first launch: a call that is refused has changed nothing
    if (t == nullptr || t->lp == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    const ge2_lp_desc& d = *t->lp;
    size_t need = 0;
    int rc = ge2_lp_workspace_bytes(&d, &need);  // also: is the descriptor a valid one?
    if (rc != GE2_OK) return rc;
    need = lp_make_layout(d, nullptr, false).bytes;  // what ge2_lp_step can do with
    if (d.workspace == nullptr || ((uintptr_t)d.workspace & 255) != 0 || d.workspace_bytes < need) return GE2_ERR_WORKSPACE;
    if (t->edges == nullptr || t->cols <= 0 || t->n_deg < 0 || t->n_deg > d.N || t->domain <= 0 || t->table_rows <= 0) return GE2_ERR_INVALID_ARGUMENT;
    if (t->packed == nullptr || t->unique == nullptr || t->inverse == nullptr || t->count == nullptr || (t->n_deg > 0 && t->deg_rows == nullptr))
        return GE2_ERR_INVALID_ARGUMENT;
    if (t->n_ids != 2 * (int64_t)d.B + (d.use_inverse ? 2 : 1) * (int64_t)d.C * d.N) return GE2_ERR_INVALID_ARGUMENT;  // what the sampler packs
    if (t->twin_begin < 0 || t->twin_len < 0 || (t->twin_len > 0 && t->twin_begin + 2 * t->twin_len > t->n_ids)) return GE2_ERR_INVALID_ARGUMENT;
    if (d.deg_sample_rows != nullptr && d.deg_sample_rows == t->deg_rows && d.n_deg != t->n_deg) return GE2_ERR_INVALID_ARGUMENT;
    if (t->table == nullptr || t->state == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    // the two halves of the row update, the finish kernel's and the scatter's, share the rows out by the same bytes and have one rate, table and state
    const bool fused = (d.flags & GE2_LP_HAS_ROW_UPDATE) != 0 && d.node_state != nullptr;
    if (t->shared != (fused ? d.row_shared : nullptr)) return GE2_ERR_INVALID_ARGUMENT;
    if (fused && (d.node_emb != t->table || d.node_state != t->state || d.row_index != t->unique || d.emb_stride != d.D || d.node_lr != t->lr ||
                  d.table_rows != t->table_rows))
        return GE2_ERR_INVALID_ARGUMENT;
    if (t->num_dense < 0 || t->num_dense > 2 || t->dense_numel < 0) return GE2_ERR_INVALID_ARGUMENT;
    for (int k = 0; k < t->num_dense && t->dense_numel > 0; k++)
        if (t->dense_param[k] == nullptr || t->dense_state[k] == nullptr || t->dense_grad[k] == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    const int64_t mapped = std::min(t->domain, t->table_rows);  // ids past the table get no local id: they are flagged, and no later kernel meets them
    if (t->unique_ws == nullptr || ((uintptr_t)t->unique_ws & 255) != 0 || t->unique_ws_bytes < ge2_unique_workspace_bytes(mapped)) return GE2_ERR_WORKSPACE;

    ge2_front_desc f = {};
    f.edges = t->edges, f.cols = t->cols, f.seed = t->seed, f.batch_index = t->batch_index;
    f.B = d.B, f.C = d.C, f.N = d.N, f.n_deg = t->n_deg, f.domain = t->domain, f.want_src_negs = d.use_inverse;
    f.packed = t->packed, f.deg_rows = t->deg_rows, f.mapped = mapped;
    f.unique_ws = t->unique_ws, f.unique_ws_bytes = t->unique_ws_bytes;
    f.unique = t->unique, f.inverse = t->inverse, f.count = t->count, f.shared = t->shared;
    // the sampler's own marking counts a negative that both sides share once
    const bool twins = t->shared == nullptr || (d.use_inverse ? t->twin_begin == 2 * (int64_t)d.B && t->twin_len == (int64_t)d.C * d.N : t->twin_len == 0);
    if (twins && (t->cols == 2 || t->cols == 3)) {
        rc = ge2_sample_unique(&f, stream);
    } else {
        rc = ge2_sample_negatives(t->edges, t->edges + t->cols - 1, t->cols, d.B, d.C, d.N, t->n_deg, t->domain, d.use_inverse, t->seed, t->batch_index,
                                  t->packed, t->deg_rows, stream);
        if (rc == GE2_OK)
            rc = ge2_unique_bitmap_shared(t->packed, t->n_ids, mapped, t->unique_ws, t->unique_ws_bytes, t->unique, t->inverse, t->count, t->shared,
                                          t->twin_begin, t->twin_len, stream);
    }
    if (rc != GE2_OK) return rc;
    rc = ge2_lp_step(&d, stream);
    if (rc != GE2_OK) return rc;
    return ge2_adagrad_step(t->table, t->state, t->table_rows, t->unique, d.U, t->count, d.node_grad, d.D, t->lr, t->shared, d.status, t->num_dense, t->dense_param,
                            t->dense_state, t->dense_grad, t->dense_numel, t->dense_lr, 1e-10f, t->grad_scale, stream);
}
