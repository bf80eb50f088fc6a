// Link-prediction training step (forward scores, softmax cross-entropy, backward) -- gather / scatter halves.
// The contraction-heavy middle lives in lp_scores_fp32.cu / lp_scores_f16.cu.
//
// Follows, in the reference project: Model::train_batch up to loss.backward() (cpp/src/nn/model.cpp:362-397),
// mod_node_corrupt_forward RNS branch (cpp/src/nn/decoders/edge/decoder_methods.cpp:724-806,933-946,1089-1097),
// relation operators (relation_operators.cpp:3-31), apply_score_filter (cpp/src/data/samplers/negative.cpp:570-575)
// and SoftmaxCrossEntropy with SUM reduction (cpp/src/nn/loss.cpp:46-63).
#include <algorithm>
#include <cstddef>
#include <cstring>

#include "adagrad.cuh"
#include "lp_internal.cuh"

namespace ge2 {
namespace {

// The row of a local node id; the first row in the place of one that the table does not have (the finish kernel reports it and leaves its
// gradient out).  Dropping what was read instead, here, is a dozen instructions more a row: 0.5 us of a step of 88.
__device__ __forceinline__ const float* emb_row(const ge2_lp_desc& d, int64_t local) {
    const int64_t row = d.row_index != nullptr ? __ldg(&d.row_index[local]) : local;
    return d.node_emb + ((uint64_t)row < (uint64_t)d.table_rows ? row : 0) * d.emb_stride;
}

// ---------------------------------------------------------------------------------------------------
// mask: one int per (side, chunk, column) = the batch row whose score there is overwritten with -1e9
// ---------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) mask_from_pairs_kernel(const int64_t* __restrict__ pairs, int64_t F, int npc, int Bp, int N,
                                                              int32_t* __restrict__ mask, int32_t* status) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; f < F; f += stride) {
        const int64_t row = pairs[2 * f], col = pairs[2 * f + 1];
        if (row < 0 || row >= Bp || col < 0 || col >= N) {
            or_status(status, GE2_STATUS_BAD_INDEX);
            continue;
        }
        const int c = (int)(row / npc);
        const int32_t old = atomicCAS(&mask[(int64_t)c * N + col], -1, (int32_t)row);
        if (old != -1 && old != (int32_t)row) or_status(status, GE2_STATUS_FILTER_COLLISION);
    }
}

// ---------------------------------------------------------------------------------------------------
// A row of D columns is spread over ld / 4 lanes (16 or 32), four values a lane.
//   plain   : lane l holds columns [4l, 4l + 4), or (V == 1) columns l, l + ld / 4, l + 2 ld / 4, l + 3 ld / 4, so that scalar accesses
//             of neighbouring lanes are neighbours
//   ComplEx : coordinates 2l and 2l + 1 of the h = D / 2 complex ones, or (V == 1) l and l + ld / 4: .x .y their real parts (columns k, k'),
//             .z .w their imaginary parts (columns h + k, h + k'), so the relation operator and its backward need no other lane's values
// V is the widest access that the row length and the pointers allow (4 only for plain rows); columns past the row read as zero.
// ---------------------------------------------------------------------------------------------------
template <int V, bool CPLX>
__device__ __forceinline__ float4 load_row(const float* __restrict__ row, int l, int D) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    const int k = CPLX ? 2 * l : 4 * l, h = D >> 1;
    if constexpr (CPLX) {
        if constexpr (V == 2) {
            if (k < h) {
                const float2 a = __ldg(reinterpret_cast<const float2*>(row + k)), b = __ldg(reinterpret_cast<const float2*>(row + h + k));
                v = make_float4(a.x, a.y, b.x, b.y);
            }
        } else {
            const int n = lp_row_ld(D) >> 2;
            if (l < h) v.x = __ldg(row + l), v.z = __ldg(row + h + l);
            if (l + n < h) v.y = __ldg(row + l + n), v.w = __ldg(row + h + l + n);
        }
    } else if constexpr (V == 4) {
        if (k < D) v = __ldg(reinterpret_cast<const float4*>(row + k));
    } else if constexpr (V == 2) {
        if (k < D) {
            const float2 a = __ldg(reinterpret_cast<const float2*>(row + k));
            v.x = a.x, v.y = a.y;
        }
        if (k + 2 < D) {
            const float2 b = __ldg(reinterpret_cast<const float2*>(row + k + 2));
            v.z = b.x, v.w = b.y;
        }
    } else {
        const int n = lp_row_ld(D) >> 2;
        if (l < D) v.x = __ldg(row + l);
        if (l + n < D) v.y = __ldg(row + l + n);
        if (l + 2 * n < D) v.z = __ldg(row + l + 2 * n);
        if (l + 3 * n < D) v.w = __ldg(row + l + 3 * n);
    }
    return v;
}

struct PutStore {
    static __device__ __forceinline__ void one(float* p, float a) { *p = a; }
    static __device__ __forceinline__ void two(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
    static __device__ __forceinline__ void four(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
};
struct PutAdd {  // reductions at L2, as wide as the row allows
    static __device__ __forceinline__ void one(float* p, float a) { atomicAdd(p, a); }
    static __device__ __forceinline__ void two(float* p, float a, float b) { atomicAdd(reinterpret_cast<float2*>(p), make_float2(a, b)); }
    static __device__ __forceinline__ void four(float* p, float4 v) { atomicAdd(reinterpret_cast<float4*>(p), v); }
};
template <int V, bool CPLX, typename Put>
__device__ __forceinline__ void put_row(float* row, int l, int D, float4 v) {
    const int k = CPLX ? 2 * l : 4 * l, h = D >> 1;
    if constexpr (CPLX) {
        if constexpr (V == 2) {
            if (k < h) Put::two(row + k, v.x, v.y), Put::two(row + h + k, v.z, v.w);
        } else {
            const int n = lp_row_ld(D) >> 2;
            if (l < h) Put::one(row + l, v.x), Put::one(row + h + l, v.z);
            if (l + n < h) Put::one(row + l + n, v.y), Put::one(row + h + l + n, v.w);
        }
    } else if constexpr (V == 4) {
        if (k < D) Put::four(row + k, v);
    } else if constexpr (V == 2) {
        if (k < D) Put::two(row + k, v.x, v.y);
        if (k + 2 < D) Put::two(row + k + 2, v.z, v.w);
    } else {
        const int n = lp_row_ld(D) >> 2;
        if (l < D) Put::one(row + l, v.x);
        if (l + n < D) Put::one(row + l + n, v.y);
        if (l + 2 * n < D) Put::one(row + l + 2 * n, v.z);
        if (l + 3 * n < D) Put::one(row + l + 3 * n, v.w);
    }
}

// the relation operator: element-wise product, or product of complex numbers
template <bool CPLX>
__device__ __forceinline__ float4 rel_mul(float4 a, float4 r) {
    if constexpr (CPLX) return make_float4(a.x * r.x - a.z * r.z, a.y * r.y - a.w * r.w, a.x * r.z + a.z * r.x, a.y * r.w + a.w * r.y);
    else return make_float4(a.x * r.x, a.y * r.y, a.z * r.z, a.w * r.w);
}
// ... and its transpose: the gradient of a from that of a x r (and of r from it, with a in the place of r)
template <bool CPLX>
__device__ __forceinline__ float4 rel_mul_t(float4 g, float4 r) {
    if constexpr (CPLX) return make_float4(g.x * r.x + g.z * r.z, g.y * r.y + g.w * r.w, -g.x * r.z + g.z * r.x, -g.y * r.w + g.w * r.y);
    else return make_float4(g.x * r.x, g.y * r.y, g.z * r.z, g.w * r.w);
}
__device__ __forceinline__ float4 axpy4(float a, float4 x, float4 y) { return make_float4(a * x.x + y.x, a * x.y + y.y, a * x.z + y.z, a * x.w + y.w); }
__device__ __forceinline__ float4 add4(float4 x, float4 y) { return make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w); }
__device__ __forceinline__ float4 scale4(float a, float4 x) { return make_float4(a * x.x, a * x.y, a * x.z, a * x.w); }
__device__ __forceinline__ float dot4(float4 x, float4 y) { return x.x * y.x + x.y * y.y + x.z * y.z + x.w * y.w; }

__device__ __forceinline__ void store_half4(__half* dst, float4 v) {
    const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
    uint2 pk;
    pk.x = *reinterpret_cast<const uint32_t*>(&lo);
    pk.y = *reinterpret_cast<const uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(dst) = pk;
}

// an fp32 value as the sum of three bf16 values, exactly (24 bits as 8 + 8 + 8; rounded to nearest, so the parts alternate in sign and
// the later ones are at most 2^-8 and 2^-16 of it)
__device__ __forceinline__ void store_split4(__nv_bfloat16* dst, int64_t plane, float4 v) {
    const float x[4] = {v.x, v.y, v.z, v.w};
    float r[4];
#pragma unroll
    for (int e = 0; e < 4; e++) r[e] = x[e];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const __nv_bfloat162 a = __floats2bfloat162_rn(r[0], r[1]), b = __floats2bfloat162_rn(r[2], r[3]);
        uint2 pk;
        pk.x = *reinterpret_cast<const uint32_t*>(&a);
        pk.y = *reinterpret_cast<const uint32_t*>(&b);
        *reinterpret_cast<uint2*>(dst + k * plane) = pk;
        const float2 fa = __bfloat1622float2(a), fb = __bfloat1622float2(b);
        r[0] -= fa.x, r[1] -= fa.y, r[2] -= fb.x, r[3] -= fb.y;
    }
}

// one row in the lanes' layout as an operand row of the scores kernels: fp16, or (plane > 0) the three bf16 planes
template <int V, bool CPLX, bool HALF>
__device__ __forceinline__ void store_operand(void* rows, int64_t plane, int64_t row, int ld, int l, int D, float4 v) {
    if constexpr (!CPLX && V == 1) {
        const int n = ld >> 2;
        float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
            uint16_t* p = (uint16_t*)rows + row * ld + l + e * n;
            if constexpr (HALF) {
                *p = __half_as_ushort(__float2half_rn(x[e]));
            } else {
#pragma unroll
                for (int t = 0; t < 3; t++, p += plane) {
                    const __nv_bfloat16 b = __float2bfloat16_rn(x[e]);
                    *p = __bfloat16_as_ushort(b);
                    x[e] -= __bfloat162float(b);
                }
            }
        }
    } else if constexpr (!CPLX) {
        if constexpr (HALF) store_half4((__half*)rows + row * ld + 4 * l, v);
        else store_split4((__nv_bfloat16*)rows + row * ld + 4 * l, plane, v);
    } else {
        const int k = 2 * l, h = D >> 1, n = ld >> 2;
        uint16_t* p = (uint16_t*)rows + row * ld;
        if constexpr (HALF) {
            const __half2 re = __floats2half2_rn(v.x, v.y), im = __floats2half2_rn(v.z, v.w);
            if constexpr (V == 2) {
                if (k < h) *reinterpret_cast<__half2*>(p + k) = re, *reinterpret_cast<__half2*>(p + h + k) = im;
            } else {  // an odd h leaves the imaginary parts on odd columns
                if (l < h) p[l] = __half_as_ushort(re.x), p[h + l] = __half_as_ushort(im.x);
                if (l + n < h) p[l + n] = __half_as_ushort(re.y), p[h + l + n] = __half_as_ushort(im.y);
            }
            for (int c = D + k; c < ld; c += ld >> 1) *reinterpret_cast<uint32_t*>(p + c) = 0u;  // the padding of the row
        } else {
#pragma unroll
            for (int t = 0; t < 3; t++, p += plane) {
                const __nv_bfloat162 re = __floats2bfloat162_rn(v.x, v.y), im = __floats2bfloat162_rn(v.z, v.w);
                if constexpr (V == 2) {
                    if (k < h) *reinterpret_cast<__nv_bfloat162*>(p + k) = re, *reinterpret_cast<__nv_bfloat162*>(p + h + k) = im;
                } else {
                    if (l < h) p[l] = __bfloat16_as_ushort(re.x), p[h + l] = __bfloat16_as_ushort(im.x);
                    if (l + n < h) p[l + n] = __bfloat16_as_ushort(re.y), p[h + l + n] = __bfloat16_as_ushort(im.y);
                }
                for (int c = D + k; c < ld; c += ld >> 1) *reinterpret_cast<uint32_t*>(p + c) = 0u;
                const float2 fr = __bfloat1622float2(re), fi = __bfloat1622float2(im);
                v.x -= fr.x, v.y -= fr.y, v.z -= fi.x, v.w -= fi.y;
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------
// prep: the operands of the scores kernels.  A group of ld / 4 lanes takes one edge (both corruption sides: four rows in, two
// operand rows and two positive scores out) or two columns of negatives (one row in and both sides' rows out where the sides share the
// node) at a time.
// Bound by the chain id -> row index -> row on small batches (and by fetching the kernel's own code: 80 KB of it, with more rows a
// group unrolled, ran no faster than one row at a time), by L2 and HBM on large ones.  10 000 edges, 2 x 10 000 negatives, ComplEx 100:
// 10.8 us; 100 000 edges, 2 x 200 000 negatives, DistMult 128: 85 us (eight lanes a row and side: 12.8 and 168 us).
// ---------------------------------------------------------------------------------------------------
constexpr int kPrepNegs = 2;

template <int V, bool CPLX, bool REL, bool HALF>
__global__ void __launch_bounds__(256, 5) lp_prep_kernel(const __grid_constant__ LpKernelArgs a, int write_mask) {
    const ge2_lp_desc& d = a.d;
    const LpLayout& L = a.L;
    const int ld = L.ld, D = d.D, lpr = ld >> 2;
    const int lane = threadIdx.x & 31, l = lane & (lpr - 1);
    const unsigned gmask = lpr == 32 ? 0xFFFFFFFFu : 0xFFFFu << (lane & 16);
    const int groups = (int)(gridDim.x * blockDim.x) / lpr;
    const int64_t neg_units = (L.CN + kPrepNegs - 1) / kPrepNegs;
    const int64_t q_plane = (int64_t)L.S * L.Bp * ld, k_plane = (int64_t)L.S * L.CN * ld;
    void* const Q = HALF ? (void*)L.Qh : (void*)L.Qs;
    void* const K = HALF ? (void*)L.Kh : (void*)L.Ks;
    const bool two = REL && L.S == 2;
    griddep_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0) *L.loss_acc = 0.0;  // the scores kernel of this step adds every row's loss term to it
#pragma unroll 1
    for (int64_t u = (int)(blockIdx.x * blockDim.x + threadIdx.x) / lpr; u < L.Bp + neg_units; u += groups) {
        if (u < L.Bp) {
            const int64_t i = u;
            bool ok = i < d.B;  // rows past B: zero rows appended by pad_and_reshape; their positive score is padded with 0
            int64_t sid = 0, did = 0, rid = 0;
            if (ok) {
                sid = __ldg(&d.src_ids[i * d.edge_stride]);
                did = __ldg(&d.dst_ids[i * d.edge_stride]);
                if (REL) rid = __ldg(&d.rel_ids[i * d.rel_stride]);
                ok = sid >= 0 && sid < d.U && did >= 0 && did < d.U && (!REL || (rid >= 0 && rid < d.R));
                if (!ok && l == 0) or_status(d.status, GE2_STATUS_BAD_INDEX);
            }
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f), t = s, r0 = s, r1 = s;
            if (ok) {
                const float *es = emb_row(d, sid), *ed = emb_row(d, did);
                if (REL) r0 = load_row<V, CPLX>(d.rel + rid * D, l, D);
                if (two) r1 = load_row<V, CPLX>(d.inv_rel + rid * D, l, D);
                s = load_row<V, CPLX>(es, l, D);
                t = load_row<V, CPLX>(ed, l, D);
            }
            const float4 q0 = REL ? rel_mul<CPLX>(s, r0) : s;
            store_operand<V, CPLX, HALF>(Q, q_plane, i, ld, l, D, q0);
            float p0 = dot4(q0, t), p1 = 0.f;
            if (two) {
                const float4 q1 = rel_mul<CPLX>(t, r1);
                store_operand<V, CPLX, HALF>(Q, q_plane, L.Bp + i, ld, l, D, q1);
                p1 = dot4(q1, s);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                if (o < lpr) {
                    p0 += __shfl_xor_sync(gmask, p0, o);
                    if (REL) p1 += __shfl_xor_sync(gmask, p1, o);
                }
            }
            if (l == 0) {
                L.pos[i] = p0;
                if (two) L.pos[L.Bp + i] = p1;
            }
        } else {
            const int64_t j0 = (u - L.Bp) * kPrepNegs;
            const float* src[2][kPrepNegs];
#pragma unroll
            for (int e = 0; e < kPrepNegs; e++) {
                const int64_t j = j0 + e < L.CN ? j0 + e : L.CN - 1;
                const int64_t i0 = __ldg(&d.dst_negs[j]), i1 = two ? __ldg(&d.src_negs[j]) : i0;
                const bool bad0 = i0 < 0 || i0 >= d.U, bad1 = i1 < 0 || i1 >= d.U;
                if ((bad0 || bad1) && l == 0) or_status(d.status, GE2_STATUS_BAD_INDEX);
                src[0][e] = bad0 ? nullptr : emb_row(d, i0);
                src[1][e] = bad1 ? nullptr : i1 == i0 ? src[0][e] : emb_row(d, i1);
            }
            if (write_mask && l < kPrepNegs && j0 + l < L.CN) {
                // the filter word of this (side, chunk, column): deg_negative_local_filter on the device (negative.cpp:215-263 of
                // the reference): entry (c, col) masks row deg_rows[c][col] when that row belongs to chunk c; the same for both
                // sides (the reference shares one filter tensor, negative.cpp:1049-1056)
                const int64_t j = j0 + l;
                int32_t m = -1;
                if (d.deg_sample_rows != nullptr) {
                    const int c = (int)((uint32_t)j / (uint32_t)d.N), col = (int)j - c * d.N;  // (C N fits 31 bits)
                    if (col < d.n_deg) {
                        const int64_t r = d.deg_sample_rows[(int64_t)c * d.n_deg + col];
                        if (r < 0 || r >= d.B) or_status(d.status, GE2_STATUS_BAD_INDEX);
                        else if ((int)((uint32_t)r / (uint32_t)L.npc) == c) m = (int32_t)r;
                    }
                }
                L.mask[j] = m;
                if (two) L.mask[L.CN + j] = m;
            }
            float4 v[2][kPrepNegs];
#pragma unroll
            for (int e = 0; e < kPrepNegs; e++) {
                v[0][e] = v[1][e] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (src[0][e] != nullptr) v[0][e] = load_row<V, CPLX>(src[0][e], l, D);
                if (REL && src[1][e] != src[0][e] && src[1][e] != nullptr) v[1][e] = load_row<V, CPLX>(src[1][e], l, D);
            }
#pragma unroll
            for (int e = 0; e < kPrepNegs; e++) {
                if (j0 + e >= L.CN) break;
                store_operand<V, CPLX, HALF>(K, k_plane, j0 + e, ld, l, D, v[0][e]);
                if (two) store_operand<V, CPLX, HALF>(K, k_plane, L.CN + j0 + e, ld, l, D, src[1][e] == src[0][e] ? v[0][e] : v[1][e]);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------
// finish: relation-operator backward and the scatter of every gradient row.
// The first CTAs take the negatives, `occ` rows of dK a warp; the others batches of kFinBatch edges, both corruption sides at once,
// with the scalars of the next batch on their way while the rows of one are worked on.  Rows that occur again among a batch's
// edges (relations always do; hub nodes of a skewed graph) or the warp's negatives are added up on chip first -- thousands of
// reductions onto the same 128 bytes would serialise in L2 -- and the rest go to the gradient tables as 16-byte reductions at L2.
// Where the caller hands over the optimizer state and says which nodes occur once in the batch (row_shared), such a node is
// finished on the spot: the whole gradient of its row is in registers here, and so is the row, so its Adagrad step costs one read
// of the state and two writes instead of a reduction, and later a read, a clearing and a second visit to the table.
// Sums are the same as the reference's index_add backward up to fp32 addition order.
// Bound by latency on small batches (ids -> rows -> reductions), by HBM on large ones.  With the sparse Adagrad pass that follows:
// 10 000 edges, 2 x 10 000 negatives, ComplEx 100: 28 us (33 us with every row through the gradient table); 50 000 edges and
// negatives, Dot 100: 104 us (143 us); 100 000 edges, 2 x 200 000 negatives, DistMult 128: 270 us (465 us).
// A node in half of the edges and of the degree negatives: the first of these 28 us (31 us with its rows summed in shared memory for a CTA's
// lifetime), the last with half of the negatives by degree 275 us (461 us).  Scalar reductions feel it most: 7919 edges, 2 x 4571 negatives,
// ComplEx 50 (25 columns a half): 20 us, 25 us with neighbouring lanes two columns apart (17 us and 17 us without such a node).
// ---------------------------------------------------------------------------------------------------
constexpr int kFinWarps = 8;
constexpr int kNoRow = 2;      // in the place of a node's "occurs again": its row is not one of the table, so nothing is done with it
constexpr int kFinBatch = 16;  // edges a batch: their 32 endpoints are the lanes of one warp when it looks for repeated nodes

struct FinScalars {
    long long id[2 * kFinBatch];   // local node ids, sources then destinations; -1: skip the edge (bad ids, flagged by prep)
    long long row[2 * kFinBatch];  // their rows of the table
    unsigned same[2 * kFinBatch];  // lanes with the same node
    int rid[kFinBatch];
    unsigned rel_same[kFinBatch];  // edges with the same relation
    float dpos[2][kFinBatch];
    unsigned char shared[2 * kFinBatch];  // the node occurs elsewhere in the batch
};

// one row's Adagrad step
template <int V, bool CPLX>
__device__ __forceinline__ void adagrad_row(float* emb, float* state, int l, int D, float4 e, float4 s, float4 g, float neg_lr) {
    // a lane without columns must not divide: 0 / 1e-10 is off the short path, and the whole warp would wait for it
    const int n = lp_row_ld(D) >> 2;
    // values of this lane that exist (at least); ComplEx: pairs of them
    const int cols = CPLX ? (V == 1 ? ((D >> 1) - l + n - 1) / n : (D >> 1) - 2 * l) : V == 1 ? (D - l + n - 1) / n : D - 4 * l;
    if (cols <= 0) return;
    if (CPLX ? cols == 1 : cols < 4) {
        if (CPLX) s.y = s.w = 1.f;
        else s.w = 1.f, s.z = cols < 3 ? 1.f : s.z, s.y = cols < 2 ? 1.f : s.y;
    }
    const float gr[4] = {g.x, g.y, g.z, g.w};
    float st[4] = {s.x, s.y, s.z, s.w}, dl[4], up[4];
    adagrad_elems<4>(gr, st, dl, up, neg_lr);
    e.x = __fadd_rn(e.x, dl[0]), e.y = __fadd_rn(e.y, dl[1]), e.z = __fadd_rn(e.z, dl[2]), e.w = __fadd_rn(e.w, dl[3]);
    put_row<V, CPLX, PutStore>(state, l, D, make_float4(st[0], st[1], st[2], st[3]));
    put_row<V, CPLX, PutStore>(emb, l, D, e);
}

template <int V, bool CPLX, bool REL>
__global__ void __launch_bounds__(kFinWarps * 32, 4) lp_finish_kernel(const __grid_constant__ LpKernelArgs a, int neg_ctas, int occ) {
    extern __shared__ __align__(16) float fin_rows[];  // [4][kFinBatch][ld]: relation, inverse relation, source, destination gradients
    __shared__ FinScalars sm;
    const ge2_lp_desc& d = a.d;
    const LpLayout& L = a.L;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int D = d.D, ld = L.ld, lpr = ld >> 2, l = lane & (lpr - 1);
    const int per_warp = 32 / lpr;            // rows a warp works on side by side
    const int sub = per_warp == 1 ? 0 : lane >> 4;
    const float gs = L.grad_unscale;  // the tensor path leaves dQ / dK scaled by a power of two
    const bool fused = d.node_state != nullptr && d.row_shared != nullptr;
    const float neg_lr = -d.node_lr;
    float* const table = const_cast<float*>(d.node_emb);
    griddep_wait();
    // loss = sum over sides and padded rows of (lse - pos), accumulated in double by the scores kernel that ran before
    if (blockIdx.x == 0 && tid == 0) *d.loss = (float)*L.loss_acc;

    if ((int)blockIdx.x < neg_ctas) {  // ---- negatives
        const int64_t w = (int64_t)blockIdx.x * kFinWarps + warp;
        const int per_side = L.S == 2 ? occ >> 1 : occ;
        const int side = lane >= per_side ? 1 : 0;
        const int64_t j = w * per_side + (lane - side * per_side);
        long long id = -1 - lane;
        int shared = 1;
        long long trow = 0;
        if (lane < occ && j < L.CN) {
            const long long v = (side == 0 ? d.dst_negs : d.src_negs)[j];
            if (v >= 0 && v < d.U) id = v;
        }
        if (id >= 0) {
            if (fused) shared = d.row_shared[id];
            trow = d.row_index != nullptr ? __ldg(&d.row_index[id]) : id;
        }
        const unsigned same = __match_any_sync(0xFFFFFFFFu, id);
        const long long dk_row = (long long)side * L.CN + j;
        const bool leads = id >= 0 && (same & ((1u << lane) - 1u)) == 0;
        const unsigned leaders = __ballot_sync(0xFFFFFFFFu, leads);
        if ((uint64_t)trow >= (uint64_t)d.table_rows) {  // (here: the row may arrive while the ids are matched)
            shared = kNoRow;
            or_status(d.status, GE2_STATUS_BAD_INDEX);
        }
#pragma unroll 1
        for (int k0 = 0; k0 < occ; k0 += per_warp) {
            if (((leaders >> k0) & ((1u << per_warp) - 1u)) == 0u) continue;
            const int k = k0 + sub;
            const unsigned members = __shfl_sync(0xFFFFFFFFu, same, k);
            const long long gid = __shfl_sync(0xFFFFFFFFu, id, k), grow = __shfl_sync(0xFFFFFFFFu, trow, k);
            const int sh = __shfl_sync(0xFFFFFFFFu, shared, k);
            const bool on = ((leaders >> k) & 1u) && sh != kNoRow;
            const bool upd = on && sh == 0;
            const long long r1 = __shfl_sync(0xFFFFFFFFu, dk_row, k);
            unsigned rest = members & (members - 1);
            const long long r2 = __shfl_sync(0xFFFFFFFFu, dk_row, rest ? __ffs((int)rest) - 1 : k);
            float4 g = make_float4(0.f, 0.f, 0.f, 0.f), g2 = g, e = g, s = g;
            if (on) g = load_row<V, CPLX>(L.dK + r1 * ld, l, D);
            if (on && rest) g2 = load_row<V, CPLX>(L.dK + r2 * ld, l, D);  // the other side's row, mostly
            if (upd) {
                e = load_row<V, CPLX>(table + grow * d.emb_stride, l, D);
                s = load_row<V, CPLX>(d.node_state + grow * d.emb_stride, l, D);
            }
            g = add4(g, g2);
            rest = on ? rest & (rest - 1) : 0u;
            while (__any_sync(0xFFFFFFFFu, rest != 0u)) {
                const long long r = __shfl_sync(0xFFFFFFFFu, dk_row, rest ? __ffs((int)rest) - 1 : 0);
                if (rest) g = add4(g, load_row<V, CPLX>(L.dK + r * ld, l, D));
                rest &= rest - 1;
            }
            g = scale4(gs, g);
            if (upd) adagrad_row<V, CPLX>(table + grow * d.emb_stride, d.node_state + grow * d.emb_stride, l, D, e, s, g, neg_lr);
            else if (on) put_row<V, CPLX, PutAdd>(d.node_grad + gid * D, l, D, g);
        }
        return;
    }

    // ---- edges
    // the scalars of one batch, a lane an endpoint (warp 0: sources, then destinations), an edge's relation (warp 1) or its d loss / d
    // pos on one side (warp 2)
    long long p_id = -1, p_row = -1;
    int p_rid = -1;
    float p_dpos = 0.f;
    int p_shared = 1;
    const int k16 = lane & (kFinBatch - 1);
    auto fetch = [&](int64_t base) {
        const int64_t i = base + k16;
        if (warp == 0) {  // lanes are endpoints: sources, then destinations
            p_id = p_row = -1;
            p_shared = 1;
            if (i < d.B) p_id = (lane < kFinBatch ? d.src_ids : d.dst_ids)[i * d.edge_stride];
            if (p_id >= d.U || p_id < 0) p_id = -1;
            if (p_id >= 0) {
                p_row = d.row_index != nullptr ? __ldg(&d.row_index[p_id]) : p_id;
                if (fused) p_shared = d.row_shared[p_id];
            }
        } else if (warp == 1 && REL) {
            p_rid = -1;
            if (i < d.B) {
                const int64_t r = d.rel_ids[i * d.rel_stride];
                if (r >= 0 && r < d.R) p_rid = (int)r;
            }
        } else if (warp == 2) {
            const int side = lane / kFinBatch;
            if (side < L.S && i < d.B) {
                const int64_t qrow = (int64_t)side * L.Bp + i;
                p_dpos = __expf(L.pos[qrow] - L.lse[qrow]) - 1.0f;  // d loss / d pos_i = softmax prob of the positive - 1
            }
        }
    };
    auto usable = [&](int k) { return sm.id[k] >= 0 && sm.id[kFinBatch + k] >= 0 && (!REL || sm.rid[k] >= 0); };
    const int group = warp * per_warp + sub, groups = kFinWarps * per_warp;
    const int plane = kFinBatch * ld;
    const bool two = REL && L.S == 2;
    const int64_t step = (int64_t)(gridDim.x - neg_ctas) * kFinBatch;
    int64_t base = (int64_t)((int)blockIdx.x - neg_ctas) * kFinBatch;
    fetch(base);
#pragma unroll 1
    for (; base < d.B; base += step) {
        if (warp == 0) {
            if (p_id >= 0 && (uint64_t)p_row >= (uint64_t)d.table_rows) {  // (here and not where it is fetched: the load is not waited for until now)
                p_id = -1;
                or_status(d.status, GE2_STATUS_BAD_INDEX);
            }
            sm.id[lane] = p_id, sm.row[lane] = p_row, sm.shared[lane] = (unsigned char)p_shared;
        }
        else if (warp == 1 && REL && lane < kFinBatch) sm.rid[lane] = p_rid;
        else if (warp == 2) sm.dpos[lane / kFinBatch][k16] = p_dpos;
        __syncthreads();
        if (warp == 0) {
            sm.same[lane] = __match_any_sync(0xFFFFFFFFu, usable(k16) ? p_id : -1ll - lane);
        } else if (warp == 1 && REL) {
            const unsigned m = __match_any_sync(0xFFFFFFFFu, usable(k16) ? p_rid : -1 - lane);
            if (lane < kFinBatch) sm.rel_same[lane] = m & ((1u << kFinBatch) - 1u);
        }
        fetch(base + step);
        __syncthreads();
#pragma unroll 1
        for (int k = group; k < kFinBatch; k += groups) {
            if (!usable(k)) continue;
            const int64_t i = base + k;
            const int64_t srow = sm.row[k] * d.emb_stride, drow = sm.row[kFinBatch + k] * d.emb_stride;
            // one edge, both corruption sides at once: side 0 applies the relation to the source and compares with the
            // destination, side 1 the inverse relation to the destination and compares with the source, so each endpoint
            // receives one combined row instead of two
            const float4 es = load_row<V, CPLX>(table + srow, l, D), ed = load_row<V, CPLX>(table + drow, l, D);
            float4 g0 = load_row<V, CPLX>(L.dQ + i * ld, l, D), g1 = g0, r0 = g0, r1 = g0, ss = g0, sd = g0;
            const int rid = REL ? sm.rid[k] : 0;
            if (REL) r0 = load_row<V, CPLX>(d.rel + (int64_t)rid * D, l, D);
            if (two) {
                g1 = load_row<V, CPLX>(L.dQ + (L.Bp + i) * ld, l, D);
                r1 = load_row<V, CPLX>(d.inv_rel + (int64_t)rid * D, l, D);
            }
            if (!sm.shared[k]) ss = load_row<V, CPLX>(d.node_state + srow, l, D);
            if (!sm.shared[kFinBatch + k]) sd = load_row<V, CPLX>(d.node_state + drow, l, D);
            // gradient with respect to the relation-adjusted embedding q = op(a, r): from the negatives (dQ) and the positive
            const float p0 = sm.dpos[0][k];
            g0 = axpy4(p0, ed, scale4(gs, g0));
            float4 gsrc = g0, gdst = scale4(p0, es);
            float* const buf = fin_rows + k * ld + 4 * l;
            if (REL) {
                gsrc = rel_mul_t<CPLX>(g0, r0);
                gdst = scale4(p0, rel_mul<CPLX>(es, r0));
                float4 vr0 = rel_mul_t<CPLX>(g0, es), vr1 = vr0;
                if (two) {
                    const float p1 = sm.dpos[1][k];
                    g1 = axpy4(p1, es, scale4(gs, g1));
                    gdst = add4(gdst, rel_mul_t<CPLX>(g1, r1));
                    gsrc = add4(gsrc, scale4(p1, rel_mul<CPLX>(ed, r1)));
                    vr1 = rel_mul_t<CPLX>(g1, ed);
                }
                if ((sm.rel_same[k] & (sm.rel_same[k] - 1u)) == 0u) {
                    put_row<V, CPLX, PutAdd>(d.rel_grad + (int64_t)rid * D, l, D, vr0);
                    if (two) put_row<V, CPLX, PutAdd>(d.inv_rel_grad + (int64_t)rid * D, l, D, vr1);
                } else {
                    *reinterpret_cast<float4*>(buf) = vr0;
                    *reinterpret_cast<float4*>(buf + plane) = vr1;
                }
            }
            float4 g = gsrc, e = es, st = ss;
            int64_t at = srow;
#pragma unroll 1
            for (int side = 0; side < 2; side++) {  // the two endpoints
                const int kk = side * kFinBatch + k;
                if (!sm.shared[kk]) adagrad_row<V, CPLX>(table + at, d.node_state + at, l, D, e, st, g, neg_lr);
                else if ((sm.same[kk] & (sm.same[kk] - 1u)) == 0u) put_row<V, CPLX, PutAdd>(d.node_grad + sm.id[kk] * D, l, D, g);
                else *reinterpret_cast<float4*>(buf + (2 + side) * plane) = g;
                g = gdst, e = ed, st = sd, at = drow;
            }
        }
        __syncthreads();
        // the repeated rows: their first occurrence adds them up and sends the sum
        const int rel_tasks = REL ? L.S * kFinBatch : 0;
#pragma unroll 1
        for (int t = group; t < rel_tasks + 2 * kFinBatch; t += groups) {
            const bool is_rel = t < rel_tasks;
            const int k = is_rel ? t & (kFinBatch - 1) : t - rel_tasks, side = is_rel ? t / kFinBatch : 2;
            unsigned m = is_rel ? sm.rel_same[k] : sm.same[k];
            if ((m & (m - 1u)) == 0u || __ffs((int)m) - 1 != k || (!is_rel && !sm.shared[k])) continue;
            const float* rows = fin_rows + side * plane + 4 * l;  // (the destinations follow the sources)
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            while (m != 0u) {
                v = add4(v, *reinterpret_cast<const float4*>(rows + (__ffs((int)m) - 1) * ld));
                m &= m - 1u;
            }
            float* grow = is_rel ? (side == 0 ? d.rel_grad : d.inv_rel_grad) + (int64_t)sm.rid[k] * D : d.node_grad + sm.id[k] * D;
            put_row<V, CPLX, PutAdd>(grow, l, D, v);
        }
        __syncthreads();  // the scalars are overwritten by the next batch
    }
}

// the widest access all rows of a step allow: 16 bytes when rows are multiples of it and every table starts on one (8 for ComplEx, whose
// halves need not), else 8, else 4
int row_access(const ge2_lp_desc& d) {
    const bool cplx = d.has_relations && d.decoder == GE2_DECODER_COMPLEX;
    const uintptr_t bits = (uintptr_t)d.node_emb | (uintptr_t)d.node_grad | (uintptr_t)d.rel | (uintptr_t)d.inv_rel | (uintptr_t)d.rel_grad |
                           (uintptr_t)d.inv_rel_grad | (uintptr_t)d.node_state | (uintptr_t)(d.emb_stride * 4);
    if (cplx) return d.D % 4 == 0 && (bits & 7) == 0 ? 2 : 1;
    if (d.D % 4 == 0 && (bits & 15) == 0) return 4;
    return d.D % 2 == 0 && (bits & 7) == 0 ? 2 : 1;
}

using PrepKernel = void (*)(LpKernelArgs, int);
using FinishKernel = void (*)(LpKernelArgs, int, int);
template <bool HALF>
PrepKernel prep_kernel_of(const ge2_lp_desc& d) {
    const int V = row_access(d);
    if (d.has_relations && d.decoder == GE2_DECODER_COMPLEX) return V == 2 ? lp_prep_kernel<2, true, true, HALF> : lp_prep_kernel<1, true, true, HALF>;
    if (d.has_relations) return V == 4 ? lp_prep_kernel<4, false, true, HALF> : V == 2 ? lp_prep_kernel<2, false, true, HALF> : lp_prep_kernel<1, false, true, HALF>;
    return V == 4 ? lp_prep_kernel<4, false, false, HALF> : V == 2 ? lp_prep_kernel<2, false, false, HALF> : lp_prep_kernel<1, false, false, HALF>;
}
FinishKernel finish_kernel_of(const ge2_lp_desc& d) {
    const int V = row_access(d);
    if (d.has_relations && d.decoder == GE2_DECODER_COMPLEX) return V == 2 ? lp_finish_kernel<2, true, true> : lp_finish_kernel<1, true, true>;
    if (d.has_relations) return V == 4 ? lp_finish_kernel<4, false, true> : V == 2 ? lp_finish_kernel<2, false, true> : lp_finish_kernel<1, false, true>;
    return V == 4 ? lp_finish_kernel<4, false, false> : V == 2 ? lp_finish_kernel<2, false, false> : lp_finish_kernel<1, false, false>;
}

__global__ void __launch_bounds__(256) copy_pos_kernel(const float* __restrict__ pos, int Bp, float* __restrict__ out0, float* __restrict__ out1,
                                                       int S) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < Bp) {
        if (out0 != nullptr) out0[i] = pos[i];
        if (S == 2 && out1 != nullptr) out1[i] = pos[Bp + i];
    }
}

// the descriptor as the kernels see it: what the caller did not say it has is zero
ge2_lp_desc whole_desc(const ge2_lp_desc* d) {
    ge2_lp_desc whole = {};
    memcpy(&whole, d, (d->flags & GE2_LP_HAS_ROW_UPDATE) ? sizeof(whole) : offsetof(ge2_lp_desc, node_state));
    if (whole.table_rows == 0) whole.table_rows = INT64_MAX;  // not told: every row is taken for one of the table
    return whole;
}

int validate(const ge2_lp_desc* d) {
    if (d == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    if (d->B <= 0 || d->C <= 0 || d->N <= 0 || d->D <= 0 || d->U <= 0) return GE2_ERR_INVALID_ARGUMENT;
    if (d->decoder != GE2_DECODER_DISTMULT && d->decoder != GE2_DECODER_COMPLEX) return GE2_ERR_INVALID_ARGUMENT;
    if (d->precision != GE2_PRECISION_FP32 && d->precision != GE2_PRECISION_F16) return GE2_ERR_INVALID_ARGUMENT;
    if (d->use_inverse && !d->has_relations) return GE2_ERR_INVALID_ARGUMENT;
    if (d->D > 128) return GE2_ERR_UNSUPPORTED;
    // the reference's complex operator splits the row in D/2 and D - D/2 columns and multiplies them element-wise: D must be even
    if (d->decoder == GE2_DECODER_COMPLEX && d->has_relations && (d->D & 1)) return GE2_ERR_INVALID_ARGUMENT;
    if (d->node_emb == nullptr || d->src_ids == nullptr || d->dst_ids == nullptr || d->dst_negs == nullptr || d->node_grad == nullptr ||
        d->loss == nullptr || d->edge_stride <= 0 || d->emb_stride < d->D)
        return GE2_ERR_INVALID_ARGUMENT;
    if (d->has_relations && (d->rel_stride <= 0 || d->rel_ids == nullptr || d->rel == nullptr || d->rel_grad == nullptr || d->R <= 0)) return GE2_ERR_INVALID_ARGUMENT;
    if (d->use_inverse && (d->src_negs == nullptr || d->inv_rel == nullptr || d->inv_rel_grad == nullptr)) return GE2_ERR_INVALID_ARGUMENT;
    if (d->dst_filter_n < 0 || d->src_filter_n < 0 || (d->dst_filter_n > 0 && d->dst_filter == nullptr) ||
        (d->src_filter_n > 0 && d->src_filter == nullptr))
        return GE2_ERR_INVALID_ARGUMENT;
    if (d->deg_sample_rows != nullptr && (d->n_deg <= 0 || d->n_deg > d->N)) return GE2_ERR_INVALID_ARGUMENT;
    if (d->flags & GE2_LP_HAS_ROW_UPDATE) {
        if ((d->node_state == nullptr) != (d->row_shared == nullptr) || d->table_rows < 0) return GE2_ERR_INVALID_ARGUMENT;
        if (d->node_state != nullptr && d->table_rows == 0) return GE2_ERR_INVALID_ARGUMENT;  // rows are written only where they are known to exist
    }
    if (d->deg_sample_rows != nullptr && (d->dst_filter_n > 0 || d->src_filter_n > 0)) return GE2_ERR_INVALID_ARGUMENT;
    return GE2_OK;
}

}  // namespace
}  // namespace ge2

using namespace ge2;

extern "C" int ge2_lp_workspace_bytes(const ge2_lp_desc* desc, size_t* bytes) {
    if (bytes == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    int rc = validate(desc);
    if (rc != GE2_OK) return rc;
    *bytes = lp_make_layout(*desc, nullptr).bytes;
    return GE2_OK;
}

extern "C" int ge2_lp_idle_sms(const ge2_lp_desc* desc, int32_t* sms) {
    if (sms == nullptr) return GE2_ERR_INVALID_ARGUMENT;
    const int rc = validate(desc);
    if (rc != GE2_OK) return rc;
    *sms = kNumSMs - scores_ctas(scores_units(*desc, desc->has_relations && desc->use_inverse ? 2 : 1));
    return GE2_OK;
}

extern "C" int ge2_lp_step(const ge2_lp_desc* desc, ge2_stream_t stream_) {
    int rc = validate(desc);
    if (rc != GE2_OK) return rc;
    LpKernelArgs a;
    a.d = whole_desc(desc);
    if (desc->workspace == nullptr || ((uintptr_t)desc->workspace & 255) != 0) return GE2_ERR_WORKSPACE;
    a.L = lp_make_layout(*desc, desc->workspace);
    // no room for the streaming form's parts (a workspace for a larger batch that takes the other form, or of an earlier version's size)
    if (desc->workspace_bytes < a.L.bytes) a.L = lp_make_layout(*desc, desc->workspace, false);
    if (desc->workspace_bytes < a.L.bytes) return GE2_ERR_WORKSPACE;
    const LpLayout& L = a.L;
    cudaStream_t stream = as_stream(stream_);

    const int phases = desc->phases == 0 ? 7 : desc->phases;
    if ((phases & 4) && !(desc->flags & GE2_LP_NODE_GRAD_IS_ZERO))
        GE2_CUDA_TRY(cudaMemsetAsync(desc->node_grad, 0, (size_t)desc->U * desc->D * 4, stream));
    if (phases & 1) {
    // without explicit filter pairs the prepare kernel writes every filter word itself
    const bool pairs = desc->dst_filter_n > 0 || desc->src_filter_n > 0;
    if (pairs) {
        GE2_CUDA_TRY(cudaMemsetAsync(L.mask, 0xFF, (size_t)L.S * L.CN * 4, stream));
        if (desc->dst_filter_n > 0) {
            mask_from_pairs_kernel<<<stream_grid(desc->dst_filter_n, 256), 256, 0, stream>>>(desc->dst_filter, desc->dst_filter_n, L.npc, L.Bp,
                                                                                           desc->N, L.mask, desc->status);
            GE2_LAUNCH_CHECK();
        }
        if (L.S == 2 && desc->src_filter_n > 0) {
            mask_from_pairs_kernel<<<stream_grid(desc->src_filter_n, 256), 256, 0, stream>>>(desc->src_filter, desc->src_filter_n, L.npc, L.Bp,
                                                                                           desc->N, L.mask + L.CN, desc->status);
            GE2_LAUNCH_CHECK();
        }
    }

    const int64_t units = L.Bp + ceil_div<int64_t>(L.CN, kPrepNegs);
    const PrepKernel prep = desc->precision == GE2_PRECISION_F16 ? prep_kernel_of<true>(a.d) : prep_kernel_of<false>(a.d);
    GE2_CUDA_TRY(launch_after(prep, dim3((unsigned)stream_grid(units, 1024 / L.ld, 5)), dim3(256), 0, stream, a, pairs ? 0 : 1));
    }

    if (phases & 2) {
        rc = desc->precision == GE2_PRECISION_FP32 ? lp_scores_fp32(a, stream) : L.o_part != nullptr ? lp_flash_f16(a, stream) : lp_scores_f16(a, stream);
        if (rc != GE2_OK) return rc;
    }
    if (!(phases & 4)) return GE2_OK;

    // negatives a warp: as few as fill the GPU once, since a warp goes through them one by one (3000 of them in groups of 16: 28 us, a
    // step of 55 us instead of 40), but at least four and up to the 32 that one lane each can hold: more of them together
    // merge more repeated nodes (9000 drawn half by degree: 15.4 us in groups of 2, 12.5 in groups of 8)
    const int64_t neg_rows = (int64_t)L.S * L.CN;
    int occ = 4;
    while (occ < 32 && neg_rows / occ > (int64_t)kNumSMs * 4 * kFinWarps) occ *= 2;
    // As many as are resident together.  More (one batch each) take 5 % off this kernel alone and put 4 % on the pipelined step, whose
    // sampler and unique-map for the next batch run beside it.
    const int edge_ctas = std::min(ceil_div(desc->B, kFinBatch), kNumSMs * 4);
    const int64_t neg_ctas = ceil_div<int64_t>(ceil_div<int64_t>(L.CN, occ / L.S), kFinWarps);
    const size_t fin_smem = (size_t)4 * kFinBatch * L.ld * 4;
    GE2_CUDA_TRY(launch_after(finish_kernel_of(a.d), dim3((unsigned)(edge_ctas + neg_ctas)), dim3(kFinWarps * 32), fin_smem, stream, a, (int)neg_ctas, occ));
    if (desc->pos_scores != nullptr || desc->inv_pos_scores != nullptr) {
        copy_pos_kernel<<<ceil_div(L.Bp, 256), 256, 0, stream>>>(L.pos, L.Bp, desc->pos_scores, desc->inv_pos_scores, L.S);
        GE2_LAUNCH_CHECK();
    }
    return GE2_OK;
}
