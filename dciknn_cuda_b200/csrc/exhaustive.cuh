// Queries whose stop rule provably never fires: every point of every partition is a candidate, so the answer is
// the exact k nearest rows by (distance, id) and nothing of the index is needed.  Two ways to it, with the
// distance chain of the traversal (ascending fma, IEEE square root), hence the same bits:
//   exact_scan_kernel     every row, one query a CTA; for small problems and few queries
//   nearest_groups_kernel for large ones: distance_bounds_kernel gives a lower bound for every (query, group of
//                         rows); one CTA per query works out the groups with the smallest bounds, which gives a
//                         k-th distance, and then only the groups whose bound does not exceed it.
#pragma once
#include "common.cuh"
#include "distance_bounds.cuh"
#include "traverse.cuh"

namespace dci {

struct ExactParams {
    const float *data, *query;      // query: first query of this launch
    int n, dim, nq, knn, topk_cap;  // topk_cap: power of two >= knn + blockDim.x
    int vec4, vec8;
    int slice_rows, slices;         // exact_scan_kernel: rows per CTA, CTAs per query
    uint64_t *lists;                // slices > 1: [nq][slices][knn]
    int *out_ids;                   // slices == 1: the result itself, [nq][knn] ...
    float *out_dists;
    uint64_t *out_packed;           // ... or packed keys instead, when not null
    const uint32_t *lb;             // nearest_groups_kernel: [num_groups][nq] bounds, rows per group
    const int *failed;
    int num_groups, group_rows, first;
};

__device__ __forceinline__ void write_result(const ExactParams &p, int q, const uint64_t *res) {
    for (int j = threadIdx.x; j < p.knn; j += blockDim.x) {
        const uint64_t key = res[j];
        const size_t o = (size_t)q * p.knn + j;
        if (p.out_packed) { p.out_packed[o] = key; continue; }
        p.out_ids[o] = key == kEmptySlot ? -1 : (int)(uint32_t)key;
        p.out_dists[o] = key == kEmptySlot ? __int_as_float(0x7F800000) : __uint_as_float((uint32_t)(key >> 32));
    }
}

// Distances of the rows row_of(0 .. count) to the query in shared memory, offered to topk; rows beyond the k-th
// distance known so far are abandoned.  All threads call; row_of may return a row >= p.n (none).
template <typename RowOf>
__device__ __forceinline__ void offer_rows(const ExactParams &p, const float *qv, CtaTopK &topk, int count, RowOf row_of) {
    for (int base = 0; base < count; base += blockDim.x) {
        const int j = base + threadIdx.x;
        float bd = __int_as_float(0x7F800000), bsq = bd;
        const uint64_t th = *topk.thresh;       // set at compactions only, the same for all threads here
        if (th != kEmptySlot && (uint32_t)(th >> 32) < 0x7F7F7F7Fu) {
            bd = __uint_as_float((uint32_t)(th >> 32));
            const float up = __uint_as_float((uint32_t)(th >> 32) + 1u);
            bsq = __fmul_ru(up, up);            // sq > bsq  =>  sqrt(sq) > bd
        }
        uint64_t key = kEmptySlot;
        if (j < count) {
            const long long r = row_of(j);
            if (r < p.n) {
                const float *row = p.data + (size_t)r * p.dim;
                const float d = p.vec8 ? dist_sequential_v8(row, qv, p.dim, bsq) : dist_sequential(row, qv, p.dim, p.vec4);
                if (d >= 0.0f && d <= bd) key = ((uint64_t)__float_as_uint(d) << 32) | (uint32_t)r;      // a NaN is no candidate
            }
        }
        topk.offer(key);
    }
}

constexpr int kScanThreads = 512;

// grid (queries, slices).  Dynamic shared memory: selection buffers | query.  Tiles of four and eight queries per CTA,
// which read a row once for all of them, were slower for the few queries this kernel is for: every offer of a row's
// keys is a CTA-wide step per query (2 000 x 100 rows, 500 queries: 68 us with four, 97 us with eight).
__global__ void __launch_bounds__(kScanThreads, 2)
exact_scan_kernel(const ExactParams p) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    __shared__ uint32_t s_sel[2][256];
    __shared__ uint32_t s_res[4];
    __shared__ int s_count;
    __shared__ uint64_t s_thresh;
    const int q = blockIdx.x, tid = threadIdx.x;
    float *qv = reinterpret_cast<float *>(dyn_smem + (size_t)p.topk_cap * 16);
    for (int c = tid; c < p.dim; c += blockDim.x) qv[c] = p.query[(size_t)q * p.dim + c];
    CtaTopK topk;
    topk.init(reinterpret_cast<uint64_t *>(dyn_smem), &s_count, &s_thresh, s_sel, s_res, p.topk_cap, p.knn);
    const long long r0 = (long long)blockIdx.y * p.slice_rows;
    offer_rows(p, qv, topk, (int)max(0ll, min((long long)p.n - r0, (long long)p.slice_rows)), [r0](int j) { return r0 + j; });
    topk.finish();
    if (p.slices == 1) { write_result(p, q, topk.result()); return; }
    uint64_t *out = p.lists + ((size_t)q * p.slices + blockIdx.y) * p.knn;
    for (int j = tid; j < p.knn; j += blockDim.x) out[j] = topk.result()[j];
}

constexpr int kNgThreads = 512;
constexpr int kNgList = 1024;        // groups collected before they are worked out

// One CTA per query.  Dynamic shared memory: selection buffers | query.
__global__ void __launch_bounds__(kNgThreads, 2)
nearest_groups_kernel(const ExactParams p) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    __shared__ uint32_t s_sel[2][256];
    __shared__ uint32_t s_res[4];
    __shared__ int s_count, s_listed;
    __shared__ uint64_t s_thresh;
    __shared__ int s_group[kNgList + kNgThreads];
    __shared__ double s_sum[2][kNgThreads / 32];
    const int q = blockIdx.x, tid = threadIdx.x;
    uint64_t *bufs = reinterpret_cast<uint64_t *>(dyn_smem);
    float *qv = reinterpret_cast<float *>(dyn_smem + (size_t)p.topk_cap * 16);
    double s = 0.0, t = 0.0;
    for (int c = tid; c < p.dim; c += blockDim.x) {
        const float v = p.query[(size_t)q * p.dim + c];
        const float e = bounds_residual(v);
        qv[c] = v;
        s += (double)v * v;
        t += (double)e * e;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { s += __shfl_xor_sync(0xFFFFFFFFu, s, o); t += __shfl_xor_sync(0xFFFFFFFFu, t, o); }
    if ((tid & 31) == 0) { s_sum[0][tid >> 5] = s; s_sum[1][tid >> 5] = t; }
    if (tid == 0) s_listed = 0;
    CtaTopK topk;
    topk.init(bufs, &s_count, &s_thresh, s_sel, s_res, p.topk_cap, p.knn);      // ends with a barrier
    double q2 = 0.0, dq2 = 0.0;
    for (int w = 0; w < kNgThreads / 32; ++w) { q2 += s_sum[0][w]; dq2 += s_sum[1][w]; }

    const uint32_t *lb = p.lb + q;
    const size_t stride = (size_t)p.nq;
    uint32_t first = 0xFFFFFFFFu;               // groups with bounds up to `first` come first
    if (!*p.failed) {
        uint32_t out[2];
        cta_select2([lb, stride](int j) { return lb[(size_t)j * stride]; }, p.num_groups, p.first, p.first, 32, s_sel, s_res, out);
        first = out[0];
    }
    auto work = [&]() {
        offer_rows(p, qv, topk, s_listed * p.group_rows,
                   [&](int j) { return (long long)s_group[j / p.group_rows] * p.group_rows + j % p.group_rows; });
        __syncthreads();
        if (tid == 0) s_listed = 0;
        __syncthreads();
    };
    float limit = __int_as_float(0x7F800000);
    for (int round = 0; round < 2; ++round) {
        if (round == 1) {
            if (first == 0xFFFFFFFFu) break;    // everything has been worked out
            topk.compact();                     // k-th distance of the first groups
            const uint64_t th = s_thresh;
            const float d = __uint_as_float((uint32_t)(th >> 32));
            if (th != kEmptySlot && d < __int_as_float(0x7F800000) && q2 <= 1.0e30)     // as in select_work_kernel
                limit = __double2float_ru((double)d * d * (1.0 + (p.dim + 8.0) / 8388608.0) + 1.0e-18 - bounds_query_term(q2, dq2, p.dim));
            __syncthreads();
        }
        for (int g0 = 0; g0 < p.num_groups; g0 += blockDim.x) {
            const int g = g0 + tid;
            bool take = false;
            if (g < p.num_groups) {
                const uint32_t v = lb[(size_t)g * stride];
                take = round == 0 ? v <= first : (v > first && !(ordered_to_float(v) > limit));
            }
            const int slot = warp_append_slot(take, &s_listed);
            if (take) s_group[slot] = g;
            __syncthreads();
            const bool full = s_listed >= kNgList;
            __syncthreads();
            if (full) work();
        }
        if (s_listed > 0) work();
    }
    topk.finish();
    write_result(p, q, topk.result());
}

}  // namespace dci
