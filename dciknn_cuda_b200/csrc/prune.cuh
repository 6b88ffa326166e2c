// Which (query, partition) pairs have to be traversed.
//
// Only a query's k nearest candidates over all partitions reach its result, so a partition whose nearest row
// lies strictly beyond k candidates that are already known cannot change the answer.  distance_bounds_kernel
// gives a rigorous lower bound of the nearest row of every partition; the pairs are then traversed in rounds.
// Round 1: per query the partitions with the smallest bounds, about as many as hold the k nearest rows when rows
// are spread evenly.  Every later round: of the remaining partitions those whose bound does not exceed the k-th best
// candidate so far -- all of them when fewer than k were found --, in the last round all of these, in a round before
// it only those with the next smallest bounds.  A pair that is left out keeps an empty list.  Nothing is assumed about
// the data: clustered rows only make the lists shorter, and a distribution on which the index finds few near
// neighbours (a loose k-th candidate) makes the last round traverse more.
// 1M x 128, 10 000 queries, k = 10, 100 partitions (398 ms when every pair is traversed): two rounds with 8, 10, 12 and
// 15 partitions first 145, 71, 60 and 73 ms; the rounds of a quarter each make that choice matter less.
#pragma once
#include "common.cuh"
#include "distance_bounds.cuh"

namespace dci {

struct SelectParams {
    const uint32_t *lb;           // [num_groups][q_stride], see distance_bounds.cuh
    const int *failed;            // not 0: the bounds are unusable, every pair is traversed in round 1
    const float *query;           // rows q0 .. of the call's queries
    uint64_t *part_topk;          // [nq][num_groups][kpart], empty lists where nothing was traversed
    uint32_t *thresh;             // [3][nq] largest bound of each round before the last, as found in round 1
    uint32_t *qbound;             // [nq] the shared distance bound of the traversal
    int *cnt, *offs, *list;       // [num_groups] (starts as 0), [num_groups + 1], [num_groups][q_stride]
    int *ticket;                  // starts as 0
    int nq, num_groups, q_stride, knn, kpart, dim;
    int first, step;              // partitions of round 1, and at most of each later round but the last
    int round, last;              // 1, 2, ..; last: 1 in the last round
    int per_item;                 // queries of a partition that a traversal CTA takes together: offs counts such items
};

// Starting values of everything the rounds use, in one launch: empty lists, no bound yet, bounds and counters.
__global__ void prune_init_kernel(uint4 *topk, size_t topk16, uint32_t *lb, size_t lb_words, uint32_t *qbound, int nq,
                                  int *zero, int zero_words) {
    const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
    for (size_t i = i0; i < topk16; i += step) topk[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    for (size_t i = i0; i < lb_words; i += step) lb[i] = ~0u;
    for (size_t i = i0; i < (size_t)nq; i += step) qbound[i] = 0x7F7F7F7Fu;      // no bound yet
    for (size_t i = i0; i < (size_t)zero_words; i += step) zero[i] = 0;
}

// |q|^2 and |dq|^2 (distance_bounds.cuh) of one query, by a CTA of 128 threads; every thread gets both.
__device__ __forceinline__ void query_norms(const float *__restrict__ q, int dim, double (*sums)[4], double *q2, double *dq2) {
    double s = 0.0, t = 0.0;
    for (int c = threadIdx.x; c < dim; c += blockDim.x) {
        const float v = q[c], e = bounds_residual(v);
        s += (double)v * v;
        t += (double)e * e;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { s += __shfl_xor_sync(0xFFFFFFFFu, s, o); t += __shfl_xor_sync(0xFFFFFFFFu, t, o); }
    if ((threadIdx.x & 31) == 0) { sums[0][threadIdx.x >> 5] = s; sums[1][threadIdx.x >> 5] = t; }
    __syncthreads();
    *q2 = (sums[0][0] + sums[0][1]) + (sums[0][2] + sums[0][3]);
    *dq2 = (sums[1][0] + sums[1][1]) + (sums[1][2] + sums[1][3]);
}

// The bounds themselves, for tests: out[g][q] <= |x - q|^2 for every row x of group g; -inf where none is claimed.
__global__ void __launch_bounds__(128)
bounds_value_kernel(const uint32_t *__restrict__ lb, const float *__restrict__ query, int dim, int num_groups, int nq, double *__restrict__ out) {
    __shared__ double s_sum[2][4];
    const int q = blockIdx.x;
    double q2, dq2;
    query_norms(query + (size_t)q * dim, dim, s_sum, &q2, &dq2);
    for (int g = threadIdx.x; g < num_groups; g += blockDim.x) {
        const size_t o = (size_t)g * nq + q;
        out[o] = q2 <= 1.0e30 ? (double)ordered_to_float(lb[o]) + bounds_query_term(q2, dq2, dim) : -(double)__int_as_float(0x7F800000);
    }
}

// One CTA per query.  Appends the query to the work lists of the partitions it has to visit in this round; the
// last CTA to finish turns the list lengths into offsets.
template <bool FIRST>
__global__ void __launch_bounds__(128) select_work_kernel(const SelectParams p) {
    __shared__ uint32_t s_sel[2][256];
    __shared__ uint32_t s_res[4];
    __shared__ double s_sum[2][4];
    __shared__ int s_last;
    __shared__ uint32_t s_scratch[40];
    const int q = blockIdx.x, tid = threadIdx.x;
    const uint32_t *lb = p.lb + q;
    const size_t stride = (size_t)p.q_stride;
    uint32_t lo = 0u;                 // later rounds: bounds above lo ...
    float limit = __int_as_float(0x7F800000);      // ... and not beyond limit are taken
    uint32_t hi = 0xFFFFFFFFu;        // bounds up to hi are taken
    if (FIRST) {
        uint32_t cut[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
        if (!*p.failed && p.first < p.num_groups) {
            auto get = [lb, stride](int j) { return lb[(size_t)j * stride]; };
            cta_select2(get, p.num_groups, p.first, min(p.first + p.step, p.num_groups), 32, s_sel, s_res, cut);
            cta_select2(get, p.num_groups, min(p.first + 2 * p.step, p.num_groups), min(p.first + 2 * p.step, p.num_groups), 32,
                        s_sel, s_res, cut + 2);
            hi = cut[0];
        }
        if (tid < 3) p.thresh[(size_t)tid * p.nq + q] = tid == 0 ? cut[0] : (tid == 1 ? cut[1] : cut[2]);
    } else {
        lo = p.thresh[(size_t)(p.round - 2) * p.nq + q];
        if (!p.last) hi = p.thresh[(size_t)(p.round - 1) * p.nq + q];
        if (lo != 0xFFFFFFFFu) {      // the same for every thread
            // k-th best candidate so far
            const uint64_t *lists = p.part_topk + (size_t)q * p.num_groups * p.kpart;
            const int total = p.num_groups * p.kpart;
            uint32_t kth = 0xFFFFFFFFu;
            if (p.knn <= total) {
                uint32_t out[2];
                cta_select2([lists](int j) { return (uint32_t)(lists[j] >> 32); }, total, p.knn, p.knn, 32, s_sel, s_res, out);
                kth = out[0];
            }
            double q2, dq2;
            query_norms(p.query + (size_t)q * p.dim, p.dim, s_sum, &q2, &dq2);
            const float d = __uint_as_float(kth);              // an empty slot reads as NaN
            if (d < __int_as_float(0x7F800000) && q2 <= 1.0e30) {
                // a row is strictly beyond d when its squared distance exceeds d^2 by more than the rounding of
                // the distance chain (about (dim + 4) 2^-24, twice that taken); 1e-18 covers underflow
                limit = __double2float_ru((double)d * d * (1.0 + (p.dim + 8.0) / 8388608.0) + 1.0e-18 - bounds_query_term(q2, dq2, p.dim));
                if (tid == 0) atomicMin(p.qbound + q, kth);
            }
        }
    }
    if (FIRST || lo != 0xFFFFFFFFu) {
        for (int g = tid; g < p.num_groups; g += blockDim.x) {
            const uint32_t v = lb[(size_t)g * stride];
            const bool take = v <= hi && (FIRST || (v > lo && !(ordered_to_float(v) > limit)));
            if (take) p.list[(size_t)g * stride + atomicAdd(p.cnt + g, 1)] = q;
        }
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(p.ticket, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (s_last) {
        __threadfence();
        // exclusive scan of the list lengths, blockDim.x of them at a time
        int run = 0;
        for (int g0 = 0; g0 < p.num_groups; g0 += blockDim.x) {
            const int g = g0 + tid, lane = tid & 31;
            const int c = g < p.num_groups ? (__ldcg(p.cnt + g) + p.per_item - 1) / p.per_item : 0;
            int inc = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= o) inc += t;
            }
            if (lane == 31) s_scratch[tid >> 5] = (uint32_t)inc;
            __syncthreads();
            int before = run, total = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
                if (w < (tid >> 5)) before += (int)s_scratch[w];
                total += (int)s_scratch[w];
            }
            if (g < p.num_groups) p.offs[g] = before + inc - c;
            run += total;
            __syncthreads();
        }
        if (tid == 0) p.offs[p.num_groups] = run;
    }
}

}  // namespace dci
