// Lower bounds of the distances between all queries and groups of consecutive rows, on the 5th-generation
// tensor cores.  A group is a partition of the index (pruning: a partition whose nearest row is provably
// farther than the k-th candidate found so far cannot change a query's answer, so it is not traversed), or a
// run of 32 or more rows (exhaustive queries).  No value computed here reaches a result: every returned
// distance is the fixed fp32 chain of the traversal.
//
// For query q and group g the kernel produces
//     v[g][q] = min over rows x of the group of  row_term(x) - 2 s^2 <x~, q~>
// where x~, q~ are the tf32 values that the tensor core makes of fp32 operands (it ignores the low 13 mantissa
// bits: truncation) and s undoes the mean loss of that.  With x' = s x~, q' = s q~ and the residuals dx = x - x',
// dq = q - q',
//     <x, q> = <x', q'> + <dx, q> + <x', dq>,   so   | <x, q> - s^2 <x~, q~> | <= |dx||q| + |x'||dq|,
// and for any r > 0:  2 |dx||q| <= |dx|^2 / r + r |q|^2,  2 |x'||dq| <= r |x'|^2 + |dq|^2 / r.  Hence
//     |x - q|^2 = |x|^2 + |q|^2 - 2 <x, q>  >=  v + query_term(q)
//     row_term(x) = keep |x|^2 - |dx|^2 / r,   query_term(q) = keep |q|^2 - |dq|^2 / r,
// keep = 1 - r (with |x'| <= (1 + 2^-9) |x|) less the accumulation of the products (dim * 2^-22 of |x||q|; the MMAs add
// eight products a step in fp32) and the rounding of the norms and of the sums.  The residuals are computed, not
// bounded: about 0.2 * 2^-10 of the norm for mantissas without a pattern, which is what r is set to, against the 2^-9
// of both operands' largest truncation (1.25M x 96 mixture, |x| about ten times the distances between neighbours,
// 1 000 queries: 10.1 -> 6.9 ms).  Rows whose squared norm exceeds 1e30 count as -inf (never pruned); rows with a NaN
// have no distance and are ignored.
//
// One persistent CTA per SM, warp-specialised like project_tf32x3_persistent_kernel: tiles of 128 queries x
// 256 rows, 32 coordinates a stage (48 KB), four stages, accumulators double buffered in tensor memory
// (2 x 256 columns), so that the minimum of one tile is taken while the next one is multiplied.  Queries are
// the tensor-memory lanes: a thread keeps one query and walks the 256 rows as columns, so the minimum needs no
// exchange between threads.  A work unit is one tile of rows against up to `qt_per_unit` query tiles.
// Roles: warp 0 requests tiles by TMA, warp 1 issues the MMAs, warps 4..7 take the minima, warps 8..15 sum
// the squared norms of the rows as their coordinates pass through shared memory (first query tile of a unit).
// PLAIN: rows that a tensor map cannot describe (dim not a multiple of 4, unaligned): warps 8..15 stage the
// tiles with ordinary loads in the same swizzled layout.
#pragma once
#include "common.cuh"
#include "project_tf32.cuh"

namespace dci {

constexpr int kLbQueries = 128;       // M of the MMA tile
constexpr int kLbRows = 256;          // N of the MMA tile
constexpr int kLbK = 32;              // coordinates per stage
constexpr int kLbThreads = 512;
constexpr int kLbNormWarps = 8;
constexpr size_t kLbABytes = (size_t)kLbQueries * 128, kLbBBytes = (size_t)kLbRows * 128;
// MT query tiles share a tile of rows: 48 KB x 4 stages for one, 64 KB x 3 for two
__host__ __device__ constexpr int lb_stages(int mt) { return mt == 1 ? 4 : 3; }
__host__ __device__ constexpr size_t lb_stage_bytes(int mt) { return mt * kLbABytes + kLbBBytes; }
__host__ __device__ constexpr size_t lb_smem(int mt) { return lb_stages(mt) * lb_stage_bytes(mt) + 1024; }
constexpr float kLbMaxNorm = 1.0e30f;

struct BoundsParams {
    const float *data, *query;        // PLAIN only; the TMA variant reads through the tensor maps
    int n, dim, nq;                   // rows, coordinates, queries (of this launch)
    int group_rows, num_groups;       // group g holds the rows [g * group_rows, (g + 1) * group_rows)
    int q_stride;                     // out is [num_groups][q_stride]
    int qt_per_unit, units_q;         // query tiles per work unit (a multiple of MT, or all), units per tile of rows
    uint32_t *out;                    // ordered fp32 (float_to_ordered), starts as all ones
    int *failed;                      // set when a bounded wait ran out: the bounds must then not be used
};

constexpr float kLbScale = 1.0f + 0.3214f / 1024;       // s: E[t x] / E[x^2] of truncation errors t for mantissas spread over [1, 2)
constexpr float kLbRatio = 0.2f / 1024;                 // r

__host__ __device__ inline float bounds_keep(int dim) {
    return (float)(1.0 - kLbRatio * (1.0 + 1.0 / 256) - (double)dim / (1 << 22) - (double)dim / (1 << 23) - 1.0 / (1 << 20));
}

// Residual of a coordinate.
__device__ __forceinline__ float bounds_residual(float x) {
    return __fmaf_rn(-kLbScale, __uint_as_float(__float_as_uint(x) & 0xFFFFE000u), x);
}

// query_term from |q|^2 and |dq|^2 (computed in double).
__device__ __forceinline__ double bounds_query_term(double q2, double dq2, int dim) {
    return (double)bounds_keep(dim) * q2 - dq2 * (1.001 / kLbRatio);
}

// MT = 2: two query tiles against every staged tile of rows, an accumulator each (so none to spare for the next tile,
// whose products wait for the minima of this one).  A third fewer bytes per product through L2, which is what bounds
// one tile (91 bytes per SM and cycle at the full tensor rate); it pays where rows are long, see launch_bounds.
template <bool PLAIN, int MT>
__global__ void __launch_bounds__(kLbThreads, 1)
distance_bounds_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_q,
                       const BoundsParams prm) {
    static_assert(!PLAIN || MT == 1, "ordinary loads stage one query tile");
    constexpr int kLbStages = lb_stages(MT);
    constexpr size_t kLbStageBytes = lb_stage_bytes(MT);
    extern __shared__ __align__(16) unsigned char lb_dyn[];
    __shared__ __align__(8) unsigned long long full_bar[kLbStages], empty_bar[kLbStages];
    __shared__ __align__(8) unsigned long long acc_full[2], acc_empty[2], norm_full[2], norm_empty[2];
    __shared__ __align__(16) float s_norm[2][kLbRows];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t s0 = smem_u32(lb_dyn);
    unsigned char *base = lb_dyn + (((s0 + 1023u) & ~1023u) - s0);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(2u * kLbRows));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 0) {
        abort_flag = 0;
        auto init = [](unsigned long long *bar, int count) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
        };
        for (int s = 0; s < kLbStages; ++s) {
            init(&full_bar[s], PLAIN ? kLbNormWarps * 32 : 1);
            init(&empty_bar[s], PLAIN ? 1 : 1 + kLbNormWarps);
        }
        for (int a = 0; a < 2; ++a) {
            init(&acc_full[a], 1); init(&acc_empty[a], 128);
            init(&norm_full[a], kLbNormWarps * 32); init(&norm_empty[a], 128);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_slot;
    // roles of whole warps decide together, so that a warp never splits around a warp-wide operation
    auto warp_ok = [](bool ok) { return __all_sync(0xFFFFFFFFu, ok) != 0; };
    const int nchunks = (prm.dim + kLbK - 1) / kLbK;
    const int row_tiles = (prm.n + kLbRows - 1) / kLbRows, q_tiles = (prm.nq + kLbQueries - 1) / kLbQueries;
    const int units = row_tiles * prm.units_q;
    const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(kLbRows >> 3) << 17) |
                           ((uint32_t)(kLbQueries >> 4) << 24);

    if (!PLAIN && warp == 0 && lane == 0) {
        // ---- producer
        uint32_t s_no = 0;
        for (int u = blockIdx.x; u < units && !abort_flag; u += gridDim.x) {
            const int rt = u / prm.units_q, qt0 = (u % prm.units_q) * prm.qt_per_unit;
            const int qt1 = min(qt0 + prm.qt_per_unit, q_tiles);
            for (int qt = qt0; qt < qt1 && !abort_flag; qt += MT)
                for (int c = 0; c < nchunks; ++c, ++s_no) {
                    const int st = (int)(s_no % kLbStages);
                    const uint32_t use = s_no / kLbStages;
                    if (use > 0 && !mbar_wait(smem_u32(&empty_bar[st]), (use - 1) & 1u)) { abort_flag = 1; break; }
                    const uint32_t a = smem_u32(base + (size_t)st * kLbStageBytes), bar = smem_u32(&full_bar[st]);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)kLbStageBytes)
                                 : "memory");
#pragma unroll
                    for (int m = 0; m < MT; ++m)             // (a tile beyond the queries reads as zeros)
                        asm volatile(
                            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
                                "r"(a + (uint32_t)(m * kLbABytes)), "l"(&map_q), "r"(c * kLbK), "r"((qt + m) * kLbQueries), "r"(bar)
                            : "memory");
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
                            "r"(a + (uint32_t)(MT * kLbABytes)), "l"(&map_x), "r"(c * kLbK), "r"(rt * kLbRows), "r"(bar)
                        : "memory");
                }
        }
        // a stage that was requested must land before the CTA may leave
        for (uint32_t back = 0; back < kLbStages && back < s_no; ++back) {
            const uint32_t j = s_no - 1 - back;
            mbar_wait(smem_u32(&full_bar[j % kLbStages]), (j / kLbStages) & 1u);
        }
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issuer
        uint32_t s_no = 0, t = 0;
        for (int u = blockIdx.x; u < units && !abort_flag; u += gridDim.x) {
            const int qt0 = (u % prm.units_q) * prm.qt_per_unit, qt1 = min(qt0 + prm.qt_per_unit, q_tiles);
            for (int qt = qt0; qt < qt1 && !abort_flag; qt += MT, ++t) {
                const int a = MT == 1 ? (int)(t & 1u) : 0;
                const uint32_t earlier = MT == 1 ? t >> 1 : t;       // tiles that used this accumulator before
                if (earlier > 0)
                    for (int m = 0; m < MT; ++m)
                        if (!mbar_wait(smem_u32(&acc_empty[a + m]), (earlier - 1) & 1u)) { abort_flag = 1; break; }
                if (abort_flag) break;
                const uint32_t tmem_d = tmem_base + (uint32_t)(a * kLbRows);
                for (int c = 0; c < nchunks; ++c, ++s_no) {
                    const int st = (int)(s_no % kLbStages);
                    if (!mbar_wait(smem_u32(&full_bar[st]), (s_no / kLbStages) & 1u)) { abort_flag = 1; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t as = smem_u32(base + (size_t)st * kLbStageBytes), bs = as + (uint32_t)(MT * kLbABytes);
#pragma unroll
                    for (int kk = 0; kk < kLbK / 8; ++kk)
#pragma unroll
                        for (int m = 0; m < MT; ++m)
                            umma_tf32(tmem_d + m * kLbRows, umma_desc_sw128(as + (uint32_t)(m * kLbABytes) + kk * 32),
                                      umma_desc_sw128(bs + kk * 32), idesc, (c | kk) ? 1u : 0u);
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                     smem_u32(&empty_bar[st])) : "memory");
                }
                if (abort_flag) break;
                for (int m = 0; m < MT; ++m)
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                     smem_u32(&acc_full[a + m])) : "memory");
            }
        }
    } else if (warp >= 8) {
        // ---- row norms (and, in the PLAIN variant, staging)
        const int wi = warp - 8, row = wi * 32 + lane;           // the row of the tile whose norm this thread sums
        uint32_t s_no = 0, un = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x, ++un) {
            const int rt = u / prm.units_q, qt0 = (u % prm.units_q) * prm.qt_per_unit;
            const int qt1 = min(qt0 + prm.qt_per_unit, q_tiles);
            float nx = 0.0f, dx = 0.0f;          // |x|^2, |dx|^2
            for (int qt = qt0; qt < qt1 && ok; qt += MT) {
                for (int c = 0; c < nchunks; ++c, ++s_no) {
                    const int st = (int)(s_no % kLbStages);
                    const uint32_t use = s_no / kLbStages;
                    unsigned char *as = base + (size_t)st * kLbStageBytes, *bs = as + MT * kLbABytes;
                    if (PLAIN) {
                        ok = warp_ok(use == 0 || mbar_wait(smem_u32(&empty_bar[st]), (use - 1) & 1u));
                        if (!ok) break;
                        const int col = c * kLbK + lane;         // a warp reads 32 consecutive coordinates of one row
                        auto stage = [&](unsigned char *tile, const float *src, int r0, int rows, int limit, int first) {
#pragma unroll 8
                            for (int r = 0; r < rows; ++r) {
                                const int rr = first + r;        // row of the tile
                                const uint32_t gr = (uint32_t)r0 + (uint32_t)rr;
                                const float v = (gr < (uint32_t)limit && col < prm.dim) ? __ldg(src + (size_t)gr * prm.dim + col) : 0.0f;
                                *reinterpret_cast<float *>(tile + rr * 128 + (((lane >> 2) ^ (rr & 7)) << 4) + (lane & 3) * 4) = v;
                            }
                        };
                        stage(bs, prm.data, rt * kLbRows, 32, prm.n, wi * 32);
                        stage(as, prm.query, qt * kLbQueries, kLbQueries / kLbNormWarps, prm.nq, wi * (kLbQueries / kLbNormWarps));
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                    } else {
                        ok = warp_ok(mbar_wait(smem_u32(&full_bar[st]), use & 1u));
                        if (!ok) break;
                    }
                    if (qt == qt0) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float4 v = *reinterpret_cast<const float4 *>(bs + row * 128 + ((j ^ (row & 7)) << 4));
                            nx = __fmaf_rn(v.x, v.x, nx); nx = __fmaf_rn(v.y, v.y, nx);
                            nx = __fmaf_rn(v.z, v.z, nx); nx = __fmaf_rn(v.w, v.w, nx);
                            const float ex = bounds_residual(v.x), ey = bounds_residual(v.y);
                            const float ez = bounds_residual(v.z), ew = bounds_residual(v.w);
                            dx = __fmaf_rn(ex, ex, dx); dx = __fmaf_rn(ey, ey, dx);
                            dx = __fmaf_rn(ez, ez, dx); dx = __fmaf_rn(ew, ew, dx);
                        }
                    }
                    if (PLAIN) {
                        mbar_arrive(smem_u32(&full_bar[st]));
                    } else {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(smem_u32(&empty_bar[st]));
                    }
                }
                if (ok && qt == qt0) {
                    const int nb = (int)(un & 1u);
                    ok = warp_ok(un <= 1 || mbar_wait(smem_u32(&norm_empty[nb]), ((un >> 1) - 1) & 1u));
                    if (!ok) break;
                    const bool live = (uint32_t)rt * kLbRows + (uint32_t)row < (uint32_t)prm.n;
                    s_norm[nb][row] = !live ? __int_as_float(0x7F800000)
                                            : (nx <= kLbMaxNorm ? __fmaf_rn(dx, -1.001f / kLbRatio, bounds_keep(prm.dim) * nx)
                                                               : __int_as_float(0xFF800000));
                    mbar_arrive(smem_u32(&norm_full[nb]));
                }
            }
        }
        if (!ok) abort_flag = 1;
    } else if (warp >= 4) {
        // ---- minima: thread = query (tensor-memory lane), columns = rows
        uint32_t t = 0, un = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x, ++un) {
            const int rt = u / prm.units_q, qt0 = (u % prm.units_q) * prm.qt_per_unit;
            const int qt1 = min(qt0 + prm.qt_per_unit, q_tiles);
            const int nb = (int)(un & 1u);
            ok = warp_ok(mbar_wait(smem_u32(&norm_full[nb]), (un >> 1) & 1u));
            if (!ok) break;
            const int r0 = rt * kLbRows;
            const int g_first = r0 / prm.group_rows;
            const int end_first = (int)min((long long)(g_first + 1) * prm.group_rows - r0, (long long)prm.n);   // column at which that group ends
            // one accumulator after the other; with MT = 2 a unit that ends on an odd tile still has both (zeros)
            const int tiles = (qt1 - qt0 + MT - 1) / MT * MT;
            for (int qt = qt0; qt < qt0 + tiles; ++qt, ++t) {
                const int a = (int)(t & 1u);
                ok = warp_ok(mbar_wait(smem_u32(&acc_full[a]), (t >> 1) & 1u));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t taddr = tmem_base + (uint32_t)(a * kLbRows) + ((uint32_t)((warp & 3) * 32) << 16);
                const int q = qt * kLbQueries + (warp & 3) * 32 + lane;
                float run = __int_as_float(0x7F800000);
                int g = g_first, gend = end_first;
                auto flush = [&]() {
                    if (q < prm.nq && g < prm.num_groups) atomicMin(prm.out + (size_t)g * prm.q_stride + q, float_to_ordered(run));
                };
#pragma unroll 1
                for (int ch = 0; ch < kLbRows / 32; ++ch) {
                    uint32_t r[32];
                    tmem_ld_32(r, taddr + ch * 32);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    const float4 *nv = reinterpret_cast<const float4 *>(&s_norm[nb][ch * 32]);
                    float m0 = __int_as_float(0x7F800000), m1 = m0;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float4 v = nv[j];
                        m0 = fminf(m0, fminf(__fmaf_rn(-2.0f * kLbScale * kLbScale, __uint_as_float(r[4 * j]), v.x),
                                             __fmaf_rn(-2.0f * kLbScale * kLbScale, __uint_as_float(r[4 * j + 1]), v.y)));
                        m1 = fminf(m1, fminf(__fmaf_rn(-2.0f * kLbScale * kLbScale, __uint_as_float(r[4 * j + 2]), v.z),
                                             __fmaf_rn(-2.0f * kLbScale * kLbScale, __uint_as_float(r[4 * j + 3]), v.w)));
                    }
                    const float m = fminf(m0, m1);
                    run = fminf(run, m);
                    // groups that end in this chunk; one that begins inside it takes the whole chunk's minimum
                    // (a smaller value is still a lower bound)
                    while (gend <= ch * 32 + 32) {
                        flush();
                        run = gend < ch * 32 + 32 ? m : __int_as_float(0x7F800000);
                        ++g;
                        gend += prm.group_rows;
                        if (g >= prm.num_groups) gend = 0x7FFFFFFF;
                    }
                }
                flush();
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                mbar_arrive(smem_u32(&acc_empty[a]));
            }
            mbar_arrive(smem_u32(&norm_empty[nb]));
        }
        if (!ok) abort_flag = 1;
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0 && abort_flag) atomicExch(prm.failed, 1);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2u * kLbRows));
}

}  // namespace dci
