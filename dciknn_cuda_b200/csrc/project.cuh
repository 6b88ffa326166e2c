// Exact fp32 projection: out[i][p] = sum_k proj[i][k] * x[p][k], one fused
// multiply-add per term, k ascending, accumulator starting at +0.  This fixed
// order is the library's definition of a projected key; it replaces the
// cublasSgemm calls of the reference (src/util_kernel.cu:45-80, called from
// src/dci_cuda_kernel.cu:167-169 for data and :802-803 for queries).
// HBM-bound: reads 4*dim bytes and writes 4*L*S bytes per point.
#pragma once
#include "common.cuh"

namespace dci {

constexpr int kProjThreads = 128;  // threads per CTA
constexpr int kProjPerThread = 2;  // points per thread: a direction value read from shared memory feeds both
constexpr int kProjPoints = kProjThreads * kProjPerThread;   // points per CTA tile
constexpr int kProjK = 32;         // k-chunk staged through shared memory
constexpr int kProjPad = 36;       // row stride of the staged x tile: 16-byte aligned, conflict-free float4 reads

// Two fused multiply-adds in one instruction (sm_100 packed fp32): each half is an ordinary IEEE
// fma, so results do not change.
__device__ __forceinline__ void fma2(float2 &acc, const float2 a, const float2 b) {
    unsigned long long c = *reinterpret_cast<unsigned long long *>(&acc);
    asm("fma.rn.f32x2 %0, %1, %2, %0;"
        : "+l"(c)
        : "l"(*reinterpret_cast<const unsigned long long *>(&a)), "l"(*reinterpret_cast<const unsigned long long *>(&b)));
    acc = *reinterpret_cast<float2 *>(&c);
}

// Each thread owns two points (tid and tid + 128 of the tile) and DIRS accumulators for each,
// kept as pairs of neighbouring directions.  The directions are staged coordinate-major, so one
// 128-bit shared-memory load brings one coordinate of four directions: two packed operands that
// feed two packed multiply-adds per point with the point's coordinate in both halves.  A
// coordinate is finished for every direction before the next one starts, so every accumulator
// still adds its terms in ascending coordinate order and the result is unchanged; coordinates
// beyond the end of a row are zero in both operands and add nothing (an accumulator that starts
// at +0 is never -0).  DIRS is a multiple of 4.
template <int DIRS>
__global__ void __launch_bounds__(kProjThreads)
project_exact_kernel(const float *__restrict__ x, long long n, int dim,
                     const float *__restrict__ proj, int num_indices, float *__restrict__ out) {
    static_assert(DIRS % 4 == 0, "directions are handled four at a time");
    __shared__ __align__(16) float xs[kProjPoints][kProjPad];
    __shared__ __align__(16) float ps[kProjK][DIRS];
    const int tid = threadIdx.x;
    const long long p0 = (long long)blockIdx.x * kProjPoints;
    const bool vec_ok = (dim % 4 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
    for (int i0 = 0; i0 < num_indices; i0 += DIRS) {
        float2 acc[kProjPerThread][DIRS / 2];
#pragma unroll
        for (int u = 0; u < kProjPerThread; ++u)
#pragma unroll
            for (int d = 0; d < DIRS / 2; ++d) acc[u][d] = make_float2(0.0f, 0.0f);
        for (int k0 = 0; k0 < dim; k0 += kProjK) {
            const int kn = min(kProjK, dim - k0);
            // stage the x tile: 256 rows x 32 columns, 8 threads (float4 each) per row; columns
            // beyond the row's end are zero
            if (vec_ok) {
                const int c4 = (tid & 7) * 4;
                for (int r = tid >> 3; r < kProjPoints; r += kProjThreads / 8) {
                    const long long p = p0 + r;
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (p < n && c4 < kn)
                        v = __ldg(reinterpret_cast<const float4 *>(x + p * dim + k0 + c4));
                    *reinterpret_cast<float4 *>(&xs[r][c4]) = v;
                }
            } else {
                const int c = tid & 31;
                for (int r = tid >> 5; r < kProjPoints; r += kProjThreads / 32) {
                    const long long p = p0 + r;
                    xs[r][c] = (p < n && c < kn) ? __ldg(x + p * dim + k0 + c) : 0.0f;
                }
            }
            for (int e = tid; e < DIRS * kProjK; e += kProjThreads) {
                const int d = e / kProjK, c = e % kProjK;          // coalesced reads of the directions' rows
                ps[c][d] = (i0 + d < num_indices && c < kn) ? __ldg(proj + (size_t)(i0 + d) * dim + k0 + c) : 0.0f;
            }
            __syncthreads();
            const int kn4 = (kn + 3) & ~3;
            for (int c = 0; c < kn4; c += 4) {
                float4 xv[kProjPerThread];
#pragma unroll
                for (int u = 0; u < kProjPerThread; ++u)
                    xv[u] = *reinterpret_cast<const float4 *>(&xs[tid + u * kProjThreads][c]);
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    float2 xb[kProjPerThread];
#pragma unroll
                    for (int u = 0; u < kProjPerThread; ++u) {
                        const float v = cc == 0 ? xv[u].x : (cc == 1 ? xv[u].y : (cc == 2 ? xv[u].z : xv[u].w));
                        xb[u] = make_float2(v, v);
                    }
#pragma unroll
                    for (int d4 = 0; d4 < DIRS / 4; ++d4) {
                        const float4 pv = *reinterpret_cast<const float4 *>(&ps[c + cc][4 * d4]);
#pragma unroll
                        for (int u = 0; u < kProjPerThread; ++u) {
                            fma2(acc[u][2 * d4], make_float2(pv.x, pv.y), xb[u]);
                            fma2(acc[u][2 * d4 + 1], make_float2(pv.z, pv.w), xb[u]);
                        }
                    }
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int u = 0; u < kProjPerThread; ++u) {
            const long long p = p0 + tid + u * kProjThreads;
            if (p < n) {
#pragma unroll
                for (int d = 0; d < DIRS / 2; ++d) {
                    if (i0 + 2 * d < num_indices) out[(size_t)(i0 + 2 * d) * n + p] = acc[u][d].x;
                    if (i0 + 2 * d + 1 < num_indices) out[(size_t)(i0 + 2 * d + 1) * n + p] = acc[u][d].y;
                }
            }
        }
    }
}

// Few points: the kernel above gives 256 points to a CTA, so a query batch ran on a handful of SMs and took as long
// as one CTA needs for its tile (20 us for up to 256 queries x 128 coordinates x 20 directions; 1 000 points in 4 CTAs).
// Here a CTA has 32 points and a thread one direction of four of them: per four coordinates four 128-bit broadcast
// reads of the points and four reads of the direction (rows padded to an odd stride, so the lanes' directions lie on
// different banks) feed sixteen multiply-adds.  The next 64 coordinates are copied (cp.async) while these are added.
// Bound by the latency of those copies; the same chain per key, hence the same bits.
constexpr int kPsmRows = 32, kPsmK = 64, kPsmXPad = 68, kPsmPPad = 65, kPsmMaxIndices = 48;

__host__ __device__ inline size_t psm_buffer_floats(int num_indices) {      // a multiple of 4: the points' rows are read as float4
    return (size_t)kPsmRows * kPsmXPad + (((size_t)num_indices * kPsmPPad + 3) & ~(size_t)3);
}

__global__ void __launch_bounds__(kPsmMaxIndices * 8)
project_small_kernel(const float *__restrict__ x, long long n, int dim, const float *__restrict__ proj, int num_indices,
                     float *__restrict__ out) {
    extern __shared__ __align__(16) float psm_smem[];
    const int tid = threadIdx.x;
    const long long p0 = (long long)blockIdx.x * kPsmRows;
    const int rows = (int)min((long long)kPsmRows, n - p0);
    const size_t buf = psm_buffer_floats(num_indices);
    auto load = [&](int k0, float *xs) {
        auto copy = [](float *dst, const float *src, bool live) {      // 4 bytes, zero when not live
            const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(live ? 4 : 0) : "memory");
        };
        float *ps = xs + kPsmRows * kPsmXPad;
        for (int e = tid; e < rows * kPsmK; e += blockDim.x) {
            const int r = e / kPsmK, k = e % kPsmK;
            const bool live = k0 + k < dim;
            copy(xs + r * kPsmXPad + k, x + (p0 + r) * dim + (live ? k0 + k : 0), live);
        }
        for (int e = tid; e < num_indices * kPsmK; e += blockDim.x) {
            const int d = e / kPsmK, k = e % kPsmK;
            const bool live = k0 + k < dim;
            copy(ps + d * kPsmPPad + k, proj + (size_t)d * dim + (live ? k0 + k : 0), live);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int d = tid % num_indices, r0 = tid / num_indices * 4;
    const bool active = r0 < rows;
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    load(0, psm_smem);
    for (int k0 = 0, c = 0; k0 < dim; k0 += kPsmK, ++c) {
        if (k0 + kPsmK < dim) {
            load(k0 + kPsmK, psm_smem + (size_t)((c + 1) & 1) * buf);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        if (active) {
            const float *xs = psm_smem + (size_t)(c & 1) * buf;
            const float *ps = xs + kPsmRows * kPsmXPad + d * kPsmPPad;
            xs += r0 * kPsmXPad;
            const int kn = min(kPsmK, (dim - k0 + 3) & ~3);         // coordinates beyond the row's end are zero
#pragma unroll 4
            for (int k = 0; k < kn; k += 4) {
                float4 xv[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) xv[u] = *reinterpret_cast<const float4 *>(xs + u * kPsmXPad + k);
                const float a = ps[k], b = ps[k + 1], e = ps[k + 2], f = ps[k + 3];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    acc[u] = __fmaf_rn(a, xv[u].x, acc[u]);
                    acc[u] = __fmaf_rn(b, xv[u].y, acc[u]);
                    acc[u] = __fmaf_rn(e, xv[u].z, acc[u]);
                    acc[u] = __fmaf_rn(f, xv[u].w, acc[u]);
                }
            }
        }
        __syncthreads();
    }
    if (active) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (r0 + u < rows) out[(size_t)d * n + p0 + r0 + u] = acc[u];
    }
}

}  // namespace dci
