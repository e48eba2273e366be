// Block-level building blocks of the kernels that keep one FP64 matrix K
// (n x m, row stride ldk even, columns m .. ldk - 1 zero) through many
// products: each block owns a run of rows, forms their dot products with a
// vector, then its part of the column products, and after a barrier of all
// blocks merges a run of columns over the blocks.
//
// FP64 issue bounds these kernels, not memory: a GB300 SM starts two FP64
// operations a clock, so a warp's FP64 instruction holds its quarter of the
// SM for 64 clocks whatever the number of active lanes. Hence the layouts:
// full warps, few reduction levels (they cost as much as full-width work),
// and no FP64 comparison where a look at the exponent bits will do.
#pragma once

#include "device_util.cuh"
#include "grid_sync.cuh"

namespace regot {

constexpr int kResThreads = 512;
constexpr int kResWarps = kResThreads / 32;

// Rows / columns owned by block b of G.
__device__ __forceinline__ int own_begin(int len, int b, int G) {
    return (int)((long long)len * b / G);
}

// 2^-lim <= |x| <= 2^lim, by the exponent bits (false for NaN, 0, infinity).
__device__ __forceinline__ bool exponent_within(double x, int lim) {
    const int e = ((__double2hiint(x) >> 20) & 0x7ff) - 1023;
    return e >= -lim && e <= lim;
}

// s_sum[r] = sum_j K[r0 + r][j] s_x[j], r < R. s_x: ldk entries in shared
// memory. Whole rows a warp; with fewer rows than warps, equal column
// segments of a row. Synchronises the block before the segments are added;
// the caller synchronises before it reads s_sum.
__device__ __forceinline__ void rows_dot(const double* __restrict__ K, long long ldk, int r0, int R,
                                         const double* s_x, double* s_part, double* s_sum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int P = (int)(ldk >> 1);
    int S = 1;
    if (R > 0 && R < kResWarps) {
        const int by_width = P / 64 > 0 ? P / 64 : 1;
        S = kResWarps / R < by_width ? kResWarps / R : by_width;
    }
    const double2* x2 = reinterpret_cast<const double2*>(s_x);
    for (int unit = warp; unit < R * S; unit += kResWarps) {
        const int row = unit / S, seg = unit - row * S;
        const double2* k2 = reinterpret_cast<const double2*>(K + (long long)(r0 + row) * ldk);
        const int p1 = (int)((long long)P * (seg + 1) / S);
        int p = (int)((long long)P * seg / S) + lane;
        double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
        for (; p + 96 < p1; p += 128) {
            const double2 q0 = __ldg(k2 + p), q1 = __ldg(k2 + p + 32), q2 = __ldg(k2 + p + 64),
                          q3 = __ldg(k2 + p + 96);
            const double2 y0 = x2[p], y1 = x2[p + 32], y2 = x2[p + 64], y3 = x2[p + 96];
            a0 = fma(q0.x, y0.x, a0);
            a1 = fma(q0.y, y0.y, a1);
            a2 = fma(q1.x, y1.x, a2);
            a3 = fma(q1.y, y1.y, a3);
            a0 = fma(q2.x, y2.x, a0);
            a1 = fma(q2.y, y2.y, a1);
            a2 = fma(q3.x, y3.x, a2);
            a3 = fma(q3.y, y3.y, a3);
        }
        for (; p < p1; p += 32) {
            const double2 q0 = __ldg(k2 + p);
            const double2 y0 = x2[p];
            a0 = fma(q0.x, y0.x, a0);
            a1 = fma(q0.y, y0.y, a1);
        }
        const double v = warp_sum_d((a0 + a1) + (a2 + a3));
        if (lane == 0) s_part[unit] = v;
    }
    __syncthreads();
    for (int r = threadIdx.x; r < R; r += kResThreads) {
        double v = s_part[r * S];
        for (int k = 1; k < S; ++k) v += s_part[r * S + k];
        s_sum[r] = v;
    }
}

// out[j] = sum_{r < R} K[r0 + r][j] s_u[r], j < ldk (out in global memory,
// written past L1). A thread owns a pair of adjacent columns; narrow
// matrices split the rows over the warps left over (s_q: 2 kResThreads
// doubles). Synchronises the block when it splits.
__device__ __forceinline__ void cols_dot(const double* __restrict__ K, long long ldk, int r0, int R,
                                         const double* s_u, double* out, double* s_q) {
    const int P = (int)(ldk >> 1);
    const int pw = (P + 31) & ~31;
    int Q = pw <= kResThreads / 2 ? kResThreads / pw : 1;
    if (Q > R) Q = R > 0 ? R : 1;
    const double2* k2 = reinterpret_cast<const double2*>(K + (long long)r0 * ldk);
    const long long ld2 = ldk >> 1;
    auto column = [&](int p, int first, int step) {
        double2 c = make_double2(0.0, 0.0);
        int r = first;
        const double2* src = k2 + p;
        for (; r + 7 * step < R; r += 8 * step) {
            double2 q[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) q[k] = __ldg(src + (long long)(r + k * step) * ld2);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const double u = s_u[r + k * step];
                c.x = fma(q[k].x, u, c.x);
                c.y = fma(q[k].y, u, c.y);
            }
        }
        for (; r < R; r += step) {
            const double2 q = __ldg(src + (long long)r * ld2);
            const double u = s_u[r];
            c.x = fma(q.x, u, c.x);
            c.y = fma(q.y, u, c.y);
        }
        return c;
    };
    double2* out2 = reinterpret_cast<double2*>(out);
    if (Q == 1) {
        for (int p = threadIdx.x; p < P; p += kResThreads) __stcg(out2 + p, column(p, 0, 1));
        return;
    }
    double2* sq2 = reinterpret_cast<double2*>(s_q);
    const int q = threadIdx.x / pw, p = threadIdx.x - q * pw;
    if (q < Q && p < P) sq2[q * pw + p] = column(p, q, Q);
    __syncthreads();
    if (threadIdx.x < P) {
        double2 c = sq2[threadIdx.x];
        for (int k = 1; k < Q; ++k) {
            const double2 d = sq2[k * pw + threadIdx.x];
            c.x += d.x;
            c.y += d.y;
        }
        __stcg(out2 + threadIdx.x, c);
    }
}

// Columns [j0, j1) summed over the G rows of part (stride ldk), one warp for
// CPW adjacent columns and 32 / CPW groups of rows: use(j, sum) in one lane
// per column. Called by `warps` whole warps, this one being number `warp`.
template <int CPW, typename F>
__device__ __forceinline__ void merge_columns_w(const double* part, long long ldk, int G, int j0,
                                                int j1, int warp, int warps, F&& use) {
    const int lane = threadIdx.x & 31;
    const int c = lane % CPW, g0 = lane / CPW;
    constexpr int GS = 32 / CPW;
    for (int jb = j0 + warp * CPW; jb < j1; jb += warps * CPW) {
        const int j = jb + c;
        const bool ok = j < j1;
        double s0 = 0.0, s1 = 0.0;
        if (ok) {
            int g = g0;
            for (; g + 3 * GS < G; g += 4 * GS) {
                double v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = __ldcg(part + (long long)(g + k * GS) * ldk + j);
                s0 += v[0];
                s1 += v[1];
                s0 += v[2];
                s1 += v[3];
            }
            for (; g < G; g += GS) s0 += __ldcg(part + (long long)g * ldk + j);
        }
        double s = s0 + s1;
#pragma unroll
        for (int o = 16; o >= CPW; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (ok && g0 == 0) use(j, s);
    }
}
// Few columns a block: two a warp, so that the chain of additions is short;
// many: four, whose loads fill whole 32-byte sectors.
template <typename F>
__device__ __forceinline__ void merge_columns(const double* part, long long ldk, int G, int j0,
                                              int j1, int warp, int warps, F&& use) {
    if (j1 - j0 <= 2 * warps) merge_columns_w<2>(part, ldk, G, j0, j1, warp, warps, use);
    else merge_columns_w<4>(part, ldk, G, j0, j1, warp, warps, use);
}

// ---- launches: one cluster of 16 blocks for small problems, else a block an SM ----

// Problems of at most this many entries run in one cluster.
constexpr long long kClusterEntries = 64 * 1024;
// A stored plan doubles the memory of the cost matrix; beyond this size the
// solvers keep to the dense passes.
constexpr double kPlanMaxBytes = 32.0 * (1ULL << 30);

inline size_t max_block_smem() {
    int dev = 0, optin = 0;
    REGOT_CUDA(cudaGetDevice(&dev));
    REGOT_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    return (size_t)optin - 1024;  // static shared memory of the kernels
}

inline cudaLaunchConfig_t resident_config(cudaLaunchAttribute* at, bool cluster, int blocks,
                                          size_t smem, cudaStream_t st) {
    if (cluster) {
        at->id = cudaLaunchAttributeClusterDimension;
        at->val.clusterDim.x = (unsigned)blocks;
        at->val.clusterDim.y = at->val.clusterDim.z = 1;
    } else {
        at->id = cudaLaunchAttributeCooperative;
        at->val.cooperative = 1;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kResThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// Whether `kernel` runs n m = entries entries in one cluster of 16 blocks.
template <typename P>
bool resident_cluster(void (*kernel)(P), long long entries, size_t smem) {
    if (entries > kClusterEntries || smem > max_block_smem()) return false;
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = resident_config(at, true, 16, smem, nullptr);
    int clusters = 0;
    const bool ok =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
            cudaSuccess &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) ==
            cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0;
    if (!ok) cudaGetLastError();
    return ok;
}

// Whether a cooperative launch of `kernel` holds one block on every SM.
template <typename P>
bool resident_grid(void (*kernel)(P), size_t smem) {
    int dev = 0, coop = 0, occ = 0;
    REGOT_CUDA(cudaGetDevice(&dev));
    REGOT_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop || smem > max_block_smem()) return false;
    REGOT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    REGOT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, kResThreads, smem));
    return occ >= 1;
}

template <typename P>
void launch_resident(void (*kernel)(P), bool cluster, int blocks, size_t smem, cudaStream_t st,
                     const P& params) {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = resident_config(at, cluster, blocks, smem, st);
    REGOT_CUDA(cudaLaunchKernelEx(&cfg, kernel, params));
    count_launch();
}

}  // namespace regot
