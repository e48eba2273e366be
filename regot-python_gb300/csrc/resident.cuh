// Block-level building blocks of the kernels that keep one FP64 matrix K
// (n x m, row stride ldk even, columns m .. ldk - 1 zero) through many
// products: each block owns a run of rows, forms their dot products with a
// vector, then its part of the column products, and after a barrier of all
// blocks merges a run of columns over the blocks.
//
// FP64 issue bounds these kernels, not memory: on a GB300 an FP64 instruction
// holds its quarter of the SM for 64 to 77 clocks, whether one of the warp's
// lanes is active or all (measured: dependent or not, 71 clocks an addition,
// 630 a division, 2150 a logarithm, 610 a five-level shuffle sum). Hence: as
// few FP64 instructions as possible, packed into full warps - divisions of a
// block's rows or columns together in one warp, lane sums of several rows
// added side by side - and no FP64 comparison where a look at the exponent
// bits will do.
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

// Sum over the lanes congruent modulo `keep`, valid in lanes 0 .. keep - 1.
__device__ __forceinline__ double warp_sum_low(double v, int keep = 1) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (o < keep) break;
        v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    return v;
}

// Sum of p[g * stride], g < G, over the warp (valid in lane 0): five loads a
// lane under way together.
__device__ __forceinline__ double warp_sum_strided(const double* p, int G, int stride) {
    const int lane = threadIdx.x & 31;
    double s = 0.0;
    for (int g = lane; g < G; g += 160) {
        double v[5];
#pragma unroll
        for (int k = 0; k < 5; ++k)
            v[k] = g + 32 * k < G ? __ldcg(p + (long long)(g + 32 * k) * stride) : 0.0;
#pragma unroll
        for (int k = 0; k < 5; ++k)
            if (g + 32 * k < G) s += v[k];
    }
    __syncwarp();
    return warp_sum_low(s);
}

// Sums of p[g].x and p[g].y, g < G, over the warp, in every lane: each half
// of the warp finishes one of the two.
__device__ __forceinline__ double2 warp_sum_pairs(const double2* p, int G) {
    const int lane = threadIdx.x & 31;
    double a = 0.0, b = 0.0;
    for (int g = lane; g < G; g += 160) {
        double2 v[5];
#pragma unroll
        for (int k = 0; k < 5; ++k)
            v[k] = g + 32 * k < G ? __ldcg(p + g + 32 * k) : make_double2(0.0, 0.0);
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            if (g + 32 * k < G) {
                a += v[k].x;
                b += v[k].y;
            }
        }
    }
    __syncwarp();
    const bool upper = (lane & 16) != 0;
    const double send = upper ? a : b;
    double s = (upper ? b : a) + __shfl_xor_sync(0xffffffffu, send, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return make_double2(__shfl_sync(0xffffffffu, s, 0), __shfl_sync(0xffffffffu, s, 16));
}

// s_sum[r] = sum_j K[r0 + r][j] s_x[j], r < R. s_x: ldk entries in shared
// memory. A warp takes a row, or one of S equal column segments of it, with S
// as it leaves the fewest FP64 instructions on a quarter of the SM. The lanes'
// sums of up to kRowUnits segments go through shared memory, so that several
// rows are added side by side; beyond that many a warp adds its own.
// Synchronises the block before the last additions; the caller synchronises
// before it reads s_sum. s_part: rows_part_size(R) doubles.
constexpr int kRowUnits = 64;
__host__ __device__ constexpr int rows_part_size(int R) {
    return R > kRowUnits * 33 ? R : kRowUnits * 33;
}
__device__ __forceinline__ int row_segments(int P, int R) {
    int best = 1, cost = 1 << 30;
    for (int S = 1; S <= 16; S <<= 1) {
        if (S > 1 && (R * S > kRowUnits || P < 64 * S)) break;
        const int c = ((R * S + 3) / 4) * (2 * ((P + 32 * S - 1) / (32 * S)) + 4);
        if (c < cost) {
            cost = c;
            best = S;
        }
    }
    return best;
}
__device__ __forceinline__ void rows_dot(const double* __restrict__ K, long long ldk, int r0, int R,
                                         int S, const double* s_x, double* s_part, double* s_sum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int P = (int)(ldk >> 1);
    const double2* x2 = reinterpret_cast<const double2*>(s_x);
    const int units = R * S, len = (P + S - 1) / S;
    const bool own = units > kRowUnits;  // then S == 1
    for (int unit = warp; unit < units; unit += kResWarps) {
        const int row = S == 1 ? unit : unit / S, seg = unit - row * S;
        const double2* k2 = reinterpret_cast<const double2*>(K + (long long)(r0 + row) * ldk);
        const int p1 = (seg + 1) * len < P ? (seg + 1) * len : P;
        int p = seg * len + lane;
        double a0 = 0.0, a1 = 0.0;
        // the next loads are under way while these are multiplied
        double2 q[4];
        auto load = [&](int at) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                q[k] = at + 32 * k < p1 ? __ldg(k2 + at + 32 * k) : make_double2(0.0, 0.0);
        };
        load(p);
        for (; p < p1; p += 128) {
            const double2 c0 = q[0], c1 = q[1], c2 = q[2], c3 = q[3];
            load(p + 128);
            const double2 y0 = x2[p];
            a0 = fma(c0.x, y0.x, a0);
            a1 = fma(c0.y, y0.y, a1);
            if (p + 32 < p1) {
                const double2 y1 = x2[p + 32];
                a0 = fma(c1.x, y1.x, a0);
                a1 = fma(c1.y, y1.y, a1);
            }
            if (p + 64 < p1) {
                const double2 y2 = x2[p + 64];
                a0 = fma(c2.x, y2.x, a0);
                a1 = fma(c2.y, y2.y, a1);
            }
            if (p + 96 < p1) {
                const double2 y3 = x2[p + 96];
                a0 = fma(c3.x, y3.x, a0);
                a1 = fma(c3.y, y3.y, a1);
            }
        }
        __syncwarp();
        const double v = a0 + a1;
        if (own) {
            const double t = warp_sum_low(v);
            if (lane == 0) s_sum[row] = t;
        } else {
            s_part[unit * 33 + lane] = v;
        }
    }
    __syncthreads();
    if (own) return;
    // eight threads a row: four lane sums of each of its segments, then a tree
    for (int g = threadIdx.x; g < ((8 * R + 31) & ~31); g += kResThreads) {
        const int row = g >> 3, e = g & 7;
        double v = 0.0;
        if (row < R) {
            const double* src = s_part + row * S * 33 + e;
            v = (src[0] + src[8]) + (src[16] + src[24]);
            for (int k = 1; k < S; ++k) {
                src += 33;
                v += (src[0] + src[8]) + (src[16] + src[24]);
            }
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (e == 0 && row < R) s_sum[row] = v;
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
// CPW adjacent columns and 32 / CPW groups of rows, five loads a lane under
// way together: use(j, sum) in one lane per column. Called by `warps` whole
// warps, this one being number `warp`.
template <int CPW, typename F>
__device__ __forceinline__ void merge_columns_w(const double* part, long long ldk, int G, int j0,
                                                int j1, int warp, int warps, F&& use) {
    const int lane = threadIdx.x & 31;
    const int c = lane % CPW, g0 = lane / CPW;
    constexpr int GS = 32 / CPW, NL = 5;
    for (int jb = j0 + warp * CPW; jb < j1; jb += warps * CPW) {
        const int j = jb + c;
        const bool ok = j < j1;
        double s = 0.0;
        for (int g = g0; g < G; g += NL * GS) {
            double v[NL];
#pragma unroll
            for (int k = 0; k < NL; ++k)
                v[k] = ok && g + k * GS < G ? __ldcg(part + (long long)(g + k * GS) * ldk + j) : 0.0;
#pragma unroll
            for (int k = 0; k < NL; ++k)
                if (g + k * GS < G) s += v[k];
        }
        __syncwarp();
        s = warp_sum_low(s, CPW);
        if (ok && g0 == 0) use(j, s);
    }
}
// Few columns a block: one a warp, so that the chain of additions is short;
// many: four, whose loads fill whole 32-byte sectors.
template <typename F>
__device__ __forceinline__ void merge_columns(const double* part, long long ldk, int G, int j0,
                                              int j1, int warp, int warps, F&& use) {
    if (j1 - j0 <= 2 * warps) merge_columns_w<1>(part, ldk, G, j0, j1, warp, warps, use);
    else merge_columns_w<4>(part, ldk, G, j0, j1, warp, warps, use);
}

// ---- launches: one cluster of 16 blocks for small problems, else a block an SM ----

// Problems of at most this many entries run in one cluster: its barrier takes a
// third of the grid's, its 16 SMs nine times the products. FP64, cluster against
// grid, us (sinkhorn_bcd / newton / ssns): 64 x 64 508 / 3210 / 1642 against 570 /
// 3457 / 1760, 128 x 128 500 / 3750 / 1778 against 490 / 3689 / 1845, 160 x 150
// 500 / 3735 / 1824 against 500 / 3798 / 1837, 250 x 250 508 / 4456 / 2036 against
// 413 / 3956 / 1837.
constexpr long long kClusterEntries = 24 * 1024;
// A stored plan doubles the memory of the cost matrix; beyond this size the
// solvers keep to the dense passes.
constexpr double kPlanMaxBytes = 32.0 * (1ULL << 30);

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
    if (entries > kClusterEntries ||
        smem > max_block_smem(reinterpret_cast<const void*>(kernel)))
        return false;
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = resident_config(at, true, 16, smem, nullptr);
    int clusters = 0;
    const bool ok =
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
    if (!coop || smem > max_block_smem(reinterpret_cast<const void*>(kernel))) return false;
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
