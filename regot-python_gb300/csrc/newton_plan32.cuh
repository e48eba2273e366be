// Mixed-precision Newton systems on a stored FP32 plan (included by
// erot_newton.cu).
//
// The HVP pass recomputes T = ex2(...) for every CG step and is bound by that
// arithmetic; here T (FP32, the same bits) is stored once per system and one
// cooperative launch runs the whole CG. Before: four kernels and their
// boundaries a step, 33 us at n = m = 4096, of which the pass took 15.5.
//
// A block of 16 warps is two groups of 8; a group takes tiles of 64 rows x 512
// columns of T (the dense passes' tile, with the same FP32 sums in the same
// order, so each product is what the HVP pass gives) through per-warp rings of
// row buffers filled by cp.async four rows ahead - across tiles and across
// steps, as T does not change, so the first rows of a step are in flight
// during the barriers before it. Odd steps walk the tiles backwards: what the
// end of a step left in L2 is read first by the next. Tiles of one slab that
// follow each other in a group share the column entries of the direction.
// (Rows straight into registers, two or four ahead, took longer than the ring:
// a pair of tiles about 30 instead of 20 thousand clocks.)
//
// A step has three barriers (the captured step had four kernel boundaries):
// the next direction's entries are formed where they are used, from the
// published z and the previous direction. CG on products with FP32 rounding
// amplifies any difference to the level of that rounding within ten steps, so
// everything here keeps the captured step's arithmetic bit for bit: the merges
// of the tiles' sums (merge_2d), the FP64 vector updates, and the order of the
// scalar sums, whose groups of 32 items (k_cg_a's blocks: rows, then columns)
// and 64 items (k_cg_b's) are dealt out to the blocks whole.
#pragma once

#include "resident.cuh"

namespace regot {
namespace {

constexpr int kCg32CW = 512, kCg32Stages = 4, kCg32Rows = 8;  // rows a warp of a tile
constexpr int kCg32Groups = kResWarps / 8;

struct PlanCg32Params {
    const float* T;
    long long ldt;
    int n, m;
    const double *rhs, *hdiag;
    double sign, reg, tol;
    double *x, *z, *p, *y;  // [N], [N], [2][N], [N]
    float *rowpart, *colpart;
    double *parts_a, *parts_b;  // sums of the 32-item and (two) of the 64-item groups
    unsigned* count;
    int* err;        // set when a barrier gives up
    unsigned polls;  // before it does
    NewtonState* st;
};

inline size_t plan_cg32_smem(int N, int G) {
    const size_t I = 64 * ((size_t)((N + 63) / 64) / G + 1);
    return (size_t)kResWarps * kCg32Stages * kCg32CW * sizeof(float) +
           (size_t)kCg32Groups * (4 * kCg32CW + kCg32CW + kRB) * sizeof(float) +
           5 * I * sizeof(double);
}

template <bool CLUSTER>
__global__ void __launch_bounds__(kResThreads, 1) k_plan_cg32(const PlanCg32Params p) {
    constexpr int CW = kCg32CW, NS = kCg32Stages, RPW = kCg32Rows, GT = 256;
    extern __shared__ __align__(128) unsigned char s_dyn32[];
    __shared__ int s_ok, s_stop;
    __shared__ double s_sc, s_w[2][kResWarps];
    __shared__ float2 s_m[kCg32Groups][8][33];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = warp >> 3, wg = warp & 7, gt = tid & (GT - 1);
    const int b = blockIdx.x, G = gridDim.x;
    const int n = p.n, m = p.m, N = n + m;
    // vector items: 64-item groups [vb, ve); merged products: 32-item groups
    const int nvb = (N + 63) / 64, vb = own_begin(nvb, b, G), ve = own_begin(nvb, b + 1, G);
    const int i0 = 64 * vb, items = 64 * (ve - vb);
    const int nar = (n + 31) / 32, nab = nar + (m + 31) / 32;
    const int ab = own_begin(nab, b, G), ae = own_begin(nab, b + 1, G);
    const int Im = 64 * (nvb / G + 1);
    float* ring = reinterpret_cast<float*>(s_dyn32) + (size_t)warp * NS * CW;
    float* s_cred = reinterpret_cast<float*>(s_dyn32) + (size_t)kResWarps * NS * CW +
                    (size_t)group * 4 * CW;
    float* s_cx = reinterpret_cast<float*>(s_dyn32) + (size_t)kResWarps * NS * CW +
                  (size_t)kCg32Groups * 4 * CW + (size_t)group * (CW + kRB);
    float* s_rx = s_cx + CW;
    double* s_h = reinterpret_cast<double*>(s_cx + (size_t)(kCg32Groups - group) * (CW + kRB));
    double* s_p = s_h + Im;
    double* s_x = s_p + Im;
    double* s_r = s_x + Im;
    double* s_z = s_r + Im;
    GridBarrier<CLUSTER> bar(p.count, p.err, p.polls, &s_ok);
    auto group_sync = [&]() {
        asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(GT) : "memory");
    };

    const int nslabs = (m + CW - 1) / CW, nrb = (n + kRB - 1) / kRB, ntiles = nslabs * nrb;
    const int gid = b * kCg32Groups + group, gtot = G * kCg32Groups;
    const int my_tiles = gid < ntiles ? (ntiles - 1 - gid) / gtot + 1 : 0;
    auto tile_at = [&](int s, int k) {
        return gid + ((s & 1) ? my_tiles - 1 - k : k) * gtot;
    };

    // ---- the row ring: row q of the warp, in the order of use over all steps ----
    int ps = 0, pk = 0, pu = 0, pq = 0;
    auto issue = [&]() {
        if (my_tiles > 0) {
            const int t = tile_at(ps, pk);
            const int slab = t % nslabs, rb = t / nslabs;
            const long long c0 = (long long)slab * CW, row = (long long)rb * kRB + wg * RPW + pu;
            if (row < n) {
                const int seg = (int)((p.ldt - c0) < CW ? (p.ldt - c0) : CW);
                const float* src = p.T + row * p.ldt + c0;
                float* dst = ring + (pq % NS) * CW;
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const int off = (v * 32 + lane) * 4;
                    if (off < seg)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                         (unsigned)__cvta_generic_to_shared(dst + off)),
                                     "l"(src + off)
                                     : "memory");
                }
            }
            ++pq;
            if (++pu == RPW) {
                pu = 0;
                if (++pk == my_tiles) {
                    pk = 0;
                    ++ps;
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int q = 0; q < NS; ++q) issue();
    // nothing may be in flight when the block ends
    auto drain = []() { asm volatile("cp.async.wait_all;" ::: "memory"); };

    // Sums over the warp of v0 (in the lower lanes) and v1 (in the upper), each in
    // warp_sum_d's order: half the additions of two such sums.
    auto pair_sum = [&](double v0, double v1) {
        const bool upper = (lane & 16) != 0;
        const double send = upper ? v0 : v1;
        double s = (upper ? v1 : v0) + __shfl_xor_sync(0xffffffffu, send, 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
    };
    // Two sums over all items, one value each a thread and round of 512 items
    // (v0, v1 by item), as grid_reduce<2> forms them over blocks of 64 threads:
    // publish the groups' sums; after a barrier, final_sums leaves the totals
    // in lane 0 of warp 0.
    auto publish2 = [&](int t, double v0, double v1) {
        const double v = pair_sum(v0, v1);
        if ((lane & 15) == 0) s_w[lane >> 4][warp] = v;
        __syncthreads();
        if ((tid & 63) < 2 && t - (tid & 63) < items) {
            const int q = tid & 63, w = warp & ~1;
            __stcg(p.parts_b + 2 * (size_t)(vb + (t >> 6)) + q, s_w[q][w] + s_w[q][w + 1]);
        }
        __syncthreads();
    };
    auto final_sums = [&](double& o0, double& o1) {
        if (warp < 2) {
            double a0 = 0.0, a1 = 0.0;
            for (int g = tid; g < nvb; g += 64) {
                const double2 q = __ldcg(reinterpret_cast<const double2*>(p.parts_b) + g);
                a0 += q.x;
                a1 += q.y;
            }
            __syncwarp();
            const double a = pair_sum(a0, a1);
            if ((lane & 15) == 0) s_w[lane >> 4][warp] = a;
        }
        __syncthreads();
        o0 = tid == 0 ? s_w[0][0] + s_w[0][1] : 0.0;
        o1 = tid == 0 ? s_w[1][0] + s_w[1][1] : 0.0;
    };

    // ---- r = sign rhs, z = r / diag(H) ----
    if (b == 0 && tid == 0) p.st->cg_done = 0;
    for (int t0 = 0; t0 < items; t0 += kResThreads) {
        const int t = t0 + tid;
        double v0 = 0.0, v1 = 0.0;
        if (t < items && i0 + t < N) {
            const double ri = p.sign * p.rhs[i0 + t], h = p.hdiag[i0 + t];
            const double zi = ri / h;
            s_h[t] = h;
            s_r[t] = ri;
            s_z[t] = zi;
            s_x[t] = 0.0;
            __stcg(p.z + i0 + t, zi);
            v0 = ri * zi;
            v1 = ri * ri;
        }
        publish2(t, v0, v1);
    }
    bar.arrive();
    if (!bar.wait()) {
        drain();
        return;
    }
    const int cg_max = p.st->cg_max;
    double rz, rr, thresh2 = 0.0;  // thread 0
    final_sums(rz, rr);
    if (tid == 0) {
        thresh2 = fmax(p.tol * p.tol * rr, 2.2250738585072014e-308);
        s_stop = rr == 0.0 || rr < thresh2 ? 1 : 0;
        s_sc = 0.0;
    }
    __syncthreads();
    int it = 0;

#pragma unroll 1
    while (!s_stop) {
        const double beta = s_sc;
        const double* p_old = p.p + (size_t)(it & 1) * N;
        double* p_new = p.p + (size_t)((it + 1) & 1) * N;
        // the own items of the direction
        for (int t = tid; t < items; t += kResThreads) {
            if (i0 + t >= N) break;
            const double pv = it == 0 ? s_z[t] : fma(beta, s_p[t], s_z[t]);
            s_p[t] = pv;
            __stcg(p_new + i0 + t, pv);
        }
        auto direction = [&](int at) {
            const double z = __ldcg(p.z + at);
            return it == 0 ? z : fma(beta, __ldcg(p_old + at), z);
        };
        int cx_slab = -1;  // whose entries s_cx holds
#pragma unroll 1
        for (int k = 0; k < my_tiles; ++k) {
            const int t = tile_at(it, k);
            const int slab = t % nslabs, rb = t / nslabs;
            const int c0 = slab * CW, r0 = rb * kRB;
            const int seg = (int)((p.ldt - c0) < CW ? (p.ldt - c0) : CW);
            if (slab != cx_slab) {
                cx_slab = slab;
                for (int c = gt; c < CW; c += GT)
                    s_cx[c] = c0 + c < m ? (float)direction(n + c0 + c) : 0.f;
            }
            if (gt < kRB) s_rx[gt] = r0 + gt < n ? (float)direction(r0 + gt) : 0.f;
            group_sync();
            float cx[16], cacc[16], rowv[RPW];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const float4 c = *reinterpret_cast<const float4*>(s_cx + (v * 32 + lane) * 4);
                cx[4 * v] = c.x;
                cx[4 * v + 1] = c.y;
                cx[4 * v + 2] = c.z;
                cx[4 * v + 3] = c.w;
            }
#pragma unroll
            for (int q = 0; q < 16; ++q) cacc[q] = 0.f;
#pragma unroll
            for (int u = 0; u < RPW; ++u) {
                rowv[u] = 0.f;
                asm volatile("cp.async.wait_group %0;" ::"n"(NS - 1) : "memory");
                float4 mv[4];
                const bool have = r0 + wg * RPW + u < n;
                const float* buf = ring + ((pq - NS) % NS) * CW;
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const int off = (v * 32 + lane) * 4;
                    mv[v] = have && off < seg ? *reinterpret_cast<const float4*>(buf + off)
                                              : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                issue();
                if (have) {
                    const float rx = s_rx[wg * RPW + u];
                    const float2 rx2 = make_float2(rx, rx);
                    float2 racc = make_float2(0.f, 0.f);
#pragma unroll
                    for (int q = 0; q < 16; q += 2) {
                        const float4 w = mv[q / 4];
                        const float2 T2 = q % 4 == 0 ? make_float2(w.x, w.y) : make_float2(w.z, w.w);
                        racc = __ffma2_rn(T2, make_float2(cx[q], cx[q + 1]), racc);
                        const float2 c = __ffma2_rn(T2, rx2, make_float2(cacc[q], cacc[q + 1]));
                        cacc[q] = c.x;
                        cacc[q + 1] = c.y;
                    }
                    rowv[u] = racc.x + racc.y;
                }
            }
            // row sums: lane 4 r holds row r of the warp's eight
#pragma unroll
            for (int lvl = 0; lvl < 3; ++lvl) {
                const int o = 16 >> lvl, K = RPW >> lvl;
                const bool upper = (lane & o) != 0;
#pragma unroll
                for (int q = 0; q < K / 2; ++q) {
                    const float send = upper ? rowv[q] : rowv[q + K / 2];
                    const float keep = upper ? rowv[q + K / 2] : rowv[q];
                    rowv[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            float rsum = rowv[0];
            rsum += __shfl_xor_sync(0xffffffffu, rsum, 2);
            rsum += __shfl_xor_sync(0xffffffffu, rsum, 1);
            if ((lane & 3) == 0) {
                const int r = wg * RPW + (lane >> 2);
                if (r0 + r < n) __stcg(p.rowpart + (size_t)slab * n + r0 + r, rsum);
            }
            // column sums of the group's warps, in the dense pass's order
            if (wg >= 4) {
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    *reinterpret_cast<float4*>(s_cred + (wg - 4) * CW + (v * 32 + lane) * 4) =
                        make_float4(cacc[4 * v], cacc[4 * v + 1], cacc[4 * v + 2], cacc[4 * v + 3]);
            }
            group_sync();
            if (wg < 4) {
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    float4* slot = reinterpret_cast<float4*>(s_cred + wg * CW + (v * 32 + lane) * 4);
                    float4 w = *slot;
                    w.x += cacc[4 * v];
                    w.y += cacc[4 * v + 1];
                    w.z += cacc[4 * v + 2];
                    w.w += cacc[4 * v + 3];
                    *slot = w;
                }
            }
            group_sync();
            for (int c = gt; c < CW; c += GT) {
                if (c0 + c >= m) continue;
                float s = s_cred[c];
                s += s_cred[CW + c];
                s += s_cred[2 * CW + c];
                s += s_cred[3 * CW + c];
                __stcg(p.colpart + (size_t)rb * m + c0 + c, s);
            }
            group_sync();
        }
        bar.arrive();
        if (!bar.wait()) {
            drain();
            return;
        }
        // ---- y = H p of 32-item groups: eight warps merge a group's sums ----
        for (int g0 = ab; g0 < ae; g0 += kCg32Groups) {
            const int g = g0 + group;
            const bool row = g < nar;
            const int item = (row ? g : g - nar) * 32 + lane;
            const bool ok = g < ae && (row ? item < n : item < m - 1);
            const int at = row ? item : n + item;
            const bool have = g < ae && (row ? item < n : item < m);
            // under way while the partials are added
            double pv = 0.0, hd = 0.0;
            if (wg == 0 && have) {
                pv = __ldcg(p_new + at);
                hd = __ldg(p.hdiag + at);
            }
            float sum = 0.f, err = 0.f;
            if (ok) {
                const float* src = row ? p.rowpart + item : p.colpart + item;
                const int cnt = row ? nslabs : nrb;
                const size_t stride = row ? (size_t)n : (size_t)m;
                for (int q = wg; q < cnt; q += 64) {
                    float v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        v[e] = q + 8 * e < cnt ? __ldcg(src + (size_t)(q + 8 * e) * stride) : 0.f;
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        if (q + 8 * e < cnt) {
                            float t, er;
                            two_sum_f(sum, v[e], t, er);
                            sum = t;
                            err += er;
                        }
                    }
                }
            }
            s_m[group][wg][lane] = make_float2(sum, err);
            group_sync();
            if (wg == 0) {
                float ss = 0.f, cc = 0.f;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float2 v = s_m[group][q][lane];
                    float t, er;
                    two_sum_f(ss, v.x, t, er);
                    ss = t;
                    cc += er + v.y;
                }
                const double tp = (double)ss + (double)cc;
                double py = 0.0;
                if (have) {
                    const double y = ok ? fma(hd, pv, tp / p.reg) : 0.0;
                    __stcg(p.y + at, y);
                    py = pv * y;
                }
                __syncwarp();
                py = warp_sum_d(py);
                if (lane == 0 && g < ae) __stcg(p.parts_a + g, py);
            }
            group_sync();
        }
        bar.arrive();
        if (!bar.wait()) {
            drain();
            return;
        }
        // the first round's y, under way while alpha is formed
        double y0 = 0.0;
        if (tid < items && i0 + tid < N) y0 = __ldcg(p.y + i0 + tid);
        if (warp == 0) {
            double s = 0.0;
            for (int g = lane; g < nab; g += 32 * 8) {
                double v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    v[e] = g + 32 * e < nab ? __ldcg(p.parts_a + g + 32 * e) : 0.0;
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (g + 32 * e < nab) s += v[e];
            }
            __syncwarp();
            s = warp_sum_d(s);
            if (lane == 0) s_sc = rz / s;
        }
        __syncthreads();
        // ---- x, r, z of the own items ----
        {
            const double alpha = s_sc;
            for (int t0 = 0; t0 < items; t0 += kResThreads) {
                const int t = t0 + tid;
                double v0 = 0.0, v1 = 0.0;
                if (t < items && i0 + t < N) {
                    s_x[t] = fma(alpha, s_p[t], s_x[t]);
                    const double yv = t0 == 0 ? y0 : __ldcg(p.y + i0 + t);
                    const double ri = fma(-alpha, yv, s_r[t]);
                    s_r[t] = ri;
                    const double zi = ri / s_h[t];
                    s_z[t] = zi;
                    __stcg(p.z + i0 + t, zi);
                    v0 = ri * zi;
                    v1 = ri * ri;
                }
                publish2(t, v0, v1);
            }
        }
        bar.arrive();
        if (!bar.wait()) {
            drain();
            return;
        }
        ++it;
        double rzn;
        final_sums(rzn, rr);
        if (tid == 0) {
            if (rr < thresh2 || it >= cg_max || !(rr == rr)) s_stop = 1;
            s_sc = rzn / rz;
            rz = rzn;
        }
        __syncthreads();
    }
    drain();
    for (int t = tid; t < items; t += kResThreads)
        if (i0 + t < N) p.x[i0 + t] = s_x[t];
    if (b == 0 && tid == 0) {
        p.st->cg_it = it;
        p.st->cg_done = 1;
    }
}

// T_ij in FP32 as the mixed passes form it (exact hi sum, scaled low parts, one
// FMA, ex2.approx), zero in the padding columns; *zero = 0.
__global__ void __launch_bounds__(256) k_plan32(const float* __restrict__ M, long long ldm, int n,
                                                int m, const float4* __restrict__ rs,
                                                const float4* __restrict__ cs, float kexp,
                                                float* T, unsigned* zero) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *zero = 0u;
    const int per_row = (int)(ldm >> 2);
    const int rows_step = gridDim.y;
    const int v = blockIdx.x * 256 + threadIdx.x;
    if (v >= per_row) return;
    float hi[4], lo[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float4 c = 4 * v + e < m ? cs[4 * v + e] : make_float4(-INFINITY, 0.f, 0.f, 0.f);
        hi[e] = c.x;
        lo[e] = __fmul_rn(c.y, kexp);
    }
    for (int i = blockIdx.y; i < n; i += rows_step) {
        const float4 r = rs[i];
        const float rl = __fmul_rn(r.y, kexp);
        const float4 c = __ldcs(reinterpret_cast<const float4*>(M + (long long)i * ldm) + v);
        const float a[4] = {c.x, c.y, c.z, c.w};
        float o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float z = fmaf((r.x + hi[e]) - a[e], kexp, __fadd_rn(rl, lo[e]));
            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(o[e]) : "f"(z));
        }
        reinterpret_cast<float4*>(T + (long long)i * ldm)[v] = make_float4(o[0], o[1], o[2], o[3]);
    }
}

// One CG system after another on the stored plan of a problem.
struct PlanCg32 {
    bool ok = false, cluster = false;
    int blocks = 0;
    size_t smem = 0;
    DBuf<float> T;
    DBuf<double> buf;
    PlanCg32Params p{};
    regot_dproblem* P = nullptr;

    void init(regot_dproblem* prob, ErotOps& ops, NewtonState* S, cudaStream_t st) {
        P = prob;
        const int n = P->n, m = P->m, N = n + m;
        if ((double)n * P->ldm * sizeof(float) > kPlanMaxBytes) return;
        const long long tiles = (long long)cdiv(m, kCg32CW) * cdiv(n, kRB);
        // one cluster where it holds all tiles at once (two a block): against the
        // grid 4.76 and 5.23 ms at 30 x 20, 5.71 and 6.68 at 300 x 260, 4.21 and 4.25
        // at 1000 x 1000 (32 tiles); with two rounds of tiles 6.00 and 4.49 at 1024 x
        // 1500 (sinkhorn_newton, mixed)
        cluster = tiles <= 16 * kCg32Groups &&
                  resident_cluster(k_plan_cg32<true>, 0, smem = plan_cg32_smem(N, 16));
        blocks = 16;
        if (!cluster) {
            const long long want = std::max<long long>((tiles + kCg32Groups - 1) / kCg32Groups,
                                                       cdiv(N, 32 * kCg32Groups));
            blocks = (int)std::min<long long>(want, device_sm_count());
            smem = plan_cg32_smem(N, blocks);
            if (!resident_grid(k_plan_cg32<false>, smem)) return;
        }
        try {
            T.alloc((size_t)n * P->ldm, st);
            buf.alloc(4 * (size_t)N + (size_t)(cdiv(n, 32) + cdiv(m, 32)) + 2 * (size_t)cdiv(N, 64) + 4,
                      st);
        } catch (const Error&) {  // no room for a second matrix
            cudaGetLastError();
            T.release();
            return;
        }
        p.T = T.get();
        p.ldt = P->ldm;
        p.n = n;
        p.m = m;
        p.reg = ops.reg();
        p.z = buf.get();  // z, p (two), y: 4 N doubles
        p.p = p.z + N;
        p.y = p.p + 2 * (size_t)N;
        p.parts_b = p.y + N;  // read in pairs: 4 N doubles from the start, so on 16 bytes
        p.parts_a = p.parts_b + 2 * (size_t)cdiv(N, 64);
        p.count = reinterpret_cast<unsigned*>(p.parts_a + cdiv(n, 32) + cdiv(m, 32));
        p.rowpart = reinterpret_cast<float*>(ops.buf().rowpart.get());
        p.colpart = reinterpret_cast<float*>(ops.buf().colpart.get());
        p.err = &S->err;
        p.polls = grid_polls();
        p.st = S;
        ok = true;
    }
    // Gives the memory back, for the plan's output; nothing can be solved any more.
    void release() {
        T.release();
        ok = false;
    }
    // H x = sign rhs at the duals split in rs, cs (H's diagonal given).
    void solve(const float4* rs, const float4* cs, const double* rhs, double sign,
               const double* hdiag, double tol, double* x, cudaStream_t st) {
        const int gx = cdiv(P->ldm / 4, 256);
        const int gy = std::max(1, std::min(p.n, 8 * device_sm_count() / gx));
        k_plan32<<<dim3(gx, std::min(gy, 65535)), 256, 0, st>>>(
            static_cast<const float*>(P->M), P->ldm, p.n, p.m, rs, cs,
            (float)(1.4426950408889634 / p.reg), T.get(), p.count);
        count_launch();
        REGOT_CHECK_LAUNCH();
        p.rhs = rhs;
        p.sign = sign;
        p.hdiag = hdiag;
        p.tol = tol;
        p.x = x;
        if (cluster) launch_resident(k_plan_cg32<true>, true, blocks, smem, st, p);
        else launch_resident(k_plan_cg32<false>, false, blocks, smem, st, p);
    }
};

}  // namespace
}  // namespace regot
