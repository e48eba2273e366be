// FP64 Schur-complement CG of the sparsified Hessian in one cooperative launch
// (included by erot_ssns.cu): the direction d with (H_s + shift) d = -g and its
// products g'd, d'H_s d.
//
// Before: five kernels a CG step in a captured graph, 38 us a step at
// 1000 x 800 where the sparse products themselves take a few. Here blocks own
// rows and columns, a warp takes a row's (column's) stored entries, and a step
// has two barriers: after the row products, whose published u = (S p) / (h1 +
// shift) every block then holds whole for its columns, and after the vector
// updates. As in newton_plan.cuh the step length is known at the first,
//     p' Delta p = sum (h2 + shift) p^2 - sum (S p) u,
// and every block updates its own copy of the direction from the published
// residual. All arithmetic is FP64.
#pragma once

#include "resident.cuh"

namespace regot {
namespace {

struct SchurCgParams {
    Sparse S;
    const double *gsrc;      // right-hand side -gsrc
    const double *g, *h;     // gradient (for g'd), (h1, h2)
    double shift, tol;
    int max_it, jacobi;
    double* dir;             // d_alpha [n], d_beta~ [m - 1], 0
    double *ubuf, *wbuf;     // [n]
    double* zbuf;            // [m - 1]
    double* red;             // [2][G][2]
    unsigned* count;
    int* err;        // set when a barrier gives up
    unsigned polls;  // before it does
    SsnState* st;
};

inline size_t schur_cg_smem(int n, int m1, int G) {
    const size_t R = (size_t)(n + G - 1) / G + 1, C = (size_t)(m1 + G - 1) / G + 1;
    return sizeof(double) * ((size_t)n + m1 + 2 * R + 6 * C + 2 * kResWarps);
}

// sum_k v[k] x[c[k]] over the warp, x in shared memory; eight entries a lane
// under way.
__device__ __forceinline__ double stored_dot(const double* __restrict__ v, const int* __restrict__ c,
                                             int cnt, const double* s_x) {
    double s0 = 0.0, s1 = 0.0;
    for (int k = threadIdx.x & 31; k < cnt; k += 256) {
        double vv[8];
        int cc[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const bool in = k + 32 * e < cnt;
            vv[e] = in ? __ldg(v + k + 32 * e) : 0.0;
            cc[e] = in ? __ldg(c + k + 32 * e) : 0;
        }
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
            if (k + 32 * e < cnt) s0 = fma(vv[e], s_x[cc[e]], s0);
            if (k + 32 * e + 32 < cnt) s1 = fma(vv[e + 1], s_x[cc[e + 1]], s1);
        }
    }
    __syncwarp();
    return warp_sum_d(s0 + s1);
}

template <bool CLUSTER>
__global__ void __launch_bounds__(kResThreads, 1) k_schur_cg(const SchurCgParams p) {
    extern __shared__ __align__(16) double s_dyn_s[];
    __shared__ int s_ok, s_stop;
    __shared__ double s_sc;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.x, G = gridDim.x;
    const Sparse& S = p.S;
    const int n = S.n, m1 = S.m1;
    const int r0 = own_begin(n, b, G), R = own_begin(n, b + 1, G) - r0;
    const int j0 = own_begin(m1, b, G), C = own_begin(m1, b + 1, G) - j0;
    const int Rm = (n + G - 1) / G + 1, Cm = (m1 + G - 1) / G + 1;
    double* s_x = s_dyn_s;    // [m1] direction, at last the solution
    double* s_u = s_x + m1;   // [n]
    double* s_w = s_u + n;    // [Rm] 1 / (h1 + shift)
    double* s_s = s_w + Rm;   // [Rm] row products
    double* s_d = s_s + Rm;   // [Cm] h2 + shift
    double* s_id = s_d + Cm;  // [Cm] 1 / preconditioner
    double* s_xs = s_id + Cm;
    double* s_r = s_xs + Cm;
    double* s_z = s_r + Cm;
    double* s_c = s_z + Cm;   // column products
    double* s_v = s_c + Cm;   // [2][kResWarps]
    GridBarrier<CLUSTER> bar(p.count, p.err, p.polls, &s_ok);
    const int items = R > C ? R : C;
    const int iwarps = (items + 31) / 32 < kResWarps ? (items + 31) / 32 : kResWarps;
    const double shift = p.shift, inv_reg = S.inv_reg;

    auto publish = [&](int slot, double v0, double v1) {
        if (warp < iwarps) {
            const bool upper = (lane & 16) != 0;
            const double send = upper ? v0 : v1;
            double s = (upper ? v1 : v0) + __shfl_xor_sync(0xffffffffu, send, 16);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if ((lane & 15) == 0) s_v[(lane >> 4) * kResWarps + warp] = s;
        }
        __syncthreads();
        if (tid < 2) {
            double s = iwarps > 0 ? s_v[tid * kResWarps] : 0.0;
            for (int w = 1; w < iwarps; ++w) s += s_v[tid * kResWarps + w];
            __stcg(p.red + ((size_t)slot * G + b) * 2 + tid, s);
        }
    };
    auto total = [&](int slot) {
        return warp_sum_pairs(reinterpret_cast<const double2*>(p.red) + (size_t)slot * G, G);
    };
    auto rows = [&]() {  // s_s = S s_x (without 1 / reg)
        for (int r = warp; r < R; r += kResWarps) {
            const int i = r0 + r;
            const double s = stored_dot(static_cast<const double*>(S.rvals) + (size_t)i * S.ldr,
                                        S.rcols + (size_t)i * S.ldr, __ldg(S.rcount + i), s_x);
            if (lane == 0) s_s[r] = s;
        }
    };
    auto columns = [&](int w, int warps) {  // s_c = S' s_u (without 1 / reg)
        for (int c = w; c < C; c += warps) {
            const int j = j0 + c;
            const double s = stored_dot(static_cast<const double*>(S.cvals) + (size_t)j * S.ldc,
                                        S.crows + (size_t)j * S.ldc, __ldg(S.ccount + j), s_u);
            if (lane == 0) s_c[c] = s;
        }
    };

    // ---- right-hand side of the Schur system, its diagonal, first residual ----
    if (b == 0 && tid == 0) p.st->done = 0;
    for (int r = tid; r < R; r += kResThreads) {
        const double w = 1.0 / (p.h[r0 + r] + shift);
        s_w[r] = w;
        __stcg(p.wbuf + r0 + r, w);
        __stcg(p.ubuf + r0 + r, -p.gsrc[r0 + r] * w);
    }
    bar.arrive();
    if (!bar.wait()) return;
    for (int i = tid; i < n; i += kResThreads) s_u[i] = __ldcg(p.ubuf + i);
    __syncthreads();
    columns(warp, kResWarps);
    for (int c = warp; c < C; c += kResWarps) {
        const int j = j0 + c;
        const double dj = p.h[n + j] + shift;
        double d = 1.0;
        if (p.jacobi) {
            const double* v = static_cast<const double*>(S.cvals) + (size_t)j * S.ldc;
            const int* q = S.crows + (size_t)j * S.ldc;
            const int cnt = __ldg(S.ccount + j);
            double s = 0.0;
            for (int k = lane; k < cnt; k += 32) {
                const double sv = v[k] * inv_reg;
                s = fma(sv * sv, __ldcg(p.wbuf + q[k]), s);
            }
            __syncwarp();
            s = warp_sum_d(s);
            const double dd = dj - s;
            d = dd > 1e-3 * dj ? dd : dj;
        }
        if (lane == 0) {
            s_d[c] = dj;
            s_id[c] = 1.0 / d;
        }
    }
    __syncthreads();
    {
        double rr = 0.0, rz = 0.0;
        for (int c = tid; c < C; c += kResThreads) {
            const double r = -p.gsrc[n + j0 + c] - s_c[c] * inv_reg, z = r * s_id[c];
            s_xs[c] = 0.0;
            s_r[c] = r;
            s_z[c] = z;
            __stcg(p.zbuf + j0 + c, z);
            rr = fma(r, r, rr);
            rz = fma(r, z, rz);
        }
        __syncwarp();
        publish(0, rr, rz);
    }
    bar.arrive();
    if (!bar.wait()) return;
    double rz = 0.0, rr = 0.0, thresh2 = 0.0;  // lane 0 of warp 0
    if (warp == 0) {
        const double2 q = total(0);
        rr = q.x;
        rz = q.y;
        if (lane == 0) {
            thresh2 = fmax(p.tol * p.tol * rr, 2.2250738585072014e-308);
            s_stop = rr == 0.0 || rr < thresh2 ? 1 : 0;
            s_sc = 0.0;
        }
        __syncwarp();
    }
    __syncthreads();
    int it = 0;

#pragma unroll 1
    while (!s_stop) {
        const double beta = s_sc;
        for (int j = tid; j < m1; j += kResThreads) {
            const double z = __ldcg(p.zbuf + j);
            s_x[j] = it == 0 ? z : fma(beta, s_x[j], z);
        }
        __syncthreads();
        rows();
        __syncthreads();
        {
            double v = 0.0;
            for (int r = tid; r < R; r += kResThreads) {
                const double s = s_s[r] * inv_reg, u = s * s_w[r];
                __stcg(p.ubuf + r0 + r, u);
                v = fma(-s, u, v);
            }
            for (int c = tid; c < C; c += kResThreads) {
                const double pc = s_x[j0 + c];
                v = fma(s_d[c] * pc, pc, v);
            }
            __syncwarp();
            publish(1, v, 0.0);
        }
        bar.arrive();
        if (!bar.wait()) return;
        // the step length in warp 0 (some three thousand clocks of additions and a
        // division), u and the columns' products in the others
        if (warp == 0) {
            const double pq = total(1).x;
            if (lane == 0) s_sc = rz / pq;
            __syncwarp();
        } else {
            for (int i = tid - 32; i < n; i += kResThreads - 32) s_u[i] = __ldcg(p.ubuf + i);
            asm volatile("bar.sync 1, %0;" ::"n"(kResThreads - 32) : "memory");
            columns(warp - 1, kResWarps - 1);
        }
        __syncthreads();
        {
            const double alpha = s_sc;
            double v0 = 0.0, v1 = 0.0;
            for (int c = tid; c < C; c += kResThreads) {
                const double pc = s_x[j0 + c];
                const double q = fma(s_d[c], pc, -s_c[c] * inv_reg);
                s_xs[c] = fma(alpha, pc, s_xs[c]);
                const double r = fma(-alpha, q, s_r[c]), z = r * s_id[c];
                s_r[c] = r;
                s_z[c] = z;
                __stcg(p.zbuf + j0 + c, z);
                v0 = fma(r, r, v0);
                v1 = fma(r, z, v1);
            }
            __syncwarp();
            publish(0, v0, v1);
        }
        bar.arrive();
        if (!bar.wait()) return;
        ++it;
        if (warp == 0) {
            const double2 q = total(0);
            rr = q.x;
            if (lane == 0) {
                if (rr < thresh2 || it >= p.max_it || !(rr == rr)) s_stop = 1;
                s_sc = q.y / rz;
                rz = q.y;
            }
            __syncwarp();
        }
        __syncthreads();
    }
    // ---- d_beta whole in every block, then d_alpha = (-g - S d_beta) / (h1 + shift) ----
    for (int c = tid; c < C; c += kResThreads) __stcg(p.zbuf + j0 + c, s_xs[c]);
    bar.arrive();
    if (!bar.wait()) return;
    for (int j = tid; j < m1; j += kResThreads) s_x[j] = __ldcg(p.zbuf + j);
    __syncthreads();
    rows();
    __syncthreads();
    {
        double dhd = 0.0, gtd = 0.0;
        for (int r = tid; r < R; r += kResThreads) {
            const int i = r0 + r;
            const double s = s_s[r] * inv_reg, d = (-p.gsrc[i] - s) * s_w[r];
            p.dir[i] = d;
            dhd = fma(d, fma(p.h[i], d, 2.0 * s), dhd);
            gtd = fma(p.g[i], d, gtd);
        }
        for (int c = tid; c < C; c += kResThreads) {
            const int j = n + j0 + c;
            const double d = s_xs[c];
            p.dir[j] = d;
            dhd = fma(p.h[j] * d, d, dhd);
            gtd = fma(p.g[j], d, gtd);
        }
        __syncwarp();
        publish(1, dhd, gtd);
    }
    bar.arrive();
    if (!bar.wait()) return;
    if (b == 0 && warp == 0) {
        const double2 q = total(1);
        if (lane == 0) {
            p.st->dhd = q.x;
            p.st->gtd = q.y;
            p.st->it = it;
            p.st->rr = rr;
            p.st->done = 1;
            p.dir[n + m1] = 0.0;
        }
    }
}

struct SchurCg {
    bool ok = false, cluster = false;
    int blocks = 0;
    size_t smem = 0;
    DBuf<double> buf;
    SchurCgParams p{};

    void init(const Sparse& S, SsnState* st, cudaStream_t stream) {
        if (S.m1 <= 0) return;
        blocks = 16;
        smem = schur_cg_smem(S.n, S.m1, blocks);
        cluster = resident_cluster(k_schur_cg<true>, (long long)S.n * S.m1, smem);
        if (!cluster) {
            blocks = std::min(std::max(S.n, S.m1), device_sm_count());
            smem = schur_cg_smem(S.n, S.m1, blocks);
            if (!resident_grid(k_schur_cg<false>, smem)) return;
        }
        const size_t nn = ((size_t)S.n + 1) & ~(size_t)1, mm = ((size_t)S.m1 + 1) & ~(size_t)1;
        try {
            buf.alloc(4 * (size_t)blocks + 2 * nn + mm + 2, stream);
        } catch (const Error&) {  // no room: the captured steps
            cudaGetLastError();
            return;
        }
        p.S = S;
        p.red = buf.get();  // first: read in pairs
        p.ubuf = p.red + 4 * (size_t)blocks;
        p.wbuf = p.ubuf + nn;
        p.zbuf = p.wbuf + nn;
        p.count = reinterpret_cast<unsigned*>(p.zbuf + mm);
        p.err = &st->err;
        p.polls = grid_polls();
        p.st = st;
        ok = true;
    }
    void solve(const double* gsrc, const double* g, const double* h, double shift, double tol,
               int max_it, bool jacobi, double* dir, cudaStream_t stream) {
        p.gsrc = gsrc;
        p.g = g;
        p.h = h;
        p.shift = shift;
        p.tol = tol;
        p.max_it = max_it;
        p.jacobi = jacobi ? 1 : 0;
        p.dir = dir;
        REGOT_CUDA(cudaMemsetAsync(p.count, 0, sizeof(unsigned), stream));
        if (cluster) launch_resident(k_schur_cg<true>, true, blocks, smem, stream, p);
        else launch_resident(k_schur_cg<false>, false, blocks, smem, stream, p);
    }
};

}  // namespace
}  // namespace regot
