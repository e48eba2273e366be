// FP64 Newton systems on a stored plan (included by erot_newton.cu).
//
// T = T(gamma) is formed once per Newton iterate (launch_plan64) and kept;
// one cooperative launch then evaluates the gradient and Hessian diagonal
// (T 1, T' 1) and runs the preconditioned conjugate gradients, every product
// H p as two matrix-vector products with T (two FP64 multiply-adds an entry,
// where a dense pass recomputes an exponential of about twenty FP64
// operations). Blocks own rows and columns as in bcd_scaled.cuh. A CG step has
// two barriers:
//   * p'H p = sum h p^2 + (2 / reg) p_alpha' (T p_beta) needs the row products
//     only, so the step length is known after the barrier that the column
//     products need anyway;
//   * every block holds p_beta whole and updates it itself from the published
//     z_beta, so the new direction needs no third barrier.
#pragma once

#include "erot_ops.cuh"
#include "newton_state.h"
#include "resident.cuh"

namespace regot {
namespace {

struct PlanCgParams {
    const double* T;
    long long ldk;
    int n, m;
    const double *a, *b, *gamma;  // gradient mode (rhs null): H x = -g
    const double* rhs;            // else H x = rhs
    double reg, grad_tol, cg_tol;
    double *g, *x;    // gradient (gradient mode) and solution, n + m (last 0)
    double* part;     // [G][ldk]
    double* zbuf;     // [ldk]
    double* red;      // [3][G][2]: pairs of block sums
    unsigned* count;
    int* err;        // set when a barrier gives up
    unsigned polls;  // before it does
    NewtonState* st;
    double *hobj, *hmar, *htime;  // gradient mode: this iterate's record (or null)
    double* hdiag;                // gradient alone: diag(H) [n + m] out, no solve
};

inline size_t plan_cg_smem(int n, long long ldk, int m, int G) {
    const size_t R = (size_t)(n + G - 1) / G + 1, C = (size_t)(m + G - 1) / G + 1;
    return sizeof(double) * ((size_t)ldk + 2 * kResThreads + 2 * R + rows_part_size((int)R) +
                             7 * (R + C) + 4 * kResWarps);
}

template <bool CLUSTER>
__global__ void __launch_bounds__(kResThreads, 1) k_plan_cg(const PlanCgParams p) {
    extern __shared__ __align__(16) double s_dyn_n[];
    __shared__ int s_ok, s_stop;
    __shared__ double s_sc;  // beta, then alpha, of the step
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.x, G = gridDim.x;
    const int n = p.n, m = p.m;
    const long long ldk = p.ldk;
    const int r0 = own_begin(n, b, G), R = own_begin(n, b + 1, G) - r0;
    const int j0 = own_begin(m, b, G), j1 = own_begin(m, b + 1, G), C = j1 - j0;
    const int Rm = (n + G - 1) / G + 1, Cm = (m + G - 1) / G + 1, Im = Rm + Cm;
    double* s_x = s_dyn_n;                  // [ldk] p_beta (ones at first)
    double* s_q = s_x + ldk;              // [2 kResThreads]
    double* s_u = s_q + 2 * kResThreads;  // [Rm] p_alpha of the own rows (ones at first)
    double* s_sum = s_u + Rm;             // [Rm]
    double* s_part = s_sum + Rm;
    // own items: rows 0 .. R - 1, columns R .. R + C - 1
    double* s_h = s_part + rows_part_size(Rm);  // diag(H)
    double* s_ih = s_h + Im;                    // 1 / diag(H)
    double* s_p = s_ih + Im;
    double* s_xs = s_p + Im;  // the solution
    double* s_r = s_xs + Im;
    double* s_z = s_r + Im;
    double* s_y = s_z + Im;   // (T'p)_j of the own columns, at R + j
    double* s_w = s_y + Im;   // [2][kResWarps]
    GridBarrier<CLUSTER> bar(p.count, p.err, p.polls, &s_ok);
    const double reg = p.reg;
    const int S = row_segments((int)(ldk >> 1), R);
    const int items = R + C, iwarps = (items + 31) / 32 < kResWarps ? (items + 31) / 32 : kResWarps;

    // Pairs (v0, v1) summed over the block's item threads into red[slot][b]:
    // called by all threads (the warps without items only synchronise). A slot is
    // written again only behind a barrier of all blocks that follows its last
    // total(): slot 0 of a step is written in the phase after the residual's
    // totals are read, so those (of the first residual too) are in slot 1.
    auto publish = [&](int slot, double v0, double v1) {
        if (warp < iwarps) {
            const bool upper = (lane & 16) != 0;
            const double send = upper ? v0 : v1;
            double s = (upper ? v1 : v0) + __shfl_xor_sync(0xffffffffu, send, 16);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if ((lane & 15) == 0) s_w[(lane >> 4) * kResWarps + warp] = s;
        }
        __syncthreads();
        if (tid < 2) {
            double s = iwarps > 0 ? s_w[tid * kResWarps] : 0.0;
            for (int w = 1; w < iwarps; ++w) s += s_w[tid * kResWarps + w];
            __stcg(p.red + ((size_t)slot * G + b) * 2 + tid, s);
        }
    };
    // After a barrier, in one warp: the totals over all blocks (the same bits
    // in every block).
    auto total = [&](int slot) {
        return warp_sum_pairs(reinterpret_cast<const double2*>(p.red) + (size_t)slot * G, G);
    };
    // Beside it, in the other warps: the own columns' products.
    auto merge = [&]() {
        merge_columns(p.part, ldk, G, j0, j1, warp - 1, kResWarps - 1,
                      [&](int j, double c) { s_y[R + j - j0] = c; });
    };
    auto publish_z = [&]() {
        for (int c = tid; c < C; c += kResThreads) __stcg(p.zbuf + j0 + c, s_z[R + c]);
    };

    if (b == 0 && tid == 0) p.st->cg_done = 0;
    // ---- row and column sums: gradient, objective, diag(H), first residual ----
    for (int j = tid; j < ldk; j += kResThreads) s_x[j] = j < m ? 1.0 : 0.0;
    for (int r = tid; r < R; r += kResThreads) s_u[r] = 1.0;
    __syncthreads();
    rows_dot(p.T, ldk, r0, R, S, s_x, s_part, s_sum);
    cols_dot(p.T, ldk, r0, R, s_u, p.part + (long long)b * ldk, s_q);
    bar.arrive();
    if (!bar.wait()) return;
    if (warp > 0) merge();
    __syncthreads();
    {
        double v[4] = {0.0, 0.0, 0.0, 0.0};  // rr, rz, sum r, sum gamma (a, b)
        for (int t = tid; t < items; t += kResThreads) {
            const bool row = t < R;
            const int gi = row ? r0 + t : n + j0 + (t - R);
            const bool last = gi == n + m - 1;
            const double s = row ? s_sum[t] : s_y[t];
            double ri = 0.0;
            if (p.rhs) {
                ri = last ? 0.0 : p.rhs[gi];
            } else if (!last) {
                const double w = row ? p.a[gi] : p.b[gi - n];
                const double gr = s - w;
                p.g[gi] = gr;
                ri = -gr;
                if (row) v[2] += s;
                v[3] = fma(p.gamma[gi], w, v[3]);
            } else {
                p.g[gi] = 0.0;
            }
            const double h = last ? 1.0 : s / reg;
            const double ih = 1.0 / h, z = ri * ih;
            s_h[t] = h;
            s_ih[t] = ih;
            if (p.hdiag) p.hdiag[gi] = h;
            s_r[t] = ri;
            s_z[t] = z;
            s_p[t] = z;
            s_xs[t] = 0.0;
            v[0] = fma(ri, ri, v[0]);
            v[1] = fma(ri, z, v[1]);
        }
        __syncthreads();
        publish_z();
        publish(1, v[0], v[1]);
        __syncthreads();
        publish(2, v[2], v[3]);
    }
    bar.arrive();
    if (!bar.wait()) return;
    // scalars of the iteration: lane 0 of warp 0, broadcast through s_sc
    double rz = 0.0, thresh2 = 0.0;
    const int cg_max = p.st->cg_max;
    if (warp == 0) {
        const double2 q1 = total(1), q2 = total(2);
        const double rr0 = q1.x, sr = q2.x, sg = q2.y;
        rz = q1.y;
        if (lane == 0) {
            thresh2 = fmax(p.cg_tol * p.cg_tol * rr0, 2.2250738585072014e-308);
            int stop = rr0 == 0.0 || rr0 < thresh2 ? 1 : 0;
            if (!p.rhs) {
                const double f = reg * sr - sg, gnorm = sqrt(rr0);
                // the caller stops here
                if (gnorm < p.grad_tol || !isfinite(f) || p.hdiag) stop = 2;
                if (b == 0) {
                    p.st->f = f;
                    p.st->gnorm = gnorm;
                    if (p.hobj) {
                        *p.hobj = f;
                        *p.hmar = gnorm;
                        *p.htime = (double)(globaltimer_ns() - p.st->t0) * 1e-6;
                    }
                    if (stop == 2) p.st->cg_done = 2;
                }
            }
            s_stop = stop;
            s_sc = 0.0;
        }
        __syncwarp();
    }
    __syncthreads();
    if (s_stop == 2) return;
    const double inv_reg = 1.0 / reg;
    int it = 0;

#pragma unroll 1
    while (!s_stop) {
        // the direction: p_beta whole, p_alpha of the own rows
        const double beta = s_sc;
        for (int j = tid; j < m - 1; j += kResThreads) {
            const double z = __ldcg(p.zbuf + j);
            s_x[j] = it == 0 ? z : fma(beta, s_x[j], z);
        }
        if (it == 0) {
            for (int j = m - 1 + tid; j < ldk; j += kResThreads) s_x[j] = 0.0;
        } else {
            for (int t = tid; t < items; t += kResThreads) s_p[t] = fma(beta, s_p[t], s_z[t]);
        }
        __syncthreads();
        rows_dot(p.T, ldk, r0, R, S, s_x, s_part, s_sum);
        __syncthreads();
        {
            double v = 0.0;
            for (int t = tid; t < items; t += kResThreads) {
                const double pt = s_p[t];
                double y = s_h[t] * pt;
                if (t < R) y = fma(2.0 * inv_reg, s_sum[t], y);
                v = fma(pt, y, v);
            }
            __syncwarp();
            publish(0, v, 0.0);
        }
        cols_dot(p.T, ldk, r0, R, s_p, p.part + (long long)b * ldk, s_q);
        bar.arrive();
        if (!bar.wait()) return;
        if (warp == 0) {
            const double pap = total(0).x;
            if (lane == 0) s_sc = rz / pap;
            __syncwarp();
        } else {
            merge();
        }
        __syncthreads();
        {
            const double alpha = s_sc;
            double v[2] = {0.0, 0.0};
            for (int t = tid; t < items; t += kResThreads) {
                const bool last = t >= R && j0 + (t - R) == m - 1;
                const double tp = t < R ? s_sum[t] : s_y[t];
                const double pt = s_p[t];
                const double y = last ? 0.0 : fma(s_h[t], pt, tp * inv_reg);
                s_xs[t] = fma(alpha, pt, s_xs[t]);
                const double ri = fma(-alpha, y, s_r[t]);
                s_r[t] = ri;
                const double z = ri * s_ih[t];
                s_z[t] = z;
                v[0] = fma(ri, ri, v[0]);
                v[1] = fma(ri, z, v[1]);
            }
            __syncthreads();
            publish_z();
            publish(1, v[0], v[1]);
        }
        bar.arrive();
        if (!bar.wait()) return;
        ++it;
        if (warp == 0) {
            const double2 q = total(1);
            const double rr = q.x, rzn = q.y;
            if (lane == 0) {
                s_sc = rzn / rz;
                rz = rzn;
                if (rr < thresh2 || it >= cg_max || !(rr == rr)) s_stop = 1;
            }
            __syncwarp();
        }
        __syncthreads();
    }
    for (int t = tid; t < items; t += kResThreads) {
        const int gi = t < R ? r0 + t : n + j0 + (t - R);
        p.x[gi] = s_xs[t];
    }
    if (b == 0 && tid == 0) {
        p.st->cg_it = it;
        p.st->cg_done = 1;
    }
}

// totals[s] = sum_ij T_ij phi(steps[s] w_ij), w = (d_i + d_j) / reg,
// phi(x) = e^x - 1 - x, for the line search; FP64 issue bounds it (about twenty
// instructions an entry and step).
struct PlanLsParams {
    const double* T;
    long long ldk;
    int n, m;
    const double* d;  // n + m, last 0
    double inv_reg;
    double steps[4];
    int nsteps;
    double* parts;  // [grid][4]
    double* out;    // [4]
    NewtonState* st;
    int skip;       // nothing to do where the last gradient stopped the solve
    Exp64 ex;
};

__global__ void __launch_bounds__(256) k_plan_ls(const PlanLsParams p) {
    if (p.skip && p.st->cg_done == 2) return;  // the gradient already met the tolerance
    const unsigned per_row = (unsigned)(p.ldk >> 1);
    const long long total = (long long)p.n * per_row;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long i = total <= 0xffffffffLL ? (long long)((unsigned)t / per_row) : t / per_row;
        const int j = 2 * (int)(t - i * per_row);
        const double2 q = __ldg(reinterpret_cast<const double2*>(p.T + i * p.ldk + j));
        const double di = p.d[i];
        const double w0 = (di + p.d[p.n + j]) * p.inv_reg;
        const bool two = j + 1 < p.m;
        const double w1 = two ? (di + p.d[p.n + j + 1]) * p.inv_reg : 0.0;
#pragma unroll 1
        for (int s = 0; s < p.nsteps; ++s) {
            double a = q.x * phi_tabled(p.steps[s] * w0, p.ex);
            if (two) a = fma(q.y, phi_tabled(p.steps[s] * w1, p.ex), a);
            if (s == 0) v[0] += a;
            else if (s == 1) v[1] += a;
            else if (s == 2) v[2] += a;
            else v[3] += a;
        }
    }
    double out[4];
    if (grid_reduce<4>(v, p.parts, &p.st->counter, out)) {
        for (int s = 0; s < 4; ++s) p.out[s] = out[s];
    }
}

// Launch shape, as in bcd_scaled.cuh.
struct PlanCgLaunch {
    bool ok = false, cluster = false;
    int blocks = 0;
    size_t smem = 0;
    long long ldk = 0;
    DBuf<double> T, part, buf, lsparts;
    PlanCgParams p{};

    // Room and launch for n x m, or ok = false.
    void init(regot_dproblem* P, double reg, NewtonState* S, cudaStream_t st) {
        const int n = P->n, m = P->m;
        ldk = ((long long)m + 1) & ~1LL;
        if ((double)n * ldk * sizeof(double) > kPlanMaxBytes) return;
        cluster = resident_cluster(k_plan_cg<true>, (long long)n * m, smem = plan_cg_smem(n, ldk, m, 16));
        blocks = 16;
        if (!cluster) {
            blocks = n < device_sm_count() ? n : device_sm_count();
            smem = plan_cg_smem(n, ldk, m, blocks);
            if (!resident_grid(k_plan_cg<false>, smem)) return;
        }
        try {
            T.alloc((size_t)n * ldk, st);
            part.alloc((size_t)blocks * ldk, st);
            buf.alloc((size_t)ldk + 8 * (size_t)blocks + 8, st);
            lsparts.alloc(4 * (size_t)(8 * device_sm_count()), st);
        } catch (const Error&) {  // no room for a second matrix
            cudaGetLastError();
            T.release();
            return;
        }
        p.T = T.get();
        p.ldk = ldk;
        p.n = n;
        p.m = m;
        p.a = P->a;
        p.b = P->b;
        p.reg = reg;
        p.part = part.get();
        p.red = buf.get();
        p.zbuf = p.red + 8 * (size_t)blocks;
        p.count = reinterpret_cast<unsigned*>(p.zbuf + ldk);
        p.err = &S->err;
        p.polls = grid_polls();
        p.st = S;
        ok = true;
    }
    // Gives the memory back, for the plan's output; nothing can be solved any more.
    void release() {
        T.release();
        part.release();
        ok = false;
    }
    // Blocks of the line search: at most eight an SM, with the items dealt out
    // evenly over their rounds.
    int ls_blocks() const {
        const long long need = ((long long)p.n * (ldk / 2) + 255) / 256, cap = 8LL * device_sm_count();
        const long long rounds = (need + cap - 1) / cap;
        return (int)((need + rounds - 1) / rounds);
    }
    void form_plan(regot_dproblem* P, const double* gamma, cudaStream_t st) {
        launch_plan64(static_cast<const double*>(P->M), P->ldm, p.n, p.m, gamma, gamma + p.n, p.reg,
                      T.get(), ldk, p.count, st);
    }
    // The gradient and the CG solve, right after form_plan.
    void solve(cudaStream_t st) {
        if (cluster) launch_resident(k_plan_cg<true>, true, blocks, smem, st, p);
        else launch_resident(k_plan_cg<false>, false, blocks, smem, st, p);
    }
    // The gradient, objective and diag(H) alone, right after form_plan.
    void gradient(const double* gamma, double* g, double* h, cudaStream_t st) {
        p.gamma = gamma;
        p.rhs = nullptr;
        p.g = g;
        p.hdiag = h;
        solve(st);
    }
    void line_search(const double* d, const double* steps, int nsteps, double* out, bool skip,
                     cudaStream_t st) {
        PlanLsParams q{};
        q.T = p.T;
        q.ldk = ldk;
        q.n = p.n;
        q.m = p.m;
        q.d = d;
        q.inv_reg = 1.0 / p.reg;
        for (int s = 0; s < nsteps; ++s) q.steps[s] = steps[s];
        q.nsteps = nsteps;
        q.parts = lsparts.get();
        q.out = out;
        q.st = p.st;
        q.skip = skip ? 1 : 0;
        q.ex = exp64_for(p.reg);
        k_plan_ls<<<ls_blocks(), 256, 0, st>>>(q);
        count_launch();
        REGOT_CHECK_LAUNCH();
    }
};

}  // namespace
}  // namespace regot
