// FP64 sweeps of sinkhorn_bcd on a stored plan (included by erot_bcd.cu).
//
// K = T(alpha0, beta0) = exp((alpha0_i + beta0_j - M_ij) / reg) is formed
// once and kept; the iterates are scalings of it, T = diag(u) K diag(v) with
// u = exp((alpha - alpha0) / reg), v = exp((beta - beta0) / reg), so a sweep
// is two matrix-vector products
//     s = K v,  u = a / s,      c = K' u,  v = b / c
// (the stabilised scaling iteration of Schmitzer, "Stabilized sparse scaling
// algorithms for entropy regularized transport problems", SIAM J. Sci.
// Comput. 41, 2019) in place of two exponentials an entry. All arithmetic is
// FP64. The base duals move ("absorption": K is rebuilt at the current
// duals) when a scaling leaves 2^-kScaleLim .. 2^kScaleLim, so that what K
// loses to underflow stays far below the rounding of any sum.
//
// One cooperative launch runs the sweeps to the stop, one block an SM (or one
// cluster of 16 blocks for small problems, whose barrier is cheaper): blocks
// own rows; a sweep has two barriers, before and after the column merge. What
// bounds it: two FP64 multiply-adds an entry at two a clock and SM, and the
// two barriers.
#pragma once

#include "resident.cuh"

namespace regot {
namespace {

constexpr int kScaleLim = 100;   // scalings stay within 2^-100 .. 2^100
constexpr int kSumLim = 896;     // sums within 2^-896 .. 2^896 are exact enough
constexpr double kMinMarginal = 1e-150;

struct ScaledParams {
    const double* K;
    long long ldk;
    int n, m;
    const double *a, *b;
    double *alpha, *beta;  // base duals in, the last complete iterate out
    double* alpha_next;    // column sums out of range: alpha_{k+1}
    double reg, sum_a, sum_bt;
    double* part;     // [G][ldk] column products of each block
    double* vbuf;     // [ldk] column scalings
    double* red;      // [G][4]: sum g^2, sum r, sum a alpha, sum b beta~
    int* redf;        // [G] flags
    double* blast;    // beta_{m-1}
    unsigned* count;  // grid barrier
    int* err;
    BcdState* st;
    double *hobj, *hmar, *htime;
    int first_col;  // start with v = b / K'1 (beta0 is an anchor, alpha0 = 0)
};

enum : int { SC_ROW = 1, SC_COL = 2, SC_RANGE = 4 };

inline size_t scaled_smem(int n, long long ldk, int m, int G) {
    const size_t R = (size_t)(n + G - 1) / G + 1, C = (size_t)(m + G - 1) / G + 1;
    return sizeof(double) * ((size_t)ldk + 3 * R + (R > kResWarps ? R : kResWarps) +
                             2 * kResThreads + 2 * C + 2 * kResWarps);
}

template <bool CLUSTER>
__global__ void __launch_bounds__(kResThreads, 1) k_bcd_scaled(const ScaledParams p) {
    extern __shared__ __align__(16) double s_dyn[];
    __shared__ int s_ok, s_exit, s_flags, s_colflags;
    __shared__ double s_gsum, s_bl;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.x, G = gridDim.x;
    const int n = p.n, m = p.m;
    const long long ldk = p.ldk;
    const int r0 = own_begin(n, b, G), R = own_begin(n, b + 1, G) - r0;
    const int j0 = own_begin(m, b, G), j1 = own_begin(m, b + 1, G);
    const int Rm = (n + G - 1) / G + 1, Cm = (m + G - 1) / G + 1;
    double* s_v = s_dyn;               // [ldk] column scalings of the current iterate
    double* s_q = s_v + ldk;           // [2 kResThreads]
    double* s_u = s_q + 2 * kResThreads;  // [Rm] row scalings of the current iterate
    double* s_un = s_u + Rm;           // [Rm] ... of the next
    double* s_sum = s_un + Rm;         // [Rm]
    double* s_part = s_sum + Rm;       // [max(Rm, kResWarps)]
    double* s_vp = s_part + (Rm > kResWarps ? Rm : kResWarps);  // [Cm] own columns, previous v
    double* s_vn = s_vp + Cm;          // [Cm] own columns, next v
    double* s_wa = s_vn + Cm;          // [kResWarps] sums of a alpha
    double* s_wb = s_wa + kResWarps;   // [kResWarps] sums of b beta~
    GridBarrier<CLUSTER> bar(p.count, p.err, &s_ok);

    for (int j = tid; j < ldk; j += kResThreads) s_v[j] = j < m ? 1.0 : 0.0;
    for (int r = tid; r < R; r += kResThreads) s_u[r] = s_un[r] = 1.0;
    for (int j = j0 + tid; j < j1; j += kResThreads) s_vp[j - j0] = 1.0;
    if (tid < kResWarps) s_wa[tid] = s_wb[tid] = 0.0;
    if (tid == 0) {
        s_colflags = 0;
        s_exit = 0;
    }
    __syncthreads();

    // Sums of a alpha (row scalings u) and b beta~ (column scalings v) over
    // the block's own rows and columns; only warps that own any take part.
    auto alpha_terms = [&](const double* u) {
        if (warp * 32 < R) {
            double v = 0.0;
            for (int r = tid; r < R; r += kResThreads)
                v += p.a[r0 + r] * (p.alpha[r0 + r] + p.reg * log(u[r]));
            v = warp_sum_d(v);
            if (lane == 0) s_wa[warp] = v;
        }
    };
    auto beta_terms = [&](const double* v0) {  // v0[j - j0]
        if (warp * 32 < j1 - j0) {
            double v = 0.0;
            for (int j = j0 + tid; j < j1; j += kResThreads) {
                const double be = p.beta[j] + p.reg * log(v0[j - j0]);
                if (j < m - 1) v += p.b[j] * be;
                else s_bl = be;
            }
            v = warp_sum_d(v);
            if (lane == 0) s_wb[warp] = v;
        }
    };
    auto in_sum_range = [](double s) { return s > 0.0 && exponent_within(s, kSumLim); };
    // After a barrier: the own columns' new scalings into vbuf and s_vn.
    auto merge = [&](int warps) {
        merge_columns(p.part, ldk, G, j0, j1, warp, warps, [&](int j, double c) {
            const double v = p.b[j] / c;
            if (!in_sum_range(c)) atomicOr(&s_colflags, SC_COL);
            if (!exponent_within(v, kScaleLim)) atomicOr(&s_colflags, SC_RANGE);
            __stcg(p.vbuf + j, v);
            s_vn[j - j0] = v;
        });
    };
    auto stage_v = [&]() {
        for (int j = j0 + tid; j < j1; j += kResThreads) s_vp[j - j0] = s_v[j];
        __syncthreads();
        for (int j = tid; j < m; j += kResThreads) s_v[j] = __ldcg(p.vbuf + j);
    };

    if (p.first_col) {
        cols_dot(p.K, ldk, r0, R, s_un, p.part + (long long)b * ldk, s_q);
        bar.arrive();
        if (!bar.wait()) return;
        merge(kResWarps);
        // the columns' range is not checked: beta0 is an anchor, and the sums
        // are between 1 and n
        __syncthreads();
        if (tid == 0) s_colflags = 0;
        bar.arrive();
        beta_terms(s_vn);
        if (!bar.wait()) return;
        stage_v();
        __syncthreads();
    } else {
        beta_terms(s_vp);
        alpha_terms(s_u);
    }
    const double gb2_start = p.st->gb2_once;
    unsigned long long t0 = p.st->t0;
    if (p.first_col && b == 0) t0 = globaltimer_ns();
    int k = p.st->iter;
    const int max_iter = p.st->max_iter;
    const double tol = p.st->tol;
    double gb2 = gb2_start;

#pragma unroll 1
    for (;;) {
        // ---- rows: s = K v, u_next = a / s ----
        __syncthreads();
        rows_dot(p.K, ldk, r0, R, s_v, s_part, s_sum);
        __syncthreads();
        for (int r = tid; r < R; r += kResThreads) s_un[r] = p.a[r0 + r] / s_sum[r];
        __syncthreads();
        // ---- columns of the own rows, and the block's share of the sums ----
        if (warp == kResWarps - 1) {
            double g2 = 0.0, rs = 0.0;
            int f = 0;
            for (int r = lane; r < R; r += 32) {
                const double s = s_sum[r];
                const double t = s_u[r] * s;
                const double g = t - p.a[r0 + r];
                g2 = fma(g, g, g2);
                rs += t;
                if (!in_sum_range(s)) f |= SC_ROW;
                if (!exponent_within(s_u[r], kScaleLim)) f |= SC_RANGE;
            }
            f = __reduce_or_sync(0xffffffffu, f);
            g2 = warp_sum_d(g2);
            rs = warp_sum_d(rs);
            if (lane == 0) {
                double sa = 0.0, sb = 0.0;
                const int wr = (R + 31) / 32 < kResWarps ? (R + 31) / 32 : kResWarps;
                const int wc = (j1 - j0 + 31) / 32 < kResWarps ? (j1 - j0 + 31) / 32 : kResWarps;
                for (int w = 0; w < wr; ++w) sa += s_wa[w];
                for (int w = 0; w < wc; ++w) sb += s_wb[w];
                double2* red = reinterpret_cast<double2*>(p.red + 4 * (size_t)b);
                __stcg(red, make_double2(g2, rs));
                __stcg(red + 1, make_double2(sa, sb));
                __stcg(p.redf + b, f | s_colflags);
                if (j0 < m && j1 == m) __stcg(p.blast, s_bl);
            }
        }
        cols_dot(p.K, ldk, r0, R, s_un, p.part + (long long)b * ldk, s_q);
        bar.arrive();
        alpha_terms(s_un);  // for the next iterate, while the others arrive
        if (!bar.wait()) return;
        // ---- the stop, decided by every block from the same numbers ----
        if (warp == kResWarps - 1) {
            double g2 = 0.0;
            int f = 0;
            for (int g = lane; g < G; g += 32) {
                g2 += __ldcg(p.red + 4 * (size_t)g);
                f |= __ldcg(p.redf + g);
            }
            g2 = warp_sum_d(g2);
            f = __reduce_or_sync(0xffffffffu, f);
            if (lane == 0) {
                const double gnorm = sqrt(g2 + gb2);
                s_gsum = gnorm;
                s_flags = f;
                s_exit = ((f & (SC_ROW | SC_COL)) == 0 && (gnorm < tol || k >= max_iter)) ? 1
                         : f ? 2 : 0;
            }
        } else {
            if (tid == 0) s_colflags = 0;
            __syncwarp();
            // the flags of the new scalings are raised after this reset
            asm volatile("bar.sync 1, %0;" ::"n"(kResThreads - 32) : "memory");
            merge(kResWarps - 1);
        }
        __syncthreads();
        if (b == 0 && warp == 0) {
            double v[3] = {0.0, 0.0, 0.0};
            for (int g = lane; g < G; g += 32) {
                const double2 q0 = __ldcg(reinterpret_cast<const double2*>(p.red + 4 * (size_t)g));
                const double2 q1 = __ldcg(reinterpret_cast<const double2*>(p.red + 4 * (size_t)g) + 1);
                v[0] += q0.y;
                v[1] += q1.x;
                v[2] += q1.y;
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) v[q] = warp_sum_d(v[q]);
            if (lane == 0) {
                const double bl = __ldcg(p.blast);
                const int f = s_flags;
                if (!(f & (SC_ROW | SC_COL))) {
                    const double gnorm = s_gsum;
                    p.hobj[k] = p.reg * v[0] - v[1] - bl * p.sum_a - v[2] + bl * p.sum_bt;
                    p.hmar[k] = gnorm;
                    p.htime[k] = (double)(globaltimer_ns() - t0) * 1e-6;
                    p.st->hist_len = k + 1;
                    p.st->last_gnorm = gnorm;
                    p.st->gb2_once = 0.0;
                }
                if (s_exit) {
                    p.st->iter = (f & SC_COL) ? k - 1 : k;
                    p.st->bad = (f & SC_COL) ? SC_COL : (f & SC_ROW) ? SC_ROW : 0;
                    p.st->sum_bb = v[2];
                    p.st->beta_last = bl;
                    p.st->t0 = t0;
                    if (s_exit == 1) {
                        p.st->done = 1;
                        p.st->niter = k;
                    }
                }
            }
        }
        if (s_exit) break;
        gb2 = 0.0;
        bar.arrive();
        beta_terms(s_vn);
        if (!bar.wait()) return;
        stage_v();
        for (int r = tid; r < R; r += kResThreads) s_u[r] = s_un[r];
        ++k;
    }
    // ---- the last complete iterate: (alpha_k, beta_k); after column sums out
    // of range, alpha_k and beta_{k-1} ----
    const bool colbad = (s_flags & SC_COL) != 0;
    for (int r = tid; r < R; r += kResThreads) {
        const double al = p.alpha[r0 + r] + p.reg * log(s_u[r]);
        p.alpha[r0 + r] = al;
        p.alpha_next[r0 + r] = al;
    }
    for (int j = j0 + tid; j < j1; j += kResThreads)
        p.beta[j] += p.reg * log(colbad ? s_vp[j - j0] : s_v[j]);
}

// Launch shape of the sweeps: one cluster for problems whose products are
// short against a barrier of the whole grid, else a block an SM.
struct ScaledPlan {
    bool ok = false, cluster = false;
    int blocks = 0;
    size_t smem = 0;
};

inline ScaledPlan scaled_plan(int n, int m, long long ldk) {
    ScaledPlan s;
    s.blocks = 16;
    s.smem = scaled_smem(n, ldk, m, s.blocks);
    s.ok = s.cluster = resident_cluster(k_bcd_scaled<true>, (long long)n * m, s.smem);
    if (s.ok) return s;
    s.blocks = n < device_sm_count() ? n : device_sm_count();
    s.smem = scaled_smem(n, ldk, m, s.blocks);
    s.ok = resident_grid(k_bcd_scaled<false>, s.smem);
    return s;
}

inline void launch_scaled(const ScaledPlan& s, const ScaledParams& p, cudaStream_t st) {
    launch_resident(s.cluster ? k_bcd_scaled<true> : k_bcd_scaled<false>, s.cluster, s.blocks, s.smem,
                    st, p);
}

}  // namespace
}  // namespace regot
