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
// duals) when a scaling leaves 2^-kScaleLim .. 2^kScaleLim, and no sum beyond
// 2^-kSumLim .. 2^kSumLim is used, so that what K loses to underflow stays far
// below the rounding of any sum.
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

constexpr int kScaleLim = 100;   // scalings beyond 2^-100 .. 2^100 end a launch
// Sums beyond 2^-kSumLim .. 2^kSumLim go to the max-anchored updates. A launch ends
// one sweep after a scaling left its range, so that scaling, up to a / s, meets K
// once more: an entry of K is off by up to 2^-1075 (what underflow loses), n of
// them times a scaling of 2^480 by n 2^-595, which a sum of at least 2^-480 has
// 115 - log2 n bits below its leading one. (Sums down to 2^-896 were taken before:
// a row at 2^-866 got the scaling 2^865, and a column whose largest entry it was
// came out of what was left, wrong by hundreds of reg in its dual.)
constexpr int kSumLim = 480;
constexpr double kMinMarginal = 1e-150;

struct ScaledParams {
    const double* K;
    long long ldk;
    int n, m;
    const double *a, *b;
    double *alpha, *beta;  // base duals in, the last complete iterate out
    double* alpha_next;    // column sums out of range: alpha_{k+1}
    double reg, sum_a, sum_bt;
    double stop2;     // the largest x with sqrt(x) < tol
    double* part;     // [G][ldk] column products of each block
    double* vbuf;     // [ldk] column scalings
    double* red;      // [G][4]: sum g^2, sum r, sum a alpha, sum b beta~
    int* redf;        // [G] flags
    double* blast;    // beta_{m-1}
    double* fin;      // [G + 1]: the last iterate's sums of b beta~, beta_{m-1}
    unsigned* count;  // grid barrier
    int* err;        // set when a barrier gives up
    unsigned polls;  // before it does
    BcdState* st;
    double *hobj, *hmar, *htime;
    int first_col;  // start with v = b / K'1 (beta0 is an anchor, alpha0 = 0)
};

enum : int { SC_ROW = 1, SC_COL = 2, SC_RANGE = 4 };

inline size_t scaled_smem(int n, long long ldk, int m, int G) {
    const size_t W = G > 1 ? G - 1 : 1;  // workers
    const size_t R = (size_t)(n + W - 1) / W + 1, C = (size_t)(m + W - 1) / W + 1;
    return sizeof(double) * ((size_t)ldk + 5 * R + rows_part_size((int)R) +
                             2 * kResThreads + 2 * C + 2 * kResWarps);
}

// The objective of iterate k needs logarithms of its scalings. They are taken
// while the block waits at the first barrier of a sweep (those of u_{k+1} and
// v_k at the barrier of iterate k), so the sums of b beta~ arrive one sweep
// later than the rest of the record, and the last objective after one barrier
// more. The last block has no rows and columns: it forms and writes the records
// (some 5000 clocks a sweep) while the others work.
template <bool CLUSTER>
__global__ void __launch_bounds__(kResThreads, 1) k_bcd_scaled(const ScaledParams p) {
    extern __shared__ __align__(16) double s_dyn_b[];
    __shared__ int s_ok, s_exit, s_flags, s_colflags;
    __shared__ double s_bl, s_rec[4];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.x, W = gridDim.x - 1;
    const bool recorder = b == W;
    const int n = p.n, m = p.m;
    const long long ldk = p.ldk;
    const int r0 = recorder ? n : own_begin(n, b, W);
    const int R = recorder ? 0 : own_begin(n, b + 1, W) - r0;
    const int j0 = recorder ? m : own_begin(m, b, W), j1 = recorder ? m : own_begin(m, b + 1, W);
    const int C = j1 - j0, Rm = (n + W - 1) / W + 1, Cm = (m + W - 1) / W + 1;
    const int S = row_segments((int)(ldk >> 1), R);
    double* s_v = s_dyn_b;                  // [ldk] column scalings of the current iterate
    double* s_q = s_v + ldk;              // [2 kResThreads]
    double* s_u = s_q + 2 * kResThreads;  // [Rm] row scalings of the current iterate
    double* s_un = s_u + Rm;              // [Rm] ... of the next
    double* s_sum = s_un + Rm;            // [Rm]
    double* s_t = s_sum + Rm;             // [Rm] row marginals
    double* s_g = s_t + Rm;               // [Rm] squared gradient entries
    double* s_part = s_g + Rm;
    double* s_vp = s_part + rows_part_size(Rm);  // [Cm] own columns, previous v
    double* s_c = s_vp + Cm;                     // [Cm] own columns' sums
    double* s_wa = s_c + Cm;                     // [kResWarps] sums of a alpha
    double* s_wb = s_wa + kResWarps;             // [kResWarps] sums of b beta~
    GridBarrier<CLUSTER> bar(p.count, p.err, p.polls, &s_ok);

    for (int j = tid; j < ldk; j += kResThreads) s_v[j] = j < m ? 1.0 : 0.0;
    for (int r = tid; r < R; r += kResThreads) s_u[r] = s_un[r] = 1.0;
    for (int j = tid; j < C; j += kResThreads) s_vp[j] = 1.0;
    if (tid < kResWarps) s_wa[tid] = s_wb[tid] = 0.0;
    if (tid == 0) s_colflags = s_exit = 0;
    __syncthreads();

    // The block's sums of a alpha (rows scaled by u) and b beta~ (columns
    // scaled by v): rows on the even warps and columns on the odd ones, so
    // that their logarithms run side by side.
    auto log_terms = [&](const double* u) {
        constexpr int H = kResWarps / 2;
        const int w = warp >> 1, t = w * 32 + lane;
        if (warp & 1) {
            if (w * 32 >= C) return;
            double v = 0.0;
            for (int j = t; j < C; j += H * 32) {
                const double be = fma(p.reg, log(s_v[j0 + j]), p.beta[j0 + j]);
                if (j0 + j < m - 1) v = fma(p.b[j0 + j], be, v);
                else s_bl = be;
            }
            __syncwarp();
            v = warp_sum_low(v);
            if (lane == 0) s_wb[w] = v;
        } else {
            if (w * 32 >= R) return;
            double v = 0.0;
            for (int r = t; r < R; r += H * 32)
                v = fma(p.a[r0 + r], fma(p.reg, log(u[r]), p.alpha[r0 + r]), v);
            __syncwarp();
            v = warp_sum_low(v);
            if (lane == 0) s_wa[w] = v;
        }
    };
    auto of_warps = [](const double* w, int items) {  // sum of the warps' sums
        double s = w[0];
        for (int k = 1; k < kResWarps / 2 && k * 32 < items; ++k) s += w[k];
        return s;
    };
    auto in_sum_range = [](double s) {
        return __double2hiint(s) > 0 && exponent_within(s, kSumLim);
    };
    auto stage_v = [&]() {
        for (int j = tid; j < C; j += kResThreads) s_vp[j] = s_v[j0 + j];
        __syncthreads();
        for (int j = tid; j < m; j += kResThreads) s_v[j] = __ldcg(p.vbuf + j);
    };

    // rows without a worker's columns leave part as it is: the recorder has none
    auto columns = [&]() {
        if (!recorder) cols_dot(p.K, ldk, r0, R, s_un, p.part + (long long)b * ldk, s_q);
    };
    if (p.first_col) {
        columns();
        bar.arrive();
        if (!bar.wait()) return;
        // the range is not checked: beta0 is an anchor, the sums are in 1 .. n
        merge_columns(p.part, ldk, W, j0, j1, warp, kResWarps,
                      [&](int j, double c) { __stcg(p.vbuf + j, p.b[j] / c); });
        bar.arrive();
        if (!bar.wait()) return;
        stage_v();
    } else {
        log_terms(s_u);
    }
    double gb2 = p.st->gb2_once;
    unsigned long long t0 = p.st->t0;
    if (p.first_col) t0 = globaltimer_ns();
    int k = p.st->iter;
    const int max_iter = p.st->max_iter;
    // the recorder's thread 0: the record of the previous iterate
    bool pending = false;
    double last_r = 0.0, last_a = 0.0;
    auto finish_record = [&](double sb, double bl) {
        if (pending)
            p.hobj[k - 1] = p.reg * last_r - last_a - bl * p.sum_a - sb + bl * p.sum_bt;
        pending = false;
    };

#pragma unroll 1
    for (;;) {
        // ---- rows: s = K v, u_next = a / s ----
        __syncthreads();
        rows_dot(p.K, ldk, r0, R, S, s_v, s_part, s_sum);
        __syncthreads();
        for (int r = tid; r < R; r += kResThreads) {
            const double a = p.a[r0 + r], sr = s_sum[r];
            const double t = s_u[r] * sr, g = t - a;
            s_un[r] = a / sr;
            s_t[r] = t;
            s_g[r] = g * g;
        }
        __syncthreads();
        // ---- columns of the own rows, and the block's share of the sums (half
        // a warp each) ----
        if (warp == kResWarps - 1 && !recorder) {
            const double* src = lane < 16 ? s_g : s_t;
            double v = 0.0;
            int f = 0;
            for (int r = lane & 15; r < R; r += 16) {
                v += src[r];
                if (!in_sum_range(s_sum[r])) f |= SC_ROW;
                if (!exponent_within(s_u[r], kScaleLim)) f |= SC_RANGE;
            }
            f = __reduce_or_sync(0xffffffffu, f);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            double* red = p.red + 4 * (size_t)b;
            if (lane == 0) {
                __stcg(red, v);
                __stcg(red + 2, of_warps(s_wa, R));
                __stcg(p.redf + b, f | s_colflags);
            }
            if (lane == 16) {
                __stcg(red + 1, v);
                __stcg(red + 3, of_warps(s_wb, C));
                if (C > 0 && j1 == m) __stcg(p.blast, s_bl);
            }
            __syncwarp();
        }
        columns();
        bar.arrive();
        log_terms(s_un);
        if (!bar.wait()) return;
        // ---- the stop, decided by every block from the same numbers, beside
        // the merge of the own columns ----
        if (warp == kResWarps - 1) {
            int f = 0;
            for (int g = lane; g < W; g += 32) f |= __ldcg(p.redf + g);
            const double g2 = warp_sum_strided(p.red, W, 4);
            f = __reduce_or_sync(0xffffffffu, f);
            if (lane == 0) {
                // g2 + gb2 <= stop2 exactly where its root is below tol
                const bool stop = g2 + gb2 <= p.stop2 || k >= max_iter;
                s_flags = f;
                s_exit = (f & (SC_ROW | SC_COL)) == 0 && stop ? 1 : f ? 2 : 0;
                s_colflags = 0;
            }
        } else if (!recorder) {
            merge_columns(p.part, ldk, W, j0, j1, warp, kResWarps - 1,
                          [&](int j, double c) { s_c[j - j0] = c; });
        } else if (warp < 4) {
            const double v = warp_sum_strided(p.red + warp, W, 4);
            if (lane == 0) s_rec[warp] = v;
        }
        __syncthreads();
        for (int j = tid; j < C; j += kResThreads) {
            const double c = s_c[j], v = p.b[j0 + j] / c;
            if (!in_sum_range(c)) atomicOr(&s_colflags, SC_COL);
            if (!exponent_within(v, kScaleLim)) atomicOr(&s_colflags, SC_RANGE);
            __stcg(p.vbuf + j0 + j, v);
        }
        double bl = 0.0;
        if (recorder && tid == 0) bl = __ldcg(p.blast);
        const int leave = s_exit;
        if (!leave) bar.arrive();
        if (recorder && tid == 0) {
            finish_record(s_rec[3], bl);
            if (!(s_flags & (SC_ROW | SC_COL))) {
                const double gnorm = sqrt(s_rec[0] + gb2);
                p.hmar[k] = gnorm;
                p.htime[k] = (double)(globaltimer_ns() - t0) * 1e-6;
                p.st->hist_len = k + 1;
                p.st->last_gnorm = gnorm;
                p.st->gb2_once = 0.0;
                pending = true;
                last_r = s_rec[1];
                last_a = s_rec[2];
            }
        }
        if (leave) break;
        gb2 = 0.0;
        if (!bar.wait()) return;
        stage_v();
        for (int r = tid; r < R; r += kResThreads) s_u[r] = s_un[r];
        ++k;
    }
    // ---- the sums of b beta~ of the last iterate ----
    if (tid == 0 && !recorder) {
        __stcg(p.fin + b, of_warps(s_wb, C));
        if (C > 0 && j1 == m) __stcg(p.fin + W, s_bl);
    }
    bar.arrive();
    if (!bar.wait()) return;
    if (recorder && tid == 0) {
        double sb = 0.0;
        for (int g = 0; g < W; ++g) sb += __ldcg(p.fin + g);
        const double bl = __ldcg(p.fin + W);
        const int f = s_flags;
        if (pending) ++k;  // finish_record writes the iterate before k
        finish_record(sb, bl);
        if (!(f & (SC_ROW | SC_COL))) --k;
        p.st->iter = (f & SC_COL) ? k - 1 : k;
        p.st->bad = (f & SC_COL) ? SC_COL : (f & SC_ROW) ? SC_ROW : 0;
        p.st->sum_bb = sb;
        p.st->beta_last = bl;
        p.st->t0 = t0;
        if (s_exit == 1) {
            p.st->done = 1;
            p.st->niter = k;
        }
    }
    // ---- the last complete iterate: (alpha_k, beta_k); after column sums out
    // of range, alpha_k and beta_{k-1} ----
    const bool colbad = (s_flags & SC_COL) != 0;
    for (int r = tid; r < R; r += kResThreads) {
        const double al = fma(p.reg, log(s_u[r]), p.alpha[r0 + r]);
        p.alpha[r0 + r] = al;
        p.alpha_next[r0 + r] = al;
    }
    for (int j = tid; j < C; j += kResThreads)
        p.beta[j0 + j] = fma(p.reg, log(colbad ? s_vp[j] : s_v[j0 + j]), p.beta[j0 + j]);
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
    s.blocks = n + 1 < device_sm_count() ? n + 1 : device_sm_count();
    s.smem = scaled_smem(n, ldk, m, s.blocks);
    s.ok = s.blocks > 1 && resident_grid(k_bcd_scaled<false>, s.smem);
    return s;
}

inline void launch_scaled(const ScaledPlan& s, const ScaledParams& p, cudaStream_t st) {
    launch_resident(s.cluster ? k_bcd_scaled<true> : k_bcd_scaled<false>, s.cluster, s.blocks, s.smem,
                    st, p);
}

}  // namespace
}  // namespace regot
