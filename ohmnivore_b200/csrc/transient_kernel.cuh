// Transient kernels: a chunk of fixed backward-Euler steps, and the adaptive
// BE / TRAP run.  Instantiated per lanes per row in the transient_k*.cu units.
#pragma once

#include "internal.cuh"

namespace ohm {

// Device-side run record, accumulated by the grid leader.
struct TranDev {
    int status, steps_done, failed_step, kcode;
    long long newton_its, krylov_its;
    int fallbacks, pad;
    double max_residual;
};

struct TranArgs {
    int s0, s1;                        // steps [s0, s1) of this launch
    double t0, h;
    const uint32_t *c_rp, *c_col;
    const double *c_val;
    const int32_t *src_of_row;         // per row: index into srow_ptr, -1 none
    const uint32_t *srow_ptr, *srow_src;
    const double *srow_sign;
    const ohm_source *src;
    const double *pwl;
    const uint32_t *probe;
    int n_probes;
    double *wave;                      // n_steps x n_probes
    double *beff;                      // base rhs of the current step
    TranDev *st;
    double *states;                    // optional: x after step s at (s - state_base) * n
    int state_base;
    // Newton start of step s > 0: x_{n-1} (predict 0), the linear
    // extrapolation 2 x_{n-1} - x_{n-2} (predict 1; xpp holds x_{n-2}) or,
    // from step 2 on, the quadratic 3 x_{n-1} - 3 x_{n-2} + x_{n-3}
    // (predict 2; xppp holds x_{n-3})
    int predict;
    double *xpp, *xppp;
};

// Source waveforms, the formulas of transient_source.rs:39-118.
__device__ __forceinline__ double source_value(const ohm_source &s, double t, const double *pwl) {
    const double *p = s.p;
    switch (s.kind) {
        case OHM_TRAN_PULSE: {
            const double v1 = p[0], v2 = p[1], td = p[2], tr = p[3], tf = p[4], pw = p[5], per = p[6];
            if (t < td) return v1;
            const double trel = (per > 0.0 && per < 1.7976931348623157e308) ? fmod(t - td, per) : t - td;
            if (trel < tr) return tr > 0.0 ? v1 + (v2 - v1) * trel / tr : v2;
            if (trel < tr + pw) return v2;
            if (trel < tr + pw + tf) return tf > 0.0 ? v2 + (v1 - v2) * (trel - tr - pw) / tf : v1;
            return v1;
        }
        case OHM_TRAN_SIN: {
            const double vo = p[0], va = p[1], freq = p[2], td = p[3], theta = p[4];
            if (t < td) return vo;
            const double dt = t - td;
            const double env = theta != 0.0 ? exp(-dt * theta) : 1.0;
            return vo + va * sin(2.0 * 3.14159265358979323846 * freq * dt) * env;
        }
        case OHM_TRAN_PWL: {
            const double *q = pwl + 2 * (size_t)s.pwl_offset;
            const int m = s.pwl_count;
            if (m <= 0) return 0.0;
            if (t <= q[0]) return q[1];
            if (t >= q[2 * (m - 1)]) return q[2 * (m - 1) + 1];
            for (int i = 1; i < m; ++i) {
                if (t <= q[2 * i]) {
                    const double t0 = q[2 * (i - 1)], v0 = q[2 * (i - 1) + 1], t1 = q[2 * i], v1 = q[2 * i + 1];
                    return v0 + (v1 - v0) * ((t - t0) / (t1 - t0));
                }
            }
            return q[2 * (m - 1) + 1];
        }
        case OHM_TRAN_EXP: {
            const double v1 = p[0], v2 = p[1], td1 = p[2], tau1 = p[3], td2 = p[4], tau2 = p[5];
            if (t < td1) return v1;
            const double rise = (v2 - v1) * (1.0 - exp(-(t - td1) / tau1));
            if (t < td2) return v1 + rise;
            const double fall = (v1 - v2) * (1.0 - exp(-(t - td2) / tau2));
            return v1 + rise + fall;
        }
        default:
            return s.dc;
    }
}

template <int LPR, class Team>
__global__ void __launch_bounds__(kTeamBlock<Team>, 1) transient_kernel(const __grid_constant__ KernelArgs a,
                                                                     const __grid_constant__ TranArgs T) {
    Team g;
    g.init(a);
    if (T.st->status != 0) return;     // an earlier chunk failed (uniform: written before this launch)
    const double inv_h = 1.0 / T.h;
    for (int s = T.s0; s < T.s1; ++s) {
        const double tn = T.t0 + (double)(s + 1) * T.h;
        // ---- b_n = b(t_n) + (C/h) x_{n-1} for the rows of this block ----
        for (int i = g.r0 + threadIdx.x; i < g.r1; i += blockDim.x) {
            double bs = 0.0;
            const int q = T.src_of_row[i];
            if (q >= 0)
                for (uint32_t e = T.srow_ptr[q]; e < T.srow_ptr[q + 1]; ++e)
                    bs += T.srow_sign[e] * source_value(T.src[T.srow_src[e]], tn, T.pwl);
            double cx = 0.0;
            for (uint32_t k = T.c_rp[i]; k < T.c_rp[i + 1]; ++k) cx += T.c_val[k] * a.x[T.c_col[k]];
            const double bb = bs + cx * inv_h;
            T.beff[i] = bb;
            a.b[i] = bb;
        }
        if (!g.sync()) return;
        if (T.predict) {
            // after every block's (C/h) x_{n-1}: own rows start from the
            // extrapolation (x_{n-2} is known from step 1 of the run on)
            for (int i = g.r0 + threadIdx.x; i < g.r1; i += blockDim.x) {
                const double xp = a.x[i];
                if (T.predict == 2 && s > 1) a.x[i] = 3.0 * (xp - T.xpp[i]) + T.xppp[i];
                else if (s > 0) a.x[i] = 2.0 * xp - T.xpp[i];
                if (T.predict == 2) T.xppp[i] = T.xpp[i];
                T.xpp[i] = xp;
            }
            if (!g.sync()) return;
        }
        // ---- Newton on the companion system, from x_{n-1} ----
        RunOut o;
        RunCfg c{0.0, 1.0, 0.0, a.max_outer, a.max_krylov, false};
        if (!newton_run<LPR>(a, g, c, o)) return;
        if (g.leader()) {
            TranDev &d = *T.st;
            d.newton_its += o.outer_done;
            d.krylov_its += o.kiters;
            d.fallbacks += o.fallbacks;
            d.kcode = o.kcode;
            if (o.status == kOk) {
                d.steps_done = s + 1;
            } else {
                d.status = o.status;
                d.failed_step = s;
                d.max_residual = o.last_dmax;
            }
        }
        if (o.status != kOk) return;
        for (int k = g.gtid; k < T.n_probes; k += g.gstride)
            T.wave[(size_t)s * T.n_probes + k] = a.x[T.probe[k]];
        if (T.states) {
            double *st = T.states + (size_t)(s - T.state_base) * a.n;
            for (int i = g.r0 + threadIdx.x; i < g.r1; i += blockDim.x) st[i] = a.x[i];
        }
    }
}

// Adaptive BE / TRAP step control of the reference (transient.rs:77-178):
// the first step and the step after a rejection are BE; every other step
// solves TRAP and BE from x_{n-1}, estimates LTE = (2/3) max|x_trap - x_be|
// (compute_lte, :355-362), rejects it when LTE > 1e-3 (h *= clamp(0.9
// sqrt(tol / LTE), 0.5, 2), at least h_min) and otherwise accepts x_trap and
// takes h = clamp(h * that factor, h_min, h_max); h_min = tstep / 10^4,
// h_max = tstep.  Companion matrices A = G + (alpha / h) C (:285-323) are
// formed on the device for every solve.  TRAP's rhs is
// b(t_n) + (2/h) C x_{n-1} - f(x_{n-1}) + b(t_{n-1}) (:336-352) with
// f(x) = G x + i(x): the reference's G x_{n-1} plus, for nonlinear devices,
// their currents, taken as J(x) x - b of the system stamped at x on the base
// (G, 0), so TRAP integrates the same device equations Newton solves.
constexpr int kAdTimestep = 20;   // consecutive rejections at h_min (OhmnivoreError::Timestep)

struct AdaptDev {
    int status, accepted, rejected, points;
    long long newton_its, krylov_its;
    int solves, fallbacks, kcode, failed_kind;
    double t, h, t_fail, max_residual;
};

struct AdaptArgs {
    double tstep, tstop, tstart;
    int max_points;
    long long nnz;
    const double *g_vals;      // G, the plan's base values
    const double *cg;          // C on G's pattern (0 off C)
    const double *zeros;       // n zeros: the rhs base of the f(x) evaluation
    double *aval;              // companion base values of the current solve
    double *xs, *xt, *fdev;    // x_{n-1}, x_trap, f(x_{n-1})
    double *times;             // output times (max_points)
    AdaptDev *st;
};

template <int LPR, class Team>
__global__ void __launch_bounds__(kTeamBlock<Team>, 1) adaptive_kernel(const __grid_constant__ KernelArgs a,
                                                                    const __grid_constant__ TranArgs T,
                                                                    const __grid_constant__ AdaptArgs P) {
    Team g;
    g.init(a);
    const int r0 = g.r0, r1 = g.r1;
    const double h_min = P.tstep / 10000.0, h_max = P.tstep, lte_tol = 1e-3;
    constexpr int kMaxFailures = 10;
    // every thread holds the same control state: it changes only through
    // grid-wide results (Newton status, the all-reduced LTE)
    double t = 0.0, h = fmin(P.tstep, h_max), t_next = 0.0, h_next = 0.0;
    bool use_be = true;
    int stage = 0;               // 0: new step, 1: its TRAP solve, 2: its BE solve
    int fails = 0, points = 0, accepted = 0, rejected = 0, solves = 0, fallbacks = 0, kcode = 0;
    int status = kOk, failed_kind = 0;
    long long nits = 0, kits = 0;
    double t_fail = 0.0, max_res = 0.0;

    // output row `points` (kept only below max_points; the count continues)
    auto record = [&](double tr) {
        if (points < P.max_points) {
            for (int k = g.gtid; k < T.n_probes; k += g.gstride)
                T.wave[(size_t)points * T.n_probes + k] = a.x[T.probe[k]];
            if (g.leader()) P.times[points] = tr;
        }
        ++points;
    };
    if (P.tstart <= 0.0) record(0.0);
    while (true) {
        if (stage == 0) {
            if (!(t < P.tstop)) break;
            if (t + h > P.tstop) h = P.tstop - t;
            if (h < h_min * 0.5) break;
            t_next = t + h;
            for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) P.xs[i] = a.x[i];
            if (!use_be) {
                // f(x_{n-1}) = J x - b of the system stamped at x on (G, 0)
                for (long long k = g.gtid; k < P.nnz; k += g.gstride) {
                    a.vals64[k] = P.g_vals[k];
                    if (a.vals32) a.vals32[k] = (float)P.g_vals[k];
                }
                for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) a.b[i] = 0.0;
                if (!g.sync()) return;
                const RunCfg c0{0.0, 1.0, 0.0, 0, 0, false};
                if (!assemble(a, g, c0, P.g_vals, P.zeros)) return;
                const double *xv = a.x;
                auto x_at = [&](int j, bool) -> double { return xv[j]; };
                auto f_row = [&](int i, double ax) { P.fdev[i] = ax - a.b[i]; };
                spmv_rows<LPR, double>(a.row_ptr, a.col, a.vals64, (const uint8_t *)nullptr, r0, r1, x_at, f_row,
                                       a.longflag);
                if (!spmv_long<double>(a, g, a.col, a.vals64, (const uint8_t *)nullptr, x_at, f_row)) return;
                if (!g.sync()) return;
            }
            stage = use_be ? 2 : 1;
        }
        // companion base A = G + (alpha / h) C and the step's rhs
        const double fac = (stage == 1 ? 2.0 : 1.0) / h;
        for (long long k = g.gtid; k < P.nnz; k += g.gstride) {
            const double v = P.g_vals[k] + fac * P.cg[k];
            P.aval[k] = v;
            a.vals64[k] = v;
            if (a.vals32) a.vals32[k] = (float)v;
        }
        for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
            double bn = 0.0, bp = 0.0;
            const int q = T.src_of_row[i];
            if (q >= 0)
                for (uint32_t e = T.srow_ptr[q]; e < T.srow_ptr[q + 1]; ++e) {
                    const ohm_source &src = T.src[T.srow_src[e]];
                    bn += T.srow_sign[e] * source_value(src, t_next, T.pwl);
                    if (stage == 1) bp += T.srow_sign[e] * source_value(src, t, T.pwl);
                }
            double cx = 0.0;
            for (uint32_t k = T.c_rp[i]; k < T.c_rp[i + 1]; ++k) cx += T.c_val[k] * a.x[T.c_col[k]];
            const double bb = stage == 1 ? ((bn + fac * cx) - P.fdev[i]) + bp : bn + fac * cx;
            T.beff[i] = bb;
            a.b[i] = bb;
        }
        if (!g.sync()) return;
        RunOut o;
        const RunCfg c{0.0, 1.0, 0.0, a.max_outer, a.max_krylov, false};
        if (!newton_run<LPR>(a, g, c, o)) return;
        nits += o.outer_done;
        kits += o.kiters;
        fallbacks += o.fallbacks;
        kcode = o.kcode;
        ++solves;
        if (o.status != kOk) {
            status = o.status;
            failed_kind = stage;
            t_fail = t_next;
            max_res = o.last_dmax;
            break;
        }
        if (stage == 1) {            // keep x_trap, solve BE from x_{n-1}
            for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
                P.xt[i] = a.x[i];
                a.x[i] = P.xs[i];
            }
            if (!g.sync()) return;
            stage = 2;
            continue;
        }
        stage = 0;
        if (!use_be) {
            double mx[1] = {0.0};
            for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) mx[0] = fmax(mx[0], fabs(P.xt[i] - a.x[i]));
            if (!g.template allmax<1>(mx)) return;
            const double lte = (2.0 / 3.0) * mx[0];
            const double factor = fmin(fmax(0.9 * sqrt(lte_tol / lte), 0.5), 2.0);
            if (lte > lte_tol) {     // reject: smaller h, BE from x_{n-1}
                h = fmax(h * factor, h_min);
                ++fails;
                if (fails >= kMaxFailures && h <= h_min * 1.01) {
                    status = kAdTimestep;
                    t_fail = t;
                    break;
                }
                ++rejected;
                use_be = true;
                for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) a.x[i] = P.xs[i];
                if (!g.sync()) return;
                continue;
            }
            h_next = fmin(fmax(h * factor, h_min), h_max);
            for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) a.x[i] = P.xt[i];
            if (!g.sync()) return;
        } else {
            use_be = false;
            h_next = h;
        }
        fails = 0;
        ++accepted;
        t = t_next;
        h = h_next;
        if (t >= P.tstart) record(t);
    }
    if (g.leader()) {
        AdaptDev &d = *P.st;
        d.status = status;
        d.accepted = accepted;
        d.rejected = rejected;
        d.points = points;
        d.newton_its = nits;
        d.krylov_its = kits;
        d.solves = solves;
        d.fallbacks = fallbacks;
        d.kcode = kcode;
        d.failed_kind = failed_kind;
        d.t = t;
        d.h = h;
        d.t_fail = t_fail;
        d.max_residual = max_res;
    }
}

using TranFn = void (*)(KernelArgs, TranArgs);
using AdaptFn = void (*)(KernelArgs, TranArgs, AdaptArgs);

// Kernels for lanes per row 1, 4 or 8, with and without Krylov slices.
template <int LPR>
KernelPair<TranFn> transient_kernel_for();
template <int LPR>
KernelPair<AdaptFn> adaptive_kernel_for();
template <>
KernelPair<TranFn> transient_kernel_for<1>();
template <>
KernelPair<TranFn> transient_kernel_for<4>();
template <>
KernelPair<TranFn> transient_kernel_for<8>();
template <>
KernelPair<AdaptFn> adaptive_kernel_for<1>();
template <>
KernelPair<AdaptFn> adaptive_kernel_for<4>();
template <>
KernelPair<AdaptFn> adaptive_kernel_for<8>();

}  // namespace ohm
