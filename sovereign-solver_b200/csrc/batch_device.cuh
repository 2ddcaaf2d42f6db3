// batch_device.cuh -- an instance's check terms, decision and restart, shared
// by the batched kernels over all instances (batch_kernels.cu) and the kernel
// that runs an instance on one cluster (batch_resident.cuh).
#pragma once

#include <cmath>

#include "batch_kernels.cuh"
#include "fast_common.cuh"

namespace pdhg {
namespace {

template <class T>
__device__ __forceinline__ void inst_row_terms(const BatchView& b, const Iterates<T>& it,
                                               const BatchParams& p, int i, double act_c,
                                               double act_a, double inv, Terms& t) {
    const DevProblem& P = b.P;
    p.act_avg[i] = act_a;
    const double lo = P.rlo[i], hi = P.rhi[i];
    const double yc = static_cast<double>(it.y[i]);
    const double ya = avg_y(it, i, inv);
    t.cp = smax(t.cp, primal_term(act_c, lo, hi));
    t.ap = smax(t.ap, primal_term(act_a, lo, hi));
    t.cd = smax(t.cd, cs_term(yc, act_c, lo, hi, p.tol));
    t.ad = smax(t.ad, cs_term(ya, act_a, lo, hi, p.tol));
    const double rs = P.rs[i];
    const double lo_o = P.rlo_o[i], hi_o = P.rhi_o[i];
    const double aoc = act_c / rs, aoa = act_a / rs;
    t.ocp = smax(t.ocp, primal_term(aoc, lo_o, hi_o));
    t.oap = smax(t.oap, primal_term(aoa, lo_o, hi_o));
    t.ocd = smax(t.ocd, cs_term(yc * rs, aoc, lo_o, hi_o, p.bound_tol));
    t.oad = smax(t.oad, cs_term(ya * rs, aoa, lo_o, hi_o, p.bound_tol));
    if (p.termination_rule != 0) {
        t.dobj_c += clipped_inf(yc * rs, lo_o, hi_o);
        t.dobj_a += clipped_inf(ya * rs, lo_o, hi_o);
    }
    if (p.termination_rule == 2) {  // squares of the row violation and of y's sign violation
        const double pc = primal_term(aoc, lo_o, hi_o), pa = primal_term(aoa, lo_o, hi_o);
        const double dc = sign_violation(yc * rs, lo_o, hi_o);
        const double da = sign_violation(ya * rs, lo_o, hi_o);
        t.ppc += pc * pc;
        t.ppa += pa * pa;
        t.ddc += dc * dc;
        t.dda += da * da;
    }
}

template <class T>
__device__ __forceinline__ void inst_col_terms(const BatchView& b, const Iterates<T>& it,
                                               const BatchParams& p, double sign, int j,
                                               double aty_c, double aty_a, double inv,
                                               Terms& t) {
    const DevProblem& P = b.P;
    const double cj = P.c[j];
    const double lo = P.lo[j], hi = P.hi[j];
    const double xc = static_cast<double>(it.x[j]);
    const double xa = avg_x(it, j, inv);
    const double rc = cj - aty_c, ra = cj - aty_a;
    t.cd = smax(t.cd, cs_term(rc, xc, lo, hi, p.tol));
    t.ad = smax(t.ad, cs_term(ra, xa, lo, hi, p.tol));
    const double cs = P.cs[j];
    const double lo_o = P.lo_o[j], hi_o = P.hi_o[j];
    t.ocd = smax(t.ocd, cs_term(rc / cs, xc * cs, lo_o, hi_o, p.bound_tol));
    t.oad = smax(t.oad, cs_term(ra / cs, xa * cs, lo_o, hi_o, p.bound_tol));
    if (p.termination_rule == 2) {  // squares of the reduced cost's sign violation
        const double dc = sign_violation(rc / cs, lo_o, hi_o);
        const double da = sign_violation(ra / cs, lo_o, hi_o);
        t.ddc += dc * dc;
        t.dda += da * da;
    }
    if (p.termination_rule != 0) {
        t.pobj_c += sign * P.c_o[j] * (xc * cs);
        t.pobj_a += sign * P.c_o[j] * (xa * cs);
        t.dobj_c += clipped_inf(rc / cs, lo_o, hi_o);
        t.dobj_a += clipped_inf(ra / cs, lo_o, hi_o);
    }
}

__device__ void finish_instance(const BatchView& b, InstState& s) {
    const int left = atomicSub(&b.g->active, 1);
    if (left == 1) b.g->done = 1;
    b.g->dirty = 1;
}

// The instance's decision (kkt_residual, original_space_residual, candidate,
// termination, restart rule: pdhg.cpp:333-408) from the check's values v
// (kBatchCheckVals), by one thread. iter: the iterations completed before the
// period; stop: the host's stop request.
__device__ void batch_decide(const BatchView& b, const BatchParams& p, InstState& s, const double* v, bool halpern,
                             bool f32, long long iter, int stop) {
    const double inv = halpern ? 1.0 : 1.0 / static_cast<double>(s.since_restart + p.period);
    const double cp = v[0], cd = v[1], ap = v[2], ad = v[3];
    const double ocp = v[4], ocd = v[5], oap = v[6], oad = v[7];
    const double s0 = v[8], s1 = v[9], s2 = v[10], s3 = v[11];
    // ---- the instance's decision (as the single engine's check) ----
    double cur = smax(cp, cd), avg = smax(ap, ad);
    // termination rule 2: relative parts of the current point and the average
    // (original units, l2 norms); their l2 norm is restart rule 2's measure
    double part_c[3] = {0, 0, 0}, part_a[3] = {0, 0, 0};
    if (p.termination_rule == 2) {
        const double k0 = s.obj_sign * s.obj_const;
        const double pp[2] = {v[12], v[14]}, dd[2] = {v[13], v[15]};
        const double ps[2] = {s0 + k0, s2 + k0}, ds[2] = {s1 + k0, s3 + k0};
        for (int w = 0; w < 2; ++w) {
            double* pt = w ? part_a : part_c;
            pt[0] = sqrt(pp[w]) / (1.0 + s.bnorm2);
            pt[1] = sqrt(dd[w]) / (1.0 + s.cnorm2);
            pt[2] = fabs(ps[w] - ds[w]) / (1.0 + fabs(ps[w]) + fabs(ds[w]));
        }
        if (p.restart_rule == 2) {
            const double mc = sqrt(part_c[0] * part_c[0] + part_c[1] * part_c[1] + part_c[2] * part_c[2]);
            const double ma = sqrt(part_a[0] * part_a[0] + part_a[1] * part_a[1] + part_a[2] * part_a[2]);
            cur = isfinite(cur) ? mc : cur;
            avg = isfinite(avg) ? ma : avg;
        }
    }
    if (halpern) cur = avg;  // only T(z) is measured
    s.cur_res = cur;
    s.avg_res = avg;
    s.inv = inv;
    s.restart = 0;
    s.fold = 0;
    const long long it_idx = iter + p.period - 1;
    if (!isfinite(cur) || !isfinite(avg)) {
        s.done = 1;
        s.status = kStatusNumericalFailure;
        s.fail_kind = 1;
        s.stop_iter = it_idx;
        finish_instance(b, s);
        return;
    }
    const bool ab = halpern ? true : avg <= cur;  // Halpern: the candidate is T(z)
    s.avg_better = ab ? 1 : 0;
    const double op = ab ? oap : ocp, od = ab ? oad : ocd;
    const double orig = smax(op, od);
    s.orig_res = orig;
    if (!isfinite(orig)) {
        s.done = 1;
        s.status = kStatusNumericalFailure;
        s.fail_kind = 2;
        s.stop_iter = it_idx;
        finish_instance(b, s);
        return;
    }
    double rel = 0.0;
    if (p.termination_rule == 2) {
        const double* pt = ab ? part_a : part_c;
        rel = smax(smax(pt[0], pt[1]), pt[2]);
    } else if (p.termination_rule == 1) {
        // the objective constant shifts both objectives
        const double ps = (ab ? s2 : s0) + s.obj_sign * s.obj_const;
        const double ds = (ab ? s3 : s1) + s.obj_sign * s.obj_const;
        const double gap = fabs(ps - ds) / (1.0 + fabs(ps) + fabs(ds));
        rel = smax(smax(op / (1.0 + s.bnorm), od / (1.0 + s.cnorm)), gap);
    }
    s.rel_kkt = rel;
    const bool conv = (p.termination_rule != 0) ? (rel < p.tol) : (orig < p.tol);
    if (conv) {
        s.done = 1;
        s.converged = 1;
        s.status = kStatusOptimal;
        s.stop_iter = it_idx + 1;
        finish_instance(b, s);
        return;
    }
    if (p.restart_rule == 0) {
        if (!isfinite(s.res_last)) s.res_last = cur;
        if (avg <= p.restart_decrease * s.res_last) {
            s.restart = 1;
            s.restart_to_avg = 1;
            s.res_last = avg;
            s.since_restart = 0;
            s.restarts += 1;
        } else {
            s.since_restart += p.period;
        }
    } else {
        const double cand = ab ? avg : cur;
        if (!isfinite(s.res_last)) s.res_last = cur;
        const long long span = s.since_restart + p.period;
        const long long total = iter + p.period;
        const bool sufficient = cand <= 0.2 * s.res_last;
        const bool necessary = cand <= 0.8 * s.res_last && cand > s.res_prev_cand;
        const bool artificial = static_cast<double>(span) >= 0.36 * static_cast<double>(total);
        s.res_prev_cand = cand;
        if (sufficient || necessary || artificial) {
            s.restart = 1;
            s.restart_to_avg = ab ? 1 : 0;
            s.res_last = cand;
            s.since_restart = 0;
            s.restarts += 1;
        } else {
            s.since_restart = span;
        }
    }
    s.fresh = s.restart;
    s.fold = f32 && !halpern ? 1 : 0;
    if (p.allow_switch) {  // no 2% gain in 25 checks: the FP32 phase of this instance ends
        // under rule 2 only at FP32's precision floor (as the single engine:
        // plateaus above kFp32Zone are the method's own)
        const double r = p.termination_rule != 0 ? rel : orig;
        if (p.termination_rule == 2 && r > kFp32Zone) {
            s.since_improve = 0;
            if (r < s.best_res) s.best_res = r;
        } else if (r < 0.98 * s.best_res) {
            s.best_res = r;
            s.since_improve = 0;
        } else if (++s.since_improve >= 25) {
            s.done = 1;
            s.stalled = 1;
            s.status = kBatchStalled;
            s.stop_iter = it_idx + 1;
            finish_instance(b, s);
            return;
        }
    }
    if (stop != 0) {
        s.done = 1;
        s.status = stop;
        s.stop_iter = it_idx + 1;
        finish_instance(b, s);
    }
}

// A restart of one column / row (to the average or the current point; the
// Halpern anchor with it) and the fold of the mixed mode's period sums; its
// squared distance from the last restart point, for the primal weight.
template <class T>
__device__ __forceinline__ double restart_col(const Iterates<T>& it, const BatchParams& p, const PV<T>& pv, int j,
                                              int restart, bool to_avg, double inv) {
    double d = 0.0;
    if (restart && to_avg) it.x[j] = clampT<T>(static_cast<T>(avg_x(it, j, inv)), pv.lo[j], pv.hi[j]);
    if (restart && it.halpern) it.xa[j] = it.x[j];  // the new anchor
    if (restart && p.primal_weight_update) {
        const double xn = static_cast<double>(it.x[j]);
        d = xn - p.x_last[j];
        p.x_last[j] = xn;
    }
    if constexpr (std::is_same<T, float>::value)
        it.xsum[j] = restart ? 0.0 : it.xsum[j] + static_cast<double>(it.psx[j]);
    return d * d;
}
template <class T>
__device__ __forceinline__ double restart_row(const Iterates<T>& it, const BatchParams& p, const PV<T>& pv, int i,
                                              int restart, bool to_avg, double inv) {
    double d = 0.0;
    if (restart && to_avg) {
        it.y[i] = static_cast<T>(avg_y(it, i, inv));
        it.s[i] = clampT<T>(static_cast<T>(p.act_avg[i]), pv.rlo[i], pv.rhi[i]);
    }
    if (restart && it.halpern) {
        it.ya[i] = it.y[i];
        it.sa[i] = it.s[i];
    }
    if (restart && p.primal_weight_update) {
        const double yn = static_cast<double>(it.y[i]);
        d = yn - p.y_last[i];
        p.y_last[i] = yn;
    }
    if constexpr (std::is_same<T, float>::value)
        it.ysum[i] = restart ? 0.0 : it.ysum[i] + static_cast<double>(it.psy[i]);
    return d * d;
}
// The distance that such a restart moves a column / row, before it does.
template <class T>
__device__ __forceinline__ double restart_move_col(const Iterates<T>& it, const BatchParams& p, const PV<T>& pv, int j,
                                                   bool to_avg, double inv) {
    const T x = to_avg ? clampT<T>(static_cast<T>(avg_x(it, j, inv)), pv.lo[j], pv.hi[j]) : it.x[j];
    return static_cast<double>(x) - p.x_last[j];
}
template <class T>
__device__ __forceinline__ double restart_move_row(const Iterates<T>& it, const BatchParams& p, int i, bool to_avg,
                                                   double inv) {
    const T y = to_avg ? static_cast<T>(avg_y(it, i, inv)) : it.y[i];
    return static_cast<double>(y) - p.y_last[i];
}
__device__ __forceinline__ void restart_weight(InstState& s, double dx2, double dy2) {
    const double dx = sqrt(dx2), dy = sqrt(dy2);
    if (dx > 1e-10 && dy > 1e-10) {
        s.omega = sqrt(s.omega * (dy / dx));
        s.tau = s.eta / s.omega;
        s.sigma = s.eta * s.omega;
    }
}

}  // namespace
}  // namespace pdhg
