// pms_plasticity.cu -- general elastoplastic stress update, batched: one thread per IP.
//
// Replaces Elastoplastic::update_stress (reference src/material/elastoplastic.rs:539-641) with the
// von Mises plasticity model (PlasticityTrait for VonMises, src/material/von_mises.rs:229-282),
// the only model that Elastoplastic::new accepts (elastoplastic.rs:129-135).  Per IP:
//
//   1. yield function f = sigma_d - z (von_mises.rs:236-240) at the start;
//   2. case selection (select_case, elastoplastic.rs:437-499): inside (A) or on/outside (B);
//      going inside when (df/dsigma) : D_e : deps < 0 (going_inside, :379-389); the crossings of
//      the yield surface along the elastic path (intersection_finding, :394-435) give the cases
//      AE, AXB(t), BE, BXP(t), BP with the pseudo-time tolerance 1e-7;
//   3. the elastic part: sigma(t) = sigma0 + t D_e : deps;
//   4. the elastoplastic part: the ODE dsigma/dt = D_ep : deps, dz/dt = Lambda_d H
//      (ode_system_ep, :159-205) from t_int (or 0) to 1.
//
// Two departures from the reference's numerics, both because the B200 path needs no host-side
// solver objects and both exact for this model:
//   * the elastic path is linear in t (linear elasticity), so f(t) = 0 is the root of a quadratic
//     in t, solved in closed form; the reference finds the same roots with a Chebyshev interpolant
//     of f (30 points, truncated at 1e-8) and its companion-matrix root finder;
//   * the ODE is integrated with the Dormand-Prince 5(4) pair (Dormand & Prince 1980, 7 stages,
//     first-same-as-last) and the standard step-size controller (Hairer, Norsett & Wanner, Solving
//     ODEs I, II.4); the reference uses russell_ode's DoPri8.  Along a radial path D_ep : deps is
//     constant and every Runge-Kutta method is exact; elsewhere both are accurate to the tolerance.
//
// The tangent of this model is not built: the reference's Elastoplastic::stiffness returns
// Err("TODO") (elastoplastic.rs:528-537).
// Roofline: HBM-bound for elastic and radial IPs (reads sigma, z, deps: 13 doubles in 3D; writes
// sigma, z, flag); FP64-bound otherwise (about 330 instructions for each ODE step of a plastic IP).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>

#include "../../include/pms.h"
#include "pms_device.cuh"

using namespace pms;

namespace {

constexpr double NUMERATOR_TOL = 1e-8;     // elastoplastic.rs:17
constexpr double PSEUDO_TIME_TOL = 1e-7;   // elastoplastic.rs:23
constexpr double SIGMA_D_SINGULAR = 1e-10;  // df/dsigma is undefined at sigma_d = 0

enum EpErr : int {
    E_DF_DSIGMA = PMS_ERR_DF_DSIGMA,
    E_NUMERATOR = PMS_ERR_NUMERATOR,
    E_ODE = PMS_ERR_ODE,
    E_INTERSECTION = PMS_ERR_INTERSECTION,
};

struct EpConst {
    double rtol, atol, h_ini;
    int max_steps;
};

__device__ __forceinline__ void report(int32_t* status, int code, int64_t ip) {
    if (status == nullptr || code == OK) return;
    if (atomicCAS(status, 0, code) == 0) {
        status[1] = (int32_t)(ip & 0x7fffffff);
        status[2] = (int32_t)(ip >> 31);
    }
}

// deviator of a Mandel vector (the shear components are already deviatoric)
template <int NC>
__device__ __forceinline__ void deviator(const double* v, double* d) {
    const double m = (v[0] + v[1] + v[2]) / 3.0;
    d[0] = v[0] - m;
    d[1] = v[1] - m;
    d[2] = v[2] - m;
#pragma unroll
    for (int i = 3; i < NC; i++) d[i] = v[i];
}

template <int NC>
__device__ __forceinline__ double ddot(const double* a, const double* b) {
    double r = 0.0;
#pragma unroll
    for (int i = 0; i < NC; i++) r = fma(a[i], b[i], r);
    return r;
}

// The flow in the plane of two deviators.  With an isotropic elastic law and n = 3/2 s / sigma_d the ODE
// of elastoplastic.rs:159-205 reads (D_e : n = 2G n, n : D_e : n = 3G, ds_e = dev(D_e : deps) constant)
//   ds/dt = ds_e - k s,   k = 3G/(H + 3G) (3/2 s:ds_e)/sigma_d^2,   dz/dt = H/(H + 3G) max(0, n : D_e : deps)
// and a constant rate of the mean stress.  So s stays in the plane of its start value s_a and of
// s_b = ds_e: s = alpha s_a + beta s_b, dalpha/dt = -k alpha, dbeta/dt = 1 - k beta, where
// sigma_d^2 and s:ds_e come from the three products of s_a and s_b.  A Runge-Kutta step commutes with
// this linear map, so the steps (sizes, rejections, errors) are those of the stress components
// up to rounding, at two scalars a stage instead of 2*NDIM + 1 with a division for each component.
struct EpPlane {
    double aa, ab, bb;  // 3/2 s_a:s_a, 3/2 s_a:s_b, 3/2 s_b:s_b
    double kap, hz;     // 3G/(H + 3G), H/(H + 3G)
};

struct EpRate {
    double a, b, z;  // dalpha/dt, dbeta/dt, dz/dt
};

__device__ __forceinline__ int ep_rates(const EpPlane& g, double al, double be, EpRate& o) {
    const double u = fma(al, g.aa, be * g.ab), p = fma(al, g.ab, be * g.bb);  // 3/2 s:s_a, 3/2 s:s_b
    const double q = fma(al, u, be * p);                                      // sigma_d^2
    if (!(q > SIGMA_D_SINGULAR * SIGMA_D_SINGULAR)) return E_DF_DSIGMA;
    const double r = rsqrt(q);
    const double num = p * r;  // n : D_e : deps
    if (num < -NUMERATOR_TOL) return E_NUMERATOR;
    const double k = g.kap * num * r;
    o.a = -k * al;
    o.b = fma(-k, be, 1.0);
    o.z = g.hz * fmax(0.0, num);
    return OK;
}

// v^(-1/10) by Newton's method on y^-10 = v (y += y (1 - v y^10) / 10) from a single-precision start:
// the relative error e becomes 11/2 e^2, so two rounds take 1e-6 to rounding.
__device__ __forceinline__ double inv_tenth_root(double v) {
    double y = (double)exp2f(-0.1f * log2f((float)v));
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const double y2 = y * y, y4 = y2 * y2, y10 = y4 * y4 * y2;
        y = fma(0.1 * y, fma(-v, y10, 1.0), y);
    }
    return y;
}

// Sum of (e_i/s_i)^2 over up to four entries with one division; entries whose products leave the
// range (scales beyond 1e+-35) are divided one by one.
template <int N>
__device__ __forceinline__ double sum_of_squares(const double* e, const double* s) {
    double num = e[0] * e[0], den = s[0] * s[0];
#pragma unroll
    for (int i = 1; i < N; i++) {
        const double s2 = s[i] * s[i];
        num = fma(num, s2, e[i] * e[i] * den);
        den *= s2;
    }
    if (den > 1e-280 && den < 1e280 && num < 1e280) return num / den;
    double t = 0.0;
#pragma unroll
    for (int i = 0; i < N; i++) t += (e[i] / s[i]) * (e[i] / s[i]);
    return t;
}

// One IP on its way through the plastic part: Dormand-Prince 5(4) with the standard controller, from t0
// to 1.
template <int NC>
struct EpPoint {
    EpPlane g;
    double sa[NC], sb[NC];  // the deviators that span the flow
    double m0, dm, t0;      // mean stress at t0 and its rate
    double al, be, z;       // the state
    double y[NC];           // |sigma_i| of the state (error scales)
    EpRate k1;
    double t, h;
    int steps;
    bool rejected;

    __device__ __forceinline__ double mean(double tt) const { return fma(tt - t0, dm, m0); }
    __device__ __forceinline__ double sigma(int i, double a, double b, double m) const {
        return fma(a, sa[i], fma(b, sb[i], i < 3 ? m : 0.0));
    }

    // sig0: the stress at t0; sb is filled already
    __device__ __forceinline__ int begin(const MatConst& mc, const EpConst& e, double start, const double* sig0,
                                         const double* dse, double zz) {
        t = t0 = start;
        m0 = (sig0[0] + sig0[1] + sig0[2]) / 3.0;
        dm = (dse[0] + dse[1] + dse[2]) / 3.0;
        deviator<NC>(sig0, sa);
        g.aa = 1.5 * ddot<NC>(sa, sa);
        g.ab = 1.5 * ddot<NC>(sa, sb);
        g.bb = 1.5 * ddot<NC>(sb, sb);
        const double hp = mc.hh + 3.0 * mc.gg;
        g.kap = 3.0 * mc.gg / hp;
        g.hz = mc.hh / hp;
        al = 1.0;
        be = 0.0;
        z = zz;
#pragma unroll
        for (int i = 0; i < NC; i++) y[i] = fabs(sig0[i]);
        h = fmin(e.h_ini, 1.0 - t0);
        steps = 0;
        rejected = false;
        return ep_rates(g, al, be, k1);
    }

    // One step.  Returns an Err code; the IP is done when t has reached 1.
    __device__ __forceinline__ int step(const EpConst& e) {
        // Butcher tableau (Dormand & Prince 1980); the 5th-order weights equal row 7 (FSAL)
        constexpr double a21 = 1.0 / 5.0;
        constexpr double a31 = 3.0 / 40.0, a32 = 9.0 / 40.0;
        constexpr double a41 = 44.0 / 45.0, a42 = -56.0 / 15.0, a43 = 32.0 / 9.0;
        constexpr double a51 = 19372.0 / 6561.0, a52 = -25360.0 / 2187.0, a53 = 64448.0 / 6561.0, a54 = -212.0 / 729.0;
        constexpr double a61 = 9017.0 / 3168.0, a62 = -355.0 / 33.0, a63 = 46732.0 / 5247.0, a64 = 49.0 / 176.0,
                         a65 = -5103.0 / 18656.0;
        constexpr double b1 = 35.0 / 384.0, b3 = 500.0 / 1113.0, b4 = 125.0 / 192.0, b5 = -2187.0 / 6784.0,
                         b6 = 11.0 / 84.0;
        // error weights: 5th-order minus 4th-order weights
        constexpr double e1 = 71.0 / 57600.0, e3 = -71.0 / 16695.0, e4 = 71.0 / 1920.0, e5 = -17253.0 / 339200.0,
                         e6 = 22.0 / 525.0, e7 = -1.0 / 40.0;
        if (steps >= e.max_steps) return E_ODE;
        steps++;
        const bool last = t + h >= 1.0;
        if (last) h = 1.0 - t;
        EpRate k2, k3, k4, k5, k6, k7;
        int rc;
        if ((rc = ep_rates(g, fma(h, a21 * k1.a, al), fma(h, a21 * k1.b, be), k2)) != OK) return rc;
        if ((rc = ep_rates(g, fma(h, a31 * k1.a + a32 * k2.a, al), fma(h, a31 * k1.b + a32 * k2.b, be), k3)) != OK)
            return rc;
        if ((rc = ep_rates(g, fma(h, a41 * k1.a + a42 * k2.a + a43 * k3.a, al),
                           fma(h, a41 * k1.b + a42 * k2.b + a43 * k3.b, be), k4)) != OK)
            return rc;
        if ((rc = ep_rates(g, fma(h, a51 * k1.a + a52 * k2.a + a53 * k3.a + a54 * k4.a, al),
                           fma(h, a51 * k1.b + a52 * k2.b + a53 * k3.b + a54 * k4.b, be), k5)) != OK)
            return rc;
        if ((rc = ep_rates(g, fma(h, a61 * k1.a + a62 * k2.a + a63 * k3.a + a64 * k4.a + a65 * k5.a, al),
                           fma(h, a61 * k1.b + a62 * k2.b + a63 * k3.b + a64 * k4.b + a65 * k5.b, be), k6)) != OK)
            return rc;
        const double al5 = fma(h, b1 * k1.a + b3 * k3.a + b4 * k4.a + b5 * k5.a + b6 * k6.a, al);
        const double be5 = fma(h, b1 * k1.b + b3 * k3.b + b4 * k4.b + b5 * k5.b + b6 * k6.b, be);
        const double z5 = fma(h, b1 * k1.z + b3 * k3.z + b4 * k4.z + b5 * k5.z + b6 * k6.z, z);
        if ((rc = ep_rates(g, al5, be5, k7)) != OK) return rc;
        const double ea = h * (e1 * k1.a + e3 * k3.a + e4 * k4.a + e5 * k5.a + e6 * k6.a + e7 * k7.a);
        const double eb = h * (e1 * k1.b + e3 * k3.b + e4 * k4.b + e5 * k5.b + e6 * k6.b + e7 * k7.b);
        // mean square of the error of (sigma, z) over its scales (the mean stress has no error)
        double y5[NC], ei[NC + 1], sc[NC + 1];
        const double m5 = mean(t + h);
#pragma unroll
        for (int i = 0; i < NC; i++) {
            y5[i] = fabs(sigma(i, al5, be5, m5));
            ei[i] = fma(ea, sa[i], eb * sb[i]);
            sc[i] = fma(e.rtol, fmax(y[i], y5[i]), e.atol);
        }
        ei[NC] = h * (e1 * k1.z + e3 * k3.z + e4 * k4.z + e5 * k5.z + e6 * k6.z + e7 * k7.z);
        sc[NC] = fma(e.rtol, fmax(fabs(z), fabs(z5)), e.atol);
        constexpr int N1 = (NC + 1) / 2;
        const double v = (sum_of_squares<N1>(ei, sc) + sum_of_squares<NC + 1 - N1>(ei + N1, sc + N1)) *
                         (1.0 / (NC + 1));
        // new step: h * min(fac_max, max(fac_min, 0.9 err^(-1/5))), err = sqrt(v); the factor is clamped to
        // [0.2, 10], which v outside [1e-12, 1e8] is already
        double fac = v > 0.0 ? 0.9 * inv_tenth_root(fmin(fmax(v, 1e-12), 1e8)) : 10.0;
        if (v <= 1.0) {
            t = last ? 1.0 : t + h;
            al = al5;
            be = be5;
            z = z5;
            k1 = k7;
#pragma unroll
            for (int i = 0; i < NC; i++) y[i] = y5[i];
            fac = fmin(rejected ? 1.0 : 10.0, fmax(0.2, fac));
            rejected = false;
        } else {
            fac = fmin(1.0, fmax(0.2, fac));
            rejected = true;
        }
        h *= fac;
        return OK;
    }
};

// Case selection of one IP.  Returns an Err code; an elastic IP (cases AE, BE) is done: sig is its new
// stress.  Otherwise pt is at the start of its plastic part.
template <int NC>
__device__ __forceinline__ int ep_select(const MatConst& m, const EpConst& e, double* sig, double z,
                                         const double* deps, int& cs, EpPoint<NC>& pt) {
    double dse[NC];
#pragma unroll
    for (int i = 0; i < NC; i++) dse[i] = 0.0;
    hooke_add<NC>(m, dse, deps);  // D_e : deps
    double s0[NC];
    double* ds = pt.sb;
    deviator<NC>(sig, s0);
    deviator<NC>(dse, ds);
    // along sigma(t) = sigma0 + t dse with z frozen: 3/2 |s0 + t ds|^2 = z^2  <=>
    // a t^2 + 2 b t + cp = 0, a = ds:ds, b = s0:ds, cp = s0:s0 - 2/3 z^2
    const double a = ddot<NC>(ds, ds), b = ddot<NC>(s0, ds), c = ddot<NC>(s0, s0);
    const double cp = c - (2.0 / 3.0) * z * z;
    const double f0 = sqrt(1.5 * c) - z;
    double t_int = 0.0;
    if (f0 < 0.0) {
        // A: inside.  cp < 0, so g(t) = a t^2 + 2 b t + cp has one positive root (a > 0)
        bool root = false;
        if (a > 0.0) {
            const double sq = sqrt(b * b - a * cp);
            t_int = b >= 0.0 ? -cp / (b + sq) : (sq - b) / a;
            root = t_int <= 1.0;
        }
        if (!root) cs = PMS_EP_AE;
        else if (t_int <= PSEUDO_TIME_TOL) cs = PMS_EP_BP;
        else if (t_int >= 1.0 - PSEUDO_TIME_TOL) cs = PMS_EP_AE;
        else cs = PMS_EP_AXB;
    } else {
        // B: on or outside.  going inside: (df/dsigma) : D_e : deps = 3/2 (s0 : dse) / sigma_d < 0
        const double sd0 = f0 + z;
        if (!(sd0 > SIGMA_D_SINGULAR)) return E_DF_DSIGMA;
        // loading tangent to the surface (indicator zero up to rounding, |s0:ds| <= 1e-10 |s0||ds|)
        // is not going inside: the reference's own tangent path (update_stress_von_mises_5) is BP
        const double indicator = 1.5 * b / sd0;
        if (indicator < -1e-10 * 1.5 * sqrt(a * c) / sd0) {
            // b < 0 and cp >= 0 (up to rounding): the smaller root is the start point (counted as
            // a crossing, t1 ~ 0), the larger one is where the path leaves the surface again
            int nroot = 0;
            double t2 = 2.0;
            const double disc = b * b - a * cp;
            if (a > 0.0 && disc >= 0.0) {
                const double q = sqrt(disc) - b;  // > 0
                const double t1 = cp / q;
                t2 = q / a;
                // a second crossing at t = 1 up to rounding still counts (it ends the path on the surface)
                nroot = (t1 <= 1.0 ? 1 : 0) + (t2 >= 0.0 && t2 <= 1.0 + PSEUDO_TIME_TOL ? 1 : 0);
            }
            if (nroot == 2) {
                t_int = t2;
                if (t_int <= PSEUDO_TIME_TOL) cs = PMS_EP_BP;
                else if (t_int >= 1.0 - PSEUDO_TIME_TOL) cs = PMS_EP_BE;
                else cs = PMS_EP_BXP;
            } else {
                // no way back out: the trial point must lie inside (elastoplastic.rs:484)
                const double f1 = sqrt(1.5 * (a + 2.0 * b + c)) - z;
                if (f1 > 0.0) return E_INTERSECTION;
                cs = PMS_EP_BE;
            }
        } else {
            cs = PMS_EP_BP;
        }
    }
    if (cs == PMS_EP_AE || cs == PMS_EP_BE) {
#pragma unroll
        for (int i = 0; i < NC; i++) sig[i] += dse[i];
        return OK;
    }
    const double t0 = (cs == PMS_EP_BP) ? 0.0 : t_int;
#pragma unroll
    for (int i = 0; i < NC; i++) sig[i] += t0 * dse[i];
    return pt.begin(m, e, t0, sig, dse, z);
}

// One lane per IP.  The steps of the ODE differ from IP to IP (31 on average, up to 94, on the timed
// set), so a lane that is done takes the warp's next IP instead of waiting for the longest of 32:
// warp w of nwarp owns the runs of 32 IPs w, w + nwarp, ... and hands out their IPs in order, once
// REFILL lanes are idle (the selection costs about as much as a step, for one lane or for 32;
// REFILL = 4, 8 and 12 measured 1.44, 1.45 and 1.49 ms, no refill before all are done 2.15 ms).
// Bound by the FP64 pipe (49% busy in 3D) and its latency: about 330 instructions a step, 12 warps per SM in 3D (162
// registers; 16 warps with spills and 10 without measured the same or slower), 16 in 2D.
// 1,048,576 IPs, half of them on the yield surface, the others inside it: 28.4 ms in 3D and 5.3 ms in
// 2D with all stress components integrated, one IP a thread; 1.45 and 0.88 ms here.  4,000 3D IPs:
// 1.13 and 0.11 ms.
constexpr int EP_THREADS = 64;
constexpr int REFILL = 8;
__host__ __device__ constexpr int ep_blocks_per_sm(int nc) { return nc == 6 ? 6 : 8; }

template <int NC>
__global__ void __launch_bounds__(EP_THREADS, ep_blocks_per_sm(NC))
ep_update_kernel(MatConst m, EpConst e, int64_t n, double* __restrict__ sig, double* __restrict__ z,
                 uint8_t* __restrict__ elastic, const double* __restrict__ deps, int32_t* __restrict__ cases,
                 int32_t* __restrict__ steps, int32_t* status) {
    const int lane = threadIdx.x & 31;
    const int64_t w = ((int64_t)blockIdx.x * EP_THREADS + threadIdx.x) >> 5;
    const int64_t nwarp = ((int64_t)gridDim.x * EP_THREADS) >> 5;
    const int64_t nrun = (n + 31) >> 5;
    const int64_t end = w < nrun ? ((nrun - w + nwarp - 1) / nwarp) << 5 : 0;  // IPs of this warp's runs
    int64_t next = 0;
    EpPoint<NC> pt;
    int64_t i = 0;
    int cs = -1;
    bool busy = false;
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !busy);
        const int nidle = __popc(idle);
        if (next < end && nidle >= REFILL) {
            if (!busy) {
                const int64_t j = next + __popc(idle & ((1u << lane) - 1u));
                i = (((j >> 5) * nwarp + w) << 5) + (j & 31);
                if (j < end && i < n) {
                    double s[NC], de[NC];
#pragma unroll
                    for (int c = 0; c < NC; c++) {
                        s[c] = sig[(int64_t)c * n + i];
                        de[c] = deps[(int64_t)c * n + i];
                    }
                    cs = -1;
                    const int rc = ep_select<NC>(m, e, s, z[i], de, cs, pt);
                    busy = rc == OK && cs != PMS_EP_AE && cs != PMS_EP_BE;
                    if (!busy) {
                        if (rc != OK) {
                            report(status, rc, i);
                        } else {
#pragma unroll
                            for (int c = 0; c < NC; c++) sig[(int64_t)c * n + i] = s[c];
                            elastic[i] = 1;
                        }
                        if (cases) cases[i] = rc == OK ? cs : -1;
                        if (steps) steps[i] = 0;
                    }
                }
            }
            next += nidle;
            continue;
        }
        if (nidle == 32) break;
        if (busy) {
            const int rc = pt.t < 1.0 ? pt.step(e) : OK;
            if (rc != OK || !(pt.t < 1.0)) {
                if (rc != OK) {
                    report(status, rc, i);
                } else {
                    const double mean = pt.mean(pt.t);
#pragma unroll
                    for (int c = 0; c < NC; c++) sig[(int64_t)c * n + i] = pt.sigma(c, pt.al, pt.be, mean);
                    z[i] = pt.z;
                    elastic[i] = 0;
                }
                if (cases) cases[i] = rc == OK ? cs : -1;
                if (steps) steps[i] = pt.steps;
                busy = false;
            }
        }
    }
}

}  // namespace

extern "C" int pms_ep_update_stress_batch(const pms_material* mat, int32_t ndim, int64_t n, double* sig, double* z,
                                          uint8_t* elastic, const double* deps, const pms_ep_settings* settings,
                                          int32_t* cases, int32_t* steps, int32_t* status, void* stream) {
    if (!mat || (ndim != 2 && ndim != 3) || n < 0) return PMS_ERR_INVALID;
    if (mat->model != PMS_VON_MISES) return PMS_ERR_INVALID;  // elastoplastic.rs:131-134
    if (!(mat->young > 0.0) || !(mat->poisson > -1.0 && mat->poisson < 0.5) || !(mat->hh >= 0.0))
        return PMS_ERR_INVALID;
    if (n == 0) return PMS_OK;
    if (!sig || !z || !elastic || !deps) return PMS_ERR_INVALID;
    EpConst e;
    e.rtol = settings ? settings->tol_rel : 1e-10;
    e.atol = settings ? settings->tol_abs : 1e-10;
    e.h_ini = settings ? settings->h_ini : 1.0;
    e.max_steps = settings ? settings->max_steps : 1000;
    if (!(e.rtol > 0.0) || !(e.atol > 0.0) || !(e.h_ini > 0.0) || e.max_steps < 1) return PMS_ERR_INVALID;
    const MatConst m = make_matconst(PMS_VON_MISES, mat->young, mat->poisson, mat->hh, mat->z_ini);
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t blocks = std::min<int64_t>((n + EP_THREADS - 1) / EP_THREADS, (int64_t)sms * ep_blocks_per_sm(2 * ndim));  // one wave
    cudaStream_t st = (cudaStream_t)stream;
    if (ndim == 2)
        ep_update_kernel<4><<<(unsigned)blocks, EP_THREADS, 0, st>>>(m, e, n, sig, z, elastic, deps, cases, steps, status);
    else
        ep_update_kernel<6><<<(unsigned)blocks, EP_THREADS, 0, st>>>(m, e, n, sig, z, elastic, deps, cases, steps, status);
    return cudaGetLastError() == cudaSuccess ? PMS_OK : PMS_ERR_CUDA;
}

namespace {
// device staging of the host-buffer entry, grown on demand and kept until exit
struct EpStage {
    std::mutex mu;
    void* buf = nullptr;
    size_t bytes = 0;
    cudaStream_t stream = nullptr;
} g_ep_stage;
}  // namespace

extern "C" int pms_ep_update_stress_host(const pms_material* mat, int32_t ndim, int64_t n, double* sig, double* z,
                                         uint8_t* elastic, const double* deps, const pms_ep_settings* settings,
                                         int32_t* cases, int32_t* steps) {
    if (!mat || (ndim != 2 && ndim != 3) || n < 0) return PMS_ERR_INVALID;
    if (n == 0) return PMS_OK;
    if (!sig || !z || !elastic || !deps) return PMS_ERR_INVALID;
    const size_t nc = 2 * (size_t)ndim, b_sig = nc * n * 8, b_n = (size_t)n * 8, b_i = (size_t)n * 4;
    const size_t need = 64 + 2 * b_sig + b_n + (cases ? b_i : 0) + (steps ? b_i : 0) + (size_t)n;
    std::lock_guard<std::mutex> lock(g_ep_stage.mu);
    if (!g_ep_stage.stream && cudaStreamCreateWithFlags(&g_ep_stage.stream, cudaStreamNonBlocking) != cudaSuccess)
        return PMS_ERR_CUDA;
    if (g_ep_stage.bytes < need) {
        if (g_ep_stage.buf) cudaFree(g_ep_stage.buf);
        g_ep_stage.buf = nullptr;
        g_ep_stage.bytes = 0;
        if (cudaMalloc(&g_ep_stage.buf, need) != cudaSuccess) return PMS_ERR_NOMEM;
        g_ep_stage.bytes = need;
    }
    char* p = (char*)g_ep_stage.buf;
    int32_t* d_status = (int32_t*)p; p += 64;
    double* d_sig = (double*)p; p += b_sig;
    double* d_deps = (double*)p; p += b_sig;
    double* d_z = (double*)p; p += b_n;
    int32_t* d_cases = nullptr;
    if (cases) { d_cases = (int32_t*)p; p += b_i; }
    int32_t* d_steps = nullptr;
    if (steps) { d_steps = (int32_t*)p; p += b_i; }
    uint8_t* d_el = (uint8_t*)p;
    cudaStream_t s = g_ep_stage.stream;
    cudaMemsetAsync(d_status, 0, 16, s);
    cudaMemcpyAsync(d_sig, sig, b_sig, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(d_deps, deps, b_sig, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(d_z, z, b_n, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(d_el, elastic, (size_t)n, cudaMemcpyHostToDevice, s);
    int rc = pms_ep_update_stress_batch(mat, ndim, n, d_sig, d_z, d_el, d_deps, settings, d_cases, d_steps,
                                        d_status, s);
    if (rc) {
        cudaStreamSynchronize(s);
        return rc;
    }
    cudaMemcpyAsync(sig, d_sig, b_sig, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(z, d_z, b_n, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(elastic, d_el, (size_t)n, cudaMemcpyDeviceToHost, s);
    if (cases) cudaMemcpyAsync(cases, d_cases, b_i, cudaMemcpyDeviceToHost, s);
    if (steps) cudaMemcpyAsync(steps, d_steps, b_i, cudaMemcpyDeviceToHost, s);
    int32_t hst[4] = {0, 0, 0, 0};
    cudaMemcpyAsync(hst, d_status, 16, cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) return PMS_ERR_CUDA;
    return hst[0];
}
