// integrands.cuh -- built-in device integrands, selected by id.
//
// In the reference an integrand is a std::function (Vegas.hh:27-28,
// Integrand.hh:41-47) and cannot cross to the device; the workloads' own
// integrands are compiled in and chosen by chili_integrand_kind.
#pragma once

#include <cmath>

#include "chili_gpu.h"
#include "common.cuh"

namespace chili_dev {

struct IntegrandDesc {
    int32_t kind;
    int32_t nparams;
    int32_t pre;  // chili_preprocess_kind
    int32_t n_ext;  // external legs (CHILI_PRE_CUTS)
    double p[CHILI_MAX_INTEGRAND_PARAMS];
    double cut[4];  // CHILI_PRE_CUTS: sqrts, ptmin, etamax, delta_r
    double sure[3];  // set_cut_bounds
};

// Bounds that decide most cuts of CHILI_PRE_CUTS without the transverse
// angles: |z| / pT below which |eta| <= etamax surely holds, and
// cosh(deta) - cos(dphi) above which a pair's Delta R surely reaches delta_r
// (at most cosh(R) - 1 on the circle of radius R) and below which it surely
// does not (at least 1 - cos(R), R <= pi).  The margins are far above the
// rounding of both sides; what they leave open takes the angles themselves.
inline void set_cut_bounds(IntegrandDesc &f) {
    const double eta = f.cut[2], r = f.cut[3];
    f.sure[0] = eta > 700.0 ? 1e300 : std::sinh(eta) * (1.0 - 1e-9) - 1e-9;
    f.sure[1] = r > 3.0 ? 1e300 : (std::cosh(r) - 1.0) * (1.0 + 1e-6) + 1e-9;
    f.sure[2] = r > 3.0 ? -1.0 : (1.0 - std::cos(r)) * (1.0 - 1e-6) - 1e-9;
}

// f(x) = N [exp(-|x-a|^2/s^2) + exp(-|x-b|^2/s^2)]; params {s, N, a[D], b[D]};
// s2 = s^2 and its reciprocal given (once per thread, not per point).
__device__ __forceinline__ double camel(const IntegrandDesc *__restrict__ f, const double *x, int dims, double s2,
                                        double rs2) {
    double d1 = 0, d2 = 0;
    for (int i = 0; i < dims; ++i) {
        double t = x[i] - f->p[2 + i];
        d1 += t * t;
        t = x[i] - f->p[2 + dims + i];
        d2 += t * t;
    }
    return f->p[1] * (exp(div_by(-d1, s2, rs2)) + exp(div_by(-d2, s2, rs2)));
}

// Pair Breit-Wigner sum (or product of the two largest) times the t-channel
// factors over the outgoing legs; params {M, G, m}.
__device__ __forceinline__ double propagator(const IntegrandDesc *__restrict__ f, const V4 *mom, int n_ext,
                                             bool top2) {
    const double m = f->p[0], g = f->p[1], mt = f->p[2];
    const double m2 = m * m, mw2 = m * m * g * g, mt2 = mt * mt;
    double sum = 0, big1 = 0, big2 = 0;
    for (int i = 2; i < n_ext; ++i) {
        for (int j = i + 1; j < n_ext; ++j) {
            const double d = mass2(mom[i] + mom[j]) - m2;
            const double bw = 1.0 / (d * d + mw2);
            sum += bw;
            if (bw > big1) {
                big2 = big1;
                big1 = bw;
            } else if (bw > big2) {
                big2 = bw;
            }
        }
    }
    double tprod = 1;
    for (int j = 2; j < n_ext; ++j) tprod *= 1.0 / (fabs(mass2(mom[0] + mom[j])) + mt2);
    return (top2 ? big1 * big2 : sum) * tprod;
}

__device__ __forceinline__ double eval_momenta(const IntegrandDesc *__restrict__ f, const V4 *mom, int n_ext) {
    switch (f->kind) {
    case CHILI_FUNC_PROPAGATOR: return propagator(f, mom, n_ext, false);
    case CHILI_FUNC_PROPAGATOR_TOP2: return propagator(f, mom, n_ext, true);
    default: return 1.0;
    }
}

// The eta and Delta R cuts of CHILI_PRE_CUTS on legs whose pT passed.
__device__ __noinline__ inline bool pass_angles(const IntegrandDesc *__restrict__ f, const V4 *mom) {
    const double etamax = f->cut[2], dr2 = f->cut[3] * f->cut[3];
    const int ne = f->n_ext;
    double eta[CHILI_MAX_EXT], phi[CHILI_MAX_EXT];
    for (int i = 2; i < ne; ++i) {
        const V4 q = mom[i];
        eta[i] = asinh(q.z / sqrt(q.x * q.x + q.y * q.y));
        if (!(fabs(eta[i]) <= etamax)) return false;
        phi[i] = atan2(q.y, q.x);
    }
    for (int i = 2; i < ne; ++i)
        for (int j = i + 1; j < ne; ++j) {
            double dphi = fabs(phi[i] - phi[j]);
            if (dphi > kPi) dphi = 2.0 * kPi - dphi;
            const double deta = eta[i] - eta[j];
            if (!(deta * deta + dphi * dphi >= dr2)) return false;
        }
    return true;
}

// The physical region and the cuts of CHILI_PRE_CUTS (include/chili_gpu.h).
// NaN momenta fail every comparison.  The bounds replace an asinh and an
// atan2 per leg by two roots: the forward pass of 1.7e6 2->4 points 0.59 ->
// 0.54 ms (with sincos; the angles inside the pair loop instead of behind it:
// 0.63 ms, some lane of a warp always took them).
__device__ __forceinline__ bool pass_cuts(const IntegrandDesc *__restrict__ f, const V4 *mom) {
    const double half = 0.5 * f->cut[0] * (1.0 + 1e-12);
    if (!(-mom[0].e <= half) || !(-mom[1].e <= half)) return false;
    const double pt2min = f->cut[1] * f->cut[1];
    const int ne = f->n_ext;
    double pabs[CHILI_MAX_EXT], ptr[CHILI_MAX_EXT];  // |p|, pT
    bool open = false;  // a cut that the bounds do not decide
    for (int i = 2; i < ne; ++i) {
        const V4 q = mom[i];
        const double t2 = q.x * q.x + q.y * q.y;
        if (!(t2 >= pt2min) || !(t2 > 0)) return false;
        ptr[i] = sqrt(t2);
        pabs[i] = sqrt(p2(q));
        open = open || !(fabs(q.z) < f->sure[0] * ptr[i]);
    }
    for (int i = 2; i < ne; ++i) {
        const V4 q = mom[i];
        for (int j = i + 1; j < ne; ++j) {
            // (|p_i| |p_j| - p_i p_j) / (pT_i pT_j) = cosh(deta) - cos(dphi);
            // its rounding error is a few ulps of |p_i| |p_j|
            const double pp = pabs[i] * pabs[j], tt = ptr[i] * ptr[j];
            const double v = pp - dot3(q, mom[j]);
            const bool sound = pp < 1e5 * tt;
            if (sound && v < f->sure[2] * tt) return false;
            open = open || !(sound && v > f->sure[1] * tt);
        }
    }
    return !open || pass_angles(f, mom);
}

// PreProcess (MultiChannel.hh:219-223); CHILI_PRE_FINITE follows the first
// check of src/example.cc:26-29.
__device__ __forceinline__ bool preprocess(const IntegrandDesc *__restrict__ f, const V4 *mom) {
    if (f->pre == CHILI_PRE_FINITE) return !isnan(mom[0].e);
    if (f->pre == CHILI_PRE_CUTS) return pass_cuts(f, mom);
    return true;
}

}  // namespace chili_dev
