// common.cuh — shared device helpers for libflame3d_b200 (sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <type_traits>

#include "../../include/flame3d_b200.h"

#include <nvtx3/nvToolsExt.h>  // header-only; a no-op unless a profiler is attached

namespace flame {

constexpr double kEps = 2.220446049250313e-16;  // CUDA.eps(Float64), utils.jl:100
// Scheme constants, run.jl:51-57.
constexpr double kWenoEps = 1e-26;
constexpr double kHybrid1 = 1e-3;
constexpr double kHybrid2 = 0.1;
constexpr double kUP7_2 = 17.0 / 600, kUP7_3 = -23.0 / 120, kUP7_4 = 22.0 / 30, kUP7_5 = 0.5,
                 kUP7_6 = -0.075, kUP7_7 = 0.005;  // UP7[1] is 0 (run.jl:57)

// Extents of a ghosted grid; every array index is computed in 64-bit.
struct Dims {
    int nx, ny, nz, ng, ns;
    long long tx, ty, tz, np;
    __host__ __device__ long long P(long long i, long long j, long long k) const {
        return i + tx * (j + ty * k);
    }
};

inline Dims make_dims(const FlameGrid &g) {
    Dims d;
    d.nx = g.nx, d.ny = g.ny, d.nz = g.nz, d.ng = g.ng, d.ns = g.ns;
    d.tx = g.nx + 2LL * g.ng, d.ty = g.ny + 2LL * g.ng, d.tz = g.nz + 2LL * g.ng;
    d.np = d.tx * d.ty * d.tz;
    return d;
}

__device__ __forceinline__ double jmax(double a, double b) {  // Julia max: NaN-propagating
    if (a != a || b != b) return __longlong_as_double(0x7ff8000000000000LL);
    return a > b ? a : b;
}

__device__ __forceinline__ int64_t tag_at(const int64_t *tag, long long p) {
    return tag ? tag[p] : 0;
}

// Reciprocal and reciprocal square root for the fused FP64 paths: the hardware's approximation
// (PTX rcp.approx.ftz.f64 / rsqrt.approx.ftz.f64) refined by one step of third order, without the
// branches of the correctly rounded forms.  With e = 1 - d x the reciprocal is x / (1 - e), and
// Householder's method (A. S. Householder, The Numerical Treatment of a Single Nonlinear Equation,
// 1970) cuts the series after x (1 + e + e^2): a seed good to 2^-20 gives 2^-57 before rounding.
// fast_rcp and fast_rsqrt are for the sweeps, whose arguments are normal (rsqrt: positive) with a
// normal result: for zero and infinity they give NaN, and a reciprocal below the normal range is
// flushed to zero.
__device__ __forceinline__ double fast_rcp(double d) {
    double x;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(d));
    const double e = fma(-d, x, 1.0);
    return fma(x, fma(e, e, e), x);
}
// The same where a zero or an infinity can occur: the seed is exact there, and the step that is
// then NaN is left out.
__device__ __forceinline__ double full_rcp(double d) {
    double x;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(d));
    const double e = fma(-d, x, 1.0), r = fma(x, fma(e, e, e), x);
    return r == r ? r : x;
}
// a / b: the quotient by the refined reciprocal and one correction from its residual (P. Markstein,
// Computation of elementary functions on the IBM RISC System/6000 processor, 1990), which leaves it
// within rounding of the correctly rounded one (no branch and no call, so a kernel near its register
// limit does not spill around it).  b is normal with a normal reciprocal, a finite.
__device__ __forceinline__ double fast_div(double a, double b) {
    const double r = fast_rcp(b), q = a * r;
    return fma(fma(-b, q, a), r, q);
}
// The same for any operands: a zero or infinite one, or a quotient that overflows, gives what a
// division gives, by the seed; a quotient or reciprocal below the normal range may come out as zero.
__device__ __forceinline__ double full_div(double a, double b) {
    double x;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(b));
    const double e = fma(-b, x, 1.0), r = fma(x, fma(e, e, e), x), q = a * r;
    const double c = fma(fma(-b, q, a), r, q);
    return fabs(c) > 0 ? c : a * x;  // not a number, or a zero, whose sign is the seed's too
}
// x (1 + e/2 + 3 e^2 / 8) with e = 1 - d x^2, the series of x / sqrt(1 - e) cut after the second
// order.  The rounding of d x leaves 2^-54 before that of the last multiply-add.
__device__ __forceinline__ double fast_rsqrt(double d) {
    double x;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(d));
    const double e = fma(-d * x, x, 1.0);
    return fma(x * e, fma(0.375, e, 0.5), x);
}

// ------------------------------------------------------------------ NASA-7 thermo (thermo.jl)
// h_specs, thermo.jl:107-133 (J/kg)
__device__ __forceinline__ double h_spec(const FlameThermo &th, int n, double T, double T2,
                                         double T3, double T4, double T5) {
    const double *lo = th.coeffs_lo + 7 * n;
    double h;
    if (T < th.coeffs_sep[n]) {
        h = lo[0] * T + lo[1] * T2 + lo[2] * T3 + lo[3] * T4 + lo[4] * T5;
    } else {
        const double *hc = th.coeffs_hi + 7 * n;
        h = hc[0] * T + hc[1] * T2 + hc[2] * T3 + hc[3] * T4 + hc[4] * T5 + (hc[5] - lo[5]);
    }
    return h * (th.Ru / th.mw[n]);
}

// cp_specs, thermo.jl:82-104 (dimensionless cp/R)
__device__ __forceinline__ double cp_spec(const FlameThermo &th, int n, double T, double T2,
                                          double T3, double T4) {
    const double *c = (T < th.coeffs_sep[n]) ? th.coeffs_lo + 7 * n : th.coeffs_hi + 7 * n;
    return c[0] + c[1] * T + c[2] * T2 + c[3] * T3 + c[4] * T4;
}

// ei_specs, thermo.jl:136-160 (dimensionless e/R)
__host__ __device__ __forceinline__ double ei_spec(const FlameThermo &th, int n, double T, double T2,
                                          double T3, double T4, double T5) {
    const double *lo = th.coeffs_lo + 7 * n;
    if (T < th.coeffs_sep[n])
        return (lo[0] - 1) * T + lo[1] * T2 + lo[2] * T3 + lo[3] * T4 + lo[4] * T5;
    const double *hc = th.coeffs_hi + 7 * n;
    return (hc[0] - 1) * T + hc[1] * T2 + hc[2] * T3 + hc[3] * T4 + hc[4] * T5 + (hc[5] - lo[5]);
}

// InternalEnergy, thermo.jl:219-228 (J/m^3)
template <int NS>
__host__ __device__ __forceinline__ double internal_energy(const FlameThermo &th, int ns, double T,
                                                  const double *rhoi) {
    double T2 = 0.5 * T * T;
    double T3 = 2.0 / 3.0 * T2 * T;
    double T4 = T2 * T2;
    double T5 = 0.8 * T4 * T;
    double r = 0;
    const int n_end = NS > 0 ? NS : ns;
#pragma unroll
    for (int n = 0; n < (NS > 0 ? NS : FLAME_MAX_NS); ++n) {
        if (n >= n_end) break;
        r += rhoi[n] * ei_spec(th, n, T, T2, T3, T4, T5) / th.mw[n];
    }
    return r * th.Ru;
}

// CV, thermo.jl:194-203 (J/(m^3 K))
template <int NS>
__device__ __forceinline__ double heat_cv(const FlameThermo &th, int ns, double T,
                                          const double *rhoi) {
    double T2 = T * T, T3 = T2 * T, T4 = T2 * T2;
    double r = 0;
    const int n_end = NS > 0 ? NS : ns;
#pragma unroll
    for (int n = 0; n < (NS > 0 ? NS : FLAME_MAX_NS); ++n) {
        if (n >= n_end) break;
        r += (cp_spec(th, n, T, T2, T3, T4) - 1) * rhoi[n] / th.mw[n];
    }
    return r * th.Ru;
}

// GetT, thermo.jl:231-282: Newton on e(T) with ±100 K step clamp and break-before-update.
template <int NS>
__device__ double get_T(const FlameThermo &th, int ns, double ein, const double *rhoi) {
    const double tol = 1e-3;
    const double tmin = th.min_temp, tmax = th.max_temp;
    const int n_end = NS > 0 ? NS : ns;
    double emin = internal_energy<NS>(th, ns, tmin, rhoi);
    double emax = internal_energy<NS>(th, ns, tmax, rhoi);
    if (ein < emin) return tmin - (emin - ein) / heat_cv<NS>(th, ns, tmin, rhoi);
    if (ein > emax) return tmax - (emax - ein) / heat_cv<NS>(th, ns, tmax, rhoi);
    double As = 0;
    for (int n = 0; n < n_end; ++n) As += (th.coeffs_lo[7 * n] - 1) * th.Ru / th.mw[n] * rhoi[n];
    double t1 = ein / As;
    if (t1 < tmin || t1 > tmax) t1 = tmin + (tmax - tmin) / (emax - emin) * (ein - emin);
    for (int it = 0; it < 30; ++it) {
        double e1 = internal_energy<NS>(th, ns, t1, rhoi);
        double cv = heat_cv<NS>(th, ns, t1, rhoi);
        double dt = (ein - e1) / cv;
        if (dt > 100.0)
            dt = 100.0;
        else if (dt < -100.0)
            dt = -100.0;
        else if (fabs(dt) < tol)
            break;
        else if (t1 + dt == t1)
            break;
        t1 += dt;
    }
    return t1;
}

// GetT for the fused stages: the same iteration as get_T (start, clamps, tolerance, break
// before the update), with e(T) and cv(T) of the mixture evaluated from its own polynomial.
// e/R and cv/R are linear in the species weights w_n = ρ_n / W_n, so the per-species NASA-7
// coefficients are summed once per cell into the mixture's coefficients for the low and the
// high range; an iteration then costs one polynomial instead of ns.  Where T lies between
// separators of different species the per-species sums are used.  The result differs from
// get_T by round-off only.
template <int NS>
struct MixPoly {
    double lo[5], hi[5], off, smin, smax;  // e/R = Σ_a c_a T_a (+ off in the high range)
    double wsum;                           // Σ_n w_n, so that Σ_n w_n cp_n = cv + Ru wsum
    const FlameThermo *th;
    const double *rhoi;
    __device__ __forceinline__ MixPoly(const FlameThermo &t, const double *r) : th(&t), rhoi(r) {
#pragma unroll
        for (int a = 0; a < 5; ++a) lo[a] = 0.0, hi[a] = 0.0;
        off = 0.0, wsum = 0.0;
        smin = smax = t.coeffs_sep[0];
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            const double w = fast_div(r[n], t.mw[n]);
            wsum += w;
            const double *L = t.coeffs_lo + 7 * n, *H = t.coeffs_hi + 7 * n;
            lo[0] += w * (L[0] - 1), hi[0] += w * (H[0] - 1);
#pragma unroll
            for (int a = 1; a < 5; ++a) lo[a] += w * L[a], hi[a] += w * H[a];
            off += w * (H[5] - L[5]);
            smin = fmin(smin, t.coeffs_sep[n]), smax = fmax(smax, t.coeffs_sep[n]);
        }
    }
    __device__ __forceinline__ double e(double T) const {  // InternalEnergy, J/m^3
        if (T >= smin && T < smax) return internal_energy<NS>(*th, NS, T, rhoi);
        const double T2 = 0.5 * T * T, T3 = 2.0 / 3.0 * T2 * T, T4 = T2 * T2, T5 = 0.8 * T4 * T;
        const double *c = T < smin ? lo : hi;
        const double r = c[0] * T + c[1] * T2 + c[2] * T3 + c[3] * T4 + c[4] * T5;
        return (T < smin ? r : r + off) * th->Ru;
    }
    __device__ __forceinline__ double cv(double T) const {  // CV, J/(m^3 K)
        if (T >= smin && T < smax) return heat_cv<NS>(*th, NS, T, rhoi);
        const double *c = T < smin ? lo : hi;
        const double T2 = T * T, T3 = T2 * T, T4 = T2 * T2;
        return (c[0] + c[1] * T + c[2] * T2 + c[3] * T3 + c[4] * T4) * th->Ru;
    }
};

template <int NS>
__device__ double get_T_mix(const MixPoly<NS> &M, const FlameThermo &th, double ein) {
    const double tol = 1e-3;
    const double tmin = th.min_temp, tmax = th.max_temp;
    const double emin = M.e(tmin), emax = M.e(tmax);
    if (ein < emin) return tmin - (emin - ein) / M.cv(tmin);
    if (ein > emax) return tmax - (emax - ein) / M.cv(tmax);
    // Σ_n (a1_n - 1) Ru / W_n ρ_n is the mixture's own; where it is zero ein / 0 lies outside as well
    double t1 = ein * fast_rcp(M.lo[0] * th.Ru);
    if (!(t1 >= tmin && t1 <= tmax)) t1 = tmin + (tmax - tmin) / (emax - emin) * (ein - emin);
    for (int it = 0; it < 30; ++it) {
        double dt = (ein - M.e(t1)) * full_rcp(M.cv(t1));
        if (dt > 100.0)
            dt = 100.0;
        else if (dt < -100.0)
            dt = -100.0;
        else if (fabs(dt) < tol)
            break;
        else if (t1 + dt == t1)
            break;
        t1 += dt;
    }
    return t1;
}

// Pmixture, thermo.jl:20-26
template <int NS>
__device__ __forceinline__ double p_mixture(const FlameThermo &th, int ns, double T,
                                            const double *rhoi) {
    double yow = 0;
    const int n_end = NS > 0 ? NS : ns;
#pragma unroll
    for (int n = 0; n < (NS > 0 ? NS : FLAME_MAX_NS); ++n) {
        if (n >= n_end) break;
        yow += rhoi[n] / th.mw[n];
    }
    return th.Ru * T * yow;
}

// ----------------------------------------------------------- hybrid reconstruction (schemes.jl)
template <typename T>
__device__ __forceinline__ T minmod(T a, T b) {  // schemes.jl:26-28
    return (a * b > 0) ? ((fabs(a) > fabs(b)) ? b : a) : T(0);
}

// WENO-Z weights and combination, schemes.jl:152-162, for the 1:1 kernels: the smoothness
// indicators come in the arithmetic type T and the weights are formed in FP64 in the reference's
// four-division form (in plain FP32, q = τ/(1e-26 + β) overflows when a one-sided split makes β
// exactly 0, and ∞·0 would poison the flux; wenoz_combine_fast below avoids that).
template <typename T>
__device__ __forceinline__ T wenoz_combine(T s11_, T s22_, T s33_, T v1, T v2, T v3) {
    const double s11 = s11_, s22 = s22_, s33 = s33_;
    const double tau = fabs(s11 - s33);
    double q, a1, a2, a3;
    q = tau / (kWenoEps + s11), a1 = (1 + q * q) * 1;
    q = tau / (kWenoEps + s22), a2 = (1 + q * q) * 6;
    q = tau / (kWenoEps + s33), a3 = (1 + q * q) * 3;
    const double invsum = 1 / (a1 + a2 + a3);
    return T((1.0 / 6.0) * invsum * (a1 * double(v1) + a2 * double(v2) + a3 * double(v3)));
}

// WENO-Z5 positive-flux reconstruction from V1..V5 = F+[c-3..c+1], schemes.jl:139-162
template <typename T>
__device__ __forceinline__ T wenoz_plus(T V1, T V2, T V3, T V4, T V5) {
    const T tmp1 = T(13.0 / 12.0), q4 = T(0.25);
    T a, b;
    a = V1 - 2 * V2 + V3, b = V1 - 4 * V2 + 3 * V3;
    const T s11 = tmp1 * (a * a) + q4 * (b * b);
    a = V2 - 2 * V3 + V4, b = V2 - V4;
    const T s22 = tmp1 * (a * a) + q4 * (b * b);
    a = V3 - 2 * V4 + V5, b = 3 * V3 - 4 * V4 + V5;
    const T s33 = tmp1 * (a * a) + q4 * (b * b);
    return wenoz_combine<T>(s11, s22, s33, 2 * V1 - 7 * V2 + 11 * V3, -V2 + 5 * V3 + 2 * V4,
                            2 * V3 + 5 * V4 - V5);
}

// WENO-Z5 negative-flux reconstruction from V1..V5 = F-[c-2..c+2], schemes.jl:164-187
template <typename T>
__device__ __forceinline__ T wenoz_minus(T V1, T V2, T V3, T V4, T V5) {
    const T tmp1 = T(13.0 / 12.0), q4 = T(0.25);
    T a, b;
    a = V5 - 2 * V4 + V3, b = V5 - 4 * V4 + 3 * V3;
    const T s11 = tmp1 * (a * a) + q4 * (b * b);
    a = V2 - 2 * V3 + V4, b = V4 - V2;
    const T s22 = tmp1 * (a * a) + q4 * (b * b);
    a = V3 - 2 * V2 + V1, b = 3 * V3 - 4 * V2 + V1;
    const T s33 = tmp1 * (a * a) + q4 * (b * b);
    return wenoz_combine<T>(s11, s22, s33, 11 * V3 - 7 * V4 + 2 * V5, -V4 + 5 * V3 + 2 * V2,
                            2 * V3 + 5 * V2 - V1);
}

// max that propagates NaN (Julia's) in the arithmetic type
template <typename T>
__device__ __forceinline__ T nmax(T a, T b) {
    return (a > b || a != a) ? a : b;
}

// WENO-Z5 of the fused FP64 paths, schemes.jl:139-187, for a stencil V1..V5 in upwind order (the
// negative flux passes its points reversed), written with the first differences e_k = V_{k+1} -
// V_k and the second differences a_k = e_{k+1} - e_k:
//   4 β_k = (13/3) a_k^2 + b_k^2,  b = a_1 + 2 e_2,  e_2 + e_3,  a_3 - 2 e_3
//   6 v_k = 6 V3 + r_k,            r = 5 e_2 - 2 e_1,  e_2 + 2 e_3,  4 e_3 - e_4
// so the face value is V3 + (1/6) Σ α_k r_k / Σ α_k, with the reference's weights
// α_k = d_k (1 + q_k^2), q_k = τ / (ε + β_k), d = 1, 6, 3 (the factor 4 cancels in q).  The
// same value in real arithmetic, with a third fewer operations than from the V_k, and the
// rounding of the weighted part only touches the correction to V3.  The sweeps are bound by FP64
// issue and latency: this, fast_rcp and the split below took an FP64 step of the 256x128x128 jet
// from 6.75 to 6.34 ms, 101x75x63 with five species from 2.00 to 1.80 ms, 32^3 from 139 to 129 us.
//
// Σ α_k r_k / Σ α_k comes as a fraction N / D without divisions: multiplying every α_k by
// b_1^2 b_2^2 b_3^2 gives A_k = d_k (b_k^2 + τ^2) Π_{j≠k} b_j^2 with the same ratios (N, of
// the order of 144 (4β)^6 sqrt(β), stays in range for β < 1e46).
__device__ __forceinline__ void weno_fraction(double V1, double V2, double V3, double V4,
                                              double V5, double &N, double &D) {
    const double e1 = V2 - V1, e2 = V3 - V2, e3 = V4 - V3, e4 = V5 - V4;
    const double s1 = e2 - e1, s2 = e3 - e2, s3 = e4 - e3;
    const double c1 = s1 + 2 * e2, c2 = e2 + e3, c3 = s3 - 2 * e3;
    const double k = 13.0 / 3.0, eps = 4 * kWenoEps;
    const double b1 = fma(k * s1, s1, fma(c1, c1, eps));  // 4 (ε + β_k)
    const double b2 = fma(k * s2, s2, fma(c2, c2, eps));
    const double b3 = fma(k * s3, s3, fma(c3, c3, eps));
    const double m = 12 * e3;  // the candidates' corrections: r_1, 6 r_2, 3 r_3 (d_k folded in)
    const double r1 = fma(5.0, e2, -2 * e1), r2 = fma(6.0, e2, m), r3 = fma(-3.0, e4, m);
    const double tau = b1 - b3;
    const double p1 = b1 * b1, p2 = b2 * b2, p3 = b3 * b3;
    const double a1 = fma(tau, tau, p1) * (p2 * p3);
    const double a2 = fma(tau, tau, p2) * (p1 * p3);
    const double a3 = fma(tau, tau, p3) * (p1 * p2);
    N = fma(a1, r1, fma(a2, r2, a3 * r3));
    D = fma(6.0, a2, fma(3.0, a3, a1));
}

// The corrections of F+ (stencil P1..P5) and F- (M1..M5, reversed) together.  Each denominator is
// a normal number (at least 10 ε^6 = 1e-155), so no branch guards its reciprocal.
__device__ __forceinline__ double weno_corrections(double P1, double P2, double P3, double P4,
                                                   double P5, double M1, double M2, double M3,
                                                   double M4, double M5) {
    double Np, Dp, Nm, Dm;
    weno_fraction(P1, P2, P3, P4, P5, Np, Dp);
    weno_fraction(M1, M2, M3, M4, M5, Nm, Dm);
    return 1.0 / 6.0 * fma(Np, fast_rcp(Dp), Nm * fast_rcp(Dm));
}

// FP32 (the mixed-precision paths), from the V_k: the rounding of the mixed path decides faces whose
// sensor lies at a branch threshold, so its operations are left as they are.  In the reference's own shape α_k = d_k (1 + q_k²),
// q_k = τ / (ε + β_k), with every step kept inside FP32 range: q_k is capped at 1e15 (a stencil
// with q_k that large already carries weight 1 to FP32 precision; when two are capped their
// candidate values agree to far below FP32 resolution, since β_k < 1e-15 τ bounds their second
// differences), the α_k are normalised by their sum before they multiply the candidates, and
// the divisions are the fast approximate ones (2 ulp), ample for weights in FP32.
__device__ __forceinline__ float wenoz_combine_fast(float s11, float s22, float s33, float v1,
                                                    float v2, float v3) {
    constexpr float eps = float(kWenoEps), qmax = 1e15f;
    const float tau = fabsf(s11 - s33);
    const float q1 = fminf(__fdividef(tau, eps + s11), qmax);
    const float q2 = fminf(__fdividef(tau, eps + s22), qmax);
    const float q3 = fminf(__fdividef(tau, eps + s33), qmax);
    const float a1 = 1.0f + q1 * q1, a2 = 6.0f * (1.0f + q2 * q2), a3 = 3.0f * (1.0f + q3 * q3);
    const float r = __fdividef(1.0f, a1 + a2 + a3);
    return (1.0f / 6.0f) * ((a1 * r) * v1 + (a2 * r) * v2 + (a3 * r) * v3);
}

__device__ __forceinline__ float wenoz_plus_fast(float V1, float V2, float V3, float V4, float V5) {
    const float tmp1 = float(13.0 / 12.0), q4 = float(0.25);
    float a, b;
    a = V1 - 2 * V2 + V3, b = V1 - 4 * V2 + 3 * V3;
    const float s11 = tmp1 * (a * a) + q4 * (b * b);
    a = V2 - 2 * V3 + V4, b = V2 - V4;
    const float s22 = tmp1 * (a * a) + q4 * (b * b);
    a = V3 - 2 * V4 + V5, b = 3 * V3 - 4 * V4 + V5;
    const float s33 = tmp1 * (a * a) + q4 * (b * b);
    return wenoz_combine_fast(s11, s22, s33, 2 * V1 - 7 * V2 + 11 * V3, -V2 + 5 * V3 + 2 * V4,
                                 2 * V3 + 5 * V4 - V5);
}

__device__ __forceinline__ float wenoz_minus_fast(float V1, float V2, float V3, float V4, float V5) {
    const float tmp1 = float(13.0 / 12.0), q4 = float(0.25);
    float a, b;
    a = V5 - 2 * V4 + V3, b = V5 - 4 * V4 + 3 * V3;
    const float s11 = tmp1 * (a * a) + q4 * (b * b);
    a = V2 - 2 * V3 + V4, b = V4 - V2;
    const float s22 = tmp1 * (a * a) + q4 * (b * b);
    a = V3 - 2 * V2 + V1, b = 3 * V3 - 4 * V2 + V1;
    const float s33 = tmp1 * (a * a) + q4 * (b * b);
    return wenoz_combine_fast(s11, s22, s33, 11 * V3 - 7 * V4 + 2 * V5, -V4 + 5 * V3 + 2 * V2,
                                 2 * V3 + 5 * V2 - V1);
}

// One face of the hybrid scheme for the fused paths: hybrid_face7 (below) with WENO-Z in
// difference form.
template <typename T>
__device__ __forceinline__ T hybrid_face_fast(const T *p, const T *m, T phif) {
    T fp, fm;
    if (phif < T(kHybrid1)) {
        fp = T(kUP7_2) * p[0] + T(kUP7_3) * p[1] + T(kUP7_4) * p[2] + T(kUP7_5) * p[3] +
             T(kUP7_6) * p[4] + T(kUP7_7) * p[5];
        fm = T(kUP7_7) * m[0] + T(kUP7_6) * m[1] + T(kUP7_5) * m[2] + T(kUP7_4) * m[3] +
             T(kUP7_3) * m[4] + T(kUP7_2) * m[5];
    } else if (phif < T(kHybrid2)) {
        if constexpr (sizeof(T) == 8) {
            return p[2] + m[3] +
                   weno_corrections(p[0], p[1], p[2], p[3], p[4], m[5], m[4], m[3], m[2], m[1]);
        } else {
            fp = wenoz_plus_fast(p[0], p[1], p[2], p[3], p[4]);
            fm = wenoz_minus_fast(m[1], m[2], m[3], m[4], m[5]);
        }
    } else {
        fp = p[2] + T(0.5) * minmod(p[3] - p[2], p[2] - p[1]);
        fm = m[3] - T(0.5) * minmod(m[4] - m[3], m[3] - m[2]);
    }
    return fp + fm;
}

// Steger-Warming splitting of one point, split.jl:17-89, for the fused paths; returns the
// contravariant velocity A·u.
//
// FP64: with h = p + e (so γ = h / e, γ - 1 = p / e and c² = γ p / ρ) the reference's terms
// collapse: ρ/(2γ) = ρ e / (2h); the acoustic kinetic terms |u ∓ c n|²/2 = k ∓ c θ + c²/2 with
// k = |u|²/2 and θ = u·n; and ρ/(2γ) (c²/2 + W2) = e / 2.  Equal in real arithmetic; one
// reciprocal of e ρ h instead of the divisions, and each half of the split costs fifteen
// operations.
__device__ __forceinline__ double split_fast(double rho, double u, double v, double w, double p,
                                             double ei, double A1, double A2, double A3,
                                             double *fp, double *fm) {
    const double hh = p + ei, er = ei * rho;
    const double inv = fast_rcp(er * hh);
    const double rh = inv * er, q1 = inv * hh;  // 1 / h and 1 / (e ρ)
    const double c2 = hh * p * q1;
    const double cs = c2 * fast_rsqrt(c2);
    const double r2 = A1 * A1 + A2 * A2 + A3 * A3;
    const double rs = fast_rsqrt(r2);
    const double E1 = A1 * u + A2 * v + A3 * w;
    const double css = cs * (r2 * rs);
    const double E2 = E1 - css, E3 = E1 + css;
    const double B1 = A1 * rs, B2 = A2 * rs, B3 = A3 * rs, th = E1 * rs;
    const double E1P = (E1 + fabs(E1)) * 0.5, E2P = (E2 + fabs(E2)) * 0.5,
                 E3P = (E3 + fabs(E3)) * 0.5;
    const double E1M = E1 - E1P, E2M = E2 - E2P, E3M = E3 - E3P;
    const double t1 = 0.5 * er * rh;         // ρ / (2γ)
    const double g2 = 2 * (p * rho) * q1;    // 2 (γ - 1)
    const double k = 0.5 * (u * u + v * v + w * w), he = 0.5 * ei;
    const double tc = t1 * cs;
    {
        const double s = E2P + E3P, d = tc * (E3P - E2P), m = t1 * fma(g2, E1P, s);
        fp[0] = m;
        fp[1] = fma(d, B1, m * u), fp[2] = fma(d, B2, m * v), fp[3] = fma(d, B3, m * w);
        fp[4] = fma(d, th, fma(m, k, he * s));
    }
    {
        const double s = E2M + E3M, d = tc * (E3M - E2M), m = t1 * fma(g2, E1M, s);
        fm[0] = m;
        fm[1] = fma(d, B1, m * u), fm[2] = fma(d, B2, m * v), fm[3] = fma(d, B3, m * w);
        fm[4] = fma(d, th, fma(m, k, he * s));
    }
    return E1;
}

// FP32: the reference's form with its divisions folded into two reciprocals and an rsqrt.  The
// outputs are STRIDE apart, so that a caller can have them stored where it stages them: through
// two arrays the compiler held all ten to the end and stored them together, and a mixed step of
// the 256x128x128 jet took 4328 us, with each stored as it is formed 4286.
template <int STRIDE = 1>
__device__ __forceinline__ float split_fast(float rho, float u, float v, float w, float p,
                                            float ei, float A1, float A2, float A3, float *fp,
                                            float *fm) {
    const float h = 0.5f;
    const float gam = p * (1.0f / ei) + 1;
    const float gm1 = gam - 1;
    const float inv = 1.0f / (rho * gam * gm1);  // 1 / (ρ γ (γ-1))
    const float cs = sqrt(gam * p * (gam * gm1 * inv));
    const float r2 = A1 * A1 + A2 * A2 + A3 * A3;
    const float rs = rsqrt(r2);
    const float ss = r2 * rs;
    const float E1 = A1 * u + A2 * v + A3 * w;
    const float E2 = E1 - cs * ss, E3 = E1 + cs * ss;
    const float B1 = A1 * rs, B2 = A2 * rs, B3 = A3 * rs;
    const float E1P = (E1 + fabs(E1)) * h, E2P = (E2 + fabs(E2)) * h, E3P = (E3 + fabs(E3)) * h;
    const float E1M = E1 - E1P, E2M = E2 - E2P, E3M = E3 - E3P;
    const float uc1 = u - cs * B1, uc2 = u + cs * B1;
    const float vc1 = v - cs * B2, vc2 = v + cs * B2;
    const float wc1 = w - cs * B3, wc2 = w + cs * B3;
    const float vvc1 = (uc1 * uc1 + vc1 * vc1 + wc1 * wc1) * h;
    const float vvc2 = (uc2 * uc2 + vc2 * vc2 + wc2 * wc2) * h;
    const float vv = gm1 * (u * u + v * v + w * w);
    const float W2 = (3 - gam) * (h * rho * gam * inv) * (cs * cs);  // (3-γ)/(2(γ-1)) c²
    const float tmp1 = h * rho * (rho * gm1 * inv);                  // ρ/(2γ)
    const float tmp2 = 2 * gm1;
    fp[0] = tmp1 * (tmp2 * E1P + E2P + E3P);
    fp[STRIDE] = tmp1 * (tmp2 * E1P * u + E2P * uc1 + E3P * uc2);
    fp[2 * STRIDE] = tmp1 * (tmp2 * E1P * v + E2P * vc1 + E3P * vc2);
    fp[3 * STRIDE] = tmp1 * (tmp2 * E1P * w + E2P * wc1 + E3P * wc2);
    fp[4 * STRIDE] = tmp1 * (E1P * vv + E2P * vvc1 + E3P * vvc2 + W2 * (E2P + E3P));
    fm[0] = tmp1 * (tmp2 * E1M + E2M + E3M);
    fm[STRIDE] = tmp1 * (tmp2 * E1M * u + E2M * uc1 + E3M * uc2);
    fm[2 * STRIDE] = tmp1 * (tmp2 * E1M * v + E2M * vc1 + E3M * vc2);
    fm[3 * STRIDE] = tmp1 * (tmp2 * E1M * w + E2M * wc1 + E3M * wc2);
    fm[4 * STRIDE] = tmp1 * (E1M * vv + E2M * vvc1 + E3M * vvc2 + W2 * (E2M + E3M));
    return E1;
}

// One face of the hybrid scheme, schemes.jl:110-199.  p[0..6] = F+[c-3..c+3] (F+[c-4] has
// weight UP7[1] = 0 and is not read), m[0..6] = F-[c-3..c+3]; the face lies between c-1 and c.
template <typename T>
__device__ __forceinline__ T hybrid_face7(const T *p, const T *m, T phif) {
    T fp, fm;
    if (phif < T(kHybrid1)) {
        fp = T(kUP7_2) * p[0] + T(kUP7_3) * p[1] + T(kUP7_4) * p[2] + T(kUP7_5) * p[3] +
             T(kUP7_6) * p[4] + T(kUP7_7) * p[5];
        fm = T(kUP7_7) * m[0] + T(kUP7_6) * m[1] + T(kUP7_5) * m[2] + T(kUP7_4) * m[3] +
             T(kUP7_3) * m[4] + T(kUP7_2) * m[5];
    } else if (phif < T(kHybrid2)) {
        fp = wenoz_plus(p[0], p[1], p[2], p[3], p[4]);
        fm = wenoz_minus(m[1], m[2], m[3], m[4], m[5]);
    } else {
        fp = p[2] + T(0.5) * minmod(p[3] - p[2], p[2] - p[1]);
        fm = m[3] - T(0.5) * minmod(m[4] - m[3], m[3] - m[2]);
    }
    return fp + fm;
}

// ---- mixtureProperties, thermo.jl:284-369 (transport law 2) in the reference's order.
// dot5, thermo.jl:284-286
__device__ __forceinline__ double dot5(double l1, double l2, double l3, double l4,
                                       const double *p) {
    return p[0] + l1 * p[1] + l2 * p[2] + l3 * p[3] + l4 * p[4];
}

// X: mole fractions; poly: visc (5, ns) | conduct (5, ns) | binarydiff (5, ns, ns).  Writes the
// mixture-averaged D_k to Dk[n * stride] and returns λ, μ.  W is an ns*ns work array.
__device__ __forceinline__ void mixture_properties(double T, double P, const double *X,
                                                   const FlameThermo &th, const double *poly,
                                                   int ns, double *W, double *mui, double *Dk,
                                                   long long stride, double &lam, double &mu) {
    const double *visc = poly, *cond = poly + 5 * ns, *bin = poly + 10 * ns;
    const double sqT = sqrt(T), sqsqT = sqrt(sqT), lgT = log(T);
    const double lgT2 = lgT * lgT, lgT3 = lgT * lgT2, lgT4 = lgT2 * lgT2;
    for (int n = 0; n < ns; ++n) mui[n] = sqT * dot5(lgT, lgT2, lgT3, lgT4, cond + 5 * n);
    double sum1 = 0, sum2 = 0;
    for (int k = 0; k < ns; ++k) sum1 += X[k] * mui[k], sum2 += X[k] / mui[k];
    lam = 0.5 * (sum1 + 1 / sum2);
    for (int n = 0; n < ns; ++n) {
        const double s = sqsqT * dot5(lgT, lgT2, lgT3, lgT4, visc + 5 * n);
        mui[n] = s * s;
    }
    for (int n = 0; n < ns; ++n) {  // Wilke, W[n*ns + l] is the reference's D[(n-1)*Nspecs+l]
        const double tmp1 = 1 / th.mw[n], tmp2 = mui[n];
        for (int l = 0; l <= n; ++l) {
            const double wr = th.mw[l] * tmp1, vr = tmp2 / mui[l];
            const double f1 = 1 + sqrt(vr * sqrt(wr));
            const double t = f1 * f1 / sqrt(8 + 8 / wr);
            W[n * ns + l] = t;
            W[l * ns + n] = t / (vr * wr);
        }
        W[n * ns + n] = 1.0;
    }
    mu = 0;
    for (int n = 0; n < ns; ++n) {
        double t = 0.0;
        for (int l = 0; l < ns; ++l) t += X[l] * W[n * ns + l];
        mu += X[n] * mui[n] / t;
    }
    for (int n = 0; n < ns; ++n)
        for (int m = n; m < ns; ++m) {
            const double t = T * sqT * dot5(lgT, lgT2, lgT3, lgT4, bin + 5 * (m + ns * n));
            W[m * ns + n] = t;
            W[n * ns + m] = t;
        }
    for (int n = 0; n < ns; ++n) {
        double s = 0.0;
        for (int m = 0; m < ns; ++m) {
            if (m == n) continue;
            s += X[m] / W[n * ns + m];
        }
        s *= P;
        Dk[n * stride] = (1 - X[n]) / (s + kEps);
    }
}

// mixtureProperties (thermo.jl:289-369) for a compile-time species count, without the ns x ns
// work array of mixture_properties: the Wilke factors W[n][l] and W[l][n] come from the same
// pair terms, and the binary-diffusion matrix is symmetric, so each pair is evaluated once and
// added to both rows' sums.  Every row sum still takes its terms in the order l = 0 .. NS-1 of
// the reference's loops (row n's terms l < n arrive in iteration n, its terms l > n in the
// later iterations, in increasing order), and each term is the reference's expression.
//
// The block's MixTables hold the terms of the Wilke factors that depend on the molar masses
// alone (for the pair (n, l) at n * NS + l: 1 / wr with wr = W_l / W_n, sqrt(wr) and
// 1 / sqrt(8 + 8 / wr), each formed in FP64).  The per-point divisions of the reference's
// expressions become products with reciprocals (1 / μ_l once per species, 1 / D_nm once per
// pair): the same formulas, each term within a few ulps of the reference's, at a third of the
// divisions and square roots.  MT is the arithmetic type: double on the FP64 path; float on the
// mixed path, which stores μ, λ and D_k in FP32 anyway (the tables then also hold the
// polynomial fits rounded to FP32 once per block).
template <int NS, typename MT>
struct MixTables {
    MT pw[3 * NS * NS];
    MT poly[sizeof(MT) == 4 ? 10 * NS + 5 * NS * NS : 1];
};

template <int NS, typename MT>
__device__ __forceinline__ void mix_tables_fill(const FlameThermo &th, const FlameTransport &tr,
                                                MixTables<NS, MT> &t) {
    for (int i = threadIdx.x; i < NS * NS; i += blockDim.x) {
        const int n = i / NS, l = i % NS;
        const double tmp1 = 1 / th.mw[n];
        const double wr = th.mw[l] * tmp1;
        t.pw[i] = MT(1 / wr);
        t.pw[NS * NS + i] = MT(sqrt(wr));
        t.pw[2 * NS * NS + i] = MT(1 / sqrt(8 + 8 / wr));
    }
    if constexpr (sizeof(MT) == 4) {
        for (int i = threadIdx.x; i < 10 * NS + 5 * NS * NS; i += blockDim.x)
            t.poly[i] = MT(tr.poly[i]);
    }
}

// Reciprocal, square root and quotient of the mixture rule: FP64 by the refined forms (arguments
// are positive and normal; mixture_exact has the other cases), FP32 the correctly rounded ones.
__device__ __forceinline__ double rule_rcp(double x) { return fast_rcp(x); }
__device__ __forceinline__ float rule_rcp(float x) { return 1 / x; }
__device__ __forceinline__ double rule_sqrt(double x) { return x * fast_rsqrt(x); }
__device__ __forceinline__ float rule_sqrt(float x) { return sqrt(x); }
__device__ __forceinline__ double rule_div(double a, double b) { return a * fast_rcp(b); }
__device__ __forceinline__ float rule_div(float a, float b) { return a / b; }

template <typename MT>
__device__ __forceinline__ MT dot5t(MT l1, MT l2, MT l3, MT l4, const MT *p) {
    return p[0] + l1 * p[1] + l2 * p[2] + l3 * p[3] + l4 * p[4];
}

// mixture_properties_pairs with exact divisions and square roots, for a point where its refined ones
// gave a value that is not a number: a transport fit may be zero (a species that does not conduct or
// diffuse), and exact divisions then make terms zero or infinite and the result finite.  A function of
// its own, since guarding each operation costs a step of 64x40x36 cells with nine species 4 % and the
// same code a second time in the caller makes it spill.  out: λ, μ, D_0 .. D_{NS-1}.
template <int NS>
__device__ __noinline__ void mixture_exact(double T, double P, const double *X, const double *pw,
                                           const double *poly, double *out) {
    const double *visc = poly, *cond = poly + 5 * NS, *bin = poly + 10 * NS;
    const double sqT = sqrt(T), sqsqT = sqrt(sqT), lgT = log(T);
    const double lgT2 = lgT * lgT, lgT3 = lgT * lgT2, lgT4 = lgT2 * lgT2;
    double mui[NS];
    double sum1 = 0, sum2 = 0;
    for (int k = 0; k < NS; ++k) {
        const double c = sqT * dot5(lgT, lgT2, lgT3, lgT4, cond + 5 * k);
        sum1 += X[k] * c, sum2 += X[k] / c;
    }
    out[0] = 0.5 * (sum1 + 1 / sum2);
    for (int n = 0; n < NS; ++n) {
        const double s = sqsqT * dot5(lgT, lgT2, lgT3, lgT4, visc + 5 * n);
        mui[n] = s * s;
    }
    double mu = 0;
    for (int n = 0; n < NS; ++n) {
        double row = 0;
        for (int l = 0; l < NS; ++l) {
            // the pair's factor t = W[hi][lo] with hi > lo, and W[lo][hi] = t / (vr wr)
            const int hi = n > l ? n : l, lo = n > l ? l : n, i = hi * NS + lo;
            const double vr = mui[hi] / mui[lo], f1 = 1 + sqrt(vr * pw[NS * NS + i]);
            const double t = f1 * f1 * pw[2 * NS * NS + i];
            row += X[l] * (l == n ? 1.0 : l < n ? t : t / vr * pw[i]);
        }
        mu += X[n] * mui[n] / row;
    }
    out[1] = mu;
    for (int n = 0; n < NS; ++n) {
        double row = 0;
        for (int m = 0; m < NS; ++m) {
            if (m == n) continue;
            const int hi = n > m ? n : m, lo = n > m ? m : n;
            row += X[m] / (T * sqT * dot5(lgT, lgT2, lgT3, lgT4, bin + 5 * (hi + NS * lo)));
        }
        out[2 + n] = (1 - X[n]) / (row * P + kEps);
    }
}

template <int NS, typename MT>
__device__ __forceinline__ void mixture_properties_pairs(MT T, MT P, const MT *X, const MT *pw,
                                                         const MT *poly, MT *Dk, MT &lam,
                                                         MT &mu) {
    const MT *visc = poly, *cond = poly + 5 * NS, *bin = poly + 10 * NS;
    const MT sqT = sqrt(T), sqsqT = sqrt(sqT), lgT = log(T);
    const MT lgT2 = lgT * lgT, lgT3 = lgT * lgT2, lgT4 = lgT2 * lgT2;
    MT mui[NS], row[NS];
#pragma unroll
    for (int n = 0; n < NS; ++n) mui[n] = sqT * dot5t<MT>(lgT, lgT2, lgT3, lgT4, cond + 5 * n);
    MT sum1 = 0, sum2 = 0;
#pragma unroll
    for (int k = 0; k < NS; ++k) sum1 += X[k] * mui[k], sum2 += rule_div(X[k], mui[k]);
    lam = MT(0.5) * (sum1 + 1 / sum2);
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        const MT s = sqsqT * dot5t<MT>(lgT, lgT2, lgT3, lgT4, visc + 5 * n);
        mui[n] = s * s;
        row[n] = 0;
    }
    MT rmu[NS];
#pragma unroll
    for (int n = 0; n < NS; ++n) rmu[n] = rule_rcp(mui[n]);
#pragma unroll
    for (int n = 0; n < NS; ++n) {  // Wilke: row[n] = Σ_l X[l] W[n][l]
#pragma unroll
        for (int l = 0; l < n; ++l) {
            const int i = n * NS + l;
            const MT vr = mui[n] * rmu[l];  // μ_n / μ_l
            const MT f1 = 1 + rule_sqrt(vr * pw[NS * NS + i]);
            const MT t = f1 * f1 * pw[2 * NS * NS + i];
            row[n] += X[l] * t;                                 // W[n][l]
            row[l] += X[n] * (t * (mui[l] * rmu[n]) * pw[i]);  // W[l][n] = t / (vr wr)
        }
        row[n] += X[n] * MT(1);  // W[n][n]
    }
    mu = 0;
#pragma unroll
    for (int n = 0; n < NS; ++n) mu += rule_div(X[n] * mui[n], row[n]);
#pragma unroll
    for (int n = 0; n < NS; ++n) row[n] = 0;  // now Σ_{m≠n} X[m] / Dbin[n][m]
#pragma unroll
    for (int n = 0; n < NS; ++n)
#pragma unroll
        for (int m = n + 1; m < NS; ++m) {
            const MT t = T * sqT * dot5t<MT>(lgT, lgT2, lgT3, lgT4, bin + 5 * (m + NS * n));
            const MT rt = rule_rcp(t);
            row[n] += X[m] * rt;
            row[m] += X[n] * rt;
        }
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        const MT s = row[n] * P;
        Dk[n] = rule_div(1 - X[n], s + MT(kEps));
    }
    if constexpr (sizeof(MT) == 8) {
        MT all = lam + mu;
#pragma unroll
        for (int n = 0; n < NS; ++n) all += Dk[n];
        if (__builtin_expect(all != all, 0)) {
            double x[NS], out[2 + NS];
#pragma unroll
            for (int n = 0; n < NS; ++n) x[n] = X[n];
            mixture_exact<NS>(T, P, x, pw, poly, out);
            lam = out[0], mu = out[1];
#pragma unroll
            for (int n = 0; n < NS; ++n) Dk[n] = out[2 + n];
        }
    }
}

// The reference's mixture kernel at one point with law 2 (thermo.jl:371-403): Y = max(ρi/ρ, 0)
// with ρ = max(Q_ρ, eps), X from Y (Y2X, thermo.jl:38-52), then mixtureProperties in MT.  The
// fused stage stores the result as μ, λ, D_0 .. D_{NS-1}.  mt: the block's MixTables.
template <int NS, typename MT>
__device__ __forceinline__ void mixture_point(const FlameThermo &th, const FlameTransport &tr,
                                              const MixTables<NS, MT> &mt, double T, double P,
                                              double rho_raw, const double *r, double &mu,
                                              double &lam, double *Dk) {
    // Y2X with correctly rounded quotients (fast_div), as the reference's: where a species is alone
    // its D_k = (1 - X_k) / (Σ + eps) is a quotient of their rounding errors
    const double rhoinv = fast_div(1.0, jmax(rho_raw, kEps));
    double X[NS];
    double yow = 0;
#pragma unroll
    for (int n = 0; n < NS; ++n)
        X[n] = fast_div(jmax(r[n] * rhoinv, 0.0), th.mw[n]), yow += X[n];
    const double yowinv = fast_div(1.0, yow);
#pragma unroll
    for (int n = 0; n < NS; ++n) X[n] *= yowinv;
    if constexpr (sizeof(MT) == 8) {
        mixture_properties_pairs<NS, double>(T, P, X, mt.pw, tr.poly, Dk, lam, mu);
    } else {
        MT Xm[NS], Dm[NS], lm, mm;
#pragma unroll
        for (int n = 0; n < NS; ++n) Xm[n] = MT(X[n]);
        mixture_properties_pairs<NS, MT>(MT(T), MT(P), Xm, mt.pw, mt.poly, Dm, lm, mm);
        lam = lm, mu = mm;
#pragma unroll
        for (int n = 0; n < NS; ++n) Dk[n] = Dm[n];
    }
}

// An NVTX range over a host-side scope (stage launches show up by name in Nsight timelines).
struct NvtxRange {
    explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange &) = delete;
    NvtxRange &operator=(const NvtxRange &) = delete;
};

}  // namespace flame

// Error plumbing shared by every C entry point (defined in capi.cu).
int flame_fail(int code, const char *fmt, ...);
int flame_check_launch(const char *what);
int flame_check_grid(const FlameGrid *g, const char *what);
