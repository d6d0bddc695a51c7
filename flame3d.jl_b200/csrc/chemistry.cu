// chemistry.cu — the finite-rate chemistry step of the reference (reactions.jl), 1:1.
//
// eval_gpu (explicit) and eval_gpu_stiff (point-implicit) advance the partial densities of every
// interior cell hotter than T_criteria by the mass production rates of the mechanism, add the
// formation-enthalpy release to the total energy, clip and rescale ρi to ρ and recover T, p, e.
// Rates follow vproductionRate / vproductionRate_Jac: Arrhenius forward rates, equilibrium
// constants from the Gibbs energy (thermo.jl:163-191), third-body and Troe falloff reactions.
//
// Built with -fmad=false, like kernels_ref.cu.  One thread per cell.  Above nine species the
// arithmetic is the oracle's, operation by operation, apart from exp / log / pow (the device math
// library against the host's), and the work arrays (ns, nreacs and ns x ns doubles) live in local
// memory, as MVector / MMatrix do in the reference.  Up to nine they live in registers, and
// reciprocals stand for some divisions, the elimination is written with fma and T comes from the
// mixture's polynomial: within 1e-12 of the oracle (tests/test_parity_chemistry.py).

#include "common.cuh"

namespace flame {
namespace chem {

constexpr int kMaxReacs = 64;

struct Mech {
    int nr;
    double atm;
    const int64_t *type, *sgm, *vf, *vr;
    const double *Arr, *ef, *loP, *Troe;
};

// x^k for the small integer stoichiometric powers (repeated multiplication, both signs)
__device__ __forceinline__ double ipow(double x, long long k) {
    double r = 1.0;
    const long long m = k < 0 ? -k : k;
    for (long long i = 0; i < m; ++i) r *= x;
    return k < 0 ? 1.0 / r : r;
}

// gibbs, thermo.jl:163-191 (dimensionless g/RT per species)
__device__ void gibbs(double *gi, double T, double lgT, double invT, const FlameThermo &th,
                      int ns) {
    const double mlogT = 1 - lgT;
    const double T1 = 0.5 * T;
    const double T2 = 1.0 / 6.0 * T * T;
    const double T3 = T1 * T2;
    const double T4 = 1.8 * T2 * T2;
    for (int n = 0; n < ns; ++n) {
        const double *c = T < th.coeffs_sep[n] ? th.coeffs_lo + 7 * n : th.coeffs_hi + 7 * n;
        gi[n] = c[0] * mlogT - c[1] * T1 - c[2] * T2 - c[3] * T3 - c[4] * T4 + c[5] * invT - c[6];
    }
}

// vproductionRate (reactions.jl:311-380) and, with JAC, vproductionRate_Jac (:383-462):
// wdot [mol/(cm^3 s)] from the concentrations sc [mol/cm^3]; A (ns x ns, column-major) gets
// the Jacobian of wdot with respect to sc.
template <bool JAC>
__device__ void production(double *wdot, const double *sc, double *A, double T,
                           const FlameThermo &th, const Mech &M, int ns) {
    double gi[FLAME_MAX_NS], kf[kMaxReacs], Kc[kMaxReacs];
    const double lgT = log(T);
    const double invT = 1.0 / T;
    for (int n = 0; n < M.nr; ++n)
        kf[n] = M.Arr[3 * n] * exp(M.Arr[3 * n + 1] * lgT - M.Arr[3 * n + 2] * invT);
    gibbs(gi, T, lgT, invT, th, ns);
    const double RsT = th.Ru / M.atm * 1e6 * T;
    for (int n = 0; n < M.nr; ++n) {
        double dg = 0;
        for (int m = 0; m < ns; ++m) dg += gi[m] * double(M.vf[m + ns * n] - M.vr[m + ns * n]);
        Kc[n] = ipow(RsT, M.sgm[n]) * exp(dg);
    }
    for (int n = 0; n < M.nr; ++n) {
        double qf = kf[n];
        double qr = qf / Kc[n];
        for (int m = 0; m < ns; ++m) {
            const long long vf = M.vf[m + ns * n], vr = M.vr[m + ns * n];
            if (vf != 0) qf *= ipow(sc[m], vf);
            if (vr != 0) qr *= ipow(sc[m], vr);
        }
        double mix = 0.0;
        if (M.type[n] == 2) {  // three-body
            for (int m = 0; m < ns; ++m) mix += M.ef[m + ns * n] * sc[m];
            qf *= mix;
            qr *= mix;
        } else if (M.type[n] == 3) {  // falloff, Troe form
            for (int m = 0; m < ns; ++m) mix += M.ef[m + ns * n] * sc[m];
            const double *lo = M.loP + 3 * n, *tr = M.Troe + 4 * n;
            const double redP = mix / kf[n] * lo[0] * exp(lo[1] * lgT - lo[2] * invT);
            const double logPred = log10(redP);
            const double a = tr[0];
            const double logFcent =
                log10((1 - a) * exp(-T / tr[1]) + a * exp(-T / tr[2]) + exp(-tr[3] * invT));
            const double troe_c = -0.4 - 0.67 * logFcent;
            const double troe_n = 0.75 - 1.27 * logFcent;
            const double troe = (troe_c + logPred) / (troe_n - 0.14 * (troe_c + logPred));
            const double F = pow(10.0, logFcent / (1.0 + troe * troe));
            const double k1 = (redP / (1.0 + redP)) * F;
            qf *= k1;
            qr *= k1;
        }
        for (int m = 0; m < ns; ++m) {
            const double nu = double(M.vr[m + ns * n] - M.vf[m + ns * n]);
            wdot[m] += (qf - qr) * nu;
            if constexpr (JAC) {
                const double invsc = 1 / (sc[m] + kEps);
                const double Awf = double(M.vf[m + ns * n]) * qf * invsc;
                const double Awr = double(M.vr[m + ns * n]) * qr * invsc;
                for (int l = 0; l < ns; ++l)
                    A[l + ns * m] += (Awf - Awr) * double(M.vr[l + ns * n] - M.vf[l + ns * n]);
            }
        }
    }
}

// solve, reactions.jl:465-504: Gaussian elimination with partial pivoting; a (ns x ns,
// column-major) and b are overwritten.
__device__ void solve(double *x, double *a, double *b, int ns) {
#define AT(i, j) a[(i) + ns * (j)]
    for (int k = 0; k < ns - 1; ++k) {
        double fmax = fabs(AT(k, k));
        int kk = k;
        for (int i = k + 1; i < ns; ++i) {
            const double absa = fabs(AT(i, k));
            if (absa > fmax) fmax = absa, kk = i;
        }
        for (int j = k; j < ns; ++j) {
            const double t = AT(k, j);
            AT(k, j) = AT(kk, j);
            AT(kk, j) = t;
        }
        const double t = b[k];
        b[k] = b[kk];
        b[kk] = t;
        for (int i = k + 1; i < ns; ++i) {
            const double f = -AT(i, k) / AT(k, k);
            for (int j = 0; j < ns; ++j) AT(i, j) += f * AT(k, j);
            b[i] += f * b[k];
        }
    }
    x[ns - 1] = b[ns - 1] / AT(ns - 1, ns - 1);
    for (int i = ns - 2; i >= 0; --i) {
        x[i] = b[i];
        for (int j = i + 1; j < ns; ++j) x[i] -= AT(i, j) * x[j];
        x[i] /= AT(i, i);
    }
#undef AT
}

// eval_gpu (STIFF false, reactions.jl:187-232) and eval_gpu_stiff (STIFF true, :235-309)
template <bool STIFF>
__global__ void k_eval(Dims D, double *U, double *Q, double *rhoi, double dt, FlameThermo th,
                       Mech M, const int64_t *tag, double Tcrit, int transposed) {
    const long long c = blockIdx.x * 128LL + threadIdx.x;
    const long long ncell = (long long)D.nx * D.ny * D.nz;
    if (c >= ncell) return;
    const long long x = c % D.nx, y = (c / D.nx) % D.ny, z = c / ((long long)D.nx * D.ny);
    const long long p = D.P(x + D.ng, y + D.ng, z + D.ng), np = D.np;
    if (tag && tag[p] != 0) return;
    double T = Q[p + 5 * np];
    if (!(T > Tcrit)) return;
    const int ns = D.ns;
    double sc[FLAME_MAX_NS], wdot[FLAME_MAX_NS], r[FLAME_MAX_NS], dr[FLAME_MAX_NS];
    for (int n = 0; n < ns; ++n) {
        r[n] = rhoi[p + n * np];
        sc[n] = r[n] / th.mw[n] * 1e-6;
        wdot[n] = 0.0;
    }
    double dei = 0;
    if constexpr (STIFF) {
        double A[FLAME_MAX_NS * FLAME_MAX_NS], A1[FLAME_MAX_NS * FLAME_MAX_NS];
        double drho[FLAME_MAX_NS];
        for (int i = 0; i < ns * ns; ++i) A[i] = 0.0;
        production<true>(wdot, sc, A, T, th, M, ns);
        for (int l = 0; l < ns; ++l)  // I - A dt, with the mass weights
            for (int n = 0; n < ns; ++n)
                A1[n + ns * l] = (n == l ? 1.0 : 0.0) - A[n + ns * l] * th.mw[n] / th.mw[l] * dt;
        for (int n = 0; n < ns; ++n) drho[n] = wdot[n] * th.mw[n] * 1e6 * dt;
        solve(dr, A1, drho, ns);
        for (int n = 0; n < ns; ++n) {
            const double a6 = transposed ? th.coeffs_lo[n + 35] : th.coeffs_lo[5 + 7 * n];
            dei += -a6 * dr[n] * th.Ru / th.mw[n];
            r[n] += dr[n];
        }
    } else {
        production<false>(wdot, sc, nullptr, T, th, M, ns);
        for (int n = 0; n < ns; ++n) {
            const double d = wdot[n] * th.mw[n] * 1e6 * dt;
            dei += -th.coeffs_lo[5 + 7 * n] * d * th.Ru / th.mw[n];
            r[n] += d;
        }
    }
    U[p + 4 * np] += dei;
    const double rho = jmax(Q[p], kEps);
    double sum = 0.0;
    for (int n = 0; n < ns; ++n) r[n] = jmax(r[n], 0.0), sum += r[n];
    for (int n = 0; n < ns; ++n) r[n] *= rho / sum;
    for (int n = 0; n < ns; ++n) rhoi[p + n * np] = r[n];
    double ein = Q[p + 6 * np];
    ein += dei;
    T = jmax(get_T<0>(th, ns, ein, r), kEps);
    const double pr = jmax(p_mixture<0>(th, ns, T, r), kEps);
    Q[p + 4 * np] = pr;
    Q[p + 5 * np] = T;
    Q[p + 6 * np] = ein;
}

// ------------------------------------------------------------ compile-time species count
// The same step for ns <= kMaxTemplated.  The runtime-ns kernel above spends its time in local
// memory (the Jacobian, its copy and the rate arrays are indexed at run time: 4 KB per thread)
// and in converting the mechanism's 64-bit integers for every cell; here the block lays the
// mechanism out in shared memory once (stoichiometric numbers as doubles, the participants of
// a reaction as bit masks, so that a reaction touches only its own species), every array of a
// cell is indexed at compile time and lives in registers, the reactions' rate constants are
// used as they are formed, and the Newton recovery of T runs on the mixture's own polynomial
// (MixPoly).  Measured (64^3 cells, 8 species, 8 reactions, point-implicit, 80 % of the cells
// hot): 856 us -> 193 us for the call.  Elimination: a row exchange is a predicated swap, skipped when no
// lane of the warp needs one; one reciprocal per pivot.
constexpr int kMaxTemplated = 9;

template <int NS>
struct MechTables {
    double nu[kMaxReacs][NS];  // vr - vf
    double ef[kMaxReacs][NS];
    long long vf[kMaxReacs][NS], vr[kMaxReacs][NS], sgm[kMaxReacs];
    double Arr[kMaxReacs][3], loP[kMaxReacs][3], Troe[kMaxReacs][4];
    int type[kMaxReacs];
    unsigned fmask[kMaxReacs], rmask[kMaxReacs];  // species with vf / vr != 0
    double rmw[NS];                               // 1 / W_n
};

template <int NS>
__device__ __forceinline__ void fill_tables(MechTables<NS> &t, const Mech &M,
                                            const FlameThermo &th) {
    for (int n = threadIdx.x; n < M.nr; n += blockDim.x) {
        unsigned fm = 0, rm = 0;
        const int type = (int)M.type[n];
        for (int m = 0; m < NS; ++m) {
            const long long vf = M.vf[m + NS * n], vr = M.vr[m + NS * n];
            t.vf[n][m] = vf, t.vr[n][m] = vr;
            t.nu[n][m] = double(vr - vf);
            fm |= (vf != 0 ? 1u : 0u) << m, rm |= (vr != 0 ? 1u : 0u) << m;
        }
        t.fmask[n] = fm, t.rmask[n] = rm;
        t.type[n] = type, t.sgm[n] = M.sgm[n];
        for (int a = 0; a < 3; ++a) t.Arr[n][a] = M.Arr[3 * n + a];
        // only what the reaction's type uses is read, so the arrays may end with the last reaction
        // that needs them
        if (type == 2 || type == 3)
            for (int m = 0; m < NS; ++m) t.ef[n][m] = M.ef[m + NS * n];
        if (type == 3) {
            for (int a = 0; a < 3; ++a) t.loP[n][a] = M.loP[3 * n + a];
            for (int a = 0; a < 4; ++a) t.Troe[n][a] = M.Troe[4 * n + a];
        }
    }
    if (threadIdx.x < NS) t.rmw[threadIdx.x] = 1 / th.mw[threadIdx.x];
}

// production() with the tables: wdot, and with JAC A[l][m] = d wdot_l / d sc_m.
template <int NS, bool JAC>
__device__ __forceinline__ void production_ns(double (&wdot)[NS], const double (&sc)[NS],
                                              double (&A)[JAC ? NS : 1][NS], double T,
                                              const FlameThermo &th, const MechTables<NS> &M,
                                              int nr, double atm) {
    const double lgT = log(T);
    const double invT = 1.0 / T;
    double gi[NS], invsc[NS];
    gibbs(gi, T, lgT, invT, th, NS);
    if constexpr (JAC) {
#pragma unroll
        for (int m = 0; m < NS; ++m) invsc[m] = 1 / (sc[m] + kEps);
    }
    const double RsT = th.Ru / atm * 1e6 * T;
    for (int n = 0; n < nr; ++n) {
        const double kf = M.Arr[n][0] * exp(M.Arr[n][1] * lgT - M.Arr[n][2] * invT);
        double dg = 0;
#pragma unroll
        for (int m = 0; m < NS; ++m) dg -= gi[m] * M.nu[n][m];
        const double Kc = ipow(RsT, M.sgm[n]) * exp(dg);
        double qf = kf;
        double qr = qf / Kc;
        const unsigned fm = M.fmask[n], rm = M.rmask[n];
#pragma unroll
        for (int m = 0; m < NS; ++m) {
            if (fm >> m & 1) qf *= ipow(sc[m], M.vf[n][m]);
            if (rm >> m & 1) qr *= ipow(sc[m], M.vr[n][m]);
        }
        const int type = M.type[n];
        if (type == 2 || type == 3) {
            double mix = 0.0;
#pragma unroll
            for (int m = 0; m < NS; ++m) mix += M.ef[n][m] * sc[m];
            double k1 = mix;      // three-body
            if (type == 3) {      // falloff, Troe form
                const double *lo = M.loP[n], *tr = M.Troe[n];
                const double redP = mix / kf * lo[0] * exp(lo[1] * lgT - lo[2] * invT);
                const double logPred = log10(redP);
                const double a = tr[0];
                const double logFcent =
                    log10((1 - a) * exp(-T / tr[1]) + a * exp(-T / tr[2]) + exp(-tr[3] * invT));
                const double troe_c = -0.4 - 0.67 * logFcent;
                const double troe_n = 0.75 - 1.27 * logFcent;
                const double troe = (troe_c + logPred) / (troe_n - 0.14 * (troe_c + logPred));
                const double F = pow(10.0, logFcent / (1.0 + troe * troe));
                k1 = (redP / (1.0 + redP)) * F;
            }
            qf *= k1;
            qr *= k1;
        }
        const double q = qf - qr;
#pragma unroll
        for (int m = 0; m < NS; ++m) {
            if (!((fm | rm) >> m & 1)) continue;
            wdot[m] += q * M.nu[n][m];
            if constexpr (JAC) {
                const double d = (double(M.vf[n][m]) * qf - double(M.vr[n][m]) * qr) * invsc[m];
#pragma unroll
                for (int l = 0; l < NS; ++l) A[l][m] += d * M.nu[n][l];
            }
        }
    }
}

// solve() in registers: a x = b by elimination with partial pivoting; b becomes x.  Column K and
// the columns after it; a recursion rather than a loop, so that every index is a constant
// whatever the unrolling limits.
template <int NS, int K>
__device__ __forceinline__ void solve_from(double (&a)[NS][NS], double (&b)[NS]) {
    double fmax = fabs(a[K][K]);
    int kk = K;
#pragma unroll
    for (int i = K + 1; i < NS; ++i) {
        const double v = fabs(a[i][K]);
        if (v > fmax) fmax = v, kk = i;
    }
    if (kk != K) {
#pragma unroll
        for (int i = K + 1; i < NS; ++i) {
            const bool s = kk == i;
#pragma unroll
            for (int j = K; j < NS; ++j) {
                const double t = a[K][j], v = a[i][j];
                a[K][j] = s ? v : t, a[i][j] = s ? t : v;
            }
            const double t = b[K], v = b[i];
            b[K] = s ? v : t, b[i] = s ? t : v;
        }
    }
    const double rp = 1 / a[K][K];
    if constexpr (K + 1 < NS) {
#pragma unroll
        for (int i = K + 1; i < NS; ++i) {
            const double f = -a[i][K] * rp;
#pragma unroll
            for (int j = K + 1; j < NS; ++j) a[i][j] = fma(f, a[K][j], a[i][j]);
            b[i] = fma(f, b[K], b[i]);
        }
        solve_from<NS, K + 1>(a, b);
#pragma unroll
        for (int j = K + 1; j < NS; ++j) b[K] = fma(-a[K][j], b[j], b[K]);
    }
    b[K] *= rp;
}

template <int NS, bool STIFF>
__global__ void __launch_bounds__(128) k_eval_ns(Dims D, double *U, double *Q, double *rhoi,
                                                 double dt, const __grid_constant__ FlameThermo th,
                                                 Mech M, const int64_t *tag, double Tcrit,
                                                 int transposed) {
    __shared__ MechTables<NS> t;
    const long long c = blockIdx.x * 128LL + threadIdx.x;
    const long long ncell = (long long)D.nx * D.ny * D.nz;
    long long x, y, z;
    if (ncell < 1LL << 31) {  // 32-bit divisions where the cells allow
        const unsigned q = (unsigned)c / (unsigned)D.nx;
        x = (unsigned)c % (unsigned)D.nx, y = q % (unsigned)D.ny, z = q / (unsigned)D.ny;
    } else {
        x = c % D.nx, y = (c / D.nx) % D.ny, z = c / ((long long)D.nx * D.ny);
    }
    const long long p = D.P(x + D.ng, y + D.ng, z + D.ng), np = D.np;
    double T = 0.0;
    bool hot = c < ncell && !(tag && tag[p] != 0);
    if (hot) T = Q[p + 5 * np], hot = T > Tcrit;
    // A block without a hot cell leaves the mechanism alone.  Eight species, 96^3 cells, explicit /
    // point-implicit: no cell hot 25 / 33 -> 13 / 19 us (the run-time kernel, with fewer registers,
    // 15 / 15), one cell in a hundred 110 / 205 -> 87 / 179, all of them 310 / 640 -> 296 / 635; a grid
    // of a few blocks pays the load of T first (16^3 27.1 -> 28.0).  A loop over chunks in as many
    // blocks as the GPU holds spills (all hot 352 / 691).
    if (!__syncthreads_or(hot)) return;
    fill_tables<NS>(t, M, th);
    __syncthreads();
    if (!hot) return;
    double sc[NS], w[NS], r[NS];
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        r[n] = rhoi[p + n * np];
        sc[n] = r[n] * t.rmw[n] * 1e-6;
        w[n] = 0.0;
    }
    const double rho = jmax(Q[p], kEps);
    double ein = Q[p + 6 * np];
    const double u4 = U[p + 4 * np];
    double dei = 0;
    if constexpr (STIFF) {
        double A[NS][NS];
#pragma unroll
        for (int l = 0; l < NS; ++l)
#pragma unroll
            for (int n = 0; n < NS; ++n) A[l][n] = 0.0;
        production_ns<NS, true>(w, sc, A, T, th, t, M.nr, M.atm);
#pragma unroll
        for (int n = 0; n < NS; ++n) {  // I - A dt, with the mass weights; the mass rates
#pragma unroll
            for (int l = 0; l < NS; ++l)
                A[n][l] = (n == l ? 1.0 : 0.0) - A[n][l] * (th.mw[n] * t.rmw[l] * dt);
            w[n] = w[n] * th.mw[n] * 1e6 * dt;
        }
        solve_from<NS, 0>(A, w);
    } else {
        double none[1][NS];
        production_ns<NS, false>(w, sc, none, T, th, t, M.nr, M.atm);
#pragma unroll
        for (int n = 0; n < NS; ++n) w[n] = w[n] * th.mw[n] * 1e6 * dt;
    }
    double sum = 0.0;
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        const double a6 = STIFF && transposed ? th.coeffs_lo[n + 35] : th.coeffs_lo[5 + 7 * n];
        dei += -a6 * w[n] * th.Ru * t.rmw[n];
        r[n] = jmax(r[n] + w[n], 0.0), sum += r[n];
    }
    const double scale = rho / sum;
#pragma unroll
    for (int n = 0; n < NS; ++n) r[n] *= scale, rhoi[p + n * np] = r[n];
    U[p + 4 * np] = u4 + dei;
    ein += dei;
    const MixPoly<NS> mp(th, r);
    T = jmax(get_T_mix<NS>(mp, th, ein), kEps);
    const double pr = jmax(th.Ru * T * mp.wsum, kEps);
    Q[p + 4 * np] = pr;
    Q[p + 5 * np] = T;
    Q[p + 6 * np] = ein;
}

template <int NS>
void launch_ns(bool stiff, unsigned blocks, cudaStream_t s, const Dims &D, double *U, double *Q,
               double *rhoi, double dt, const FlameThermo &th, const Mech &M, const int64_t *tag,
               double Tcrit, int transposed) {
    if (stiff)
        k_eval_ns<NS, true><<<blocks, 128, 0, s>>>(D, U, Q, rhoi, dt, th, M, tag, Tcrit, transposed);
    else
        k_eval_ns<NS, false><<<blocks, 128, 0, s>>>(D, U, Q, rhoi, dt, th, M, tag, Tcrit, 0);
}

int launch(bool stiff, const FlameGrid *g, cudaStream_t s, double *U, double *Q, double *rhoi,
           double dt, const FlameThermo *th, const FlameReactions *re, const int64_t *tag,
           double Tcrit, int transposed, const char *what) {
    if (int e = flame_check_grid(g, what)) return e;
    if (!U || !Q || !rhoi || !th || !re || !re->reaction_type || !re->sgm || !re->vf ||
        !re->vr || !re->Arr || !re->ef || !re->loP || !re->Troe)
        return flame_fail(FLAME_EINVAL, "%s: NULL argument", what);
    if (re->nreacs < 1 || re->nreacs > kMaxReacs)
        return flame_fail(FLAME_EUNSUPPORTED, "%s: %d reactions (1..%d supported)", what,
                          re->nreacs, kMaxReacs);
    if (stiff && transposed && g->ns + 35 > 7 * FLAME_MAX_NS)
        return flame_fail(FLAME_EINVAL, "%s: transposed read outside coeffs_lo", what);
    const Dims D = make_dims(*g);
    const Mech M{re->nreacs, re->atm, re->reaction_type, re->sgm, re->vf, re->vr,
                 re->Arr, re->ef, re->loP, re->Troe};
    const long long ncell = (long long)D.nx * D.ny * D.nz;
    const unsigned blocks = (unsigned)((ncell + 127) / 128);
    // up to kMaxTemplated species the cell's arrays fit in registers (9 x 9 Jacobian: 162 of 255)
    switch (D.ns) {
#define CASE(N)                                                                               \
    case N:                                                                                   \
        launch_ns<N>(stiff, blocks, s, D, U, Q, rhoi, dt, *th, M, tag, Tcrit, transposed); \
        break;
        CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9)
#undef CASE
        default:
            if (stiff)
                k_eval<true><<<blocks, 128, 0, s>>>(D, U, Q, rhoi, dt, *th, M, tag, Tcrit,
                                                    transposed);
            else
                k_eval<false><<<blocks, 128, 0, s>>>(D, U, Q, rhoi, dt, *th, M, tag, Tcrit, 0);
    }
    return flame_check_launch(what);
}

}  // namespace chem
}  // namespace flame

extern "C" int flame_eval_gpu(const FlameGrid *g, flame_stream_t s, double *U, double *Q,
                              double *rhoi, double dt, const FlameThermo *thermo,
                              const FlameReactions *react, const int64_t *tag, double T_criteria) {
    return flame::chem::launch(false, g, s, U, Q, rhoi, dt, thermo, react, tag, T_criteria, 0,
                               "flame_eval_gpu");
}

extern "C" int flame_eval_gpu_stiff(const FlameGrid *g, flame_stream_t s, double *U, double *Q,
                                    double *rhoi, double dt, const FlameThermo *thermo,
                                    const FlameReactions *react, const int64_t *tag,
                                    double T_criteria, int transposed) {
    return flame::chem::launch(true, g, s, U, Q, rhoi, dt, thermo, react, tag, T_criteria,
                               transposed, "flame_eval_gpu_stiff");
}
