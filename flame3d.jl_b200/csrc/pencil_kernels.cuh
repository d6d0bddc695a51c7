// pencil_kernels.cuh — the RK3 stage as sweeps along the grid axes (sm_100a).
//
// One stage of solver.jl:298-326, as k_prep (below), the sweeps and the finish.  In FP64 the
// sweeps are one launch, in mixed precision most are (sweep_kernels.cuh).  The rest of the mixed
// path (one species on large grids, law 2, configurations 5 and 6) and the persistent batches of
// either precision are organised for latency hiding instead of shared-memory tiling:
//   k_prep      every ghosted point: shock sensor ϕ (schemes.jl:1-24) and the mass fractions
//               Y = max(ρi / max(ρ, eps), 0) (thermo.jl:391-394) into a scratch array;
//   k_pencil<2> z sweep, k_pencil<1> y sweep, k_pencil<0> x sweep: a warp owns a pencil of 32
//               points along the sweep axis (26 owned cells plus the 3 + 3 stencil halo).  Each
//               lane splits its point once (split.jl:17-130), computes the cell-centred
//               tangential derivatives the viscous fluxes average across a face, and publishes
//               everything in the warp's slice of shared memory; the face between lanes l-1 and
//               l then forms the hybrid UP7 / WENO-Z / minmod flux (schemes.jl:86-437) minus the
//               viscous and species-diffusion flux (viscous.jl:1-665); the difference of two
//               faces is the cell's contribution.  Only __syncwarp orders the phases.
//   The z and y sweeps accumulate into a scratch right-hand side; the x sweep (lanes along x,
//   so its stores coalesce) finishes the stage: div (div.jl), RK3 combination (utils.jl:95-112),
//   c2Prim with the Newton temperature (utils.jl:2-48, thermo.jl:231-282), the transport law of
//   the new state, and the periodic ghost images.
// Configurations (flame_rk_stage_tiled) of the mixed path: 3 as above; 4 moves the finish into
// k_finish, one thread per cell; 5 and 6 are 3 and 4 with each z / y sweep split into a flow sweep (the NS = 0
// instance of the same kernel) and a species sweep (PART 2: species fluxes and the
// enthalpy-diffusion term of the energy flux, with fewer slots and registers).  The flame_batch_*
// persistent kernels at the end of the file run configuration 3 over many cases.
//
// Template parameters as in fused_stage.cu: NS species, QT storage of Q / transport, CT
// arithmetic type of split, reconstruction and viscous fluxes.  All indices are 32-bit.
//
// pencil_inst.cu is compiled once per species count and instantiates what pencil_stage.cu
// dispatches to through PencilOps (the species counts compile side by side).
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <type_traits>
#include <utility>
#include <vector>

#include "common.cuh"
#include "sweep_shape.cuh"

namespace flame {
namespace pencil {

constexpr int OWN = 26;  // cells owned by a 32-lane pencil (3 halo lanes below, 3 above)

// Warps per block.  The x sweep reads whole rows per warp; the y and z sweeps read one value per
// lane from 32 different rows, so their blocks take 16 consecutive x columns and together use
// every byte of each 128-byte line they touch.
template <int DIR>
struct Wpb {
    static constexpr int value = DIR == 0 ? 4 : 16;
};

template <typename QT>
struct Args {
    int nx, ny, nz, ng, tx, ty, tz, np, sy, sz;
    int per;  // periodic axes (FlameGrid::periodic): ghost images are written on these only
    int stage;
    double dt, ca, cb;
    double *U, *Un;
    const QT *Qi;
    QT *Qo;
    const QT *Ti;
    QT *To;
    const double *ri;
    double *ro, *rn;
    const double *met[10];
    const QT *metq;  // the metrics rounded to QT once (mixed precision), or null
    QT *aux;     // ϕ (1) and Y (NS), ghosted
    double *R;   // right-hand side accumulator (5 + NS), ghosted indexing: z sweep, then all
    double *R2;  // the y sweep's contribution (5 + NS), written, never read-modify-written
    double *xq, *xs;  // FP64 sweeps: the x sweep's contribution, flow (5) and species (NS)
    FlameThermo th;
    FlameTransport tr;
};

// Shared-memory slots of one lane's point (CT each).  REUSE (the FP64 y and z sweeps): the
// metrics are staged after the reconstruction has read the split fluxes, into their slots, so a
// point needs ten slots fewer and three 8-column blocks fit on an SM.
template <int NS, bool REUSE = false>
struct Slots {
    static constexpr int FP = 0;                // F+ flow (5), F- flow (5), F+ sp (NS), F- sp (NS)
    static constexpr int VF = 10 + 2 * NS;
    static constexpr int Q4 = VF;               // u v w T
    static constexpr int MET = REUSE ? FP : Q4 + 4;    // 9 metrics + J
    static constexpr int TR = REUSE ? Q4 + 4 : MET + 10;  // μ λ D
    static constexpr int RHO = TR + 3;
    static constexpr int Y = RHO + 1;           // NS
    static constexpr int DQ1 = Y + NS;          // tangential derivatives of u v w T along d+1
    static constexpr int DQ2 = DQ1 + 4;         // ... along d+2
    static constexpr int DY1 = DQ2 + 4;         // Y[+] - Y[-] along d+1 (NS)
    static constexpr int DY2 = DY1 + NS;        // ... along d+2 (NS)
    static constexpr int PHI = DY2 + NS;
    static constexpr int N = PHI + 1;
    static constexpr int G = FP;                // face flux, reuses the split slots (5 + NS)
    static constexpr int SPP = 10, SPM = 10 + NS;  // F+ / F- of species 0
    static constexpr int D = TR + 2, T = Q4 + 3;
};

// Slots of the species sweep (PART 2): only what the species fluxes and the enthalpy
// diffusion term of the energy flux read.  MIXD (law 2): D holds D_0 and DK the other species'
// D_1 .. D_{NS-1}.
template <int NS, bool MIXD = false>
struct SpSlots {
    static constexpr int FP = 0;                // F+ sp (NS), F- sp (NS)
    static constexpr int SPP = 0, SPM = NS;
    static constexpr int MET = 2 * NS;          // 9 metrics + J
    static constexpr int D = MET + 10;
    static constexpr int RHO = D + 1;
    static constexpr int T = RHO + 1;
    static constexpr int PHI = T + 1;
    static constexpr int Y = PHI + 1;           // NS
    static constexpr int DY1 = Y + NS;          // NS
    static constexpr int DY2 = DY1 + NS;        // NS
    static constexpr int DK = DY2 + NS;         // NS - 1 (MIXD only)
    static constexpr int N = DK + (MIXD ? NS - 1 : 0);  // 5 NS + 14 (+ NS - 1)
    static constexpr int G = FP;                // NS species fluxes + the energy term
};

// PART 0: the whole face flux; PART 2: the species fluxes and the enthalpy-diffusion term of the
// energy flux only (the flow part then runs as the NS = 0 instance of the same sweep).
template <int NS, int PART, bool MIXD = false, bool REUSE = false>
using SlotsOf = std::conditional_t<PART == 2, SpSlots<NS, MIXD>, Slots<NS, REUSE>>;

template <int NS, typename CT, int WPB>
constexpr size_t smem_bytes() {
    return sizeof(CT) * Slots<NS>::N * 32 * WPB;
}

// Asks L2 for the line holding p ahead of its use (no register is held meanwhile).
__device__ __forceinline__ void prefetch_l2(const void *p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// The kernels of a small FP64 stage are chained with programmatic dependent launch: a kernel lets
// its successor's blocks take their places as soon as all of its own have started, and waits
// itself, before it touches memory, until its predecessor has completed and its writes are
// visible.  One step of 32^3 cells 87.3 -> 80.1 us, 96x50x42 with inflow 652 -> 643, 101x75x63
// 1116 -> 1107; nothing on large grids (jet 256x128x128 6338 / 6393) or in mixed precision (32^3 86.1
// / 86.5).  Launched without the attribute the wait returns at once.
__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) {
    return v < lo ? lo : (v > hi ? hi : v);
}

template <typename CT, typename T>
__device__ __forceinline__ CT ldg(const T *p, int i) {
    return CT(__ldg(p + i));
}

// ----------------------------------------------------------------------------------- prep
template <int NS, typename QT, int PTS = 256>
__device__ __forceinline__ void prep_block(const Args<QT> &A, int bid) {
    const int c = bid * PTS + threadIdx.x;
    if (c >= A.np) return;
    const int gx = c % A.tx, gy = (c / A.tx) % A.ty, gz = c / A.sz;
    const QT *P = A.Qi + 4 * A.np;
    // the inputs of Y before any store (a later load could not pass a store it may alias)
    const double rinv = 1 / jmax(double(A.Qi[c]), kEps);
    double ri[NS];
#pragma unroll
    for (int n = 0; n < NS; ++n) ri[n] = A.ri[c + n * A.np];
    double phi = 0;
    if (gx > 0 && gx < A.tx - 1 && gy > 0 && gy < A.ty - 1 && gz > 0 && gz < A.tz - 1) {
        // schemes.jl:10-22 in the arithmetic type of Q with exact divisions, so the branch
        // thresholds see the same ϕ as the reference
        using CT = QT;
        const CT P2 = P[c];
        CT a1 = P[c - 1], a3 = P[c + 1];
        const CT phx = fabs(-a1 + 2 * P2 - a3) / (a1 + 2 * P2 + a3);
        a1 = P[c - A.sy], a3 = P[c + A.sy];
        const CT phy = fabs(-a1 + 2 * P2 - a3) / (a1 + 2 * P2 + a3);
        a1 = P[c - A.sz], a3 = P[c + A.sz];
        const CT phz = fabs(-a1 + 2 * P2 - a3) / (a1 + 2 * P2 + a3);
        phi = phx + phy + phz;
    }
    A.aux[c] = QT(phi);
#pragma unroll
    for (int n = 0; n < NS; ++n) A.aux[c + (1 + n) * A.np] = QT(jmax(ri[n] * rinv, 0.0));
}

template <int NS, typename QT>
__global__ void __launch_bounds__(256) k_prep(const __grid_constant__ Args<QT> A) {
    chain_begin();
    prep_block<NS, QT>(A, blockIdx.x);
}

// ----------------------------------------------------------------------------------- sweep
template <int DIR>
struct Dir {
    static constexpr int D1 = (DIR + 1) % 3, D2 = (DIR + 2) % 3;
};

template <int NS>
__device__ __forceinline__ void transport_point(const FlameThermo &th, const FlameTransport &tr,
                                                double T, double rho_raw, const double *r,
                                                double &mu, double &lam, double &D) {
    if (tr.law == 0) {
        mu = tr.mu_ref, lam = tr.lambda_ref, D = tr.D_ref;
        return;
    }
    const double rho = jmax(rho_raw, kEps);
    const double rinv = 1 / rho;
    const double T2 = T * T, T3 = T2 * T, T4 = T2 * T2;
    double cpm = 0;
#pragma unroll
    for (int n = 0; n < NS; ++n)
        cpm += cp_spec(th, n, T, T2, T3, T4) * jmax(r[n] * rinv, 0.0) / th.mw[n];
    cpm *= th.Ru;
    mu = tr.mu_ref * pow(T / tr.T_ref, tr.exponent);
    lam = cpm * mu / tr.Pr;
    D = lam / (rho * cpm);
}

// ---- phase A: everything the faces of a pencil need from one point, into the point's
// column of shared memory (slot stride 32).  l is the point's position along the pencil.
template <int DIR, int NS, typename QT, typename CT, bool REUSE = false>
__device__ __forceinline__ void point_phase(const Args<QT> &A, CT *S, int l, int g) {
    using SL = Slots<NS, REUSE>;
    constexpr int D1 = Dir<DIR>::D1, D2 = Dir<DIR>::D2;
    const int np = A.np;
    const int s1 = D1 == 0 ? 1 : (D1 == 1 ? A.sy : A.sz);
    const int s2 = D2 == 0 ? 1 : (D2 == 1 ? A.sy : A.sz);
    const QT *Q = A.Qi;
    const CT h = CT(0.5), c23 = CT(2.0 / 3.0), c12 = CT(1.0 / 12.0);
#define SV(slot) S[(slot) * 32 + l]
    const CT rho = CT(Q[g]), u = CT(Q[g + np]), v = CT(Q[g + 2 * np]), w = CT(Q[g + 3 * np]),
             p = CT(Q[g + 4 * np]), T = CT(Q[g + 5 * np]), ei = CT(Q[g + 6 * np]);
    CT mv[10];
    if (A.metq) {  // once-rounded copy: the same values without a conversion per load
#pragma unroll
        for (int m = 0; m < 10; ++m) mv[m] = CT(__ldg(A.metq + m * np + g));
    } else {
#pragma unroll
        for (int m = 0; m < 10; ++m) mv[m] = ldg<CT>(A.met[m], g);
    }
    const CT A1 = mv[3 * DIR], A2 = mv[3 * DIR + 1], A3 = mv[3 * DIR + 2];
    // Steger-Warming split, split.jl:17-89
    {
        CT E1;
        if constexpr (sizeof(CT) == 4) {
            E1 = split_fast<32>(rho, u, v, w, p, ei, A1, A2, A3, &SV(0), &SV(5));
        } else {
            CT fp[5], fm[5];
            E1 = split_fast(rho, u, v, w, p, ei, A1, A2, A3, fp, fm);
#pragma unroll
            for (int n = 0; n < 5; ++n) SV(n) = fp[n], SV(5 + n) = fm[n];
        }
        // species, split.jl:101-130
        const CT Ep = h * (E1 + fabs(E1)), Em = h * (E1 - fabs(E1));
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            const CT r = CT(A.ri[g + n * np]);
            SV(10 + n) = Ep * r;
            SV(10 + NS + n) = Em * r;
        }
    }
    SV(SL::Q4 + 0) = u, SV(SL::Q4 + 1) = v, SV(SL::Q4 + 2) = w, SV(SL::Q4 + 3) = T;
    if constexpr (!REUSE) {  // REUSE: staged later, into the split slots (stage_metrics)
#pragma unroll
        for (int m = 0; m < 10; ++m) SV(SL::MET + m) = mv[m];
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) SV(SL::TR + m) = CT(A.Ti[g + m * np]);
    SV(SL::RHO) = rho;
    SV(SL::PHI) = CT(A.aux[g]);
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        const QT *Y = A.aux + (1 + n) * np;
        SV(SL::Y + n) = CT(Y[g]);
        SV(SL::DY1 + n) = CT(Y[g + s1]) - CT(Y[g - s1]);
        SV(SL::DY2 + n) = CT(Y[g + s2]) - CT(Y[g - s2]);
    }
    // cell-centred 4th-order tangential derivatives of u, v, w, T; the face value the reference
    // forms (viscous.jl:36-53) is the mean of the two cells' values
    const int qv[4] = {1, 2, 3, 5};
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const QT *q = Q + qv[m] * np + g;
        SV(SL::DQ1 + m) = c23 * (CT(q[s1]) - CT(q[-s1])) - c12 * (CT(q[2 * s1]) - CT(q[-2 * s1]));
        SV(SL::DQ2 + m) = c23 * (CT(q[s2]) - CT(q[-s2])) - c12 * (CT(q[2 * s2]) - CT(q[-2 * s2]));
    }
#undef SV
}

// ---- phase B: the face between pencil positions l-1 and l; G = F_inviscid − F_viscous.
// The species part runs one species at a time in two passes (the sums of the diffusion
// velocities first, then each species' reconstruction, corrected diffusion flux and enthalpy
// flux), recomputing the few gradient terms instead of holding per-species arrays in registers.
// MIXD (the mixture-averaged law, law 2): each species has its own D_k; Dk points at D_0 of
// point l in the transport fields (field 2 + n holds D_n) and dstep is the pencil's stride, so
// point l - 1 is Dk - dstep.  The other laws use the one D of the shared-memory slots and
// compile without the per-species loads.
// MODE 0: the whole face.  With the REUSE slots the face runs in two calls, between which the
// metrics overwrite the split fluxes: MODE 1 reconstructs every flux into G, MODE 2 subtracts
// the viscous and diffusion fluxes from it (the same operations in the same order as MODE 0).
template <int DIR, int NS, typename QT, typename CT, int PART = 0, bool MIXD = false,
          int MODE = 0, bool REUSE = false>
__device__ __forceinline__ void face_phase(const Args<QT> &A, const CT *S, int l, CT *G,
                                           const QT *Dk, int dstep) {
    using SL = SlotsOf<NS, PART, MIXD, REUSE>;
    constexpr int GS = PART == 2 ? 0 : 5;  // G index of species 0
    constexpr int D1 = Dir<DIR>::D1, D2 = Dir<DIR>::D2;
    const CT h = CT(0.5), c23 = CT(2.0 / 3.0), c12 = CT(1.0 / 12.0);
#define SV(slot, ll) S[(slot) * 32 + (ll)]
    const int lm = l - 1;
    const CT phif = CT(jmax(double(SV(SL::PHI, lm)), double(SV(SL::PHI, l))));
    auto recon = [&](int vp, int vm) {
        CT pv[7], mv[7];
#pragma unroll
        for (int i = 0; i < 6; ++i) pv[i] = SV(vp, l - 3 + i), mv[i] = SV(vm, l - 3 + i);
        pv[6] = mv[6] = CT(0);
        return hybrid_face_fast<CT>(pv, mv, phif);
    };
    if constexpr (PART != 2 && MODE != 2) {
#pragma unroll
        for (int n = 0; n < 5; ++n) G[n] = recon(n, 5 + n);
    }
    if constexpr (MODE == 1) {
#pragma unroll
        for (int n = 0; n < NS; ++n) G[GS + n] = recon(SL::SPP + n, SL::SPM + n);
        return;
    }
    CT met[9];
#pragma unroll
    for (int m = 0; m < 9; ++m) met[m] = (SV(SL::MET + m, lm) + SV(SL::MET + m, l)) * h;
    const CT Jac = (SV(SL::MET + 9, lm) + SV(SL::MET + 9, l)) * h;
    const CT DL = SV(SL::D, lm), DR = SV(SL::D, l);
    const CT rho = (SV(SL::RHO, lm) + SV(SL::RHO, l)) * h;
    const CT Tf = (SV(SL::T, lm) + SV(SL::T, l)) * h;
    const CT *md = met + 3 * DIR;
    // species diffusion (viscous.jl:430-507): the diffusion velocity of species n at the face
    const CT rhoD1 = (DL + DR) * rho;  // viscous.jl:473 (no 1/2, as the reference)
    auto diffusion = [&](int n, CT &Vx, CT &Vy, CT &Vz) {
        CT rhoDi = rhoD1;
        if constexpr (MIXD && PART == 2) {  // staged with the species slots
            constexpr int dk = SpSlots<NS, true>::DK;
            if (n > 0) rhoDi = (SV(dk + n - 1, lm) + SV(dk + n - 1, l)) * rho;
        } else if constexpr (MIXD) {  // the x sweep: coalesced loads
            const QT *dn = Dk + (size_t)n * A.np;
            rhoDi = (CT(dn[-dstep]) + CT(dn[0])) * rho;
        }
        const CT y0 = SV(SL::Y + n, l), ym = SV(SL::Y + n, lm);
        const CT yp = SV(SL::Y + n, l + 1), ymm = SV(SL::Y + n, l - 2);
        CT dY[3];
        dY[DIR] = CT(1.25) * (y0 - ym) - c12 * (yp - ymm);
        dY[D1] = CT(0.25) * (SV(SL::DY1 + n, l) + SV(SL::DY1 + n, lm));
        dY[D2] = CT(0.25) * (SV(SL::DY2 + n, l) + SV(SL::DY2 + n, lm));
        Vx = (dY[0] * met[0] + dY[1] * met[3] + dY[2] * met[6]) * Jac * rhoDi;
        Vy = (dY[0] * met[1] + dY[1] * met[4] + dY[2] * met[7]) * Jac * rhoDi;
        Vz = (dY[0] * met[2] + dY[1] * met[5] + dY[2] * met[8]) * Jac * rhoDi;
        return h * (ym + y0);
    };
    CT sum1 = 0, sum2 = 0, sum3 = 0;
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        CT Vx, Vy, Vz;
        diffusion(n, Vx, Vy, Vz);
        sum1 += Vx, sum2 += Vy, sum3 += Vz;
    }
    CT fh1 = 0, fh2 = 0, fh3 = 0;
    {
        const double Td = double(Tf);
        const double T2 = 0.5 * Td * Td, T3 = 2.0 / 3.0 * T2 * Td, T4 = T2 * T2, T5 = 0.8 * T4 * Td;
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            CT Vx, Vy, Vz;
            const CT Yf = diffusion(n, Vx, Vy, Vz);
            const CT hn = CT(h_spec(A.th, n, Td, T2, T3, T4, T5));
            const CT V1 = Vx - sum1 * Yf, V2 = Vy - sum2 * Yf, V3 = Vz - sum3 * Yf;
            const CT gi = MODE == 2 ? G[GS + n] : recon(SL::SPP + n, SL::SPM + n);
            G[GS + n] = gi - (V1 * md[0] + V2 * md[1] + V3 * md[2]);
            fh1 += V1 * hn, fh2 += V2 * hn, fh3 += V3 * hn;
        }
    }
    if constexpr (PART == 2) {  // the energy flux's enthalpy-diffusion term, viscous.jl:120-141
        G[NS] = -(md[0] * fh1 + md[1] * fh2 + md[2] * fh3);
    } else {
    const CT mui = (SV(SL::TR, lm) + SV(SL::TR, l)) * h;
    const CT lami = (SV(SL::TR + 1, lm) + SV(SL::TR + 1, l)) * h;
    // momentum and energy, viscous.jl:14-141
    CT gr[4][3];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        CT dq[3];
        dq[DIR] = CT(1.25) * (SV(SL::Q4 + m, l) - SV(SL::Q4 + m, lm)) -
                  c12 * (SV(SL::Q4 + m, l + 1) - SV(SL::Q4 + m, l - 2));
        dq[D1] = h * (SV(SL::DQ1 + m, l) + SV(SL::DQ1 + m, lm));
        dq[D2] = h * (SV(SL::DQ2 + m, l) + SV(SL::DQ2 + m, lm));
#pragma unroll
        for (int x = 0; x < 3; ++x)
            gr[m][x] = (dq[0] * met[x] + dq[1] * met[3 + x] + dq[2] * met[6 + x]) * Jac;
    }
    const CT u = (SV(SL::Q4 + 0, lm) + SV(SL::Q4 + 0, l)) * h;
    const CT v = (SV(SL::Q4 + 1, lm) + SV(SL::Q4 + 1, l)) * h;
    const CT w = (SV(SL::Q4 + 2, lm) + SV(SL::Q4 + 2, l)) * h;
#undef SV
    const CT div = gr[0][0] + gr[1][1] + gr[2][2];
    const CT t11 = mui * (2 * gr[0][0] - c23 * div);
    const CT t12 = mui * (gr[0][1] + gr[1][0]);
    const CT t13 = mui * (gr[0][2] + gr[2][0]);
    const CT t22 = mui * (2 * gr[1][1] - c23 * div);
    const CT t23 = mui * (gr[2][1] + gr[1][2]);
    const CT t33 = mui * (2 * gr[2][2] - c23 * div);
    const CT E1 = u * t11 + v * t12 + w * t13 + lami * gr[3][0] + fh1;
    const CT E2 = u * t12 + v * t22 + w * t23 + lami * gr[3][1] + fh2;
    const CT E3 = u * t13 + v * t23 + w * t33 + lami * gr[3][2] + fh3;
    G[1] -= md[0] * t11 + md[1] * t12 + md[2] * t13;
    G[2] -= md[0] * t12 + md[1] * t22 + md[2] * t23;
    G[3] -= md[0] * t13 + md[1] * t23 + md[2] * t33;
    G[4] -= md[0] * E1 + md[1] * E2 + md[2] * E3;
    }
}

// ---- phase A of the species sweep: the species slots of one point.
template <int DIR, int NS, typename QT, typename CT, bool MIXD = false>
__device__ __forceinline__ void species_point_phase(const Args<QT> &A, CT *S, int l, int g) {
    using SL = SpSlots<NS, MIXD>;
    constexpr int D1 = Dir<DIR>::D1, D2 = Dir<DIR>::D2;
    const int np = A.np;
    const int s1 = D1 == 0 ? 1 : (D1 == 1 ? A.sy : A.sz);
    const int s2 = D2 == 0 ? 1 : (D2 == 1 ? A.sy : A.sz);
    const QT *Q = A.Qi;
    const CT h = CT(0.5);
#define SV(slot) S[(slot) * 32 + l]
    const CT rho = CT(Q[g]), u = CT(Q[g + np]), v = CT(Q[g + 2 * np]), w = CT(Q[g + 3 * np]);
    CT mv[10];
    if (A.metq) {
#pragma unroll
        for (int m = 0; m < 10; ++m) mv[m] = CT(__ldg(A.metq + m * np + g));
    } else {
#pragma unroll
        for (int m = 0; m < 10; ++m) mv[m] = ldg<CT>(A.met[m], g);
    }
    // species split, split.jl:101-130 (the contravariant velocity as in point_phase)
    const CT E1 = mv[3 * DIR] * u + mv[3 * DIR + 1] * v + mv[3 * DIR + 2] * w;
    const CT Ep = h * (E1 + fabs(E1)), Em = h * (E1 - fabs(E1));
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        const CT r = CT(A.ri[g + n * np]);
        SV(SL::SPP + n) = Ep * r;
        SV(SL::SPM + n) = Em * r;
    }
#pragma unroll
    for (int m = 0; m < 10; ++m) SV(SL::MET + m) = mv[m];
    SV(SL::D) = CT(A.Ti[g + 2 * np]);
    if constexpr (MIXD) {
#pragma unroll
        for (int n = 1; n < NS; ++n) SV(SL::DK + n - 1) = CT(A.Ti[g + (2 + n) * np]);
    }
    SV(SL::RHO) = rho;
    SV(SL::T) = CT(Q[g + 5 * np]);
    SV(SL::PHI) = CT(A.aux[g]);
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        const QT *Y = A.aux + (1 + n) * np;
        SV(SL::Y + n) = CT(Y[g]);
        SV(SL::DY1 + n) = CT(Y[g + s1]) - CT(Y[g - s1]);
        SV(SL::DY2 + n) = CT(Y[g + s2]) - CT(Y[g - s2]);
    }
#undef SV
}

// ---- last sweep: div, RK3 combination, c2Prim, transport, ghost images of one cell.
// LAW2: the mixture-averaged transport, written as μ, λ, D_0 .. D_{NS-1}.
// mt: the block's MixTables (LAW2 only).
template <int NS, typename QT, bool LAW2 = false>
__device__ __forceinline__ void finish_cell(const Args<QT> &A, int g, int gx, int gy, int gz,
                                            const double *rhs,
                                            const MixTables<NS, QT> *mt = nullptr) {
    const int np = A.np;
    const double Jact = A.met[9][g] * A.dt;
    // every input first: the stores below could alias them as far as the compiler knows, so
    // loads placed after a store would each wait for the one before
    double u0[5], r0[NS], un0[5], rn0[NS];
#pragma unroll
    for (int n = 0; n < 5; ++n) u0[n] = A.U[g + n * np];
#pragma unroll
    for (int n = 0; n < NS; ++n) r0[n] = A.ri[g + n * np];
    if (A.stage > 1) {
#pragma unroll
        for (int n = 0; n < 5; ++n) un0[n] = A.Un[g + n * np];
#pragma unroll
        for (int n = 0; n < NS; ++n) rn0[n] = A.rn[g + n * np];
    }
    // the RK3 update, utils.jl:95-112 (the multiply-adds spelled out, so that every kernel
    // that inlines this rounds them alike)
    double Uc[5], r[NS];
#pragma unroll
    for (int n = 0; n < 5; ++n) {
        if (A.stage == 1) A.Un[g + n * np] = u0[n];
        double un = fma(rhs[n], Jact, u0[n]);
        if (A.stage > 1) un = fma(un, A.ca, un0[n] * A.cb);
        Uc[n] = un;
        A.U[g + n * np] = un;
    }
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        if (A.stage == 1) A.rn[g + n * np] = r0[n];
        double rv = fma(rhs[5 + n], Jact, r0[n]);
        if (A.stage > 1) rv = fma(rv, A.ca, rn0[n] * A.cb);
        r[n] = rv;
    }
    // c2Prim, utils.jl:2-48
    const double rho = jmax(Uc[0], kEps);
    const double rinv = fast_div(1.0, rho);
    double sr = 0.0;
#pragma unroll
    for (int n = 0; n < NS; ++n) r[n] = jmax(r[n], 0.0), sr += r[n];
    const double sc = fast_div(rho, sr);
#pragma unroll
    for (int n = 0; n < NS; ++n) r[n] *= sc;
    const double u = Uc[1] * rinv, v = Uc[2] * rinv, w = Uc[3] * rinv;
    const double ei = jmax(Uc[4] - 0.5 * rho * (u * u + v * v + w * w), kEps);
    double mu, lam, D, Tn, p;
    double Dk[LAW2 ? NS : 1];
    if constexpr (NS < 4 && sizeof(QT) == 4) {
        // few species in mixed precision: the per-species sums, which need fewer registers than
        // the mixture's polynomials inside the x sweep (64^3, one species: 309 against 314 us)
        Tn = jmax(get_T<NS>(A.th, NS, ei, r), kEps);
        p = jmax(p_mixture<NS>(A.th, NS, Tn, r), kEps);
        if constexpr (!LAW2) transport_point<NS>(A.th, A.tr, Tn, rho, r, mu, lam, D);
    } else {  // the mixture's own polynomials (MixPoly): one evaluation per Newton iteration
        const MixPoly<NS> M(A.th, r);
        Tn = jmax(get_T_mix<NS>(M, A.th, ei), kEps);
        p = jmax(A.th.Ru * Tn * M.wsum, kEps);
        if constexpr (!LAW2) {
            if (A.tr.law == 0) {
                mu = A.tr.mu_ref, lam = A.tr.lambda_ref, D = A.tr.D_ref;
            } else {  // transport_point with cp_mix = Σ_n w_n cp_n / ρ from the same polynomials
                const double rcp = M.cv(Tn) + A.th.Ru * M.wsum;  // ρ cp
                mu = A.tr.mu_ref * pow(full_div(Tn, A.tr.T_ref), A.tr.exponent);
                lam = full_div(rcp * rinv * mu, A.tr.Pr);
                D = full_div(lam, rcp);
            }
        }
    }
    if constexpr (LAW2) {  // the next stage's mixture kernel (thermo.jl:371-403), per cell
        mixture_point<NS, QT>(A.th, A.tr, *mt, Tn, p, rho, r, mu, lam, Dk);
        D = Dk[0];
    }
    const double qv[7] = {rho, u, v, w, p, Tn, ei};
    const double tv[3] = {mu, lam, D};
    // the cell and its ghost images along the periodic axes (new: the reference fills ghosts
    // with case-specific kernels, boundary.jl:1-191, which the caller runs after the stage for
    // the other axes)
    const int ng = A.ng;
    // up to two images per axis: an axis shorter than 2 NG has cells near both ends
    int ox[3] = {0, 0, 0}, oy[3] = {0, 0, 0}, oz[3] = {0, 0, 0};
    int nxo = 1, nyo = 1, nzo = 1;
    if (A.per & 1) {
        if (gx < 2 * ng) ox[nxo++] = A.nx;
        if (gx >= A.nx) ox[nxo++] = -A.nx;
    }
    if (A.per & 2) {
        if (gy < 2 * ng) oy[nyo++] = A.ny;
        if (gy >= A.ny) oy[nyo++] = -A.ny;
    }
    if (A.per & 4) {
        if (gz < 2 * ng) oz[nzo++] = A.nz;
        if (gz >= A.nz) oz[nzo++] = -A.nz;
    }
    for (int c = 0; c < nzo; ++c)
        for (int b = 0; b < nyo; ++b)
            for (int aa = 0; aa < nxo; ++aa) {
                const int t = (gx + ox[aa]) + A.sy * (gy + oy[b]) + A.sz * (gz + oz[c]);
#pragma unroll
                for (int n = 0; n < 7; ++n) A.Qo[t + n * np] = QT(qv[n]);
#pragma unroll
                for (int n = 0; n < 3; ++n) A.To[t + n * np] = QT(tv[n]);
                if constexpr (LAW2) {
#pragma unroll
                    for (int n = 1; n < NS; ++n) A.To[t + (2 + n) * np] = QT(Dk[n]);
                }
#pragma unroll
                for (int n = 0; n < NS; ++n) A.ro[t + n * np] = r[n];
            }
}

#include "sweep_kernels.cuh"

// x sweep (lanes along x, every access coalesced); it is the last sweep.  FIN: it finishes the
// stage itself (configuration 3); otherwise it adds its differences to R and k_finish follows
// (configuration 4: the FP64 finish then runs at full occupancy, apart from the sweep's
// registers and shared memory).  Both form (R + R2) + rhs the same way, so they agree bit for
// bit.
template <int NS, typename QT, typename CT, bool FIN = true, bool MIXD = false,
          int WPB = Wpb<0>::value>
__device__ __forceinline__ void x_block(const Args<QT> &A, int bid, unsigned char *smem_raw) {
    using SL = Slots<NS>;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    CT *S = reinterpret_cast<CT *>(smem_raw) + warp * SL::N * 32;
    const int nseg = (A.nx + OWN - 1) / OWN;
    const int gw = bid * WPB + warp;
    const int seg = gw % nseg;
    const int y = (gw / nseg) % A.ny, z = (gw / nseg) / A.ny;
    if (z >= A.nz) return;
    const int a = seg * OWN - 3 + lane;
    const int gx = clampi(a + A.ng, 0, A.nx + 2 * A.ng - 1), gy = y + A.ng, gz = z + A.ng;
    const int g = gx + A.sy * gy + A.sz * gz;
    if (lane >= 3 && lane < 3 + OWN && a < A.nx) {  // what the end of this sweep reads
#pragma unroll
        for (int n = 0; n < 5 + NS; ++n) {
            prefetch_l2(A.R + g + n * A.np);
            prefetch_l2(A.R2 + g + n * A.np);
        }
        if constexpr (FIN) {
#pragma unroll
            for (int n = 0; n < 5; ++n) {
                prefetch_l2(A.U + g + n * A.np);
                if (A.stage > 1) prefetch_l2(A.Un + g + n * A.np);
            }
#pragma unroll
            for (int n = 0; n < NS; ++n) {
                prefetch_l2(A.ri + g + n * A.np);
                if (A.stage > 1) prefetch_l2(A.rn + g + n * A.np);
            }
        }
    }
    point_phase<0, NS, QT, CT>(A, S, lane, g);
    __syncwarp();
    CT G[5 + NS];
    const bool face = lane >= 3 && lane <= 3 + OWN && a <= A.nx;
    if (face) face_phase<0, NS, QT, CT, 0, MIXD>(A, S, lane, G, A.Ti + 2 * A.np + g, 1);
    __syncwarp();
    if (face) {
#pragma unroll
        for (int n = 0; n < 5 + NS; ++n) S[(SL::G + n) * 32 + lane] = G[n];
    }
    __syncwarp();
    if (lane < 3 || lane >= 3 + OWN || a >= A.nx) return;
    double rhs[5 + NS];  // the complete right-hand side: (z + y) + x, one rounding per sum
#pragma unroll
    for (int n = 0; n < 5 + NS; ++n)
        rhs[n] = (A.R[g + n * A.np] + A.R2[g + n * A.np]) +
                 (double(S[(SL::G + n) * 32 + lane]) - double(S[(SL::G + n) * 32 + lane + 1]));
    if constexpr (FIN) {
        finish_cell<NS, QT>(A, g, gx, gy, gz, rhs);
    } else {
#pragma unroll
        for (int n = 0; n < 5 + NS; ++n) A.R[g + n * A.np] = rhs[n];
    }
}

template <int NS, typename QT, typename CT, bool FIN, bool MIXD = false>
__global__ void __launch_bounds__(Wpb<0>::value * 32) k_pencil_x(const __grid_constant__ Args<QT> A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    x_block<NS, QT, CT, FIN, MIXD>(A, blockIdx.x, smem_raw);
}

// The stage's finish for configuration 4: one thread per interior cell, x fastest, with the
// complete right-hand side already in R (the x sweep summed it).
// X3: the three sweeps' parts are apart (R, R2 and get_x), to be summed as (z + y) + x.
template <int NS, typename QT, bool LAW2, bool X3 = false>
__device__ __forceinline__ void finish_thread(const Args<QT> &A, const MixTables<NS, QT> *mt,
                                              int block) {
    const int c = block * 128 + threadIdx.x;
    if (c >= A.nx * A.ny * A.nz) return;
    const int x = c % A.nx, y = (c / A.nx) % A.ny, z = c / (A.nx * A.ny);
    const int gx = x + A.ng, gy = y + A.ng, gz = z + A.ng;
    const int g = gx + A.sy * gy + A.sz * gz;
    double rhs[5 + NS];
#pragma unroll
    for (int n = 0; n < 5 + NS; ++n) {
        if constexpr (X3) rhs[n] = (A.R[g + n * A.np] + A.R2[g + n * A.np]) + get_x(A, n, g);
        else rhs[n] = A.R[g + n * A.np];
    }
    finish_cell<NS, QT, LAW2>(A, g, gx, gy, gz, rhs, mt);
}

// At most 128 registers from four species on (nine need 150: four blocks instead of three per SM).
// Its divisions are fast_div's: the correctly rounded ones bring calls, around which a kernel at
// its register limit spills (96^3, nine species: 164 -> 145 us; k_finish_mix 407 -> 237 us; HBM
// traffic alone takes 102 us).
template <int NS, typename QT, bool X3>
__global__ void __launch_bounds__(128, NS < 4 ? 6 : 4) k_finish(const __grid_constant__ Args<QT> A) {
    chain_begin();
    finish_thread<NS, QT, false, X3>(A, nullptr, blockIdx.x);
}

// The finish with the mixture-averaged law (law 2).  Its mixture rule needs up to 166 registers
// at nine species (three blocks per SM); capped at 128 (four blocks, at most 72 bytes of spill)
// it runs faster.  A separate kernel, so that the bound does not touch the other laws' finish.
template <int NS, typename QT>
__global__ void __launch_bounds__(128, 4) k_finish_mix(const __grid_constant__ Args<QT> A) {
    __shared__ MixTables<NS, QT> mt;
    chain_begin();
    mix_tables_fill<NS, QT>(A.th, A.tr, mt);
    __syncthreads();
    finish_thread<NS, QT, true, sizeof(QT) == 8>(A, &mt, blockIdx.x);
}

// Columns per block of the staged y / z sweeps.  Single precision: 16 consecutive x columns, so
// the block's loads use whole 128-byte lines; 8 when the column slots would not fit in shared
// memory.  (Sizing for two blocks per SM instead, 16/8/4 columns under 112 KB, measured 0-2 %
// faster with few species and 6 % slower with nine.)  FP64 sweeps that carry species: always 8
// columns.  With one or two species a 16-column FP64 block holds 172-199 KB, one block per SM,
// and its warps wait at the phase barriers with nothing else to run; two 8-column blocks keep
// the same warp count and one block's loads overlap the other's arithmetic (2-3 % faster on the
// 256x128x128 jet, neutral with two species); from three species on 16 columns would not fit
// anyway.  The flow-only sweep of configurations 5 and 6 (ns = 0) keeps 16 columns: 8 measured
// 8 % slower there.  Host and device use this rule: the batch planner sizes its work list with
// it.
constexpr int slots_of(int ns) { return 37 + 5 * ns; }
constexpr int staged_cols(int ns, size_t csz) {
    return (csz == 8 && ns > 0) ? 8 : (csz * slots_of(ns) * 33 * 16 <= 200 * 1024 ? 16 : 8);
}

template <int NS, typename CT, int PART = 0, bool MIXD = false>
struct Staged {
    static_assert(Slots<NS>::N == slots_of(NS), "slots_of must follow Slots");
    // FP64 sweeps with one or two species stage the metrics into the split slots once the
    // reconstruction is done: ten slots fewer per point let three blocks share an SM (more
    // species would not fit three blocks anyway)
    static constexpr bool REUSE = sizeof(CT) == 8 && PART == 0 && NS >= 1 && NS <= 2;
    static constexpr int NSLOT = SlotsOf<NS, PART, MIXD, REUSE>::N;
    static constexpr int STRIDE = NSLOT * 32 + 1;  // padded column region (bank spread)
    // (the species sweep in 8-column blocks capped at three per SM measured 7-12 % slower in
    // mixed precision: the register cap spills)
    static constexpr int COLS =
        PART == 2 ? (sizeof(CT) * NSLOT * 33 * 16 <= 200 * 1024 ? 16 : 8)
                  : staged_cols(NS, sizeof(CT));
    static constexpr size_t SMEM = sizeof(CT) * STRIDE * COLS;
};

// y or z sweep (DIR 1, 2).  The block stages the points of COLS neighbouring pencils with
// x-fastest threads (coalesced loads), then each warp works its own pencil from shared memory
// exactly like the x sweep, and the right-hand side goes back with x-fastest threads.
// PASS 0 writes R, PASS 1 adds to it.
template <int DIR, int PASS, int NS, typename QT, typename CT, int PART = 0, bool MIXD = false>
__device__ __forceinline__ void staged_block(const Args<QT> &A, int block, unsigned char *smem_raw) {
    constexpr int COLS = Staged<NS, CT, PART, MIXD>::COLS;
    constexpr int STRIDE = Staged<NS, CT, PART, MIXD>::STRIDE;
    constexpr bool REUSE = Staged<NS, CT, PART, MIXD>::REUSE;
    using SL = SlotsOf<NS, PART, MIXD, REUSE>;
    constexpr int NG_OUT = PART == 2 ? NS + 1 : 5 + NS;  // face values a lane produces
    CT *base = reinterpret_cast<CT *>(smem_raw);
    const int n_along = DIR == 1 ? A.ny : A.nz;
    const int n_c2 = DIR == 1 ? A.nz : A.ny;
    const int nseg = (n_along + OWN - 1) / OWN;
    const int nxb = (A.nx + COLS - 1) / COLS;
    int bid = block;
    const int xb = bid % nxb;
    bid /= nxb;
    const int seg = bid % nseg, c2 = bid / nseg;
    if (c2 >= n_c2) return;
    const int tid = threadIdx.x;
    if constexpr (PASS == 1 && PART == 2) {  // the energy field this thread adds to in phase C
        const int cx = tid % COLS, l = tid / COLS;
        const int x = xb * COLS + cx, ac = seg * OWN - 3 + l;
        if (l >= 3 && l < 3 + OWN && ac < n_along && x < A.nx) {
            const int gy = DIR == 1 ? ac + A.ng : c2 + A.ng;
            const int gz = DIR == 1 ? c2 + A.ng : ac + A.ng;
            prefetch_l2(A.R2 + (x + A.ng) + A.sy * gy + A.sz * gz + 4 * A.np);
        }
    }
    // ---- phase A, x-fastest: thread -> (column cx, pencil position l)
    int gA;  // the thread's phase-A point
    {
        const int cx = tid % COLS, l = tid / COLS;
        const int x = clampi(xb * COLS + cx, 0, A.nx - 1);
        const int a = seg * OWN - 3 + l;
        const int ga = clampi(a + A.ng, 0, n_along + 2 * A.ng - 1);
        const int gx = x + A.ng;
        const int gy = DIR == 1 ? ga : c2 + A.ng;
        const int gz = DIR == 1 ? c2 + A.ng : ga;
        gA = gx + A.sy * gy + A.sz * gz;
        if constexpr (PART == 2)
            species_point_phase<DIR, NS, QT, CT, MIXD>(A, base + cx * STRIDE, l, gA);
        else
            point_phase<DIR, NS, QT, CT, REUSE>(A, base + cx * STRIDE, l, gA);
    }
    __syncthreads();
    // ---- phase B, one warp per pencil (column)
    const int warp = tid >> 5, lane = tid & 31;
    CT *S = base + warp * STRIDE;
    const int a = seg * OWN - 3 + lane;
    CT G[NG_OUT];
    const bool face = lane >= 3 && lane <= 3 + OWN && a <= n_along;
    // the lane's point in the transport fields (per-species D_k of law 2)
    const int gxw = clampi(xb * COLS + warp, 0, A.nx - 1) + A.ng, gaw = a + A.ng;
    const int gl = gxw + (DIR == 1 ? A.sy * gaw + A.sz * (c2 + A.ng)
                                   : A.sy * (c2 + A.ng) + A.sz * gaw);
    if constexpr (REUSE) {
        // the reconstruction, then every warp is done with the split fluxes: the x-fastest
        // threads stage their point's metrics into those slots (coalesced loads), and the faces
        // take their viscous fluxes
        if (face)
            face_phase<DIR, NS, QT, CT, PART, MIXD, 1, true>(A, S, lane, G, A.Ti + 2 * A.np + gl,
                                                             DIR == 1 ? A.sy : A.sz);
        __syncthreads();
        {
            const int cx = tid % COLS, l = tid / COLS;
            CT *Sc = base + cx * STRIDE;
#pragma unroll
            for (int m = 0; m < 10; ++m)
                Sc[(SL::MET + m) * 32 + l] =
                    A.metq ? CT(__ldg(A.metq + m * A.np + gA)) : ldg<CT>(A.met[m], gA);
        }
        __syncthreads();
        if (face)
            face_phase<DIR, NS, QT, CT, PART, MIXD, 2, true>(A, S, lane, G, A.Ti + 2 * A.np + gl,
                                                             DIR == 1 ? A.sy : A.sz);
    } else if (face) {
        face_phase<DIR, NS, QT, CT, PART, MIXD>(A, S, lane, G, A.Ti + 2 * A.np + gl,
                                                DIR == 1 ? A.sy : A.sz);
    }
    __syncwarp();
    if (face) {
#pragma unroll
        for (int n = 0; n < NG_OUT; ++n) S[(SL::G + n) * 32 + lane] = G[n];
    }
    __syncthreads();
    // ---- phase C, x-fastest again: cell differences into R
    const int cx = tid % COLS, l = tid / COLS;
    const int x = xb * COLS + cx;
    const int ac = seg * OWN - 3 + l;
    if (l < 3 || l >= 3 + OWN || ac >= n_along || x >= A.nx) return;
    const int gy = DIR == 1 ? ac + A.ng : c2 + A.ng;
    const int gz = DIR == 1 ? c2 + A.ng : ac + A.ng;
    const int g = (x + A.ng) + A.sy * gy + A.sz * gz;
    const CT *Sc = base + cx * STRIDE;
#pragma unroll
    for (int n = 0; n < NG_OUT; ++n) {
        const double d = double(Sc[(SL::G + n) * 32 + l]) - double(Sc[(SL::G + n) * 32 + l + 1]);
        // the z sweep (PASS 0) writes R, the y sweep (PASS 1) R2; PART 2: G[n] is species n
        // (field 5 + n) and G[NS] the energy term, added to field 4, which the flow sweep of
        // the same direction wrote just before
        double *Rt = PASS == 0 ? A.R : A.R2;
        const int f = PART == 2 ? (n < NS ? 5 + n : 4) : n;
        if (PART == 2 && n == NS) Rt[g + f * A.np] += d;
        else Rt[g + f * A.np] = d;
    }
}

template <int DIR, int PASS, int NS, typename QT, typename CT, int PART = 0, bool MIXD = false>
__global__ void __launch_bounds__(Staged<NS, CT, PART, MIXD>::COLS * 32)
    k_pencil_staged(const __grid_constant__ Args<QT> A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    staged_block<DIR, PASS, NS, QT, CT, PART, MIXD>(A, blockIdx.x, smem_raw);
}

// ---------------------------------------------------------------------- batched, persistent
// Persistent launches per chunk of cases (one species count and transport family) and stage,
// over a work list of (case, block) items in phase order.  Laws 0 and 1 (configuration 3's
// shape), two launches: k_batch_sweeps<V = 0> takes the prep, z-sweep and y-sweep blocks of all
// the chunk's cases, k_batch_x<false> the x-sweep blocks, which finish the stage.  Law 2
// (configuration 6's shape, per-species D_k), four: k_batch_sweeps<V = 1> the prep blocks and
// the flow-only (ns = 0) z and y sweeps, k_batch_sweeps<V = 2> the species z and y sweeps
// (which add the enthalpy-diffusion term to the flow sweeps' energy field), k_batch_x<true> the
// x sweeps without the finish, k_batch_finish the finishing blocks with the mixture rule.
// Each launch takes its items in list order from its own atomic counter, so an item only ever
// waits for items taken before it: a case's sweep item waits until the case's prep items are
// done (a counter in device memory; every wait bounded: on timeout the batch's error word is
// set, the item is skipped and every later wait gives up at once; flame_batch_status reports
// FLAME_ETIMEOUT).  Every other order is the stream's: each launch follows the one before, so
// each kernel keeps the registers of its own phases.  Cases never read each other's data, so a
// case's result does not depend on which other cases share the batch.
struct BatchItem {
    int c, b;  // case (index within the chunk), block within the case's phase
};

struct BatchLaunch {
    const BatchItem *items;  // work list
    const int4 *need;        // per case: prep items (x)
    int *next;               // this launch's item counter (zeroed before the chunk's launches)
    int *done;               // per case: completed prep items (zeroed before the launches)
    int *err;                // the batch's error word (FLAME_ETIMEOUT)
    int lo, hi;              // this launch's items: list positions [lo, hi)
    int p1, p2;              // sweep launches: first item of the second and of the third phase
    int stall;               // test hook: case 0 waits for one prep item more than exists
};

constexpr int kWaitSpins = 1 << 22;  // x 128 ns: about half a second per wait

// Spins (thread 0) until *count >= target; false if the batch already failed or the bound ran
// out (then the error word is set).
__device__ __forceinline__ bool wait_count(const int *count, int target, int *err) {
    for (int i = 0; i < kWaitSpins; ++i) {
        if (*(volatile const int *)err) return false;
        if (*(volatile const int *)count >= target) {
            __threadfence();  // acquire: the counted items' writes are visible from here on
            return true;
        }
        __nanosleep(128);
    }
    atomicExch(err, FLAME_ETIMEOUT);
    return false;
}

// The staged sweep of a sweeps launch: V 0 the whole sweep, V 1 the flow-only sweep (the ns = 0
// instance), V 2 the species sweep with per-species D_k.
template <int NS, typename CT, int V>
using SweepOf = Staged<V == 1 ? 0 : NS, CT, V == 2 ? 2 : 0, V == 2>;

template <int NS, typename QT, typename CT, int V = 0>
struct BatchShape {
    using ST = SweepOf<NS, CT, V>;
    static constexpr int COLS = ST::COLS;
    static constexpr int NT = ST::COLS * 32;  // threads of a sweep block (prep, z, y items)
    static constexpr int XW = Wpb<0>::value;  // pencils of an x item (its warps)
    static constexpr size_t SMEM = sizeof(CT) * ST::STRIDE * ST::COLS;
    static constexpr size_t SMEM_X = smem_bytes<NS, CT, XW>();
    // x blocks per SM, as the register bound: what the shared memory allows (228 KB, 1 KB
    // reserved per block), but at most what the stand-alone x sweep's own register count gives
    // at this species count and precision (its item loop and indexed descriptors cost the
    // persistent kernel registers: unbounded it takes more and fits fewer blocks, bounded
    // tighter it spills; measured on single cases and the 64-case ensemble)
    static constexpr int FIT_X = int((228 * 1024) / (SMEM_X + 1024));
    static constexpr int CAP_X = sizeof(CT) == 8 ? (NS <= 1 ? 5 : NS == 2 ? 4 : NS <= 5 ? 3 : 2)
                                                 : (NS <= 1 ? 7 : NS <= 3 ? 5 : NS <= 7 ? 4 : 3);
    static constexpr int MINB_X = FIT_X < 1 ? 1 : (FIT_X > CAP_X ? CAP_X : FIT_X);
};

constexpr int kPrepPerThread = 4;  // points each thread of a prep item handles

// The descriptors of the cases a launch advances, in constant memory: copied (device to device)
// before each launch, so the kernels read them through the constant cache as the stand-alone
// kernels read their parameters (a descriptor read from shared or global memory costs a load
// for every field, and from global memory the compiler must also assume that stores alias it).
// One table per device context and species count: persistent batches on one device run one
// after the other.
constexpr int kConstCases = 20;
static __constant__ __align__(16) unsigned char c_batch_args[kConstCases * sizeof(Args<double>)];
static_assert(sizeof(Args<double>) == sizeof(Args<float>), "one table for both precisions");

template <typename QT>
__device__ __forceinline__ const Args<QT> &batch_args(int c) {
    return reinterpret_cast<const Args<QT> *>(c_batch_args)[c];
}

// Sweep items (list positions [L.lo, L.hi)): prep items up to L.p1, then z-sweep items up to
// L.p2, then y-sweep items.  A sweep item first waits until its case's prep items are done (in
// the species launch, V 2, which has no prep items, the prep launch before it has done them
// all and the wait ends at its first look).  Thread 0 takes the next item from the counter
// while the block works on the current one.
template <int NS, typename QT, typename CT, int V>
__global__ void __launch_bounds__(BatchShape<NS, QT, CT, V>::NT)
    k_batch_sweeps(const __grid_constant__ BatchLaunch L) {
    using BS = BatchShape<NS, QT, CT, V>;
    constexpr int SN = V == 1 ? 0 : NS;               // the species the sweeps carry
    constexpr int PART = V == 2 ? 2 : 0;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_item, s_next, s_ok;
    if (threadIdx.x == 0) s_next = L.lo + atomicAdd(L.next, 1);
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = s_next;
        __syncthreads();
        const int item = s_item;
        if (item >= L.hi) return;
        const BatchItem it = L.items[item];
        const int ph = item < L.p1 ? 0 : item < L.p2 ? 1 : 2;
        if (threadIdx.x == 0) {
            s_next = L.lo + atomicAdd(L.next, 1);  // in flight while the item runs
            s_ok = ph == 0 || wait_count(L.done + 4 * it.c,
                                         L.need[it.c].x + (L.stall && it.c == 0), L.err);
        }
        __syncthreads();
        const Args<QT> &A = batch_args<QT>(it.c);
        if (s_ok) {
            if (ph == 0) {
                if constexpr (V != 2) {
#pragma unroll
                    for (int k = 0; k < kPrepPerThread; ++k)
                        prep_block<NS, QT, BS::NT>(A, it.b * kPrepPerThread + k);
                }
            } else if (ph == 1) {
                staged_block<2, 0, SN, QT, CT, PART, V == 2>(A, it.b, smem_raw);
            } else {
                staged_block<1, 1, SN, QT, CT, PART, V == 2>(A, it.b, smem_raw);
            }
        }
        __syncthreads();  // the item's writes are done and its shared memory is free
        if (threadIdx.x == 0 && ph == 0) {
            __threadfence();  // release: publish the prep block's writes before counting it
            atomicAdd(L.done + 4 * it.c, 1);
        }
    }
}

// x-sweep items (list positions [L.lo, L.hi)), launched after the sweeps on the same stream, so
// all of every case's z and y items are done.  MIX (law 2): the x sweep with per-species D_k,
// which leaves the finish to k_batch_finish; otherwise the x sweep finishes the stage.
template <int NS, typename QT, typename CT, bool MIX>
__global__ void __launch_bounds__(BatchShape<NS, QT, CT>::XW * 32, BatchShape<NS, QT, CT>::MINB_X)
    k_batch_x(const __grid_constant__ BatchLaunch L) {
    using BS = BatchShape<NS, QT, CT>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_item, s_next;
    if (threadIdx.x == 0) s_next = L.lo + atomicAdd(L.next, 1);
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = s_next;
        __syncthreads();
        const int item = s_item;
        if (item >= L.hi) return;
        const BatchItem it = L.items[item];
        if (threadIdx.x == 0) s_next = L.lo + atomicAdd(L.next, 1);
        if (!*(volatile const int *)L.err)
            x_block<NS, QT, CT, !MIX, MIX, BS::XW>(batch_args<QT>(it.c), it.b, smem_raw);
    }
}

// Finishing items of law 2 (list positions [L.lo, L.hi)), after the x items: 128 cells each,
// with the mixture rule's tables of the item's case in shared memory (filled again when the
// block moves on to another case; items come in case order, so that is rare).
template <int NS, typename QT>
__global__ void __launch_bounds__(128, 4) k_batch_finish(const __grid_constant__ BatchLaunch L) {
    __shared__ MixTables<NS, QT> mt;
    __shared__ int s_item, s_next;
    int filled = -1;  // the case whose tables mt holds
    if (threadIdx.x == 0) s_next = L.lo + atomicAdd(L.next, 1);
    for (;;) {
        __syncthreads();  // also: every thread is done with mt before it is filled again
        if (threadIdx.x == 0) s_item = s_next;
        __syncthreads();
        const int item = s_item;
        if (item >= L.hi) return;
        const BatchItem it = L.items[item];
        if (threadIdx.x == 0) s_next = L.lo + atomicAdd(L.next, 1);
        const Args<QT> &A = batch_args<QT>(it.c);
        if (it.c != filled) {  // block-uniform
            mix_tables_fill<NS, QT>(A.th, A.tr, mt);
            __syncthreads();
            filled = it.c;
        }
        if (!*(volatile const int *)L.err) finish_thread<NS, QT, true>(A, &mt, it.b);
    }
}

template <typename QT>
Args<QT> make_args(const FlameGrid &g, int stage, double dt, const FlameStageBuffers &b,
                   const FlameMetrics &m, const FlameThermo &th, const FlameTransport &tr,
                   void *scratch) {
    Args<QT> A;
    A.nx = g.nx, A.ny = g.ny, A.nz = g.nz, A.ng = g.ng;
    A.tx = g.nx + 2 * g.ng, A.ty = g.ny + 2 * g.ng, A.tz = g.nz + 2 * g.ng;
    A.np = A.tx * A.ty * A.tz;
    A.sy = A.tx, A.sz = A.tx * A.ty;
    A.per = g.periodic & 7;
    A.stage = stage;
    A.dt = dt;
    A.ca = stage == 2 ? 0.25 : 2.0 / 3.0;
    A.cb = stage == 2 ? 0.75 : 1.0 / 3.0;
    A.U = b.U, A.Un = b.Un;
    A.Qi = static_cast<const QT *>(b.Q_in);
    A.Qo = static_cast<QT *>(b.Q_out);
    A.Ti = static_cast<const QT *>(b.trans_in);
    A.To = static_cast<QT *>(b.trans_out);
    A.ri = b.rhoi_in, A.ro = b.rhoi_out, A.rn = b.rhon;
    const double *mm[10] = {m.dxidx,   m.dxidy,   m.dxidz,   m.detadx, m.detady,
                            m.detadz,  m.dzetadx, m.dzetady, m.dzetadz, m.J};
    for (int i = 0; i < 10; ++i) A.met[i] = mm[i];
    A.metq = sizeof(QT) == 4 ? static_cast<const QT *>(b.metrics_lo) : nullptr;
    // scratch: R and R2 (5 + NS doubles per point each) first, then ϕ and Y (1 + NS of QT)
    A.R = static_cast<double *>(scratch);
    A.R2 = A.R + (size_t)(5 + g.ns) * A.np;
    A.aux = reinterpret_cast<QT *>(A.R2 + (size_t)(5 + g.ns) * A.np);
    A.xq = sizeof(QT) == 8 ? static_cast<double *>(b.Q_out) : nullptr, A.xs = b.rhoi_out;
    A.th = th, A.tr = tr;
    return A;
}

template <typename K>
int set_smem(K kernel, size_t sm, std::atomic<bool> *done) {
    int dev = 0;
    cudaGetDevice(&dev);
    // atomic flags: host threads on other streams may launch the same kernel at the same time
    // (two that both find the flag unset both set the attribute, to the same value)
    if (dev >= 0 && dev < 64 && done[dev].load(std::memory_order_acquire)) return FLAME_OK;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return flame_fail(FLAME_ELAUNCH, "pencil sweep: %zu B shared memory: %s", sm,
                          cudaGetErrorString(e));
    }
    if (dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release);
    return FLAME_OK;
}

// Launches `kernel`; with `early` so that it may start while the kernel before it on the stream
// finishes (chain_begin).  For kernels whose predecessor is the one this file launched just before.
template <typename... P, typename... A>
int launch_chained(bool early, void (*kernel)(P...), unsigned blocks, int threads, size_t smem,
                   cudaStream_t s, const char *what, const A &...args) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(blocks), c.blockDim = dim3(threads), c.dynamicSmemBytes = smem, c.stream = s;
    cudaLaunchAttribute a = {};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &a, c.numAttrs = early ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, args...);  // an error is the thread's last, read and cleared here
    return flame_check_launch(what);
}

template <int DIR, int PASS, int NS, typename QT, typename CT, int PART = 0, bool MIXD = false>
int launch_staged(const Args<QT> &A, cudaStream_t s) {
    using ST = Staged<NS, CT, PART, MIXD>;
    constexpr size_t sm = sizeof(CT) * ST::STRIDE * ST::COLS;
    static std::atomic<bool> done[64];
    const int n_along = DIR == 1 ? A.ny : A.nz;
    const int n_c2 = DIR == 1 ? A.nz : A.ny;
    const long long blocks = (long long)((A.nx + ST::COLS - 1) / ST::COLS) *
                             ((n_along + OWN - 1) / OWN) * n_c2;
    if (int e = set_smem(k_pencil_staged<DIR, PASS, NS, QT, CT, PART, MIXD>, sm, done)) return e;
    k_pencil_staged<DIR, PASS, NS, QT, CT, PART, MIXD><<<(unsigned)blocks, ST::COLS * 32, sm, s>>>(A);
    return flame_check_launch("flame_rk_stage (pencil)");
}

template <int NS, typename QT, typename CT, bool FIN, bool MIXD = false>
int launch_x(const Args<QT> &A, cudaStream_t s) {
    constexpr int WPB = Wpb<0>::value;
    constexpr size_t sm = smem_bytes<NS, CT, WPB>();
    static std::atomic<bool> done[64];
    if (int e = set_smem(k_pencil_x<NS, QT, CT, FIN, MIXD>, sm, done)) return e;
    const long long warps = (long long)A.ny * A.nz * ((A.nx + OWN - 1) / OWN);
    k_pencil_x<NS, QT, CT, FIN, MIXD><<<(unsigned)((warps + WPB - 1) / WPB), WPB * 32, sm, s>>>(A);
    return flame_check_launch("flame_rk_stage (pencil)");
}

// Whether an output array is also one of those the finish reads (the last stage's result may go
// where rhon was): then it cannot hold a sweep's part until the finish.
template <typename QT>
bool outputs_shared(const Args<QT> &A) {
    const void *out[3] = {A.Qo, A.ro, A.To}, *kept[3] = {A.U, A.Un, A.rn};
    for (const void *o : out)
        for (const void *k : kept)
            if (o == k) return true;
    return false;
}

// R += R2, R2 = 0.
static __global__ void __launch_bounds__(256) k_gather(double *R, double *R2, size_t n) {
    for (size_t i = blockIdx.x * 256 + (size_t)threadIdx.x; i < n; i += 256 * (size_t)gridDim.x)
        R[i] += R2[i], R2[i] = 0.0;
}

// FP64: prep, the three sweeps in one launch, finish; chained below 2^20 cells.
inline bool chained(const Args<double> &A) { return (long long)A.nx * A.ny * A.nz < 1 << 20; }

// The sweeps of an outputs_shared stage: z and y first, then x into R2, gathered into R in the same
// order, so that the finish sums the same values (z + y) + x.
template <int NS, bool MIXD>
int launch_shared(const Args<double> &A, const SweepShape &P, cudaStream_t s) {
    constexpr size_t sm = SweepSlots<NS, MIXD>::SMEM;
    const size_t n = (size_t)(5 + NS) * A.np;
    const unsigned blocks = (unsigned)std::min<size_t>((n + 255) / 256, 148 * 16);
    SweepShape Px = P;
    Px.y0 = Px.x0 = 0;
    k_sweeps<NS, MIXD><<<(unsigned)P.x0, P.threads, sm, s>>>(A, P);
    k_gather<<<blocks, 256, 0, s>>>(A.R, A.R2, n);
    k_sweeps<NS, MIXD><<<(unsigned)(P.blocks - P.x0), P.threads, sm, s>>>(A, Px);
    k_gather<<<blocks, 256, 0, s>>>(A.R, A.R2, n);
    return flame_check_launch("flame_rk_stage (sweeps)");
}

template <int NS, bool MIXD>
int launch_sweeps(const Args<double> &A, bool early, bool shared, cudaStream_t s) {
    constexpr size_t sm = SweepSlots<NS, MIXD>::SMEM;
    static std::atomic<bool> done[64];
    if (int e = set_smem(k_sweeps<NS, MIXD>, sm, done)) return e;
    const SweepShape P = sweep_shape<SweepSlots<NS, MIXD>>(A.nx, A.ny, A.nz);
    if (shared) return launch_shared<NS, MIXD>(A, P, s);
    return launch_chained(early, k_sweeps<NS, MIXD>, P.blocks, P.threads, sm, s, "flame_rk_stage (sweeps)",
                          A, P);
}
template <int NS>
int launch_fp64(const Args<double> &A, cudaStream_t s, bool shared = false) {
    if (!shared && outputs_shared(A)) {
        Args<double> B = A;
        B.xq = A.R2, B.xs = A.R2 + 5 * (size_t)A.np;
        return launch_fp64<NS>(B, s, true);
    }
    k_prep<NS, double><<<(unsigned)((A.np + 255) / 256), 256, 0, s>>>(A);
    if (int e = flame_check_launch("flame_rk_stage (prep)")) return e;
    const unsigned blocks = (unsigned)(((long long)A.nx * A.ny * A.nz + 127) / 128);
    const bool early = chained(A) && !shared;
    // law 2: per-species D_k (one species has the one D of the other laws)
    if (int e = A.tr.law == 2 ? launch_sweeps<NS, (NS > 1)>(A, early, shared, s)
                              : launch_sweeps<NS, false>(A, early, shared, s))
        return e;
    return launch_chained(early, A.tr.law == 2 ? k_finish_mix<NS, double> : k_finish<NS, double, true>,
                          blocks, 128, 0, s, "flame_rk_stage (finish)", A);
}

// Mixed precision: the sweeps of sweep_kernels.cuh.
template <int NS>
int launch_mixed_sweeps(const Args<float> &A, cudaStream_t s) {
    using SL = MixedSlots<NS>;
    static std::atomic<bool> done[64];
    if (int e = set_smem(k_sweeps_mixed<NS>, SL::SMEM, done)) return e;
    const SweepShape P = sweep_shape<SL>(A.nx, A.ny, A.nz);
    const int first = SL::FIN ? P.x0 : P.blocks;
    k_sweeps_mixed<NS><<<(unsigned)first, P.threads, SL::SMEM, s>>>(A, P);
    if (int e = flame_check_launch("flame_rk_stage (sweeps)")) return e;
    if constexpr (SL::FIN) {
        static std::atomic<bool> done_x[64];
        if (int e = set_smem(k_sweep_x_finish<NS>, SL::SMEM, done_x)) return e;
        k_sweep_x_finish<NS><<<(unsigned)(P.blocks - P.x0), P.threads, SL::SMEM, s>>>(A, P);
    } else {
        k_finish<NS, float, true><<<(unsigned)(((long long)A.nx * A.ny * A.nz + 127) / 128), 128, 0,
                                    s>>>(A);
    }
    return flame_check_launch("flame_rk_stage (finish)");
}

// Mixed precision: prep, then the sweeps (and, for law 2, configurations 5 and 6 and one species on
// large grids, the staged sweeps one after the other; see the top of this file).
template <int NS>
int launch_mixed(const Args<float> &A, cudaStream_t s, bool split_finish, bool split_species) {
    using T = float;
    k_prep<NS, T><<<(unsigned)((A.np + 255) / 256), 256, 0, s>>>(A);
    if (int e = flame_check_launch("flame_rk_stage (prep)")) return e;
    const unsigned blocks = (unsigned)(((long long)A.nx * A.ny * A.nz + 127) / 128);
    if (A.tr.law == 2) {  // per-species D_k: configuration 6's launches with the MIXD sweeps
        if (int e = launch_staged<2, 0, 0, T, T>(A, s)) return e;
        if (int e = launch_staged<2, 0, NS, T, T, 2, true>(A, s)) return e;
        if (int e = launch_staged<1, 1, 0, T, T>(A, s)) return e;
        if (int e = launch_staged<1, 1, NS, T, T, 2, true>(A, s)) return e;
        if (int e = launch_x<NS, T, T, false, true>(A, s)) return e;
        k_finish_mix<NS, T><<<blocks, 128, 0, s>>>(A);
        return flame_check_launch("flame_rk_stage (finish)");
    }
    if (!MixedSlots<NS>::FIN && outputs_shared(A)) split_species = true;  // parts in R and R2 only
    if (split_species) {  // configurations 5, 6: flow sweep (the NS = 0 instance) + species sweep
        if (int e = launch_staged<2, 0, 0, T, T>(A, s)) return e;
        if (int e = launch_staged<2, 0, NS, T, T, 2>(A, s)) return e;
        if (int e = launch_staged<1, 1, 0, T, T>(A, s)) return e;
        if (int e = launch_staged<1, 1, NS, T, T, 2>(A, s)) return e;
    } else if (NS > 1 || !staged_sweeps_ahead(NS, (long long)A.nx * A.ny * A.nz)) {
        return launch_mixed_sweeps<NS>(A, s);  // configurations 3, 4
    } else if constexpr (NS == 1) {
        if (int e = launch_staged<2, 0, NS, T, T>(A, s)) return e;
        if (int e = launch_staged<1, 1, NS, T, T>(A, s)) return e;
    }
    if (!split_finish) return launch_x<NS, T, T, true>(A, s);
    if (int e = launch_x<NS, T, T, false>(A, s)) return e;
    k_finish<NS, T, false><<<blocks, 128, 0, s>>>(A);
    return flame_check_launch("flame_rk_stage (finish)");
}

// The stage in the storage type QT.  FP64 runs the same three launches for every pencil
// configuration; split_finish and split_species pick the mixed path's.
template <int NS, typename QT>
int launch(const FlameGrid &g, cudaStream_t s, int stage, double dt, const FlameStageBuffers &b,
           const FlameMetrics &m, const FlameThermo &th, const FlameTransport &tr,
           void *scratch, bool split_finish, bool split_species) {
    const Args<QT> A = make_args<QT>(g, stage, dt, b, m, th, tr, scratch);
    if constexpr (sizeof(QT) == 8) return launch_fp64<NS>(A, s);
    else return launch_mixed<NS>(A, s, split_finish, split_species);
}

// ---------------------------------------------------------------- batches: one species count
constexpr int kMaxPhases = 7;

// The work-list shape of a chunk: its phases and the block sizes their item counts follow.
struct BatchDims {
    int phases = 4;  // 4 (prep, z, y, x) or, law 2, 7 (prep, flow z, flow y, species z,
                     // species y, x, finish)
    int nt = 0;      // threads of a prep item (those of the first sweeps launch's blocks)
    int cols = 0;    // staged columns of the first sweeps launch's blocks
    int cols_s = 0;  // law 2: staged columns of the species sweeps' blocks
};

struct BatchChunk {
    int ns = 0, n = 0;
    bool mix = false;            // law 2
    const void *args[6] = {};    // device Args arrays of the chunk, index (stage - 1) * 2 + parity
    const BatchItem *items = nullptr;
    const int4 *need = nullptr;  // per case: prep items (x)
    int *counters = nullptr;     // item counters (ints 0-3, one per launch), per case done[4]
                                 // from int 4 on
    int bound[kMaxPhases + 1] = {};  // first item of each phase; bound[phases] = item count
    int grid[4] = {1, 1, 1, 1};      // persistent blocks of the launches
};

template <int NS, typename QT, typename CT>
BatchDims batch_dims(bool mix) {
    BatchDims d;
    if (mix) {
        d.phases = 7;
        d.nt = BatchShape<NS, QT, CT, 1>::NT;
        d.cols = BatchShape<NS, QT, CT, 1>::COLS;
        d.cols_s = BatchShape<NS, QT, CT, 2>::COLS;
    } else {
        d.nt = BatchShape<NS, QT, CT>::NT;
        d.cols = BatchShape<NS, QT, CT>::COLS;
    }
    return d;
}

// Blocks of a persistent launch: as many as fit on the device at once, at most one per item.
template <typename K>
int persistent_grid(K kernel, int threads, size_t smem, std::atomic<bool> *done, int items,
                    int &grid) {
    int dev = 0, sms = 0, occ = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (smem)
        if (int e = set_smem(kernel, smem, done)) return e;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem);
    grid = std::max(1, std::min(items, sms * std::max(occ, 1)));
    return FLAME_OK;
}

template <int NS, typename QT, typename CT>
int batch_grid(BatchChunk &bc) {
    using B0 = BatchShape<NS, QT, CT>;
    using B1 = BatchShape<NS, QT, CT, 1>;
    using B2 = BatchShape<NS, QT, CT, 2>;
    static std::atomic<bool> d[5][64];
    const int *b = bc.bound;
    int e = FLAME_OK;
    if (!bc.mix) {
        if (!e) e = persistent_grid(k_batch_sweeps<NS, QT, CT, 0>, B0::NT, B0::SMEM, d[0], b[3] - b[0], bc.grid[0]);
        if (!e) e = persistent_grid(k_batch_x<NS, QT, CT, false>, B0::XW * 32, B0::SMEM_X, d[1], b[4] - b[3], bc.grid[1]);
    } else {
        if (!e) e = persistent_grid(k_batch_sweeps<NS, QT, CT, 1>, B1::NT, B1::SMEM, d[2], b[3] - b[0], bc.grid[0]);
        if (!e) e = persistent_grid(k_batch_sweeps<NS, QT, CT, 2>, B2::NT, B2::SMEM, d[3], b[5] - b[3], bc.grid[1]);
        if (!e) e = persistent_grid(k_batch_x<NS, QT, CT, true>, B0::XW * 32, B0::SMEM_X, d[4], b[6] - b[5], bc.grid[2]);
        if (!e) e = persistent_grid(k_batch_finish<NS, QT>, 128, 0, nullptr, b[7] - b[6], bc.grid[3]);
    }
    if (e) return e;
    return flame_check_launch("flame_batch_create");
}

template <int NS, typename QT, typename CT>
int batch_launch(const BatchChunk &bc, cudaStream_t s, int stage, int parity, int *err,
                 int stall) {
    using B0 = BatchShape<NS, QT, CT>;
    using B1 = BatchShape<NS, QT, CT, 1>;
    using B2 = BatchShape<NS, QT, CT, 2>;
    cudaError_t ce = cudaMemcpyToSymbolAsync(c_batch_args, bc.args[(stage - 1) * 2 + parity],
                                             sizeof(Args<QT>) * (size_t)bc.n, 0,
                                             cudaMemcpyDeviceToDevice, s);
    if (ce == cudaSuccess)
        ce = cudaMemsetAsync(bc.counters, 0, sizeof(int) * (4 + 4 * (size_t)bc.n), s);
    if (ce != cudaSuccess) {
        cudaGetLastError();
        return flame_fail(FLAME_ELAUNCH, "flame_batch_stage: %s", cudaGetErrorString(ce));
    }
    BatchLaunch L;
    L.items = bc.items;
    L.need = bc.need;
    L.done = bc.counters + 4;
    L.err = err;
    L.stall = stall;
    // launch k: its counter, items [lo, hi) and, for the sweeps, the starts of phases 1 and 2
    auto set = [&](int k, int lo, int hi, int p1, int p2) {
        L.next = bc.counters + k;
        L.lo = lo, L.hi = hi, L.p1 = p1, L.p2 = p2;
    };
    const int *b = bc.bound;
    if (!bc.mix) {
        set(0, b[0], b[3], b[1], b[2]);
        k_batch_sweeps<NS, QT, CT, 0><<<bc.grid[0], B0::NT, B0::SMEM, s>>>(L);
        if (int e = flame_check_launch("flame_batch_stage")) return e;
        set(1, b[3], b[4], b[4], b[4]);
        k_batch_x<NS, QT, CT, false><<<bc.grid[1], B0::XW * 32, B0::SMEM_X, s>>>(L);
        return flame_check_launch("flame_batch_stage");
    }
    set(0, b[0], b[3], b[1], b[2]);
    k_batch_sweeps<NS, QT, CT, 1><<<bc.grid[0], B1::NT, B1::SMEM, s>>>(L);
    if (int e = flame_check_launch("flame_batch_stage")) return e;
    set(1, b[3], b[5], b[3], b[4]);  // no prep phase: p1 = lo
    k_batch_sweeps<NS, QT, CT, 2><<<bc.grid[1], B2::NT, B2::SMEM, s>>>(L);
    if (int e = flame_check_launch("flame_batch_stage")) return e;
    set(2, b[5], b[6], b[6], b[6]);
    k_batch_x<NS, QT, CT, true><<<bc.grid[2], B0::XW * 32, B0::SMEM_X, s>>>(L);
    if (int e = flame_check_launch("flame_batch_stage")) return e;
    set(3, b[6], b[7], b[7], b[7]);
    k_batch_finish<NS, QT><<<bc.grid[3], 128, 0, s>>>(L);
    return flame_check_launch("flame_batch_stage");
}

// The host entries of one species count, index 0 FP64 and 1 mixed precision.
struct PencilOps {
    int (*stage[2])(const FlameGrid &g, cudaStream_t s, int stage, double dt,
                    const FlameStageBuffers &b, const FlameMetrics &m, const FlameThermo &th,
                    const FlameTransport &tr, void *scratch, bool split_finish,
                    bool split_species);
    BatchDims (*dims[2])(bool mix);
    int (*grid[2])(BatchChunk &bc);
    int (*batch[2])(const BatchChunk &bc, cudaStream_t s, int stage, int parity, int *err,
                    int stall);
};
template <int NS>
const PencilOps &pencil_ops();  // defined by pencil_inst.cu for NS = 1 .. 9

}  // namespace pencil
}  // namespace flame
