// sweep_kernels.cuh — the three FP64 sweeps of a stage in one launch (sm_100a).
//
// A block takes a few lines of points along its sweep axis: eight neighbouring x columns of up to
// 32 points (y and z sweeps), or a few whole or cut rows (x sweep).  A thread owns one point of
// them, and later one face and one cell, always with the lanes along x, so that global and shared
// accesses are contiguous in every phase.  Up to three passes go through the same shared-memory
// slots, each staged by the points and read by the faces:
//   1  the split fluxes (split.jl:17-130)             -> hybrid reconstruction (schemes.jl:86-437)
//   2  metrics, velocities and T with their tangential derivatives, transport
//                                                      -> viscous flux (viscous.jl:1-428)
//   3  mass fractions and their derivatives            -> species diffusion (viscous.jl:430-665)
// so a point needs 28 to 37 slots for any species count, where staging everything at once took
// 37 + 5 NS: three blocks of 256 threads (80 registers) share an SM with one species and with
// nine, which before ran with eight warps per SM.  The differences of two faces go to an array of
// the direction's own (R, R2, and for x the stage's output arrays), so the directions run side by
// side and the finish sums them.
//
// Bound by latency at 24 warps per SM (128x64x64 jet: 0.40 instructions per scheduler and cycle,
// FP64 pipe 41 %; barrier and long-scoreboard stalls lead), with 2000 instruction slots per cell
// and sweep where a warp per 32-point pencil took 3137.  One step, before -> after: 32^3 135 ->
// 92 us, 64^3 521 -> 402, 128^3 2896 -> 2584, jet 256x128x128 6380 -> 6313; 101x75x63 with five
// species 1784 -> 1061; 96^3 with nine species 5415 -> 2741, with per-species D 4638 -> 4019.
// Tried and not kept: two blocks per SM at 128 registers (jet 6623) and four at 64 (7810);
// everything but the metrics staged in pass 1 (6920); a prefetch of pass 2's lines to L2 (6399).

constexpr int kSweepNT = 256;  // most threads (points) of a block, and the pitch of a slot
constexpr int kSweepCols = 8;  // x columns of a y / z block

// Slots of a point.  Passes 2 and 3 are one where its slots leave room for three blocks per SM
// (ONE: up to three species, two with per-species D); the sensor keeps the last slot.
template <int NS, bool MIXD>
struct SweepSlots {
    static constexpr int FM = 5, SP = 10, SM = 10 + NS, F = 10 + 2 * NS;  // pass 1: F+ at 0
    static constexpr int YN = (MIXD ? 4 : 3) * NS;
    static constexpr int MOST = 37;
    static constexpr bool ONE = 26 + YN + 1 <= MOST;
    static constexpr int MET = 0, Q4 = 10, DQ1 = 14, DQ2 = 18, MU = 22, LAM = 23, RHO = 24, D = 25;
    static constexpr int Y = ONE ? 26 : 0, DY1 = Y + NS, DY2 = Y + 2 * NS, DK = Y + 3 * NS;
    static constexpr int a = F > 26 ? F : 26, b = a > YN ? a : YN;
    static constexpr int PHI = ONE ? Y + YN : b;
    static constexpr int N = PHI + 1;
    static constexpr size_t SMEM = sizeof(double) * N * kSweepNT;
    static_assert(N <= MOST && 3 * (SMEM + 1024) <= 228 * 1024, "three blocks per SM");
};

// How the launch is cut: own cells per line and direction, lines per x block, threads per
// block, and the first block of the y and of the x sweep (blocks [0, y0) are the z sweep's).
struct SweepShape {
    int own[3], rows, threads, y0, x0, blocks;
};

// Where the x sweep leaves field n of a cell for the finish: the stage's output arrays, whose
// interior the finish of the same cell writes after it has read this (Q_out holds seven fields
// of 8 bytes, rhoi_out one per species).
__device__ __forceinline__ double *x_field(const Args<double> &A, int n, int c) {
    return n < 5 ? A.Qo + n * A.np + c : A.ro + (n - 5) * A.np + c;
}

// ---- faces: fluxes contracted with the face normal.
// With md the metric row of the face direction and c_a = Σ_x met[a][x] md[x], a derivative
// contracted with the face normal is c · dq.  The momentum fluxes need the velocity gradient
// once more for its transpose and trace; the heat flux and every species' diffusion flux
// J_n = V_n·md (viscous.jl:463-505) need only the three products of c, where forming V_n along
// x, y and z takes nine, twice over the species.  The correction Σ V Y becomes J_n - Y_n Σ J and
// the enthalpy-diffusion term Σ h_n (J_n - Y_n Σ J).  Equal in real arithmetic.  s_* are sums over
// the face's two cells (twice the reference's means); metric rows come in the order normal,
// first, second tangent.
//
// Subtracts the momentum and energy flux, viscous.jl:14-141, from G[1..4]; dq[i]: derivatives of
// u, v, w, T along the rows' axes.
__device__ __forceinline__ void viscous_flux(const double (&m)[9], const double (&c)[3],
                                             double s_J, double s_mu, double s_lam,
                                             const double (&s_u)[3], const double (&dq)[4][3],
                                             double *G) {
    double gr[3][3];  // gr[i][x]: 2 x the gradient of velocity i along x over the Jacobian
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int x = 0; x < 3; ++x)
            gr[i][x] = dq[i][0] * m[x] + dq[i][1] * m[3 + x] + dq[i][2] * m[6 + x];
    const double d23 = 2.0 / 3.0 * (gr[0][0] + gr[1][1] + gr[2][2]);
    const double sc = 1.0 / 16.0 * s_J;  // the metrics come doubled twice, J and μ once each
    const double sm = sc * s_mu;
    double E = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double a = c[0] * dq[i][0] + c[1] * dq[i][1] + c[2] * dq[i][2];
        const double b = gr[0][i] * m[0] + gr[1][i] * m[1] + gr[2][i] * m[2];
        const double t = sm * (a + b - d23 * m[i]);
        G[1 + i] -= t;
        E += s_u[i] * t;
    }
    const double qn = c[0] * dq[3][0] + c[1] * dq[3][1] + c[2] * dq[3][2];
    G[4] -= 0.5 * E + sc * s_lam * qn;
}

// The cell-centred 4th-order tangential derivative (viscous.jl:36-53; the reference takes the
// mean over the face's two cells).
__device__ __forceinline__ double tangent4(const double *q, int s) {
    return 2.0 / 3.0 * (q[s] - q[-s]) - 1.0 / 12.0 * (q[2 * s] - q[-2 * s]);
}

// One block of a sweep.  STEP: the slot distance of two points of a line.
template <int DIR, int NS, bool MIXD>
__device__ __forceinline__ void sweep_block(const Args<double> &A, const SweepShape &P, int bid,
                                            double *S) {
    using SL = SweepSlots<NS, MIXD>;
    constexpr int NT = kSweepNT, C = kSweepCols, STEP = DIR == 0 ? 1 : C;
    constexpr int D1 = Dir<DIR>::D1, D2 = Dir<DIR>::D2;
    const int np = A.np, tid = threadIdx.x;
    const int stride[3] = {1, A.sy, A.sz};
    const int st = stride[DIR], s1 = stride[D1], s2 = stride[D2];
    const double *Q = A.Qi;
    const int n_along = DIR == 0 ? A.nx : DIR == 1 ? A.ny : A.nz;
    const int own = P.own[DIR], L = own + 6;
    const int nseg = (n_along + own - 1) / own;
    // the block's lines: its first cell along the sweep, and the interior position of a line
    const int seg = bid % nseg;
    bid /= nseg;
    const int c0 = seg * own, cells = min(own, n_along - c0);
    const int nxb = (A.nx + C - 1) / C;
    const int xb = DIR == 0 ? 0 : (bid % nxb) * C, other = DIR == 0 ? 0 : bid / nxb;
    const int row0 = DIR == 0 ? bid * P.rows : 0;
    const int all_rows = A.ny * A.nz;
    const int lines = DIR == 0 ? P.rows : C;
    // ghosted index of position a (ghosted, along the sweep) of line i, clamped into the grid
    auto at = [&](int i, int a) {
        if constexpr (DIR == 0) {
            const int r = min(row0 + i, all_rows - 1);
            return a + A.sy * (r % A.ny + A.ng) + A.sz * (r / A.ny + A.ng);
        } else {
            const int x = min(xb + i, A.nx - 1) + A.ng;
            return x + (DIR == 1 ? A.sy * a + A.sz * (other + A.ng) : A.sz * a + A.sy * (other + A.ng));
        }
    };
    const int last = n_along + 2 * A.ng - 1;
    // the thread's point, its face (left of the cell) and the face's slot
    const int li = DIR == 0 ? tid / L : tid % C, l = DIR == 0 ? tid % L : tid / C;
    const bool point = DIR == 0 ? li < lines : l < L;
    const int g = at(min(li, lines - 1), min(c0 + A.ng - 3 + l, last));
    const int F = own + 1;
    const int fi = DIR == 0 ? tid / F : tid % C, fl = (DIR == 0 ? tid % F : tid / C) + 3;
    const bool inside = DIR == 0 ? fi < lines && row0 + fi < all_rows
                                 : xb + fi < A.nx;
    const bool face = inside && fl <= cells + 3;
    const int pf = DIR == 0 ? fi * L + fl : tid + 3 * C;
    double *own_slot = S + tid;        // the point's slots
    const double *f = S + (face ? pf : 3 * STEP);  // the face's right cell
#define SV(slot, o) f[(slot) * NT + (o) * STEP]
#define SUM(slot) (SV(slot, -1) + SV(slot, 0))
    auto stage_flow = [&]() {  // velocities, T, their tangential derivatives, transport
        const int qv[4] = {1, 2, 3, 5};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const double *q = Q + qv[k] * np + g;
            own_slot[(SL::Q4 + k) * NT] = q[0];
            own_slot[(SL::DQ1 + k) * NT] = tangent4(q, s1);
            own_slot[(SL::DQ2 + k) * NT] = tangent4(q, s2);
        }
        own_slot[SL::MU * NT] = A.Ti[g], own_slot[SL::LAM * NT] = A.Ti[g + np];
        own_slot[SL::RHO * NT] = Q[g], own_slot[SL::D * NT] = A.Ti[g + 2 * np];
    };
    auto stage_species = [&]() {
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            const double *Y = A.aux + (1 + n) * np + g;
            own_slot[(SL::Y + n) * NT] = Y[0];
            own_slot[(SL::DY1 + n) * NT] = Y[s1] - Y[-s1];
            own_slot[(SL::DY2 + n) * NT] = Y[s2] - Y[-s2];
            if constexpr (MIXD) own_slot[(SL::DK + n) * NT] = A.Ti[g + (2 + n) * np];
        }
    };
    // ---- pass 1
    if (point) {
        double fp[5], fm[5];
        const double un = split_fast(Q[g], Q[g + np], Q[g + 2 * np], Q[g + 3 * np], Q[g + 4 * np],
                                     Q[g + 6 * np], __ldg(A.met[3 * DIR] + g),
                                     __ldg(A.met[3 * DIR + 1] + g), __ldg(A.met[3 * DIR + 2] + g),
                                     fp, fm);
#pragma unroll
        for (int n = 0; n < 5; ++n) own_slot[n * NT] = fp[n], own_slot[(SL::FM + n) * NT] = fm[n];
        const double Ep = 0.5 * (un + fabs(un)), Em = 0.5 * (un - fabs(un));
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            const double r = A.ri[g + n * np];
            own_slot[(SL::SP + n) * NT] = Ep * r, own_slot[(SL::SM + n) * NT] = Em * r;
        }
        own_slot[SL::PHI * NT] = A.aux[g];
    }
    __syncthreads();
    double G[5 + NS];
    if (face) {
        // schemes.jl:110-199; the branch outside the loop over the fields, so that a field's
        // loads overlap the arithmetic of the one before
        const double phif = nmax(SV(SL::PHI, -1), SV(SL::PHI, 0));
#define VP(n) ((n) < 5 ? (n) : SL::SP + (n) - 5)
#define VM(n) ((n) < 5 ? SL::FM + (n) : SL::SM + (n) - 5)
        if (phif < kHybrid1) {
            const double c7[6] = {kUP7_2, kUP7_3, kUP7_4, kUP7_5, kUP7_6, kUP7_7};
#pragma unroll
            for (int n = 0; n < 5 + NS; ++n) {
                double v = 0;
#pragma unroll
                for (int i = 0; i < 6; ++i)
                    v = fma(c7[i], SV(VP(n), i - 3) + SV(VM(n), 2 - i), v);
                G[n] = v;
            }
        } else if (phif < kHybrid2) {
#pragma unroll
            for (int n = 0; n < 5 + NS; ++n) {
                const double p2 = SV(VP(n), -1), m3 = SV(VM(n), 0);
                G[n] = p2 + m3 +
                       weno_corrections(SV(VP(n), -3), SV(VP(n), -2), p2, SV(VP(n), 0), SV(VP(n), 1),
                                        SV(VM(n), 2), SV(VM(n), 1), m3, SV(VM(n), -1), SV(VM(n), -2));
            }
        } else {
#pragma unroll
            for (int n = 0; n < 5 + NS; ++n) {
                const double p2 = SV(VP(n), -1), m3 = SV(VM(n), 0);
                G[n] = p2 + 0.5 * minmod(SV(VP(n), 0) - p2, p2 - SV(VP(n), -2)) + m3 -
                       0.5 * minmod(SV(VM(n), 1) - m3, m3 - SV(VM(n), -1));
            }
        }
#undef VP
#undef VM
    }
    __syncthreads();
    // ---- pass 2
    if (point) {
#pragma unroll
        for (int k = 0; k < 10; ++k) own_slot[(SL::MET + k) * NT] = __ldg(A.met[k] + g);
        stage_flow();
        if constexpr (SL::ONE) stage_species();
    }
    __syncthreads();
    double c[3] = {0, 0, 0}, Tf = 0;  // of the species pass: c scaled by J ρ D
    if (face) {
        double m[9];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            m[x] = SUM(SL::MET + 3 * DIR + x);
            m[3 + x] = SUM(SL::MET + 3 * D1 + x);
            m[6 + x] = SUM(SL::MET + 3 * D2 + x);
        }
        const double sJ = SUM(SL::MET + 9);
#pragma unroll
        for (int k = 0; k < 3; ++k)
            c[k] = m[3 * k] * m[0] + m[3 * k + 1] * m[1] + m[3 * k + 2] * m[2];
        double dq[4][3], su[3];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const double q0 = SV(SL::Q4 + k, 0), qm = SV(SL::Q4 + k, -1);
            dq[k][0] = 1.25 * (q0 - qm) - 1.0 / 12.0 * (SV(SL::Q4 + k, 1) - SV(SL::Q4 + k, -2));
            dq[k][1] = 0.5 * SUM(SL::DQ1 + k);
            dq[k][2] = 0.5 * SUM(SL::DQ2 + k);
            if (k < 3) su[k] = qm + q0;
            else Tf = 0.5 * (qm + q0);
        }
        viscous_flux(m, c, sJ, SUM(SL::MU), SUM(SL::LAM), su, dq, G);
        double sc = 1.0 / 16.0 * sJ * SUM(SL::RHO);
        if constexpr (!MIXD) sc *= SUM(SL::D);  // viscous.jl:473: the sum, no 1/2
        c[0] *= sc, c[1] *= 0.25 * sc, c[2] *= 0.25 * sc;
    }
    if constexpr (!SL::ONE) {  // ---- pass 3
        __syncthreads();
        if (point) stage_species();
        __syncthreads();
    }
    if (face) {
        const double T2 = 0.5 * Tf * Tf, T3 = 2.0 / 3.0 * T2 * Tf, T4 = T2 * T2, T5 = 0.8 * T4 * Tf;
        double Js = 0, HJ = 0, HY = 0;
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            const double y0 = SV(SL::Y + n, 0), ym = SV(SL::Y + n, -1);
            const double dn = 1.25 * (y0 - ym) - 1.0 / 12.0 * (SV(SL::Y + n, 1) - SV(SL::Y + n, -2));
            double J = c[0] * dn + c[1] * SUM(SL::DY1 + n) + c[2] * SUM(SL::DY2 + n);
            if constexpr (MIXD) J *= SUM(SL::DK + n);
            const double hn = h_spec(A.th, n, Tf, T2, T3, T4, T5);
            G[5 + n] -= J;
            Js += J, HJ += hn * J, HY += hn * (0.5 * (ym + y0));
        }
        G[4] += Js * HY - HJ;
#pragma unroll
        for (int n = 0; n < NS; ++n) G[5 + n] += Js * (0.5 * SUM(SL::Y + n));
    }
    __syncthreads();
    // ---- cell differences
    if (face) {
#pragma unroll
        for (int n = 0; n < 5 + NS; ++n) S[n * NT + pf] = G[n];
    }
    __syncthreads();
    if (face && fl < cells + 3) {
        const int gc = at(fi, c0 + A.ng - 3 + fl);
#pragma unroll
        for (int n = 0; n < 5 + NS; ++n) {
            const double d = G[n] - S[n * NT + pf + STEP];
            if constexpr (DIR == 0) *x_field(A, n, gc) = d;
            else (DIR == 2 ? A.R : A.R2)[gc + n * np] = d;
        }
    }
#undef SUM
#undef SV
}

template <int NS, bool MIXD>
__global__ void __launch_bounds__(kSweepNT, 3)
    k_sweeps(const __grid_constant__ Args<double> A, const __grid_constant__ SweepShape P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *S = reinterpret_cast<double *>(smem_raw);
    const int b = blockIdx.x;
    if (b < P.y0) sweep_block<2, NS, MIXD>(A, P, b, S);
    else if (b < P.x0) sweep_block<1, NS, MIXD>(A, P, b - P.y0, S);
    else sweep_block<0, NS, MIXD>(A, P, b - P.x0, S);
}

// Cuts a launch.  y and z: eight columns of n / nseg cells, at most 26 (the points of a block
// are 8 (own + 6) <= 256).  x: the rows per block and the cut of a row that need the fewest warps
// (those of the points and those of the faces) per cell.
inline SweepShape sweep_shape(int nx, int ny, int nz) {
    SweepShape P{};
    const int most = kSweepNT / kSweepCols - 6;
    const int ext[3] = {nx, ny, nz};
    for (int d = 1; d < 3; ++d) {
        const int nseg = (ext[d] + most - 1) / most;
        P.own[d] = (ext[d] + nseg - 1) / nseg;
    }
    double best = 1e300;
    for (int nseg = 1; nseg <= (nx + 25) / 26 + 1; ++nseg) {
        const int own = (nx + nseg - 1) / nseg;
        for (int rows = 1; rows * (own + 6) <= kSweepNT; ++rows) {
            const double warps = (rows * (own + 6) + 31) / 32 + (rows * (own + 1) + 31) / 32;
            const double blocks = double((ny * (long long)nz + rows - 1) / rows) * ((nx + own - 1) / own);
            if (warps * blocks < best) best = warps * blocks, P.own[0] = own, P.rows = rows;
        }
    }
    const int nxb = (nx + kSweepCols - 1) / kSweepCols;
    P.y0 = nxb * ny * ((nz + P.own[2] - 1) / P.own[2]);
    P.x0 = P.y0 + nxb * nz * ((ny + P.own[1] - 1) / P.own[1]);
    P.blocks = P.x0 + (int)((ny * (long long)nz + P.rows - 1) / P.rows) * ((nx + P.own[0] - 1) / P.own[0]);
    int t = P.rows * (P.own[0] + 6);
    for (int d = 1; d < 3; ++d) t = t > kSweepCols * (P.own[d] + 6) ? t : kSweepCols * (P.own[d] + 6);
    P.threads = (t + 31) / 32 * 32;
    return P;
}
