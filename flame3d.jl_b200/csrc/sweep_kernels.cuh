// sweep_kernels.cuh — the three sweeps of a stage in one launch, FP64 and mixed precision (sm_100a).
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
// 92 us, 64^3 521 -> 402, 128^3 2896 -> 2584, jet 256x128x128 6380 -> 5780 (its x blocks then hold
// five rows of 49 points; with one row of 92 in 256 threads 6313); 101x75x63 with five
// species 1784 -> 1061; 96^3 with nine species 5415 -> 2741, with per-species D 4638 -> 4019.
// Tried and not kept: two blocks per SM at 128 registers (jet 6623) and four at 64 (7810);
// everything but the metrics staged in pass 1 (6920); a prefetch of pass 2's lines to L2 (6399).


// Slots of a point.  Passes 2 and 3 are one where its slots leave room for three blocks per SM
// (ONE: up to three species, two with per-species D); the sensor keeps the last slot.
template <int NS, bool MIXD>
struct SweepSlots {
    // x columns of a y / z block; most points of a block (its threads) and pitch of a slot
    static constexpr int C = 8, NT = 32 * C, MINB = 3;
    static constexpr int FM = 5, SP = 10, SM = 10 + NS, F = 10 + 2 * NS;  // pass 1: F+ at 0
    static constexpr int YN = (MIXD ? 4 : 3) * NS;
    static constexpr int MOST = 37;
    static constexpr bool ONE = 26 + YN + 1 <= MOST;
    static constexpr int MET = 0, Q4 = 10, DQ1 = 14, DQ2 = 18, MU = 22, LAM = 23, RHO = 24, D = 25;
    static constexpr int Y = ONE ? 26 : 0, DY1 = Y + NS, DY2 = Y + 2 * NS, DK = Y + 3 * NS;
    static constexpr int a = F > 26 ? F : 26, b = a > YN ? a : YN;
    static constexpr int PHI = ONE ? Y + YN : b;
    static constexpr int N = PHI + 1;
    static constexpr size_t SMEM = sizeof(double) * N * NT;
    static_assert(N <= MOST && MINB * (SMEM + 1024) <= 228 * 1024, "three blocks per SM");
};

// Where the x sweep leaves field n of a cell for the finish (A.xq the five flow fields, A.xs the
// species): the stage's output arrays, whose interior the finish of the same cell writes after it
// has read this, or the second right-hand side (launch_shared).
__device__ __forceinline__ void put_x(const Args<double> &A, int n, int c, double d) {
    (n < 5 ? A.xq + n * A.np : A.xs + (n - 5) * A.np)[c] = d;
}
__device__ __forceinline__ double get_x(const Args<double> &A, int n, int c) {
    return (n < 5 ? A.xq + n * A.np : A.xs + (n - 5) * A.np)[c];
}

// A block's lines and a thread's place in them: its point, its face (left of a cell) and the
// slot of the face's right cell.
template <int DIR, int C>
struct SweepPlace {
    static constexpr int STEP = DIR == 0 ? 1 : C;  // the slot distance of two points of a line
    int sy, sz, ng, ny, line_end;  // strides, ghosts; the last line in the grid
    int first, other;              // first line (row, or x column); the third axis' position
    int c0, cells;                 // first cell along the sweep, and how many
    bool point, face;
    int g, pf, fi, fl;             // the point; the face's slot, line and position
    template <typename QT>
    __device__ __forceinline__ SweepPlace(const Args<QT> &A, const SweepShape &P, int bid)
        : sy(A.sy), sz(A.sz), ng(A.ng), ny(A.ny) {
        const int tid = threadIdx.x;
        const int n_along = DIR == 0 ? A.nx : DIR == 1 ? A.ny : A.nz;
        const int own = P.own[DIR], L = own + 6, F = own + 1;
        const int nseg = (n_along + own - 1) / own, seg = bid % nseg;
        bid /= nseg;
        c0 = seg * own, cells = min(own, n_along - c0);
        const int nxb = (A.nx + C - 1) / C, lines = DIR == 0 ? P.rows : C;
        first = DIR == 0 ? bid * P.rows : (bid % nxb) * C;
        other = DIR == 0 ? 0 : bid / nxb;
        line_end = DIR == 0 ? A.ny * A.nz - 1 : A.nx - 1;
        const int li = DIR == 0 ? tid / L : tid % C, l = DIR == 0 ? tid % L : tid / C;
        point = DIR == 0 ? li < lines : l < L;
        g = at(min(li, lines - 1), min(c0 + ng - 3 + l, n_along + 2 * ng - 1));
        fi = DIR == 0 ? tid / F : tid % C, fl = (DIR == 0 ? tid % F : tid / C) + 3;
        face = fi < lines && first + fi <= line_end && fl <= cells + 3;
        pf = face ? (DIR == 0 ? fi * L + fl : tid + 3 * C) : 3 * STEP;
    }
    // ghosted index of ghosted position a along the sweep of the block's line i, kept in the grid
    __device__ __forceinline__ int at(int i, int a) const {
        const int k = min(first + i, line_end);
        if constexpr (DIR == 0) return a + sy * (k % ny + ng) + sz * (k / ny + ng);
        else return k + ng + (DIR == 1 ? sy * a + sz * (other + ng) : sz * a + sy * (other + ng));
    }
    __device__ __forceinline__ bool cell() const { return face && fl < cells + 3; }
    __device__ __forceinline__ int cell_index() const { return at(fi, c0 + ng - 3 + fl); }
};

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

// One block of an FP64 sweep.
template <int DIR, int NS, bool MIXD>
__device__ __forceinline__ void sweep_block(const Args<double> &A, const SweepShape &P, int bid,
                                            double *S) {
    using SL = SweepSlots<NS, MIXD>;
    constexpr int NT = SL::NT, D1 = Dir<DIR>::D1, D2 = Dir<DIR>::D2;
    using Place = SweepPlace<DIR, SL::C>;
    constexpr int STEP = Place::STEP;
    const Place W(A, P, bid);
    const int np = A.np, g = W.g, pf = W.pf;
    const bool point = W.point, face = W.face;
    const int stride[3] = {1, A.sy, A.sz};
    const int s1 = stride[D1], s2 = stride[D2];
    const double *Q = A.Qi;
    double *own_slot = S + threadIdx.x;  // the point's slots
    const double *f = S + pf;            // the face's right cell
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
    if (W.cell()) {
        const int gc = W.cell_index();
#pragma unroll
        for (int n = 0; n < 5 + NS; ++n) {
            const double d = G[n] - S[n * NT + pf + STEP];
            if constexpr (DIR == 0) put_x(A, n, gc, d);
            else (DIR == 2 ? A.R : A.R2)[gc + n * np] = d;
        }
    }
#undef SUM
#undef SV
}

template <int NS, bool MIXD>
__global__ void __launch_bounds__(SweepSlots<NS, MIXD>::NT, SweepSlots<NS, MIXD>::MINB)
    k_sweeps(const __grid_constant__ Args<double> A, const __grid_constant__ SweepShape P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *S = reinterpret_cast<double *>(smem_raw);
    chain_begin();
    const int b = blockIdx.x;
    if (b < P.y0) sweep_block<2, NS, MIXD>(A, P, b, S);
    else if (b < P.x0) sweep_block<1, NS, MIXD>(A, P, b - P.y0, S);
    else sweep_block<0, NS, MIXD>(A, P, b - P.x0, S);
}
// ---- mixed precision.
// The same passes in FP32, with the arithmetic of face_phase operation by operation (its results
// to the last bit: a face whose sensor lies at a branch threshold follows every rounding of the
// state), and the differences of two faces formed in FP64.  Up to two species the x sweep is a
// launch of its own that finishes the stage; more species' finish would not fit its registers.
//
// Bound by issue (64x48x40 to 128x64x64 jets: 0.66 instructions per scheduler and cycle, 2378
// slots per cell and sweep against 2874 of the staged sweeps).  One step, staged sweeps -> these:
// 64^3 with one, two, three species 345 -> 307, 489 -> 382, 579 -> 441 us; 96^3 with four 1387 ->
// 1151; 128^3 with two 2298 -> 2114; 192^3 with nine 18.1 -> 16.1 ms.  With one species on large
// grids the staged sweeps stay ahead (96^3 756 / 758 us, 128^3 1584 / 1719, jet 256x128x128 4305 /
// 4449), so from 2^20 cells on they are launched (staged_sweeps_ahead below).  Tried and not kept:
// face fluxes in slots of their own, one barrier less (nine species at 192^3 16.1 -> 19.3 ms: the
// shared memory comes out of L1); blocks in another order (within 2 %).

// Slots of a point in FP32.  ONE: everything in one pass, where two blocks of 512 threads fit an
// SM with it (up to three species); otherwise all but the split fluxes in a second pass.  A
// point's four-byte values fill half a line with sixteen columns, which serves best until the
// species' registers spill at two blocks of 512 threads: from eight species on, three blocks of
// 256 with eight columns (80 registers instead of 64).
template <int NS>
struct MixedSlots {
    static constexpr int C = NS < 8 ? 16 : 8, NT = 32 * C, MINB = NS < 8 ? 2 : 3;
    static constexpr int FM = 5, SP = 10, SM = 10 + NS, F = 10 + 2 * NS, M = 26 + 3 * NS;
    static constexpr bool ONE = MINB * (sizeof(float) * (F + M + 1) * NT + 1024) <= 228 * 1024;
    static constexpr int MET = ONE ? F : 0, Q4 = MET + 10, DQ1 = MET + 14, DQ2 = MET + 18, TR = MET + 22,
                         RHO = MET + 25, Y = MET + 26, DY1 = Y + NS, DY2 = Y + 2 * NS,
                         PHI = Y + 3 * NS, N = PHI + 1;
    static_assert(N > F, "the sensor's slot is not the split fluxes'");
    static constexpr size_t SMEM = sizeof(float) * N * NT;
    // up to two species the finish fits the x sweep's 64 registers
    static constexpr bool FIN = NS <= 2;
};

// The x sweep's FP64 flow differences as pairs of 32-bit words in Q_out's seven fields and the
// transport's three (as floats of the same bits, so that the compiler sees the type that the finish
// stores there).
__device__ __forceinline__ float *x_word(const Args<float> &A, int k, int c) {
    return k < 7 ? A.Qo + k * A.np + c : A.To + (k - 7) * A.np + c;
}
__device__ __forceinline__ void put_x(const Args<float> &A, int n, int c, double d) {
    if (n < 5) {
        *x_word(A, 2 * n, c) = __int_as_float(__double2loint(d));
        *x_word(A, 2 * n + 1, c) = __int_as_float(__double2hiint(d));
    } else {
        A.ro[(n - 5) * A.np + c] = d;
    }
}
__device__ __forceinline__ double get_x(const Args<float> &A, int n, int c) {
    return n < 5 ? __hiloint2double(__float_as_int(*x_word(A, 2 * n + 1, c)),
                                    __float_as_int(*x_word(A, 2 * n, c)))
                 : A.ro[(n - 5) * A.np + c];
}

// FIN (x): the thread finishes its cell itself, with the z and y sweeps' parts from memory.
template <int DIR, int NS, bool FIN = false>
__device__ __forceinline__ void mixed_block(const Args<float> &A, const SweepShape &P, int bid,
                                            float *S) {
    using SL = MixedSlots<NS>;
    constexpr int NT = SL::NT, D1 = Dir<DIR>::D1, D2 = Dir<DIR>::D2;
    using Place = SweepPlace<DIR, SL::C>;
    constexpr int STEP = Place::STEP;
    const Place W(A, P, bid);
    const int np = A.np, g = W.g, pf = W.pf;
    const int stride[3] = {1, A.sy, A.sz};
    const int s1 = stride[D1], s2 = stride[D2];
    const float *Q = A.Qi;
    float *own_slot = S + threadIdx.x;
    const float *f = S + pf;
    const float h = 0.5f, c23 = float(2.0 / 3.0), c12 = float(1.0 / 12.0);
    auto metric = [&](int k) { return A.metq ? __ldg(A.metq + k * np + g) : float(__ldg(A.met[k] + g)); };
    auto stage_rest = [&]() {
#pragma unroll
        for (int k = 0; k < 10; ++k) own_slot[(SL::MET + k) * NT] = metric(k);
        const int qv[4] = {1, 2, 3, 5};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float *q = Q + qv[k] * np + g;
            own_slot[(SL::Q4 + k) * NT] = q[0];
            own_slot[(SL::DQ1 + k) * NT] = c23 * (q[s1] - q[-s1]) - c12 * (q[2 * s1] - q[-2 * s1]);
            own_slot[(SL::DQ2 + k) * NT] = c23 * (q[s2] - q[-s2]) - c12 * (q[2 * s2] - q[-2 * s2]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) own_slot[(SL::TR + k) * NT] = A.Ti[g + k * np];
        own_slot[SL::RHO * NT] = Q[g];
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            const float *Y = A.aux + (1 + n) * np + g;
            own_slot[(SL::Y + n) * NT] = Y[0];
            own_slot[(SL::DY1 + n) * NT] = Y[s1] - Y[-s1];
            own_slot[(SL::DY2 + n) * NT] = Y[s2] - Y[-s2];
        }
    };
#define SV(slot, o) f[(slot) * NT + (o) * STEP]
    if (W.point) {
        float fp[5], fm[5];
        const float E1 = split_fast(Q[g], Q[g + np], Q[g + 2 * np], Q[g + 3 * np], Q[g + 4 * np],
                                    Q[g + 6 * np], metric(3 * DIR), metric(3 * DIR + 1),
                                    metric(3 * DIR + 2), fp, fm);
#pragma unroll
        for (int n = 0; n < 5; ++n) own_slot[n * NT] = fp[n], own_slot[(SL::FM + n) * NT] = fm[n];
        const float Ep = h * (E1 + fabs(E1)), Em = h * (E1 - fabs(E1));
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            const float r = float(A.ri[g + n * np]);
            own_slot[(SL::SP + n) * NT] = Ep * r, own_slot[(SL::SM + n) * NT] = Em * r;
        }
        own_slot[SL::PHI * NT] = A.aux[g];
        if constexpr (SL::ONE) stage_rest();
    }
    __syncthreads();
    float G[5 + NS];
    if (W.face) {
        const float phif = nmax(SV(SL::PHI, -1), SV(SL::PHI, 0));
        if constexpr (NS >= 8) {
            // the branch outside the loop over the fields (192^3, nine species: 16.99 -> 16.07 ms
            // a step; with fewer species the longer code costs 1-3 %); the sums of the two
            // directions are kept apart from the products before them, as hybrid_face_fast's are
            auto P = [&](int n, int o) { return SV(n < 5 ? n : SL::SP + n - 5, o); };
            auto M = [&](int n, int o) { return SV(n < 5 ? SL::FM + n : SL::SM + n - 5, o); };
            if (phif < float(kHybrid1)) {
#pragma unroll
                for (int n = 0; n < 5 + NS; ++n) {
                    const float fp = float(kUP7_2) * P(n, -3) + float(kUP7_3) * P(n, -2) +
                                     float(kUP7_4) * P(n, -1) + float(kUP7_5) * P(n, 0) +
                                     float(kUP7_6) * P(n, 1) + float(kUP7_7) * P(n, 2);
                    const float fm = float(kUP7_7) * M(n, -3) + float(kUP7_6) * M(n, -2) +
                                     float(kUP7_5) * M(n, -1) + float(kUP7_4) * M(n, 0) +
                                     float(kUP7_3) * M(n, 1) + float(kUP7_2) * M(n, 2);
                    G[n] = __fadd_rn(fp, fm);
                }
            } else if (phif < float(kHybrid2)) {
#pragma unroll
                for (int n = 0; n < 5 + NS; ++n)
                    G[n] = __fadd_rn(wenoz_plus_fast(P(n, -3), P(n, -2), P(n, -1), P(n, 0), P(n, 1)),
                                     wenoz_minus_fast(M(n, -2), M(n, -1), M(n, 0), M(n, 1), M(n, 2)));
            } else {
#pragma unroll
                for (int n = 0; n < 5 + NS; ++n) {
                    const float p2 = P(n, -1), m3 = M(n, 0);
                    const float fp = p2 + 0.5f * minmod(P(n, 0) - p2, p2 - P(n, -2));
                    const float fm = m3 - 0.5f * minmod(M(n, 1) - m3, m3 - M(n, -1));
                    G[n] = __fadd_rn(fp, fm);
                }
            }
        } else {
#pragma unroll
            for (int n = 0; n < 5 + NS; ++n) {
                const int vp = n < 5 ? n : SL::SP + n - 5, vm = n < 5 ? SL::FM + n : SL::SM + n - 5;
                float p[7], m[7];
#pragma unroll
                for (int i = 0; i < 6; ++i) p[i] = SV(vp, i - 3), m[i] = SV(vm, i - 3);
                p[6] = m[6] = 0;
                G[n] = hybrid_face_fast<float>(p, m, phif);
            }
        }
    }
    if constexpr (!SL::ONE) {
        __syncthreads();
        if (W.point) stage_rest();
        __syncthreads();
    }
    if (W.face) {
        float met[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) met[k] = (SV(SL::MET + k, -1) + SV(SL::MET + k, 0)) * h;
        const float Jac = (SV(SL::MET + 9, -1) + SV(SL::MET + 9, 0)) * h;
        const float DL = SV(SL::TR + 2, -1), DR = SV(SL::TR + 2, 0);
        const float rho = (SV(SL::RHO, -1) + SV(SL::RHO, 0)) * h;
        const float Tf = (SV(SL::Q4 + 3, -1) + SV(SL::Q4 + 3, 0)) * h;
        const float *md = met + 3 * DIR;
        const float rhoDi = (DL + DR) * rho;  // viscous.jl:473 (no 1/2, as the reference)
        auto diffusion = [&](int n, float &Vx, float &Vy, float &Vz) {
            const float y0 = SV(SL::Y + n, 0), ym = SV(SL::Y + n, -1);
            const float yp = SV(SL::Y + n, 1), ymm = SV(SL::Y + n, -2);
            float dY[3];
            dY[DIR] = 1.25f * (y0 - ym) - c12 * (yp - ymm);
            dY[D1] = 0.25f * (SV(SL::DY1 + n, 0) + SV(SL::DY1 + n, -1));
            dY[D2] = 0.25f * (SV(SL::DY2 + n, 0) + SV(SL::DY2 + n, -1));
            Vx = (dY[0] * met[0] + dY[1] * met[3] + dY[2] * met[6]) * Jac * rhoDi;
            Vy = (dY[0] * met[1] + dY[1] * met[4] + dY[2] * met[7]) * Jac * rhoDi;
            Vz = (dY[0] * met[2] + dY[1] * met[5] + dY[2] * met[8]) * Jac * rhoDi;
            return h * (ym + y0);
        };
        float sum1 = 0, sum2 = 0, sum3 = 0;
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            float Vx, Vy, Vz;
            diffusion(n, Vx, Vy, Vz);
            sum1 += Vx, sum2 += Vy, sum3 += Vz;
        }
        float fh1 = 0, fh2 = 0, fh3 = 0;
        {
            const double Td = double(Tf);
            const double T2 = 0.5 * Td * Td, T3 = 2.0 / 3.0 * T2 * Td, T4 = T2 * T2, T5 = 0.8 * T4 * Td;
#pragma unroll
            for (int n = 0; n < NS; ++n) {
                float Vx, Vy, Vz;
                const float Yf = diffusion(n, Vx, Vy, Vz);
                const float hn = float(h_spec(A.th, n, Td, T2, T3, T4, T5));
                const float V1 = Vx - sum1 * Yf, V2 = Vy - sum2 * Yf, V3 = Vz - sum3 * Yf;
                G[5 + n] = G[5 + n] - (V1 * md[0] + V2 * md[1] + V3 * md[2]);
                fh1 += V1 * hn, fh2 += V2 * hn, fh3 += V3 * hn;
            }
        }
        const float mui = (SV(SL::TR, -1) + SV(SL::TR, 0)) * h;
        const float lami = (SV(SL::TR + 1, -1) + SV(SL::TR + 1, 0)) * h;
        // momentum and energy, viscous.jl:14-141
        float gr[4][3];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float dq[3];
            dq[DIR] = 1.25f * (SV(SL::Q4 + k, 0) - SV(SL::Q4 + k, -1)) -
                      c12 * (SV(SL::Q4 + k, 1) - SV(SL::Q4 + k, -2));
            dq[D1] = h * (SV(SL::DQ1 + k, 0) + SV(SL::DQ1 + k, -1));
            dq[D2] = h * (SV(SL::DQ2 + k, 0) + SV(SL::DQ2 + k, -1));
#pragma unroll
            for (int x = 0; x < 3; ++x)
                gr[k][x] = (dq[0] * met[x] + dq[1] * met[3 + x] + dq[2] * met[6 + x]) * Jac;
        }
        const float u = (SV(SL::Q4 + 0, -1) + SV(SL::Q4 + 0, 0)) * h;
        const float v = (SV(SL::Q4 + 1, -1) + SV(SL::Q4 + 1, 0)) * h;
        const float w = (SV(SL::Q4 + 2, -1) + SV(SL::Q4 + 2, 0)) * h;
        const float div = gr[0][0] + gr[1][1] + gr[2][2];
        const float t11 = mui * (2 * gr[0][0] - c23 * div);
        const float t12 = mui * (gr[0][1] + gr[1][0]);
        const float t13 = mui * (gr[0][2] + gr[2][0]);
        const float t22 = mui * (2 * gr[1][1] - c23 * div);
        const float t23 = mui * (gr[2][1] + gr[1][2]);
        const float t33 = mui * (2 * gr[2][2] - c23 * div);
        const float E1 = u * t11 + v * t12 + w * t13 + lami * gr[3][0] + fh1;
        const float E2 = u * t12 + v * t22 + w * t23 + lami * gr[3][1] + fh2;
        const float E3 = u * t13 + v * t23 + w * t33 + lami * gr[3][2] + fh3;
        G[1] -= md[0] * t11 + md[1] * t12 + md[2] * t13;
        G[2] -= md[0] * t12 + md[1] * t22 + md[2] * t23;
        G[3] -= md[0] * t13 + md[1] * t23 + md[2] * t33;
        G[4] -= md[0] * E1 + md[1] * E2 + md[2] * E3;
    }
#undef SV
    __syncthreads();
    if (W.face) {
#pragma unroll
        for (int n = 0; n < 5 + NS; ++n) S[n * NT + pf] = G[n];
    }
    __syncthreads();
    if (W.cell()) {
        const int gc = W.cell_index();
        double rhs[FIN ? 5 + NS : 1];
#pragma unroll
        for (int n = 0; n < 5 + NS; ++n) {
            const double d = double(G[n]) - double(S[n * NT + pf + STEP]);
            if constexpr (FIN) rhs[n] = (A.R[gc + n * np] + A.R2[gc + n * np]) + d;
            else if constexpr (DIR == 0) put_x(A, n, gc, d);
            else (DIR == 2 ? A.R : A.R2)[gc + n * np] = d;
        }
        if constexpr (FIN) {
            const int gy = gc / A.sy;
            finish_cell<NS>(A, gc, gc - gy * A.sy, gy % A.ty, gy / A.ty, rhs);
        }
    }
}

template <int NS>
__global__ void __launch_bounds__(MixedSlots<NS>::NT, MixedSlots<NS>::MINB)
    k_sweeps_mixed(const __grid_constant__ Args<float> A, const __grid_constant__ SweepShape P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float *S = reinterpret_cast<float *>(smem_raw);
    const int b = blockIdx.x;
    if (b < P.y0) mixed_block<2, NS>(A, P, b, S);
    else if (b < P.x0) mixed_block<1, NS>(A, P, b - P.y0, S);
    else mixed_block<0, NS>(A, P, b - P.x0, S);
}
// The x sweep that finishes the stage (after k_sweeps_mixed of the other two directions).
template <int NS>
__global__ void __launch_bounds__(MixedSlots<NS>::NT, MixedSlots<NS>::MINB)
    k_sweep_x_finish(const __grid_constant__ Args<float> A, const __grid_constant__ SweepShape P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    mixed_block<0, NS, true>(A, P, blockIdx.x, reinterpret_cast<float *>(smem_raw));
}

// Mixed precision: one species on at least 2^20 cells runs the staged sweeps (figures above).
constexpr bool staged_sweeps_ahead(int ns, long long cells) { return ns == 1 && cells >= 1 << 20; }
