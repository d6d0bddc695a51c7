// fused_stage.cu — host side of the fused stages: argument checks, dispatch, initial transport.
#include "fused_kernels.cuh"

int flame_pencil_stage(const FlameGrid *g, cudaStream_t s, int stage, double dt,
                       const FlameStageBuffers *b, const FlameMetrics *m, const FlameThermo *th,
                       const FlameTransport *tr, int precision, void *scratch, int split_finish,
                       int split_species);

namespace flame {
namespace fused {

FLAME_FUSED_LAUNCHES(extern, 1)
FLAME_FUSED_LAUNCHES(extern, 2)
FLAME_FUSED_LAUNCHES(extern, 3)
FLAME_FUSED_LAUNCHES(extern, 4)
FLAME_FUSED_LAUNCHES(extern, 5)
FLAME_FUSED_LAUNCHES(extern, 6)
FLAME_FUSED_LAUNCHES(extern, 7)
FLAME_FUSED_LAUNCHES(extern, 8)
FLAME_FUSED_LAUNCHES(extern, 9)

// The points whose transport a ghost fill can invalidate: with `on` set, a ghosted point is
// taken when, on an axis that is not periodic, it is a ghost or the first or last interior
// plane (the planes the reference's fills overwrite, boundary.jl:1-176); otherwise every point.
struct Shell {
    int on, tx, ty, nx, ny, nz, ng, per;
    __device__ __forceinline__ bool take(int c) const {
        if (!on) return true;
        const int gx = c % tx, gy = (c / tx) % ty, gz = c / (tx * ty);
        const auto edge = [this](int g, int n) { return g <= ng || g >= n + ng - 1; };
        return (!(per & 1) && edge(gx, nx)) || (!(per & 2) && edge(gy, ny)) ||
               (!(per & 4) && edge(gz, nz));
    }
};

// Transport of the ghosted points of a state (every point once, to start the fused stage loop;
// the boundary shell after a ghost fill).
template <int NS, typename QT>
__global__ void k_transport(int np, const QT *__restrict__ Q, const double *__restrict__ ri,
                            QT *__restrict__ To, const FlameThermo th, const FlameTransport tr,
                            const Shell sh) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= np || !sh.take(c)) return;
    double r[NS];
#pragma unroll
    for (int n = 0; n < NS; ++n) r[n] = ri[c + n * np];
    double mu, lam, D;
    transport_point<NS>(th, tr, double(Q[c + 5 * np]), double(Q[c]), r, mu, lam, D);
    To[c] = QT(mu), To[c + np] = QT(lam), To[c + 2 * np] = QT(D);
}

// The same with the mixture-averaged law (law 2): μ, λ and the per-species D_k (fields 2 + n).
template <int NS, typename QT>
__global__ void k_transport_mix(int np, const QT *__restrict__ Q, const double *__restrict__ ri,
                                QT *__restrict__ To, const FlameThermo th,
                                const FlameTransport tr, const Shell sh) {
    __shared__ MixTables<NS, QT> mt;
    mix_tables_fill<NS, QT>(th, tr, mt);
    __syncthreads();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= np || !sh.take(c)) return;
    double r[NS], Dk[NS], mu, lam;
#pragma unroll
    for (int n = 0; n < NS; ++n) r[n] = ri[c + n * np];
    mixture_point<NS, QT>(th, tr, mt, double(Q[c + 5 * np]), double(Q[c + 4 * np]), double(Q[c]), r,
                      mu, lam, Dk);
    To[c] = QT(mu), To[c + np] = QT(lam);
#pragma unroll
    for (int n = 0; n < NS; ++n) To[c + (2 + n) * np] = QT(Dk[n]);
}

template <class T, typename QT, typename CT>
int dispatch_ns(int ns, const FlameGrid &g, cudaStream_t s, int stage, double dt,
                const FlameStageBuffers &b, const FlameMetrics &m, const FlameThermo &th,
                const FlameTransport &tr) {
    switch (ns) {
#define CASE(N) \
    case N: return launch<T, N, QT, CT>(g, s, stage, dt, b, m, th, tr);
        CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9)
#undef CASE
        default:
            return flame_fail(FLAME_EUNSUPPORTED, "flame_rk_stage: ns=%d (fused path has 1..9)",
                              ns);
    }
}

template <typename QT, typename CT>
int dispatch_tile(int tile, int ns, const FlameGrid &g, cudaStream_t s, int stage, double dt,
                  const FlameStageBuffers &b, const FlameMetrics &m, const FlameThermo &th,
                  const FlameTransport &tr) {
    switch (tile) {
        case 0: return dispatch_ns<Cfg16x8x8, QT, CT>(ns, g, s, stage, dt, b, m, th, tr);
        case 1: return dispatch_ns<Cfg16x8x8b2, QT, CT>(ns, g, s, stage, dt, b, m, th, tr);
        case 2: return dispatch_ns<Cfg8x8x8, QT, CT>(ns, g, s, stage, dt, b, m, th, tr);
        case 3:
        case 4:
        case 5:
        case 6:
            return flame_pencil_stage(&g, s, stage, dt, &b, &m, &th, &tr,
                                      sizeof(QT) == 8 ? 0 : 1, b.scratch, tile == 4 || tile == 6,
                                      tile >= 5);
        default: return flame_fail(FLAME_EINVAL, "flame_rk_stage: tile config %d unknown", tile);
    }
}

template <typename QT>
int transport_ns(int ns, int np, cudaStream_t s, const void *Q, const double *ri, void *To,
                 const FlameThermo &th, const FlameTransport &tr, const Shell &sh) {
    const unsigned blocks = (unsigned)((np + 255) / 256);
    const QT *q = static_cast<const QT *>(Q);
    QT *t = static_cast<QT *>(To);
    switch (ns) {
#define CASE(N)                                                                              \
    case N:                                                                                  \
        if (tr.law == 2) k_transport_mix<N, QT><<<blocks, 256, 0, s>>>(np, q, ri, t, th, tr, sh); \
        else k_transport<N, QT><<<blocks, 256, 0, s>>>(np, q, ri, t, th, tr, sh);           \
        break;
        CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9)
#undef CASE
        default: return flame_fail(FLAME_EUNSUPPORTED, "flame_transport: ns=%d", ns);
    }
    return flame_check_launch("flame_transport");
}

}  // namespace fused
}  // namespace flame

namespace {
// Every array of the call must hold fewer than 2^31 elements (32-bit indices): `fields` is what
// the widest of them holds, at least the ten metric fields.  Extents are widened to 64 bits and
// multiplied one at a time, so absurd extents cannot wrap into a small product: before each
// multiplication the partial product is below 2^28 and the factor below 2^32.
int check_sizes(const FlameGrid *g, int fields, const char *what) {
    const long long nv = fields > 10 ? fields : 10;
    const long long ext[3] = {(long long)g->nx + 2LL * g->ng, (long long)g->ny + 2LL * g->ng,
                              (long long)g->nz + 2LL * g->ng};
    long long np = 1;
    for (long long e : ext) {
        np *= e;
        if (np * nv >= (1LL << 31))
            return flame_fail(FLAME_EINVAL,
                              "%s: %dx%dx%d cells with %lld fields exceed 2^31 elements per array",
                              what, g->nx, g->ny, g->nz, nv);
    }
    return FLAME_OK;
}
}  // namespace

static int transport_call(const FlameGrid *g, flame_stream_t s, const void *Q,
                          const double *rhoi, void *trans, const FlameThermo *th,
                          const FlameTransport *tr, int precision, bool shell,
                          const char *what) {
    if (int e = flame_check_grid(g, what)) return e;
    // law 2 stores 2 + ns transport fields
    if (int e = check_sizes(g, tr && tr->law == 2 ? 2 + g->ns : g->ns, what)) return e;
    if (!Q || !rhoi || !trans || !th || !tr) return flame_fail(FLAME_EINVAL, "%s: NULL argument", what);
    if (tr->law < 0 || tr->law > 2)
        return flame_fail(FLAME_EINVAL, "%s: transport law %d unknown", what, tr->law);
    if (tr->law == 2 && !tr->poly)
        return flame_fail(FLAME_EINVAL, "%s: law 2 needs the polynomial fits (poly)", what);
    const int np = (g->nx + 2 * g->ng) * (g->ny + 2 * g->ng) * (g->nz + 2 * g->ng);
    const flame::fused::Shell sh{shell ? 1 : 0, g->nx + 2 * g->ng, g->ny + 2 * g->ng, g->nx,
                                 g->ny, g->nz, g->ng, g->periodic & 7};
    if (shell && sh.per == 7) return FLAME_OK;  // no axis is filled by the caller
    if (precision == 0)
        return flame::fused::transport_ns<double>(g->ns, np, s, Q, rhoi, trans, *th, *tr, sh);
    if (precision == 1)
        return flame::fused::transport_ns<float>(g->ns, np, s, Q, rhoi, trans, *th, *tr, sh);
    return flame_fail(FLAME_EINVAL, "%s: precision=%d must be 0 or 1", what, precision);
}

extern "C" int flame_transport(const FlameGrid *g, flame_stream_t s, const void *Q,
                               const double *rhoi, void *trans, const FlameThermo *th,
                               const FlameTransport *tr, int precision) {
    return transport_call(g, s, Q, rhoi, trans, th, tr, precision, false, "flame_transport");
}

extern "C" int flame_transport_boundary(const FlameGrid *g, flame_stream_t s, const void *Q,
                                        const double *rhoi, void *trans, const FlameThermo *th,
                                        const FlameTransport *tr, int precision) {
    return transport_call(g, s, Q, rhoi, trans, th, tr, precision, true,
                          "flame_transport_boundary");
}

extern "C" int flame_rk_stage_tiled(const FlameGrid *g, flame_stream_t s, int stage, double dt,
                                    const FlameStageBuffers *b, const FlameMetrics *m,
                                    const FlameThermo *th, const FlameTransport *tr,
                                    int precision, int tile) {
    static const char *kNames[3] = {"flame_rk_stage 1", "flame_rk_stage 2", "flame_rk_stage 3"};
    flame::NvtxRange range(kNames[(stage >= 1 && stage <= 3) ? stage - 1 : 0]);
    if (int e = flame_check_grid(g, "flame_rk_stage")) return e;
    // the right-hand sides of the pencil configurations hold 5 + ns fields
    if (int e = check_sizes(g, tile >= 3 ? 5 + g->ns : g->ns, "flame_rk_stage")) return e;
    if (!b || !m || !th || !tr || !b->U || !b->Un || !b->Q_in || !b->Q_out || !b->rhoi_in ||
        !b->rhoi_out || !b->rhon || !b->trans_in || !b->trans_out || !m->J || !m->dxidx ||
        !m->dxidy || !m->dxidz || !m->detadx || !m->detady || !m->detadz || !m->dzetadx ||
        !m->dzetady || !m->dzetadz)
        return flame_fail(FLAME_EINVAL, "flame_rk_stage: NULL argument");
    if (stage < 1 || stage > 3)
        return flame_fail(FLAME_EINVAL, "flame_rk_stage: stage=%d must be 1, 2 or 3", stage);
    if (tr->law < 0 || tr->law > 2)
        return flame_fail(FLAME_EINVAL, "flame_rk_stage: transport law %d unknown", tr->law);
    if (tr->law == 2 && !tr->poly)
        return flame_fail(FLAME_EINVAL, "flame_rk_stage: law 2 needs the polynomial fits (poly)");
    if (tr->law == 2 && tile >= 0 && tile <= 2)
        return flame_fail(FLAME_EUNSUPPORTED,
                          "flame_rk_stage: transport law 2 (per-species D_k) runs on the pencil "
                          "configurations 3-6, not on tile configuration %d", tile);
    if (g->nx < FLAME_NG || g->ny < FLAME_NG || g->nz < FLAME_NG)
        return flame_fail(FLAME_EINVAL, "flame_rk_stage: extents must be >= %d", FLAME_NG);
    if (b->Q_in == b->Q_out || (const void *)b->rhoi_in == (const void *)b->rhoi_out ||
        b->trans_in == b->trans_out)
        return flame_fail(FLAME_EINVAL, "flame_rk_stage: in and out buffers must differ");
    if (precision == 0)
        return flame::fused::dispatch_tile<double, double>(tile, g->ns, *g, s, stage, dt, *b, *m,
                                                           *th, *tr);
    if (precision == 1)
        return flame::fused::dispatch_tile<float, float>(tile, g->ns, *g, s, stage, dt, *b, *m,
                                                         *th, *tr);
    return flame_fail(FLAME_EINVAL, "flame_rk_stage: precision=%d must be 0 or 1", precision);
}

extern "C" int flame_rk_stage(const FlameGrid *g, flame_stream_t s, int stage, double dt,
                              const FlameStageBuffers *b, const FlameMetrics *m,
                              const FlameThermo *th, const FlameTransport *tr, int precision) {
    return flame_rk_stage_tiled(g, s, stage, dt, b, m, th, tr, precision, 0);
}
