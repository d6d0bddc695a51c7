// pencil_stage.cu — host side of the pencil sweeps: dispatch by species count, and batches.
#include "pencil_kernels.cuh"

namespace flame {
namespace pencil {

// Declared here, defined by pencil_inst.cu (one object file per species count).
#define DECLARE(N) \
    template <>    \
    const PencilOps &pencil_ops<N>();
DECLARE(1) DECLARE(2) DECLARE(3) DECLARE(4) DECLARE(5) DECLARE(6) DECLARE(7) DECLARE(8) DECLARE(9)
#undef DECLARE

// The entries of species count ns, or null outside 1..9.
inline const PencilOps *ops_of(int ns) {
    switch (ns) {
#define CASE(N) \
    case N: return &pencil_ops<N>();
        CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9)
#undef CASE
        default: return nullptr;
    }
}

}  // namespace pencil
}  // namespace flame

// Entry used by fused_stage.cu's dispatcher for tile configuration 3.
int flame_pencil_stage(const FlameGrid *g, cudaStream_t s, int stage, double dt,
                       const FlameStageBuffers *b, const FlameMetrics *m, const FlameThermo *th,
                       const FlameTransport *tr, int precision, void *scratch, int split_finish,
                       int split_species) {
    if (!scratch)
        return flame_fail(FLAME_EINVAL,
                          "flame_rk_stage: the pencil configuration needs scratch (see "
                          "flame_stage_scratch_bytes)");
    const flame::pencil::PencilOps *ops = flame::pencil::ops_of(g->ns);
    if (!ops)
        return flame_fail(FLAME_EUNSUPPORTED, "flame_rk_stage: ns=%d (pencil path has 1..9)",
                          g->ns);
    return ops->stage[precision](*g, s, stage, dt, *b, *m, *th, *tr, scratch, split_finish != 0,
                                 split_species != 0);
}

// What launch_fp64 and launch_mixed issue.
extern "C" int flame_stage_launches(int ns, long long cells, int law, int precision, int tile) {
    const bool tiled = tile >= 0 && tile <= 2;
    if (ns < 1 || ns > FLAME_FUSED_MAX_NS || cells < 1 || law < 0 || law > 2 || tile < 0 || tile > 6 ||
        (precision != 0 && precision != 1) || (tiled && law == 2))
        return 0;
    if (tiled) return 1;
    if (precision == 0) return 3;                // prep, the sweeps, finish
    if (law == 2) return 7;                      // prep, flow and species sweeps of z and y, x, finish
    const int finish = tile == 4 || tile == 6;
    if (tile >= 5) return 6 + finish;
    if (!flame::pencil::staged_sweeps_ahead(ns, cells)) return 3;
    return 4 + finish;                           // prep, z, y, x
}

// SIZE_MAX when the product does not fit in size_t (then no buffer can be large enough).
extern "C" size_t flame_stage_scratch_bytes(const FlameGrid *g, int precision) {
    if (!g || g->nx < 1 || g->ny < 1 || g->nz < 1 || g->ng < 0 || g->ns < 0) return 0;
    const size_t q = precision == 0 ? sizeof(double) : sizeof(float);
    size_t bytes = 2 * (5 + (size_t)g->ns) * sizeof(double) + (1 + (size_t)g->ns) * q;
    const size_t ext[3] = {(size_t)g->nx + 2 * (size_t)g->ng, (size_t)g->ny + 2 * (size_t)g->ng,
                           (size_t)g->nz + 2 * (size_t)g->ng};
    for (size_t e : ext)
        if (__builtin_mul_overflow(bytes, e, &bytes)) return SIZE_MAX;
    return bytes;
}

// ============================================================================= batches
// A batch advances many independent cases per stage: the cases are grouped by species count and
// transport family (laws 0 and 1, or law 2) and the groups cut into chunks of at most
// kConstCases cases; per chunk and stage a copy of the chunk's descriptors into the constant
// table, a memset of its counters and its persistent launches (two, or four for law 2).
// Descriptors for the three stages and both in/out parities, the work lists and the per-case
// item counts are uploaded once, into device workspace the caller owns, so flame_batch_stage
// issues copies, memsets and launches only (capturable as a CUDA graph).
#include <array>

struct FlameBatch {
    int precision = 0;
    int *err = nullptr;  // device error word (FLAME_ETIMEOUT)
    int stall = 0;       // test hook (flame_batch_test_stall)
    std::vector<flame::pencil::BatchChunk> chunks;
    // Chunks run side by side on lanes: lane 0 is the caller's stream, the others are the batch's
    // own, forked from it and joined back to it within every stage.  A species count keeps to
    // one lane, since its chunks share a constant table.
    std::vector<int> lane;             // of each chunk
    std::vector<cudaStream_t> side;    // lanes 1, 2, ...
    std::vector<cudaEvent_t> joined;   // one per side stream
    cudaEvent_t fork = nullptr;
    ~FlameBatch() {
        for (cudaEvent_t e : joined) cudaEventDestroy(e);
        for (cudaStream_t t : side) cudaStreamDestroy(t);
        if (fork) cudaEventDestroy(fork);
    }
};

namespace flame {
namespace pencil {

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

template <typename QT>
size_t args_size() { return sizeof(Args<QT>); }

// Items of one case in each phase of a chunk of shape d.
inline void case_items(const FlameGrid &g, const BatchDims &d, int items[kMaxPhases]) {
    const long long tx = g.nx + 2LL * g.ng, ty = g.ny + 2LL * g.ng, tz = g.nz + 2LL * g.ng;
    const long long np = tx * ty * tz;
    auto zsweep = [&](int cols) { return ((g.nx + cols - 1) / cols) * ((g.nz + OWN - 1) / OWN) * g.ny; };
    auto ysweep = [&](int cols) { return ((g.nx + cols - 1) / cols) * ((g.ny + OWN - 1) / OWN) * g.nz; };
    const long long per = (long long)d.nt * kPrepPerThread;
    items[0] = (int)((np + per - 1) / per);
    items[1] = zsweep(d.cols);
    items[2] = ysweep(d.cols);
    int k = 3;
    if (d.phases == 7) items[3] = zsweep(d.cols_s), items[4] = ysweep(d.cols_s), k = 5;
    const long long warps = (long long)g.ny * g.nz * ((g.nx + OWN - 1) / OWN);
    items[k] = (int)((warps + Wpb<0>::value - 1) / Wpb<0>::value);
    if (d.phases == 7) items[6] = (int)(((long long)g.nx * g.ny * g.nz + 127) / 128);
}

// The operations of a chunk's species count, or an error.
inline int batch_ops(int ns, const PencilOps *&ops) {
    ops = ops_of(ns);
    return ops ? FLAME_OK : flame_fail(FLAME_EUNSUPPORTED, "flame_batch: ns=%d (1..9)", ns);
}

template <typename QT>
void fill_args(std::vector<unsigned char> &host, size_t at, const FlameCaseDesc &c, int stage,
               int parity) {
    FlameStageBuffers b = c.buf;
    if (parity) {  // the stage reads what the buffers call "out" and writes "in"
        const void *q = b.Q_in, *t = b.trans_in;
        const double *r = b.rhoi_in;
        b.Q_in = b.Q_out, b.Q_out = const_cast<void *>(q);
        b.rhoi_in = b.rhoi_out, b.rhoi_out = const_cast<double *>(r);
        b.trans_in = b.trans_out, b.trans_out = const_cast<void *>(t);
    }
    const Args<QT> A =
        make_args<QT>(c.grid, stage, c.dt, b, c.metrics, c.thermo, c.transport, c.buf.scratch);
    memcpy(host.data() + at, &A, sizeof(A));
}

}  // namespace pencil
}  // namespace flame

namespace {

// Chunks (cases of one species count, at most kConstCases each) and the byte layout of the
// workspace: the batch's error word, then per chunk six descriptor arrays, the work list, the
// per-case counts and the counters, each aligned to 256 bytes.
struct ChunkPlan {
    int ns = 0;
    bool mix = false;  // law 2
    flame::pencil::BatchDims dims;
    std::vector<int> members;  // case indices
    long long total = 0;
    size_t args_at[6] = {}, items_at = 0, need_at = 0, counters_at = 0;
};

struct Layout {
    std::vector<ChunkPlan> chunks;
    size_t bytes = 0;
};

// The status of a runtime call.  A failed call also leaves its error as the thread's last one, which
// the next launch check would report as its own, so it is cleared.
int batch_error(cudaError_t e, const char *what) {
    if (e == cudaSuccess) return FLAME_OK;
    cudaGetLastError();
    return flame_fail(FLAME_ELAUNCH, "%s: %s", what, cudaGetErrorString(e));
}

// Lanes of a batch.  Small cases leave the GPU idle between and inside their chunks' launches:
// ten cases of 32^3 and 48^3 with four species counts 1868 -> 1772 us a step, six of 33^3 to 60^3 1872
// -> 1652, six of 48^3 to 96^3 (2.7 million cells) 4190 -> 4122.  Beyond 2^22 cells a batch fills the
// GPU by itself (64 cases up to 128^3 lost 2 % side by side).
constexpr int kMostLanes = 4;
int make_lanes(FlameBatch &B, long long cells) {
    std::vector<int> counts;  // species counts in the order of their first chunk
    for (const flame::pencil::BatchChunk &c : B.chunks)
        if (std::find(counts.begin(), counts.end(), c.ns) == counts.end()) counts.push_back(c.ns);
    const int lanes = cells > 1 << 22 ? 1 : std::min<int>(kMostLanes, (int)counts.size());
    for (const flame::pencil::BatchChunk &c : B.chunks)
        B.lane.push_back((int)(std::find(counts.begin(), counts.end(), c.ns) - counts.begin()) % lanes);
    if (lanes == 1) return FLAME_OK;
    cudaError_t e = cudaEventCreateWithFlags(&B.fork, cudaEventDisableTiming);
    for (int k = 1; k < lanes && e == cudaSuccess; ++k) {
        cudaStream_t t;
        e = cudaStreamCreateWithFlags(&t, cudaStreamNonBlocking);
        if (e != cudaSuccess) break;
        B.side.push_back(t);
        cudaEvent_t ev;
        e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
        if (e == cudaSuccess) B.joined.push_back(ev);
    }
    return batch_error(e, "flame_batch_create");
}

// A case's group: its species count, and whether it has per-species D_k (law 2).
int group_of(const FlameCaseDesc &c) { return 2 * c.grid.ns + (c.transport.law == 2); }

int plan_layout(const FlameCaseDesc *cases, int n, int precision, Layout &L) {
    std::vector<int> groups;
    for (int i = 0; i < n; ++i)
        if (std::find(groups.begin(), groups.end(), group_of(cases[i])) == groups.end())
            groups.push_back(group_of(cases[i]));
    for (int grp : groups) {
        const int ns = grp / 2;
        const bool mix = grp % 2;
        const flame::pencil::PencilOps *ops;
        if (int e = flame::pencil::batch_ops(ns, ops)) return e;
        const flame::pencil::BatchDims dims = ops->dims[precision](mix);
        bool fresh = true;
        for (int i = 0; i < n; ++i) {
            if (group_of(cases[i]) != grp) continue;
            if (fresh || (int)L.chunks.back().members.size() == flame::pencil::kConstCases) {
                L.chunks.emplace_back();
                L.chunks.back().ns = ns, L.chunks.back().mix = mix;
                L.chunks.back().dims = dims;
                fresh = false;
            }
            ChunkPlan &c = L.chunks.back();
            c.members.push_back(i);
            int it[flame::pencil::kMaxPhases] = {};
            flame::pencil::case_items(cases[i].grid, dims, it);
            for (int ph = 0; ph < dims.phases; ++ph) c.total += it[ph];
        }
    }
    const size_t asz = precision == 0 ? flame::pencil::args_size<double>()
                                      : flame::pencil::args_size<float>();
    using flame::pencil::align256;
    size_t at = 256;  // the error word
    for (ChunkPlan &c : L.chunks) {
        if (c.total >= (1LL << 31))
            return flame_fail(FLAME_EINVAL, "flame_batch: %lld work items in one chunk", c.total);
        const size_t m = c.members.size();
        for (int v = 0; v < 6; ++v) c.args_at[v] = at, at = align256(at + asz * m);
        c.items_at = at, at = align256(at + sizeof(flame::pencil::BatchItem) * c.total);
        c.need_at = at, at = align256(at + sizeof(int4) * m);
        c.counters_at = at, at = align256(at + sizeof(int) * (4 + 4 * m));
    }
    L.bytes = at;
    return FLAME_OK;
}

int check_case(const FlameCaseDesc &c, int i) {
    if (int e = flame_check_grid(&c.grid, "flame_batch")) return e;
    if ((c.grid.periodic & 7) != 7)
        return flame_fail(FLAME_EUNSUPPORTED, "flame_batch: case %d is not periodic", i);
    if (c.grid.ns > 9) return flame_fail(FLAME_EUNSUPPORTED, "flame_batch: case %d ns > 9", i);
    if (c.grid.nx < FLAME_NG || c.grid.ny < FLAME_NG || c.grid.nz < FLAME_NG)
        return flame_fail(FLAME_EINVAL, "flame_batch: case %d extents must be >= %d", i, FLAME_NG);
    const long long np =
        ((long long)c.grid.nx + 8) * ((long long)c.grid.ny + 8) * ((long long)c.grid.nz + 8);
    // 32-bit indices: the widest arrays are the ten metric fields and the right-hand sides
    const int fields = std::max(10, 5 + c.grid.ns);
    if (c.grid.nx > (1 << 20) || c.grid.ny > (1 << 20) || c.grid.nz > (1 << 20) ||
        np * fields >= (1LL << 31))
        return flame_fail(FLAME_EINVAL, "flame_batch: case %d too large", i);
    const FlameStageBuffers &b = c.buf;
    if (!b.U || !b.Un || !b.Q_in || !b.Q_out || !b.rhoi_in || !b.rhoi_out || !b.rhon ||
        !b.trans_in || !b.trans_out || !b.scratch || !c.metrics.J || !c.metrics.dxidx)
        return flame_fail(FLAME_EINVAL, "flame_batch: case %d has a NULL buffer", i);
    if (c.transport.law < 0 || c.transport.law > 2)
        return flame_fail(FLAME_EINVAL, "flame_batch: case %d: transport law %d", i,
                          c.transport.law);
    return FLAME_OK;
}

}  // namespace

extern "C" size_t flame_batch_workspace_bytes(const FlameCaseDesc *cases, int n, int precision) {
    if (!cases || n < 1 || (precision != 0 && precision != 1)) return 0;
    for (int i = 0; i < n; ++i)
        if (check_case(cases[i], i)) return 0;
    Layout L;
    if (plan_layout(cases, n, precision, L)) return 0;
    return L.bytes;
}

extern "C" int flame_batch_create(FlameBatch **out, const FlameCaseDesc *cases, int n,
                                  int precision, void *workspace, size_t bytes,
                                  flame_stream_t s) {
    if (!out || !cases || n < 1) return flame_fail(FLAME_EINVAL, "flame_batch_create: no cases");
    if (precision != 0 && precision != 1)
        return flame_fail(FLAME_EINVAL, "flame_batch_create: precision=%d", precision);
    for (int i = 0; i < n; ++i)
        if (int e = check_case(cases[i], i)) return e;
    Layout L;
    if (int e = plan_layout(cases, n, precision, L)) return e;
    if (!workspace || bytes < L.bytes)
        return flame_fail(FLAME_EINVAL, "flame_batch_create: workspace of %zu bytes, need %zu",
                          bytes, L.bytes);
    std::vector<unsigned char> host(L.bytes, 0);
    FlameBatch *B = new FlameBatch();
    B->precision = precision;
    unsigned char *dev = static_cast<unsigned char *>(workspace);
    B->err = reinterpret_cast<int *>(dev);
    const size_t asz = precision == 0 ? flame::pencil::args_size<double>()
                                      : flame::pencil::args_size<float>();
    using flame::pencil::BatchItem;
    for (const ChunkPlan &cp : L.chunks) {
        flame::pencil::BatchChunk bc;
        bc.ns = cp.ns;
        bc.mix = cp.mix;
        bc.n = (int)cp.members.size();
        const int phases = cp.dims.phases;
        std::vector<int4> need(bc.n);
        std::vector<std::array<int, flame::pencil::kMaxPhases>> counts(bc.n);
        for (int j = 0; j < bc.n; ++j) {
            const FlameCaseDesc &c = cases[cp.members[j]];
            counts[j].fill(0);
            flame::pencil::case_items(c.grid, cp.dims, counts[j].data());
            need[j] = make_int4(counts[j][0], 0, 0, 0);
            for (int st = 1; st <= 3; ++st)
                for (int par = 0; par < 2; ++par) {
                    const size_t at = cp.args_at[(st - 1) * 2 + par] + asz * j;
                    if (precision == 0) flame::pencil::fill_args<double>(host, at, c, st, par);
                    else flame::pencil::fill_args<float>(host, at, c, st, par);
                }
        }
        // work list: phase by phase (prep, z, y, ... as BatchDims lists them), each phase's
        // items case by case
        BatchItem *items = reinterpret_cast<BatchItem *>(host.data() + cp.items_at);
        long long w = 0;
        for (int ph = 0; ph < phases; ++ph) {
            bc.bound[ph] = (int)w;
            for (int j = 0; j < bc.n; ++j)
                for (int b = 0; b < counts[j][ph]; ++b) items[w++] = BatchItem{j, b};
        }
        bc.bound[phases] = (int)w;
        memcpy(host.data() + cp.need_at, need.data(), sizeof(int4) * bc.n);
        for (int v = 0; v < 6; ++v) bc.args[v] = dev + cp.args_at[v];
        bc.items = reinterpret_cast<const BatchItem *>(dev + cp.items_at);
        bc.need = reinterpret_cast<const int4 *>(dev + cp.need_at);
        bc.counters = reinterpret_cast<int *>(dev + cp.counters_at);
        if (int e = flame::pencil::ops_of(bc.ns)->grid[precision](bc)) {
            delete B;
            return e;
        }
        B->chunks.push_back(bc);
    }
    long long cells = 0;
    for (int i = 0; i < n; ++i)
        cells += (long long)cases[i].grid.nx * cases[i].grid.ny * cases[i].grid.nz;
    if (int e = make_lanes(*B, cells)) {
        delete B;
        return e;
    }
    cudaError_t ce = cudaMemcpyAsync(workspace, host.data(), L.bytes, cudaMemcpyHostToDevice, s);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
    if (int e = batch_error(ce, "flame_batch_create: upload")) {
        delete B;
        return e;
    }
    *out = B;
    return FLAME_OK;
}

extern "C" int flame_batch_stage(FlameBatch *B, flame_stream_t s, int stage, int parity) {
    flame::NvtxRange range("flame_batch_stage");
    if (!B) return flame_fail(FLAME_EINVAL, "flame_batch_stage: NULL batch");
    if (stage < 1 || stage > 3 || (parity != 0 && parity != 1))
        return flame_fail(FLAME_EINVAL, "flame_batch_stage: stage=%d parity=%d", stage, parity);
    cudaError_t ce = cudaSuccess;
    if (!B->side.empty()) ce = cudaEventRecord(B->fork, s);
    for (cudaStream_t t : B->side)
        if (ce == cudaSuccess) ce = cudaStreamWaitEvent(t, B->fork, 0);
    int err = FLAME_OK;
    for (size_t k = 0; k < B->chunks.size() && ce == cudaSuccess && !err; ++k) {
        const flame::pencil::BatchChunk &bc = B->chunks[k];
        const cudaStream_t t = B->lane[k] ? B->side[B->lane[k] - 1] : s;
        err = flame::pencil::ops_of(bc.ns)->batch[B->precision](bc, t, stage, parity, B->err, B->stall);
    }
    for (size_t k = 0; k < B->side.size(); ++k) {  // joined whatever happened in between
        cudaError_t je = cudaEventRecord(B->joined[k], B->side[k]);
        if (je == cudaSuccess) je = cudaStreamWaitEvent(s, B->joined[k], 0);
        if (ce == cudaSuccess) ce = je;
    }
    if (ce != cudaSuccess) cudaGetLastError();
    return err ? err : batch_error(ce, "flame_batch_stage");
}

extern "C" int flame_batch_status(FlameBatch *B, flame_stream_t s) {
    if (!B) return flame_fail(FLAME_EINVAL, "flame_batch_status: NULL batch");
    int h = 0;
    cudaError_t ce = cudaMemcpyAsync(&h, B->err, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
    if (ce == cudaSuccess && h) ce = cudaMemsetAsync(B->err, 0, sizeof(int), s);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
    if (int e = batch_error(ce, "flame_batch_status")) return e;
    if (h)
        return flame_fail(FLAME_ETIMEOUT,
                          "flame_batch_stage: a wait for another work item's completion ran out; "
                          "the items after it were skipped and the cases' states are invalid");
    return FLAME_OK;
}

extern "C" int flame_batch_test_stall(FlameBatch *B, int on) {
    if (!B) return flame_fail(FLAME_EINVAL, "flame_batch_test_stall: NULL batch");
    B->stall = on != 0;
    return FLAME_OK;
}

extern "C" int flame_batch_destroy(FlameBatch *B) {
    delete B;
    return FLAME_OK;
}
