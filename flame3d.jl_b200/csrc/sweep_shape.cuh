// sweep_shape.cuh — how a launch of the sweeps (sweep_kernels.cuh) is cut into blocks.  Host code.
#pragma once

namespace flame {
namespace pencil {

// How the launch is cut: own cells per line and direction, lines per x block, threads per
// block, and the first block of the y and of the x sweep (blocks [0, y0) are the z sweep's).
struct SweepShape {
    int own[3], rows, threads, y0, x0, blocks;
};

// Cuts a launch of blocks of at most SL::NT threads with SL::C columns, SL::MINB of them on an SM.
// y and z: C columns of n / nseg cells, at most 26 (the points of a block are C (own + 6) <= 32 C).
// x: among the rows per block and the cuts of a row that need the fewest warps per cell (those of
// the points and those of the faces) the one with the fewest blocks, where those still fill two
// thirds of the SMs' places; on fewer cells the cut with the fewest warps in all, whose blocks are
// smaller.  A block holds its shared memory and registers whatever it is given, so of two cuts with
// the same warps the one with fewer, fuller blocks keeps more warps on an SM; but blocks that do not
// reach every SM are better small.  One step, smaller -> fuller: mixed precision 89x64x60 (rows of 95
// points in blocks of 512 threads, one -> five) 681 -> 448 us, 120x64x60 790 -> 574; FP64 256x64x60
// (one row of 92 points in 256 threads -> five of 49) 1576 -> 1437.  At the line, mixed: 27x48x49 (157
// blocks) 122 -> 147, 270x16x17 (165) 122 -> 145, every grid measured from 200 blocks on 3 to 33 %
// faster; FP64: 256x12x13 (192 blocks) 95 -> 101, 256x16x17 (330) 138 -> 136, 270x16x17 (408) 139 ->
// 137.  Cuts within 2 or 4 % of the fewest warps, taken for still fewer blocks, gained nothing.
template <typename SL>
inline SweepShape sweep_shape(int nx, int ny, int nz) {
    constexpr int C = SL::C, NT = SL::NT;
    SweepShape P{};
    const int most = NT / C - 6;
    const int ext[3] = {nx, ny, nz};
    for (int d = 1; d < 3; ++d) {
        const int nseg = (ext[d] + most - 1) / most;
        P.own[d] = (ext[d] + nseg - 1) / nseg;
    }
    const long long all = ny * (long long)nz;
    constexpr int kPlaces = 148 * SL::MINB;
    struct Cut {
        int own = 0, rows = 0;
        long long warps = 0, blocks = 0;
    } full, least;  // warps and blocks of `full` per `rows` rows, of `least` per launch
    const int fewest = (nx + NT - 7) / (NT - 6);  // cuts with which a row fits a block
    for (int nseg = fewest; nseg <= fewest + 24 && nseg <= (nx + 25) / 26 + 1; ++nseg) {
        const int own = (nx + nseg - 1) / nseg;
        for (int rows = 1; rows * (own + 6) <= NT; ++rows) {
            const long long s = (nx + own - 1) / own;
            const long long w = s * ((rows * (own + 6) + 31) / 32 + (rows * (own + 1) + 31) / 32);
            const long long more = w * full.rows - full.warps * rows;  // > 0: more warps per row
            if (!full.rows || more < 0 || (more == 0 && s * full.rows < full.blocks * rows))
                full = {own, rows, w, s};
            const long long times = (all + rows - 1) / rows;
            if (!least.rows || w * times < least.warps) least = {own, rows, w * times, s * times};
        }
    }
    const bool fills = 3 * full.blocks * ((all + full.rows - 1) / full.rows) >= 2 * kPlaces;
    P.own[0] = fills ? full.own : least.own, P.rows = fills ? full.rows : least.rows;
    const int nxb = (nx + C - 1) / C;
    P.y0 = nxb * ny * ((nz + P.own[2] - 1) / P.own[2]);
    P.x0 = P.y0 + nxb * nz * ((ny + P.own[1] - 1) / P.own[1]);
    P.blocks = P.x0 + (int)((all + P.rows - 1) / P.rows) * ((nx + P.own[0] - 1) / P.own[0]);
    int t = P.rows * (P.own[0] + 6);
    for (int d = 1; d < 3; ++d) t = t > C * (P.own[d] + 6) ? t : C * (P.own[d] + 6);
    P.threads = (t + 31) / 32 * 32;
    return P;
}

}  // namespace pencil
}  // namespace flame
