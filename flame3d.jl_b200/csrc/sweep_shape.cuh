// sweep_shape.cuh — how a launch of the sweeps (sweep_kernels.cuh) is cut into blocks.  Host code.
#pragma once

#include <algorithm>

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
    const int all = ny * nz;  // rows; the grid's points fit in 31 bits
    constexpr int kPlaces = 148 * SL::MINB;
    int own_full = 0, rows_full = 0, warps_full = 0, blocks_full = 0;  // per rows_full rows
    int own_least = 0, rows_least = 0;
    long long least = 0;                          // warps of the whole launch
    const int fewest = (nx + NT - 7) / (NT - 6);  // cuts with which a row fits a block
    const int last = std::min(fewest + 24, (nx + 25) / 26 + 1);
    for (int nseg = fewest; nseg <= last; ++nseg) {
        const int own = (nx + nseg - 1) / nseg, s = (nx + own - 1) / own;
        for (int rows = 1, points = own + 6, faces = own + 1; points <= NT;
             ++rows, points += own + 6, faces += own + 1) {
            const int w = s * ((points + 31) / 32 + (faces + 31) / 32);
            // fewer warps per row, or as many in fewer blocks
            const long long more = (long long)w * rows_full - (long long)warps_full * rows;
            if (!rows_full || more < 0 ||
                (more == 0 && (long long)s * rows_full < (long long)blocks_full * rows))
                own_full = own, rows_full = rows, warps_full = w, blocks_full = s;
            const long long launch = (long long)w * ((all + rows - 1) / rows);
            if (!least || launch < least) least = launch, own_least = own, rows_least = rows;
        }
    }
    const long long x_blocks = (long long)blocks_full * ((all + rows_full - 1) / rows_full);
    const bool fills = 3 * x_blocks >= 2 * kPlaces;
    P.own[0] = fills ? own_full : own_least, P.rows = fills ? rows_full : rows_least;
    const int nxb = (nx + C - 1) / C;
    P.y0 = nxb * ny * ((nz + P.own[2] - 1) / P.own[2]);
    P.x0 = P.y0 + nxb * nz * ((ny + P.own[1] - 1) / P.own[1]);
    P.blocks = P.x0 + ((all + P.rows - 1) / P.rows) * ((nx + P.own[0] - 1) / P.own[0]);
    int t = P.rows * (P.own[0] + 6);
    for (int d = 1; d < 3; ++d) t = t > C * (P.own[d] + 6) ? t : C * (P.own[d] + 6);
    P.threads = (t + 31) / 32 * 32;
    return P;
}

}  // namespace pencil
}  // namespace flame
