"""How the sweeps are cut into blocks (csrc/sweep_shape.cuh, host code, compiled here with g++): every
cell has one owner, blocks fit, and of the x cuts that need the fewest warps the fullest is taken
where its blocks fill two thirds of the SMs' places, else one of the fewest warps in the launch."""
from __future__ import annotations

import shutil
import subprocess
from fractions import Fraction
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "flame3d.jl_b200" / "csrc"
SHAPES = [(8, 256, 3), (16, 512, 2)]  # columns, threads, blocks per SM: FP64 and 8-9 mixed; mixed

MAIN = """
#include <cstdio>
#include <cstdlib>
#include "sweep_shape.cuh"
struct SL { static constexpr int C = %d, NT = %d, MINB = %d; };
int main(int argc, char **argv) {
    for (int a = 1; a + 2 < argc; a += 3) {
        const auto P = flame::pencil::sweep_shape<SL>(atoi(argv[a]), atoi(argv[a + 1]), atoi(argv[a + 2]));
        printf("%%d %%d %%d %%d %%d %%d %%d %%d\\n", P.own[0], P.own[1], P.own[2], P.rows, P.threads, P.y0,
               P.x0, P.blocks);
    }
}
"""


def _warps(own, rows):
    return -(-rows * (own + 6) // 32) + -(-rows * (own + 1) // 32)


@pytest.mark.parametrize("cols,nt,per_sm", SHAPES)
def test_cuts(tmp_path, cols, nt, per_sm):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    src, exe = tmp_path / "cut.cpp", tmp_path / "cut"
    src.write_text(MAIN % (cols, nt, per_sm))
    subprocess.run([gxx, "-std=c++17", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    grids = [(nx, ny, nz) for nx in range(4, 700) for ny, nz in ((64, 60), (12, 9))]
    grids += [(100000, 4, 4), (5, 4, 2000), (33, 1000, 7), (250, 5, 4), (251, 4, 5)]
    out = subprocess.run([str(exe), *(str(v) for g in grids for v in g)], check=True, text=True,
                         capture_output=True).stdout.splitlines()
    assert len(out) == len(grids)
    up = lambda a, b: -(-a // b)  # noqa: E731
    for (nx, ny, nz), line in zip(grids, out):
        ox, oy, oz, rows, threads, y0, x0, blocks = map(int, line.split())
        assert rows >= 1 and rows * (ox + 6) <= threads <= nt and threads % 32 == 0
        for own in (oy, oz):
            assert 1 <= own <= nt // cols - 6 and cols * (own + 6) <= threads
        assert y0 == up(nx, cols) * ny * up(nz, oz)
        assert x0 == y0 + up(nx, cols) * nz * up(ny, oy)
        assert blocks == x0 + up(ny * nz, rows) * up(nx, ox)
        if nx >= 700:
            continue
        cuts = [(up(nx, own), own, r) for own in {up(nx, s) for s in range(up(nx, nt - 6), up(nx, 26) + 2)}
                for r in range(1, nt // (own + 6) + 1)]
        per_row = min((Fraction(s * _warps(own, r), r), Fraction(s, r)) for s, own, r in cuts)
        x_blocks = {s * up(ny * nz, r) for s, own, r in cuts
                    if (Fraction(s * _warps(own, r), r), Fraction(s, r)) == per_row}
        if 3 * max(x_blocks) >= 2 * 148 * per_sm and len(x_blocks) == 1:
            assert blocks - x0 in x_blocks, (nx, ny, nz)
            assert nx < 32 or 2 * rows * (ox + 6) > nt, (nx, ny, nz, ox, rows)
        elif 3 * max(x_blocks) < 2 * 148 * per_sm:
            total = min(s * _warps(own, r) * up(ny * nz, r) for s, own, r in cuts)
            assert up(nx, ox) * _warps(ox, rows) * up(ny * nz, rows) == total, (nx, ny, nz)
