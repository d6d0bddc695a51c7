"""flame_stage_launches against the kernels a captured stage holds, on both sides of every rule that
picks a set of kernels."""
from __future__ import annotations

import pytest


def test_counts_and_refusals(f3d):
    lib = f3d.load_library()
    n = lib.flame_stage_launches
    assert [n(1, 1000, 1, 0, t) for t in range(7)] == [1, 1, 1, 3, 3, 3, 3]
    assert [n(9, 1000, 2, 0, t) for t in range(7)] == [0, 0, 0, 3, 3, 3, 3]
    assert [n(1, 2 ** 20 - 1, 1, 1, t) for t in range(7)] == [1, 1, 1, 3, 3, 6, 7]
    assert [n(1, 2 ** 20, 1, 1, t) for t in range(7)] == [1, 1, 1, 4, 5, 6, 7]
    assert [n(2, 2 ** 24, 0, 1, t) for t in range(7)] == [1, 1, 1, 3, 3, 6, 7]
    assert [n(4, 1000, 2, 1, t) for t in range(7)] == [0, 0, 0, 7, 7, 7, 7]
    assert n(10, 1000, 1, 0, 3) == n(1, 1000, 3, 0, 3) == n(1, 1000, 1, 2, 3) == n(1, 1000, 1, 0, 7) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("ns,law,precision,tiles,big", [
    (1, 1, 0, (0, 3, 6), False), (5, 2, 0, (3, 4), False), (1, 1, 1, (3, 4, 5, 6), False),
    (3, 1, 1, (2, 3, 4, 6), False), (2, 2, 1, (3, 6), False), (1, 1, 1, (3, 4), True),
])
def test_counts_match_a_captured_stage(f3d, cuda_ok, ns, law, precision, tiles, big):
    import torch
    rt = pytest.importorskip("cuda.bindings.runtime")
    S = f3d.solver_module()
    if big:  # 2^20 cells: one species leaves the sweeps for the staged ones in mixed precision
        case = f3d.curvilinear_jet(nx=128, ny=128, nz=64)
    else:
        case = f3d.random_curvilinear(n=8, ns=ns, seed=3)
        if law == 2:
            case.transport = f3d.cases.mixture_averaged_transport(case.thermo, seed=3)
    dc = S.DeviceCase(case, precision=precision)
    for tile in tiles:
        dc.set_tile(tile)
        dc.stage_fused(1)  # first-launch attributes outside the capture
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(g):
            dc.stage_fused(1)
        err, nodes, count = rt.cudaGraphGetNodes(g.raw_cuda_graph())
        err, nodes, count = rt.cudaGraphGetNodes(g.raw_cuda_graph(), count)
        kinds = [rt.cudaGraphNodeGetType(v)[1] for v in nodes[:count]]
        kernels = sum(k == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds)
        assert kernels == len(kinds) == dc.launches_per_stage(), tile
        assert dc.swept == (tile >= 3 and kernels == 3)
