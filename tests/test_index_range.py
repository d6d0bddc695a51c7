"""The fused kernels index every array in 32 bits, so a grid is refused before any launch when the
widest array of the call would reach 2^31 elements: ten metric fields, 5 + ns right-hand sides on
the pencil configurations and in batches, 2 + ns transport fields with law 2."""
from __future__ import annotations

import ctypes as C

import pytest

LIMIT = 2 ** 31


def _cube(fields, over):
    """The largest cube whose ghosted points times `fields` stay below the limit, or (over) the
    next one."""
    n = int((LIMIT / fields) ** (1 / 3)) + 2
    while n ** 3 * fields >= LIMIT:
        n -= 1
    return n - 8 + over


def _stage(f3d, lib, n, ns, precision, tile):
    """Status and message; an unknown precision (2) is refused after the size check, before any
    launch."""
    g = f3d.FlameGrid(n, n, n, 4, ns, 7)
    b = f3d.FlameStageBuffers(1, 2, 3, 4, 5, 6, 7, 8, 9, 10)
    m = f3d.FlameMetrics(*([1] * 10))
    rc = lib.flame_rk_stage_tiled(C.byref(g), None, 1, 1e-3, C.byref(b), C.byref(m),
                                  C.byref(f3d.FlameThermo()), C.byref(f3d.FlameTransport()),
                                  precision, tile)
    return rc, f3d.abi.last_error(lib)


@pytest.mark.parametrize("ns", [1, 5, 6, 9])
@pytest.mark.parametrize("tile", [0, 2, 3, 4, 5, 6])
def test_stage(f3d, ns, tile):
    lib = f3d.load_library()
    fields = max(10, 5 + ns) if tile >= 3 else 10
    rc, msg = _stage(f3d, lib, _cube(fields, 1), ns, 2, tile)
    assert rc == 1 and "2^31" in msg
    rc, msg = _stage(f3d, lib, _cube(fields, 0), ns, 2, tile)
    assert rc == 1 and "precision" in msg


@pytest.mark.parametrize("law,ns,fields", [(1, 9, 10), (2, 8, 10), (2, 9, 11)])
def test_transport(f3d, law, ns, fields):
    lib = f3d.load_library()
    tr = f3d.FlameTransport()
    tr.law, tr.poly = law, 16
    for over, word in ((1, "2^31"), (0, "precision")):
        n = _cube(fields, over)
        g = f3d.FlameGrid(n, n, n, 4, ns, 7)
        rc = lib.flame_transport(C.byref(g), None, 1, 2, 3, C.byref(f3d.FlameThermo()), C.byref(tr), 2)
        assert rc == 1 and word in f3d.abi.last_error(lib)


@pytest.mark.parametrize("ns", [1, 5, 6, 9])
def test_batch(f3d, ns):
    lib = f3d.load_library()
    for over in (0, 1):
        d = f3d.abi.FlameCaseDesc()
        n = _cube(max(10, 5 + ns), over)
        d.grid = f3d.FlameGrid(n, n, n, 4, ns, 7)
        d.buf = f3d.FlameStageBuffers(*([4096] * 10))
        d.metrics = f3d.FlameMetrics(*([4096] * 10))
        d.transport.law = 1
        assert (lib.flame_batch_workspace_bytes(C.byref(d), 1, 0) == 0) == bool(over)
