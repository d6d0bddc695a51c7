"""Configurations that launch the same kernels are timed once, as the lowest of them, and choices of
other kernels are not read back (no GPU: a fake timer stands in for the device)."""
from __future__ import annotations

import importlib
import json
from types import SimpleNamespace

import pytest


def _dc(f3d, ns, cells, precision, law=1):
    S = f3d.solver_module()
    dc = S.DeviceCase.__new__(S.DeviceCase)
    dc.lib, dc.tile, dc.precision = f3d.load_library(), 3, precision
    dc.case, dc.transport = SimpleNamespace(ns=ns, cells=cells), SimpleNamespace(law=law)
    return dc


@pytest.mark.parametrize("ns,cells,precision,law,timed", [
    (1, 32 ** 3, 0, 1, [0, 1, 2, 3]), (9, 32 ** 3, 0, 2, [0, 1, 2, 3]),
    (1, 32 ** 3, 1, 1, [0, 1, 2, 3, 5, 6]), (4, 2 ** 22, 1, 1, [0, 1, 2, 3, 5, 6]),
    (1, 2 ** 20, 1, 1, [0, 1, 2, 3, 4, 5, 6]), (3, 32 ** 3, 1, 2, [0, 1, 2, 3]),
])
def test_each_set_of_kernels_is_timed_once(f3d, tmp_path, ns, cells, precision, law, timed):
    A = importlib.import_module(f3d.__name__ + ".autotune")
    seen = []
    t = A.Autotuner(tmp_path / "a.json", measure=lambda dc, tile: seen.append(tile) or 10.0 - tile)
    assert t.choose(_dc(f3d, ns, cells, precision, law), gpu="g") == max(timed)
    assert seen == timed


def test_stored_choices_of_other_kernels_are_timed_again(f3d, tmp_path):
    A = importlib.import_module(f3d.__name__ + ".autotune")
    path = tmp_path / "b.json"
    path.write_text(json.dumps({f"g|p0|ns1|c{A.size_class(32 ** 3)}": {"tile": 0}}))
    t = A.Autotuner(path, measure=lambda dc, tile: abs(tile - 3))
    assert t.choose(_dc(f3d, 1, 32 ** 3, 0), gpu="g") == 3
    assert A.key("g", 1, 1, 2 ** 20 - 1) != A.key("g", 1, 1, 2 ** 20)
    assert A.size_class(2 ** 20 - 1) == A.size_class(2 ** 20)
