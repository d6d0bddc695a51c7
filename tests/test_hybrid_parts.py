"""Hybrid batches whose cases are all on one side of the size limit: no persistent part, or no graph
part.  Captured steps end where the same cases end in a batch of that one mode."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("small_cells,mode", [(0, "graph"), (10 ** 6, "persistent")])
def test_one_part(f3d, cuda_ok, small_cells, mode):
    import torch
    S, B = f3d.solver_module(), f3d.batch_module()
    cases = [f3d.random_curvilinear(n=8 + 2 * k, ns=k + 1, seed=k) for k in range(3)]
    one, ref = ([S.DeviceCase(c, tile=3) for c in cases] for _ in range(2))
    a, b = B.Batch(one, mode="hybrid", small_cells=small_cells), B.Batch(ref, mode=mode)
    assert [p.mode for p in a.parts] == [mode]
    for batch in (a, b):
        batch.capture()
        for _ in range(3):
            batch.step()
        batch.status()
    for x, y in zip(one, ref):
        assert x.cur == y.cur
        for u, v in ((x.U, y.U), (x.Q[x.cur], y.Q[y.cur]), (x.rhoi[x.cur], y.rhoi[y.cur])):
            assert torch.equal(u, v)
        assert torch.isfinite(x.U[:, 4:-4, 4:-4, 4:-4]).all()
    a.close()
    b.close()
