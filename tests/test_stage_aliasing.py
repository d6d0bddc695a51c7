"""The third stage may leave its result's partial densities in the rhon buffer, which nothing
reads after it: each cell reads its rhon before it writes, so the call gives the same values as
with a buffer of its own."""
from __future__ import annotations

import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tile,ns,law", [
    (0, 0, 2, 1), (0, 3, 1, 1), (0, 3, 5, 1), (0, 4, 9, 1), (0, 3, 1, 2), (0, 3, 5, 2), (1, 3, 1, 1),
    (1, 3, 3, 1), (1, 4, 9, 1), (1, 6, 4, 1), (1, 3, 5, 2),
])
def test_last_stage_into_rhon(f3d, cuda_ok, precision, tile, ns, law):
    import torch
    S = f3d.solver_module()
    case = f3d.random_curvilinear(n=10, ns=ns, seed=81)
    if law == 2:
        case.transport = f3d.cases.mixture_averaged_transport(case.thermo, seed=81)
    own, alias = (S.DeviceCase(case, precision=precision, tile=tile) for _ in range(2))
    for s in (1, 2):
        own.stage_fused(s)
        alias.stage_fused(s)
    own.stage_fused(3)
    alias.rhoi[1 - alias.cur] = alias.rhon
    alias.stage_fused(3)
    tol = 1e-13 if precision == 0 else 2e-6  # another path of the same precision
    for a, b in ((own.U, alias.U), (own.Q[own.cur], alias.Q[alias.cur]),
                 (own.rhoi[own.cur], alias.rhoi[alias.cur]), (own.T[own.cur], alias.T[alias.cur])):
        for n in range(a.shape[0]):
            x, y = a[n].double(), b[n].double()
            if a.shape[0] == 5 and a is own.U:  # interior: U's ghosts are not the stage's
                x, y = (v[4:-4, 4:-4, 4:-4] for v in (x, y))
            scale = a[n].double().abs().max() if not 1 <= n <= 3 else a[1:4].double().abs().max()
            assert torch.isfinite(y).all() and (x - y).abs().max() <= 40 * tol * scale, n
