"""The FP64 sweeps (k_sweeps) at the sizes where their cuts change, against the oracle.

y and z lines hold at most 26 own cells and eight x columns, x blocks a number of rows that
depends on nx; one to three species (two with per-species D) take two staging passes, more take
three.  The extents sit on either side of those edges, down to the smallest grid.  Bound: the
fused FP64 stage's 1e-12 relative L2 per field.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(f3d, nx, ny, nz, ns, law, seed):
    """The wavy parity case with its own extents: smooth fields, noise in a third of the box and
    a pressure jump, so that all hybrid branches occur."""
    big = f3d.random_curvilinear(n=max(nx, ny, nz, 8) + 2, ns=ns, seed=seed)
    cs = f3d.cases
    metrics, _ = cs.wavy_metrics(nx, ny, nz, 0.1)
    s = (slice(None), slice(4, 4 + nz), slice(4, 4 + ny), slice(4, 4 + nx))
    tr = cs.mixture_averaged_transport(big.thermo, seed=3) if law == 2 else big.transport
    Q = big.Q[s]
    Y = big.rhoi[s] / Q[0]
    return cs._finish(f"sweep{nx}x{ny}x{nz}", nx, ny, nz, big.thermo, tr, metrics, Q[0], Q[1], Q[2],
                      Q[3], Q[5], Y, 0.4, 1, {})


@pytest.mark.parametrize("nx,ny,nz,ns,law", [
    (4, 4, 4, 1, 1), (8, 26, 27, 1, 1), (9, 27, 26, 3, 1), (7, 53, 5, 4, 1), (33, 4, 52, 9, 1),
    (250, 5, 4, 1, 1), (251, 4, 5, 2, 1), (122, 7, 6, 4, 1), (16, 12, 28, 2, 2), (17, 28, 6, 3, 2),
    (40, 9, 11, 9, 2),
])
def test_sweeps_match_oracle(f3d, oracle, cuda_ok, nx, ny, nz, ns, law):
    case = _case(f3d, nx, ny, nz, ns, law, seed=61)
    dc = f3d.solver_module().DeviceCase(case, tile=3)
    oc = oracle.OracleCase(case)
    I = oracle.interior
    for s in (1, 2, 3):
        dc.stage_fused(s)
        oc.stage(s)
        U = dc.conserved()
        Q, r = dc.primitives()
        mom = np.linalg.norm(I(oc.U[1:4]).ravel())
        vel = np.linalg.norm(oc.Q[1:4].ravel())
        for n in range(5):
            scale = mom if 1 <= n <= 3 else np.linalg.norm(I(oc.U[n]).ravel())
            assert np.linalg.norm((I(U[n]) - I(oc.U[n])).ravel()) <= 1e-12 * scale, (s, n)
        for n in range(7):
            scale = vel if 1 <= n <= 3 else np.linalg.norm(oc.Q[n].ravel())
            assert np.linalg.norm((Q[n] - oc.Q[n]).ravel()) <= 1e-12 * scale, (s, n)
        assert np.linalg.norm((r - oc.rhoi).ravel()) <= 1e-12 * np.linalg.norm(oc.rhoi.ravel()), s


@pytest.mark.parametrize("nx,ny,nz,ns", [
    (4, 4, 4, 1), (17, 27, 26, 2), (33, 9, 53, 3), (16, 12, 28, 4), (40, 30, 7, 7), (9, 26, 27, 8),
    (251, 4, 5, 9),
])
def test_mixed_sweeps_match_the_staged_sweeps(f3d, cuda_ok, nx, ny, nz, ns):
    """Mixed precision: the sweeps in one launch against the staged ones (which the persistent
    batch runs) on the same case.  Both evaluate the same FP32 expressions, so a step agrees to
    the last bit."""
    import torch
    case = _case(f3d, nx, ny, nz, ns, 1, seed=62)
    S, B = f3d.solver_module(), f3d.batch_module()
    one, ref = (S.DeviceCase(case, precision=1, tile=3) for _ in range(2))
    batch = B.Batch([ref], mode="persistent")
    assert one.swept
    for _ in range(2):
        one.step()
        batch.step()
    batch.status()
    batch.close()
    for a, b in ((one.U, ref.U), (one.Q[one.cur], ref.Q[ref.cur]), (one.rhoi[one.cur], ref.rhoi[ref.cur]),
                 (one.T[one.cur], ref.T[ref.cur])):
        assert torch.equal(a, b)
