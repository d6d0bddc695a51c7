"""Mixed precision on the paths that the sweeps in one launch do not take: configurations 5 and 6 (flow
and species in sweeps of their own), and one species on either side of 2^20 cells, where 3 and 4 leave
the sweeps in one launch for the staged ones.  Configurations 4 and 6 run the finish in a launch of its
own and have to agree with 3 and 5 bit for bit; against the oracle the bound is mixed precision's 1e-5
relative L2 in ρ, ρu and ρE."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(dc):
    return dc.U[:, 4:-4, 4:-4, 4:-4], dc.Q[dc.cur], dc.rhoi[dc.cur], dc.T[dc.cur]


def _same(a, b):
    import torch
    return all(torch.equal(x, y) for x, y in zip(_state(a), _state(b)))


def _errors(dc, oc, oracle):
    I = oracle.interior
    U = dc.conserved()
    mom = np.linalg.norm(I(oc.U[1:4]).ravel())
    return [float(np.linalg.norm((I(U[n]) - I(oc.U[n])).ravel())
                  / (mom if 1 <= n <= 3 else np.linalg.norm(I(oc.U[n]).ravel()))) for n in range(5)]


@pytest.mark.parametrize("ns", [1, 3, 9])
def test_flow_and_species_apart(f3d, oracle, cuda_ok, ns):
    S = f3d.solver_module()
    case = f3d.random_curvilinear(n=12, ns=ns, seed=63)
    a, b = (S.DeviceCase(case, precision=1, tile=t) for t in (5, 6))
    assert (a.launches_per_stage(), b.launches_per_stage()) == (6, 7)
    oc = oracle.OracleCase(case)
    for _ in range(2):
        a.step()
        b.step()
        oc.step()
    assert _same(a, b)
    assert max(_errors(a, oc, oracle)) <= 1e-5


@pytest.mark.parametrize("nz,launches", [(63, (3, 3)), (64, (4, 5))])
def test_one_species_around_the_staged_sweeps_limit(f3d, oracle, cuda_ok, nz, launches):
    """128 x 128 x 63 cells and 128 x 128 x 64 = 2^20: one stage against the oracle, three against the
    other configuration and the persistent batch (always the staged sweeps, the same FP32 bits)."""
    S, B = f3d.solver_module(), f3d.batch_module()
    case = f3d.curvilinear_jet(nx=128, ny=128, nz=nz, pressure_noise=0.02)
    a, b, ref = (S.DeviceCase(case, precision=1, tile=t) for t in (3, 4, 3))
    assert (a.launches_per_stage(), b.launches_per_stage()) == launches
    batch = B.Batch([ref], mode="persistent")
    oc = oracle.OracleCase(case)
    for s in (1, 2, 3):
        for dc in (a, b):
            dc.stage_fused(s)
        batch.stage(s)
        if s == 1:
            oc.stage(s)
            assert max(_errors(a, oc, oracle)) <= 1e-5
    batch.status()
    assert _same(a, b) and _same(a, ref)
    batch.close()
