"""Inputs whose divisions meet a zero or an infinity, against the oracle, which divides exactly.

The fused stages and the chemistry step divide by refined reciprocals.  A zero or infinite divisor
has to give what the division gives: a species with a1 = 1 starts GetT from ein / 0 = inf
(thermo.jl:231-282), Pr = inf switches conduction and diffusion off, and zero transport fits make
single terms of mixtureProperties (thermo.jl:289-369) vanish.  Bound: the fused FP64 stage's 1e-12
relative L2 per field, 1e-5 in mixed precision.
"""
from __future__ import annotations

import ctypes as C
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(f3d, ns, transport=None, a1=None, seed=71):
    """The random parity case (12 x 8 x 6 cells), with every species' a1 set to `a1` and a2 such
    that cp/R runs from 2.5 at 300 K to 8.5 at 1500 K."""
    cs = f3d.cases
    base = f3d.random_curvilinear(n=8, ns=ns, seed=seed)
    th = base.thermo
    if a1 is not None:
        lo = np.zeros((ns, 7))
        lo[:, 0], lo[:, 1] = a1, 5e-3
        th = cs.Thermo(th.mw, lo, lo.copy(), th.sep, 200.0, 3000.0, th.Ru)
    tr = transport(th) if transport else base.transport
    s = (slice(None), slice(4, -4), slice(4, -4), slice(4, -4))
    Q = base.Q[s]
    return cs._finish("degenerate", base.nx, base.ny, base.nz, th, tr, base.metrics, Q[0], Q[1],
                      Q[2], Q[3], Q[5], base.rhoi[s] / Q[0], 0.4, 1, {})


def _agree(f3d, oracle, case, precision, tile, bound):
    dc = f3d.solver_module().DeviceCase(case, precision=precision, tile=tile)
    oc = oracle.OracleCase(case)
    for s in (1, 2, 3):
        dc.stage_fused(s)
        oc.stage(s)
    I = oracle.interior
    U, (Q, r) = dc.conserved(), dc.primitives()
    assert np.isfinite(I(oc.U)).all() and np.isfinite(oc.Q).all()
    mom, vel = np.linalg.norm(I(oc.U[1:4])), np.linalg.norm(oc.Q[1:4])
    for n in range(5):
        scale = mom if 1 <= n <= 3 else np.linalg.norm(I(oc.U[n]))
        assert np.linalg.norm(I(U[n]) - I(oc.U[n])) <= bound * scale, n
    for n in range(7):
        scale = vel if 1 <= n <= 3 else np.linalg.norm(oc.Q[n])
        assert np.linalg.norm(Q[n] - oc.Q[n]) <= bound * scale, n
    assert np.linalg.norm(r - oc.rhoi) <= bound * np.linalg.norm(oc.rhoi)
    return dc


@pytest.mark.parametrize("ns,precision,tile", [(1, 0, 3), (3, 0, 3), (4, 0, 0), (5, 0, 3), (4, 1, 3),
                                               (1, 1, 3)])
def test_unit_a1(f3d, oracle, cuda_ok, ns, precision, tile):
    _agree(f3d, oracle, _case(f3d, ns, a1=1.0), precision, tile, 1e-5 if precision else 1e-12)


@pytest.mark.parametrize("ns,precision", [(1, 0), (5, 0), (4, 1)])
def test_infinite_prandtl_number(f3d, oracle, cuda_ok, ns, precision):
    tr = f3d.cases.Transport(law=1, mu_ref=1.8e-3, T_ref=300.0, exponent=0.7, Pr=np.inf)
    dc = _agree(f3d, oracle, _case(f3d, ns, lambda th: tr), precision, 3, 1e-5 if precision else 1e-12)
    T = dc.T[dc.cur].cpu().numpy()
    assert (T[0] > 0).all() and (T[1] == 0).all() and (T[2] == 0).all()


@pytest.mark.parametrize("ns", [1, 2, 9])  # every species everywhere: an absent one makes 0 / 0
@pytest.mark.parametrize("zero", ["conductivity", "diffusion", "last viscosity"])
def test_zero_transport_fits(f3d, oracle, cuda_ok, ns, zero):
    if ns == 1 and zero == "diffusion":
        pytest.skip("one species has no pair")

    def transport(th):
        tr = f3d.cases.mixture_averaged_transport(th, seed=5)
        at = {"conductivity": slice(5 * ns, 10 * ns), "diffusion": slice(10 * ns, None),
              "last viscosity": slice(5 * (ns - 1), 5 * ns)}[zero]
        tr.poly[at] = 0.0
        return tr

    dc = _agree(f3d, oracle, _case(f3d, ns, transport), 0, 3, 1e-12)
    T = dc.T[dc.cur].cpu().numpy()
    assert np.isfinite(T).all()
    if zero == "diffusion":
        assert (T[2:] == 0).all()


@pytest.mark.parametrize("stiff", [0, 1])
def test_chemistry_with_unit_a1(f3d, oracle, cuda_ok, stiff):
    import torch
    M = importlib.import_module(f3d.__name__ + ".mechanism")
    mech = M.synthetic_mechanism()
    mech.thermo.lo[:, 0], mech.thermo.lo[:, 1] = 1.0, 2e-3
    mech.thermo.hi[:] = mech.thermo.lo
    case = f3d.random_curvilinear(n=8, ns=8, seed=7, T_range=(400.0, 2600.0))
    Q, r = M.reacting_state(mech, case)
    U = np.ascontiguousarray(case.U())
    th, g = mech.thermo.to_c(), case.grid()
    arrays, rc = mech.to_device()
    dev = [torch.from_numpy(a.copy()).cuda() for a in (U, Q, r)]
    lib = f3d.load_library()
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    a = (C.byref(g), s, *(d.data_ptr() for d in dev), 1e-9, C.byref(th), C.byref(rc), None, 500.0)
    f3d.abi.check(lib, lib.flame_eval_gpu_stiff(*a, 0) if stiff else lib.flame_eval_gpu(*a))
    torch.cuda.synchronize()
    oracle.load().oracle_eval_chem(C.byref(g), stiff, oracle.ptr(U), oracle.ptr(Q), oracle.ptr(r),
                                   1e-9, C.byref(th), C.byref(mech.to_c()), None, 500.0, 0)
    assert np.isfinite(Q).all()
    for d, h in zip(dev, (U, Q, r)):
        np.testing.assert_allclose(d.cpu().numpy(), h, rtol=1e-12, atol=1e-12 * np.abs(h).max())
