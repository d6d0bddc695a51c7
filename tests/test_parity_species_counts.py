"""The kernels that are compiled per species count (1 to 9, and one for a run-time count) at the
last compiled count and the first run-time one, against the oracle.

1:1 kernels: the checks of test_parity_kernels (bit for bit, pow() aside) with 9 and 10 species.
Chemistry: the synthetic mechanism with inert species appended, 1e-12 as in test_parity_chemistry.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import test_parity_kernels as K

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _release():
    yield
    K._KEEP.clear()


@pytest.fixture(scope="module", params=[(9, 34), (10, 35)], ids=["ns9", "ns10"])
def env(request, f3d, oracle, cuda_ok):
    return K.Env(f3d, oracle, *request.param)


test_mixture = K.test_mixture
test_viscous_and_species_diffusion = K.test_viscous_and_species_diffusion
test_div_divspecs_lincomb_c2prim = K.test_div_divspecs_lincomb_c2prim


@pytest.mark.parametrize("ns", [9, 10])
@pytest.mark.parametrize("stiff,transposed,dt", [(0, 0, 1e-9), (1, 0, 1e-7), (1, 1, 1e-7)])
def test_chemistry_with_inert_species(f3d, oracle, cuda_ok, ns, stiff, transposed, dt):
    import importlib

    import torch
    M = importlib.import_module(f3d.__name__ + ".mechanism")
    m = M.synthetic_mechanism()
    more = ns - m.thermo.ns
    wide = lambda a, v: np.ascontiguousarray(  # noqa: E731
        np.concatenate([a, np.full((a.shape[0], more), v, dtype=a.dtype)], axis=1))
    rows = lambda a: np.concatenate([a, np.repeat(a[-1:], more, axis=0)])  # noqa: E731
    t = m.thermo
    thermo = f3d.Thermo(rows(t.mw), rows(t.lo), rows(t.hi), rows(t.sep), t.min_temp, t.max_temp, t.Ru)
    mech = M.Mechanism(thermo, m.reaction_type, m.sgm, wide(m.vf, 0), wide(m.vr, 0), m.Arr,
                       wide(m.ef, 1.0), m.loP, m.Troe)
    case = f3d.random_curvilinear(n=10, ns=ns, seed=7, T_range=(400.0, 2600.0))
    Q, r = M.reacting_state(mech, case)
    U = np.ascontiguousarray(case.U())
    th, g = thermo.to_c(), case.grid()
    arrays, rc = mech.to_device()
    dU, dQ, dr = (torch.from_numpy(a.copy()).cuda() for a in (U, Q, r))
    lib = f3d.load_library()
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    a = (C.byref(g), s, dU.data_ptr(), dQ.data_ptr(), dr.data_ptr(), dt, C.byref(th), C.byref(rc), None,
         500.0)
    f3d.abi.check(lib, lib.flame_eval_gpu_stiff(*a, transposed) if stiff else lib.flame_eval_gpu(*a))
    torch.cuda.synchronize()
    before = r.copy()
    oracle.load().oracle_eval_chem(C.byref(g), stiff, oracle.ptr(U), oracle.ptr(Q), oracle.ptr(r),
                                   dt, C.byref(th), C.byref(mech.to_c()), None, 500.0, transposed)
    assert not np.array_equal(r, before)  # something reacted
    for d, h in ((dU, U), (dQ, Q), (dr, r)):
        np.testing.assert_allclose(d.cpu().numpy(), h, rtol=1e-12, atol=1e-12 * np.abs(h).max())
