"""The chemistry step over blocks without, with one and with many cells above T_criteria: a cell is
advanced if and only if it is hot and fluid, the others keep their bits."""
from __future__ import annotations

import ctypes as C
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stiff", [0, 1])
@pytest.mark.parametrize("where", ["none", "one", "last", "row", "solid"])
def test_only_hot_cells_react(f3d, oracle, cuda_ok, stiff, where):
    import torch
    M = importlib.import_module(f3d.__name__ + ".mechanism")
    mech = M.synthetic_mechanism()
    case = f3d.random_curvilinear(n=11, ns=8, seed=7, T_range=(400.0, 900.0))  # 15 x 11 x 9 cells
    case.Q[5] = np.minimum(case.Q[5], 900.0)
    I = (slice(4, -4),) * 3
    T = case.Q[5][I]
    tag = np.zeros(case.Q.shape[1:], dtype=np.int64)
    if where == "one":
        T[4, 3, 7] = 1800.0
    elif where == "last":
        T[-1, -1, -1] = 1800.0
    elif where == "row":
        T[2, 5, :] = 1700.0
    elif where == "solid":
        T[2, 5, :] = 1700.0
        tag[4 + 2, 4 + 5, 4:10] = 1
    Q, r = M.reacting_state(mech, case)
    U = np.ascontiguousarray(case.U())
    th, g = mech.thermo.to_c(), case.grid()
    arrays, rc = mech.to_device()
    dev = [torch.from_numpy(a.copy()).cuda() for a in (U, Q, r)]
    dtag = torch.from_numpy(tag).cuda()
    lib = f3d.load_library()
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    a = (C.byref(g), s, *(d.data_ptr() for d in dev), 1e-8, C.byref(th), C.byref(rc), dtag.data_ptr(),
         1000.0)
    f3d.abi.check(lib, lib.flame_eval_gpu_stiff(*a, 0) if stiff else lib.flame_eval_gpu(*a))
    torch.cuda.synchronize()
    hot = np.zeros(tag.shape, dtype=bool)
    hot[I] = (Q[5][I] > 1000.0) & (tag[I] == 0)
    assert hot.sum() == {"none": 0, "one": 1, "last": 1, "row": case.nx, "solid": case.nx - 6}[where]
    before = [h.copy() for h in (U, Q, r)]
    oracle.load().oracle_eval_chem(C.byref(g), stiff, oracle.ptr(U), oracle.ptr(Q), oracle.ptr(r),
                                   1e-8, C.byref(th), C.byref(mech.to_c()), tag.ctypes.data_as(C.c_void_p), 1000.0,
                                   0)
    for d, h, b in zip(dev, (U, Q, r), before):
        got = d.cpu().numpy()
        np.testing.assert_allclose(got, h, rtol=1e-12, atol=1e-12 * np.abs(h).max())
        assert np.array_equal(got[:, ~hot], b[:, ~hot])


@pytest.mark.parametrize("stiff", [0, 1])
@pytest.mark.parametrize("kept", [4, 7, 8])
def test_arrays_may_end_with_the_last_reaction_that_uses_them(f3d, oracle, cuda_ok, stiff, kept):
    """The third-body efficiencies are read for three-body and falloff reactions only, the falloff
    parameters for falloff reactions only: the first `kept` reactions (four Arrhenius, three
    three-body, one falloff) with arrays that hold just those rows, among values that would show."""
    import torch
    M = importlib.import_module(f3d.__name__ + ".mechanism")
    full = M.synthetic_mechanism()
    cut = lambda a, n: np.ascontiguousarray(a[:n])  # noqa: E731
    mech = M.Mechanism(full.thermo, *(cut(getattr(full, k), kept) for k in M.Mechanism.FIELDS))
    case = f3d.random_curvilinear(n=8, ns=8, seed=9, T_range=(400.0, 2600.0))
    Q, r = M.reacting_state(mech, case)
    U = np.ascontiguousarray(case.U())
    th, g = mech.thermo.to_c(), case.grid()
    arrays, rc = mech.to_device()
    rows = {"ef": kept if kept > 4 else 0, "loP": kept if kept > 7 else 0, "Troe": kept if kept > 7 else 0}
    for k, n in rows.items():  # rows past the last used one hold NaN
        arrays[k][n:] = float("nan")
    dev = [torch.from_numpy(a.copy()).cuda() for a in (U, Q, r)]
    lib = f3d.load_library()
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    a = (C.byref(g), s, *(d.data_ptr() for d in dev), 1e-8, C.byref(th), C.byref(rc), None, 500.0)
    f3d.abi.check(lib, lib.flame_eval_gpu_stiff(*a, 0) if stiff else lib.flame_eval_gpu(*a))
    torch.cuda.synchronize()
    oracle.load().oracle_eval_chem(C.byref(g), stiff, oracle.ptr(U), oracle.ptr(Q), oracle.ptr(r),
                                   1e-8, C.byref(th), C.byref(mech.to_c()), None, 500.0, 0)
    for d, h in zip(dev, (U, Q, r)):
        np.testing.assert_allclose(d.cpu().numpy(), h, rtol=1e-12, atol=1e-12 * np.abs(h).max())
