"""Mixture-averaged transport where species are absent.  D_k = (1 - X_k) / (Σ_{m≠k} X_m P / D_km + eps)
(thermo.jl:360-369) is a quotient of rounding errors where X_k is 1 to an ulp: the result is 0 or near
one half by how Y2X (thermo.jl:38-52) rounds, and a jump of species next to such a cell diffuses with it.
flame_transport therefore has to round Y2X as the oracle does."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [2, 5, 9])
def test_transport_of_pure_cells(f3d, oracle, cuda_ok, ns):
    import torch
    case = f3d.random_curvilinear(n=24, ns=ns, seed=33)
    rng = np.random.default_rng(ns)
    only = rng.integers(0, ns, case.Q.shape[1:])
    pure = rng.random(only.shape) < 0.7
    for n in range(ns):  # 70 % of the points hold one species alone
        case.rhoi[n] = np.where(pure, np.where(only == n, case.Q[0], 0.0), case.rhoi[n])
    tr = f3d.cases.mixture_averaged_transport(case.thermo, seed=4)
    g, th, lib = case.grid(), case.thermo.to_c(), f3d.load_library()
    dQ, dr, dp = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (case.Q, case.rhoi, tr.poly))
    T = torch.zeros((2 + ns,) + case.Q.shape[1:], dtype=torch.float64, device="cuda")
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    f3d.abi.check(lib, lib.flame_transport(C.byref(g), s, dQ.data_ptr(), dr.data_ptr(), T.data_ptr(),
                                           C.byref(th), C.byref(tr.to_c(dp.data_ptr())), 0))
    ref = {k: np.zeros((n,) + case.Q.shape[1:]) for k, n in (("Yi", ns), ("lam", 1), ("mu", 1), ("D", ns))}
    P = oracle.ptr
    oracle.load().oracle_mixture(C.byref(g), P(case.Q), P(case.rhoi), P(ref["Yi"]), P(ref["lam"]),
                                 P(ref["mu"]), P(ref["D"]), C.byref(th), C.byref(tr.to_c()), None)
    got = T.cpu().numpy()
    alone = np.take_along_axis(ref["D"], only[None], 0)[0][pure]  # D of the species that is alone
    assert (alone == 0).any() and (alone > 0.1).any()
    for a, b in ((got[0], ref["mu"][0]), (got[1], ref["lam"][0]), (got[2:], ref["D"])):
        np.testing.assert_allclose(a, b, rtol=1e-12, atol=0)
