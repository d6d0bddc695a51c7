"""The refined reciprocal, quotient and reciprocal square root of the FP64 paths (common.cuh) against
CUDA's own operators.

Bounds, in units of the last place of CUDA's result, from the forms themselves.  Reciprocal: the cut
series leaves 2^-57 and the last multiply-add half a unit, so the two roundings differ by at most
one; the quotient's residual step likewise.  Reciprocal square root: the rounding of d x adds half a
unit, and CUDA's 1 / sqrt rounds twice, so two.  The rule's product forms round twice: two."""
from __future__ import annotations

import ctypes as C
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OPS = {"fast_rcp": 0, "full_rcp": 1, "fast_div": 2, "fast_rsqrt": 3, "rule_sqrt": 4, "rule_div": 5,
       "full_div": 6}
ULP = {"fast_rcp": 1, "full_rcp": 1, "fast_div": 1, "fast_rsqrt": 2, "rule_sqrt": 2, "rule_div": 2,
       "full_div": 1}


def _run(f3d, name, a, b):
    import torch
    path = importlib.import_module(f3d.__name__ + ".build").build_probe()
    fn = C.CDLL(str(path)).flame_probe_refined_division
    fn.argtypes = [C.c_int, C.c_longlong] + [C.c_void_p] * 5
    d = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (a, b, np.zeros_like(a), np.zeros_like(a))]
    assert fn(OPS[name], a.size, *(v.data_ptr() for v in d), None) == 0
    torch.cuda.synchronize()
    return d[2].cpu().numpy(), d[3].cpu().numpy()


def _values(rng, n, lo, hi):
    """Magnitudes spread over powers of ten, random and all-ones / all-zeros mantissas."""
    v = 10.0 ** rng.uniform(lo, hi, n)
    m, e = np.frexp(v)
    edge = np.array([0.5, np.nextafter(0.5, 1), np.nextafter(1, 0), 0.75, np.sqrt(0.5)])
    m[::7] = edge[np.arange(m[::7].size) % edge.size]
    return np.ldexp(m, e)


@pytest.mark.parametrize("name", OPS)
def test_within_units_of_the_last_place(f3d, cuda_ok, name):
    rng = np.random.default_rng(17)
    n = 1 << 20
    positive = name in ("fast_rsqrt", "rule_sqrt")
    wide = 100 if name.endswith("_div") else 300
    for lo, hi in ((-3, 3), (-wide, wide)):
        a, b = _values(rng, n, lo, hi), _values(rng, n, lo, hi)
        if not positive:
            a *= rng.choice([-1.0, 1.0], n)
            b *= rng.choice([-1.0, 1.0], n)
        got, want = _run(f3d, name, a, b)
        off = np.abs(got - want) / np.spacing(np.abs(want))
        assert np.isfinite(want).all() and off.max() <= ULP[name], (lo, off.max())


@pytest.mark.parametrize("name", ["full_rcp", "full_div"])
def test_zero_infinity_and_nan(f3d, cuda_ok, name):
    v = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1.0, -2.5, 1e-300, 1e300])
    a, b = (x.ravel().copy() for x in np.meshgrid(v, v))
    got, want = _run(f3d, name, a, b)
    keep = (np.abs(want) >= 2.3e-308) | (want == 0) | np.isnan(want)  # a subnormal may come out as zero
    assert np.array_equal(np.isnan(got[keep]), np.isnan(want[keep]))
    ok = keep & ~np.isnan(want)
    assert np.array_equal(np.isinf(got[ok]), np.isinf(want[ok]))
    assert np.array_equal(np.signbit(got[ok]), np.signbit(want[ok]))
    fin = ok & np.isfinite(want)
    assert (np.abs(got[fin] - want[fin]) <= ULP[name] * np.spacing(np.abs(want[fin]))).all()
