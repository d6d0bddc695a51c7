"""What a program that uses this framework has it do, as cases that can be timed and compared.

A case is one call (or the calls of one step) through the public entry points, with the sizes of
this repository's configurations, tests and benchmark:

  flow       one RK3 step of one resident case (`DeviceCase.step`, the fused stages): Taylor-Green
             vortices from 32^3, the curvilinear jet, mixing layers of up to nine species, in
             plain FP64 and in mixed precision, with constant, power-law or mixture-averaged
             transport
  inflow     the same on the reference's own boundaries: three stages, each with its ghost fills
  sequence   the same step through the 1:1 entry points (the drop-in launch sequence, FP64)
  host       the call with host buffers (`DeviceCase.advance_from_host`): upload, one step, download
  batch      one RK3 step of an ensemble (`Batch.step`) from its captured CUDA graph
  chemistry  the finite-rate chemistry step between two flow steps (explicit or point-implicit)

A pass advances its case by one step, so that repeated passes walk through a simulation as a
user's program does.  `exact` is the same step written in plain 64-bit torch operations.
"""
import ctypes as C
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
NG = 4


def _package():
    if "flame3d_b200" not in sys.modules:
        pkg = ROOT / "flame3d.jl_b200"
        spec = importlib.util.spec_from_file_location("flame3d_b200", pkg / "__init__.py",
                                                      submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["flame3d_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["flame3d_b200"]


def _mechanism_module():
    return importlib.import_module(_package().__name__ + ".mechanism")


# ------------------------------------------------------------------------------------ the cases
def _flow(name, field, nx, ny, nz, ns=1, precision="f64", law=1, kind="flow"):
    c = {"kind": kind, "field": field, "nx": nx, "ny": ny, "nz": nz, "ns": ns,
         "precision": precision, "law": law}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the smallest request of the serving stream and of the ensemble: launches and latency
        _flow("tgv32_f64", "tgv", 32, 32, 32, law=0),
        # the curvilinear shock case of the benchmark (its default workload), plain FP64
        _flow("jet256_f64", "jet", 256, 128, 128),
        # the same in mixed precision
        _flow("jet256_mixed", "jet", 256, 128, 128, precision="mixed"),
        # the nine-species mixing layer at full size, mixed precision: the largest single case
        _flow("mix192_ns9_mixed", "mixing", 192, 192, 192, ns=9, precision="mixed"),
        # an ordinary multi-species case of no round size on a curvilinear grid, plain FP64
        _flow("ragged_ns5_f64", "wavy", 101, 75, 63, ns=5),
        # the reference's own mixture-averaged transport (one D per species), plain FP64
        _flow("mix96_ns9_law2_f64", "mixing", 96, 96, 96, ns=9, law=2),
        # the reference's own boundary conditions (supersonic inflow, zero-gradient copies)
        _flow("inflow_ns5_f64", "inflow", 96, 50, 42, ns=5, kind="inflow"),
        # a program that replaces the reference's kernels one by one
        _flow("sequence_jet128", "jet", 128, 64, 64, kind="sequence"),
        # a call with host buffers, every step uploaded and downloaded
        _flow("host_jet128_f64", "jet", 128, 64, 64, kind="host"),
        # a mixed ensemble (sizes and species counts of the 64-case one) as one CUDA graph a step
        {"name": "ensemble_graph_mixed", "kind": "batch", "mode": "graph", "precision": "mixed",
         "members": "32x1,32x4,48x2,48x7,48x9,64x1,64x3,64x6,96x2,96x5,96x8,128x1,128x4"},
        # the small members of such an ensemble in the persistent kernels
        {"name": "ensemble_small_mixed", "kind": "batch", "mode": "persistent",
         "precision": "mixed", "members": "32x1,32x1,32x2,32x5,32x5,32x9,48x1,48x2,48x5,48x9"},
        # the point-implicit chemistry step of a reacting flow
        {"name": "chemistry_stiff", "kind": "chemistry", "stiff": True, "nx": 64, "ny": 64,
         "nz": 64},
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["flow", "flow", "flow", "flow", "inflow", "sequence", "host", "batch",
                       "batch", "chemistry"])
    precision = rng.choice(["f64", "mixed"])
    if kind == "flow":
        field = rng.choice(["tgv", "jet", "mixing", "wavy"])
        ns = 1 if field == "jet" else rng.randint(1, 9)
        law = 0 if field == "tgv" else rng.choice([1, 1, 2]) if ns > 1 else 1
        hi = 200 if ns == 1 else 130
        if field == "tgv":
            n = _side(rng, 32, hi)
            return _flow("", field, n, n, n, ns, precision, law)
        return _flow("", field, *(_side(rng, 24, hi) for _ in range(3)), ns, precision, law)
    if kind == "inflow":
        return _flow("", "inflow", _side(rng, 24, 130), _side(rng, 16, 90), _side(rng, 16, 90),
                     rng.randint(5, 9), kind="inflow")
    if kind == "sequence":
        ns = rng.randint(1, 6)
        return _flow("", "jet" if ns == 1 else "wavy", *(_side(rng, 24, 100) for _ in range(3)),
                     ns, kind="sequence")
    if kind == "host":
        return _flow("", "jet", *(_side(rng, 24, 110) for _ in range(3)), 1, precision,
                     kind="host")
    if kind == "batch":
        mode = rng.choice(["graph", "persistent", "hybrid"])
        members = ",".join("%dx%d" % (_side(rng, 32, 96), rng.randint(1, 9))
                           for _ in range(rng.randint(4, 12)))
        return {"kind": "batch", "mode": mode, "precision": precision, "members": members}
    return {"kind": "chemistry", "stiff": rng.random() < 0.5, "nx": _side(rng, 24, 100),
            "ny": _side(rng, 24, 100), "nz": _side(rng, 24, 100)}


def _members(case):
    return [tuple(int(x) for x in m.split("x")) for m in case["members"].split(",")]


# ---------------------------------------------------------------------- inputs, made on the GPU
def _inside(nx, ny, nz):
    return (slice(NG, NG + nz), slice(NG, NG + ny), slice(NG, NG + nx))


def _pad(a, nx, ny, nz, periodic):
    """Interior field(s) (nv, nz, ny, nx) with their ghosts: periodic images or edge copies."""
    out = a.new_zeros((a.shape[0], nz + 2 * NG, ny + 2 * NG, nx + 2 * NG))
    out[(slice(None),) + _inside(nx, ny, nz)] = a
    for dim, n in ((3, nx), (2, ny), (1, nz)):
        if periodic:
            out.narrow(dim, 0, NG).copy_(out.narrow(dim, n, NG).clone())
            out.narrow(dim, n + NG, NG).copy_(out.narrow(dim, NG, NG).clone())
        else:
            out.narrow(dim, 0, NG).copy_(out.narrow(dim, NG, 1).clone().expand_as(out.narrow(dim, 0, NG)))
            out.narrow(dim, n + NG, NG).copy_(
                out.narrow(dim, n + NG - 1, 1).clone().expand_as(out.narrow(dim, n + NG, NG)))
    return out


def _make(field, nx, ny, nz, ns, law, seed):
    """A `Case` with its state and metrics on the GPU, from the seed alone."""
    f3d = _package()
    cs = f3d.cases
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    f8 = dict(dtype=torch.float64, device="cuda")

    def noise():
        return 2 * torch.rand((nz, ny, nx), generator=gen, **f8) - 1

    thermo = f3d.ideal_air() if ns == 1 else f3d.synthetic_species(9, 3).subset(ns)
    K, J, I = torch.meshgrid(*(torch.arange(n, **f8) for n in (nz, ny, nx)), indexing="ij")
    tp = 2 * math.pi
    one = torch.ones_like(I)
    cfl, inflow = 0.5, None
    mw = torch.tensor(thermo.mw, **f8)

    def gamma_r(T, Y):
        cp = float(thermo.cp_mass(np.array([T]), np.asarray(Y)[:, None])[0])
        R = thermo.Ru / (1.0 / float(np.sum(np.asarray(Y) / thermo.mw)))
        return cp / (cp - R), R, cp

    if field == "tgv":  # a Taylor-Green vortex with random-phase modes, Re and Ma of the ensemble
        h = tp / nx
        metrics = cs.cartesian_metrics(nx, ny, nz, h, h, h, device="cuda")
        Re, Ma = rng.uniform(400, 3200), rng.uniform(0.1, 0.5)
        Ya = np.ones(1) if ns == 1 else rng.dirichlet(np.ones(ns))
        T0, p0 = 300.0, 101325.0
        gam, R, cp = gamma_r(T0, Ya)
        U0 = Ma * math.sqrt(gam * R * T0)
        X, Yc, Z = I * h, J * h, K * h
        vel = [U0 * torch.sin(X) * torch.cos(Yc) * torch.cos(Z),
               -U0 * torch.cos(X) * torch.sin(Yc) * torch.cos(Z), torch.zeros_like(X)]
        for c in vel:
            for _ in range(6):
                k, ph = rng.integers(-6, 7, 3), rng.uniform(0, tp)
                c += 0.02 * U0 / 6 * torch.sin(float(k[0]) * X + float(k[1]) * Yc + float(k[2]) * Z + ph)
        rho0 = p0 / (R * T0)
        p = p0 + rho0 * U0 ** 2 / 16 * (torch.cos(2 * X) + torch.cos(2 * Yc)) * (torch.cos(2 * Z) + 2)
        T = T0 * one
        Y = torch.tensor(Ya, **f8).reshape(-1, 1, 1, 1) * one
        mu = rho0 * U0 / Re
        tr = f3d.Transport(law=0, mu_ref=mu, Pr=0.71, lambda_ref=cp * mu / 0.71,
                           D_ref=cp * mu / 0.71 / (rho0 * cp))
    else:
        tr = f3d.Transport(law=1, mu_ref=1.8e-5, T_ref=300.0, exponent=0.7, Pr=0.71)
        if field == "mixing":  # a periodic double mixing layer between two compositions
            L = 0.01
            h = L / ny
            metrics = cs.cartesian_metrics(nx, ny, nz, h, h, h, device="cuda")
            X, Yc = (I + 0.5) / nx, (J + 0.5) / ny
            g = 0.5 * (torch.tanh((Yc - 0.25) * 20) - torch.tanh((Yc - 0.75) * 20))
            Ya, Yb = rng.dirichlet(np.ones(ns)), rng.dirichlet(np.ones(ns))
            T = 300.0 + 1200.0 * g
            p = 101325.0 * one
            gam, R, _ = gamma_r(300.0, Ya)
            c0 = math.sqrt(gam * R * 300.0)
            vel = [0.3 * c0 * (g - 0.5) + 1e-3 * c0 * noise(),
                   1e-3 * c0 * torch.sin(tp * X) * torch.exp(-((Yc - 0.25) * 10) ** 2)
                   + 1e-3 * c0 * noise(), 1e-3 * c0 * noise()]
        elif field in ("jet", "inflow"):  # a Ma 1.5 round jet on the wavy curvilinear mapping
            xyz = cs.wavy_mapping(nx, ny, nz, 0.1)
            metrics = cs.metrics_from_mapping(xyz, nx, ny, nz, device="cuda")
            _, Yc, Z = xyz(I, J, K)
            r = torch.sqrt((Yc - 0.5) ** 2 + (Z - 0.5) ** 2)
            if field == "jet":
                g = 0.5 * (1 + torch.tanh((0.125 - r) / 0.025))
                T = 300.0 + 4700.0 * g
                Uj = 1.5 * math.sqrt(1.4 * thermo.Ru / thermo.mw[0] * 5000.0)
                vel = [Uj * g + 0.01 * Uj * noise(), 0.01 * Uj * noise(), 0.01 * Uj * noise()]
                p = 3596.0 * one
                Ya = Yb = np.ones(1)
            else:
                inflow = cs.reference_inflow(ns)
                g = 0.5 * (1 + torch.tanh((0.125 - r) / 0.02))
                Ya = np.array([inflow.Y[n] for n in range(ns)])
                Yb = 0.7 * Ya
                Yb[0] += 0.3
                T = inflow.T + (900.0 - inflow.T) * g
                p = inflow.P * (1 + 0.02 * noise())
                vel = [inflow.u + 1000.0 * g + 20.0 * noise(), 20.0 * noise(), 20.0 * noise()]
        else:  # "wavy": smooth fields of every species on the curvilinear mapping, light noise
            xyz = cs.wavy_mapping(nx, ny, nz, 0.1)
            metrics = cs.metrics_from_mapping(xyz, nx, ny, nz, device="cuda")
            X, Yc, Z = xyz(I, J, K)
            g = 0.5 + 0.45 * torch.sin(tp * X) * torch.cos(tp * Yc)
            Ya, Yb = rng.dirichlet(np.ones(ns)), rng.dirichlet(np.ones(ns))
            T = 300.0 + 1000.0 * g
            p = 1e5 * (1 + 0.2 * torch.sin(tp * Z) + 0.002 * noise())
            gam, R, _ = gamma_r(300.0, Ya)
            c0 = math.sqrt(gam * R * 300.0)
            vel = [c0 * (a * torch.sin(tp * b) + 0.01 * noise())
                   for a, b in ((0.3, Yc), (0.2, Z), (0.1, X))]
        Y = torch.stack([float(Ya[n]) + (float(Yb[n]) - float(Ya[n])) * g for n in range(ns)])
    if law == 2:
        tr = cs.mixture_averaged_transport(thermo, seed=3)
    yow = (Y / mw.reshape(-1, 1, 1, 1)).sum(0)
    rho = p / (thermo.Ru * T * yow)
    rhoi = rho * Y
    E = _Thermo(thermo)
    Q = torch.stack([rho, *vel, thermo.Ru * T * (rhoi / E.mw).sum(0), T, E.energy(T, rhoi)])
    periodic = 0 if inflow is not None else 7
    Q = _pad(Q, nx, ny, nz, periodic)
    rhoi = _pad(rhoi, nx, ny, nz, periodic)
    case = f3d.Case(field, nx, ny, nz, thermo, tr, metrics, Q, rhoi, 0.0, 1, periodic, {}, inflow)
    # dt from the CFL rule over the interior
    s = _inside(nx, ny, nz)
    q = [Q[k][s] for k in range(7)]
    cs_ = torch.sqrt((q[4] / q[6] + 1) * q[4] / q[0])
    rate = torch.zeros_like(cs_)
    for d in ("dxi", "deta", "dzeta"):
        m = [metrics[d + "d" + x][s] for x in "xyz"]
        rate += metrics["J"][s] * ((m[0] * q[1] + m[1] * q[2] + m[2] * q[3]).abs()
                                   + cs_ * torch.sqrt(m[0] ** 2 + m[1] ** 2 + m[2] ** 2))
    case.dt = float(cfl / rate.max())
    return case


def _make_member(n, ns, seed):
    return _make("tgv", n, n, n, ns, 0, seed)


def _chemistry_inputs(case, seed):
    """A reacting state of the synthetic eight-species mechanism: T from 400 to 2600 K."""
    mech = _mechanism_module().synthetic_mechanism()
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    shape = (nz + 2 * NG, ny + 2 * NG, nx + 2 * NG)
    f8 = dict(dtype=torch.float64, device="cuda")
    th = _Thermo(mech.thermo)
    Y = torch.rand((mech.thermo.ns,) + shape, generator=gen, **f8) + 0.02
    Y /= Y.sum(0, keepdim=True)
    T = 400.0 + 2200.0 * torch.rand(shape, generator=gen, **f8)
    p = 1e5 * (0.8 + 0.4 * torch.rand(shape, generator=gen, **f8))
    rho = p / (mech.thermo.Ru * T * (Y / th.mw).sum(0))
    rhoi = rho * Y
    vel = 100.0 * (2 * torch.rand((3,) + shape, generator=gen, **f8) - 1)
    e = th.energy(T, rhoi)
    Q = torch.stack([rho, vel[0], vel[1], vel[2], mech.thermo.Ru * T * (rhoi / th.mw).sum(0), T, e])
    U = torch.stack([rho, *(rho * v for v in vel), e + 0.5 * rho * (vel ** 2).sum(0)])
    return mech, U, Q, rhoi


_DT = {True: 1e-7, False: 1e-9}  # the chemistry step: point-implicit, explicit
_TCRIT = 500.0


def prepare(case, seed):
    f3d = _package()
    kind = case["kind"]
    if kind == "chemistry":
        mech, U, Q, rhoi = _chemistry_inputs(case, seed)
        arrays, react = mech.to_device()
        return {"kind": kind, "lib": f3d.load_library(), "check": f3d.abi.check, "arrays": arrays,
                "react": react, "thermo": mech.thermo.to_c(), "U": U, "Q": Q, "rhoi": rhoi,
                "grid": f3d.FlameGrid(case["nx"], case["ny"], case["nz"], NG, mech.thermo.ns, 7),
                "stiff": case["stiff"], "dt": _DT[case["stiff"]]}
    S = f3d.solver_module()
    precision = 1 if case["precision"] == "mixed" else 0
    if kind == "batch":
        dcs = [S.DeviceCase(_make_member(n, ns, 1000 * seed + i), precision=precision)
               for i, (n, ns) in enumerate(_members(case))]
        batch = f3d.batch_module().Batch(dcs, mode=case["mode"])
        batch.capture()
        return {"kind": kind, "batch": batch, "cases": dcs}
    c = _make(case["field"], case["nx"], case["ny"], case["nz"], case["ns"], case["law"], seed)
    st = {"kind": kind}
    if kind == "host":
        st["Q"], st["rhoi"] = c.Q.cpu().pin_memory(), c.rhoi.cpu().pin_memory()
        st["Qo"] = torch.empty(st["Q"].shape, dtype=torch.float64).pin_memory()
        st["rhoio"] = torch.empty(st["rhoi"].shape, dtype=torch.float64).pin_memory()
    st["dc"] = S.DeviceCase(c, precision=precision, sequence_buffers=kind == "sequence")
    return st


def _state(dc):
    return {"U": dc.U, "Q": dc.Q[dc.cur], "rhoi": dc.rhoi[dc.cur]}


def run(state):
    kind = state["kind"]
    if kind == "chemistry":
        s = state
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        a = (C.byref(s["grid"]), stream, s["U"].data_ptr(), s["Q"].data_ptr(),
             s["rhoi"].data_ptr(), s["dt"], C.byref(s["thermo"]), C.byref(s["react"]), None, _TCRIT)
        rc = s["lib"].flame_eval_gpu_stiff(*a, 0) if s["stiff"] else s["lib"].flame_eval_gpu(*a)
        s["check"](s["lib"], rc)
        return {"U": s["U"], "Q": s["Q"], "rhoi": s["rhoi"]}
    if kind == "batch":
        state["batch"].step()
        return [_state(dc) for dc in state["cases"]]
    dc = state["dc"]
    if kind == "host":
        dc.advance_from_host(state["Q"], state["rhoi"], 1, state["Qo"], state["rhoio"])
        return {"Q": state["Qo"], "rhoi": state["rhoio"]}
    dc.step(fused=kind != "sequence")
    return _state(dc)


def _stage_work(cells, ns, precision):
    """One stage of a perfectly fused solver: Q, the metrics, mu, lambda, D, U, Un, rho_i read
    once, U, Q and rho_i written once (32-bit Q and transport in mixed precision); the
    operations of the hybrid scheme with all faces in the WENO-Z branch."""
    d = ns if ns >= 2 else 0
    q = 8 if precision == "f64" else 4
    nbytes = q * (7 + 2 + 7 + d) + 8 * (10 + 15 + 3 * ns)
    flops = 3 * (110 * (5 + ns) + 100 + 220 + 70 * ns) + 200 + 40 * ns
    return cells * nbytes, cells * flops


def work(case):
    kind = case["kind"]
    if kind == "chemistry":
        cells = case["nx"] * case["ny"] * case["nz"]
        # U4, rho, T, e, rho_i in; U4, p, T, e, rho_i out; rates, Jacobian and elimination
        return {"bytes": cells * 8 * (4 + 8 + 4 + 8), "flops": cells * (6000 if case["stiff"] else 2500)}
    if kind == "batch":
        b = [_stage_work(n ** 3, ns, case["precision"]) for n, ns in _members(case)]
        return {"bytes": 3 * sum(x for x, _ in b), "flops": 3 * sum(x for _, x in b)}
    cells = case["nx"] * case["ny"] * case["nz"]
    b, f = _stage_work(cells, case["ns"], case["precision"])
    b, f = 3 * b, 3 * f
    if kind == "host":
        points = (case["nx"] + 2 * NG) * (case["ny"] + 2 * NG) * (case["nz"] + 2 * NG)
        b += 2 * 8 * points * (7 + case["ns"])
    return {"bytes": b, "flops": f}


# ------------------------------------------------- the same in plain 64-bit torch operations
class _Thermo:
    def __init__(self, th):
        t = lambda a: torch.tensor(np.asarray(a), dtype=torch.float64, device="cuda")  # noqa: E731
        col = lambda a: t(a).reshape(-1, 1, 1, 1)  # noqa: E731
        self.ns, self.Ru = th.ns, th.Ru
        self.mw = col(th.mw)
        self.lo = [col(th.lo[:, a]) for a in range(7)]
        self.hi = [col(th.hi[:, a]) for a in range(7)]
        self.sep = col(th.sep)
        self.tmin, self.tmax = th.min_temp, th.max_temp

    def _pick(self, T, f):
        return torch.where(T < self.sep, f(self.lo), f(self.hi))

    def e_species(self, T):
        p = lambda c: (c[0] - 1) * T + c[1] * T ** 2 / 2 + c[2] * T ** 3 / 3 + c[3] * T ** 4 / 4 \
            + c[4] * T ** 5 / 5  # noqa: E731
        return torch.where(T < self.sep, p(self.lo), p(self.hi) + (self.hi[5] - self.lo[5]))

    def cp_species(self, T):
        return self._pick(T, lambda c: c[0] + c[1] * T + c[2] * T ** 2 + c[3] * T ** 3 + c[4] * T ** 4)

    def h_species(self, T):
        """The enthalpy without the formation part, as the scheme's diffusion flux takes it."""
        p = lambda c: c[0] * T + c[1] * T ** 2 / 2 + c[2] * T ** 3 / 3 + c[3] * T ** 4 / 4 \
            + c[4] * T ** 5 / 5  # noqa: E731
        return torch.where(T < self.sep, p(self.lo), p(self.hi) + (self.hi[5] - self.lo[5])) \
            * self.Ru / self.mw

    def energy(self, T, r):
        return (r * self.e_species(T) / self.mw).sum(0) * self.Ru

    def cv(self, T, r):
        return ((self.cp_species(T) - 1) * r / self.mw).sum(0) * self.Ru

    def temperature(self, e, r):
        """Newton on e(T) with steps of at most 100 K, stopped before an update below 1e-3 K."""
        full = torch.full_like(e, self.tmin), torch.full_like(e, self.tmax)
        emin, emax = (self.energy(t, r) for t in full)
        T = e / ((self.lo[0] - 1) * self.Ru / self.mw * r).sum(0)
        out = (T < self.tmin) | (T > self.tmax)
        T = torch.where(out, self.tmin + (self.tmax - self.tmin) / (emax - emin) * (e - emin), T)
        live = (e >= emin) & (e <= emax)
        for _ in range(30):
            dt = (e - self.energy(T, r)) / self.cv(T, r)
            live = live & (dt.abs() >= 1e-3)
            if not bool(live.any()):
                break
            T = torch.where(live, T + dt.clamp(-100.0, 100.0), T)
        T = torch.where(e < emin, self.tmin - (emin - e) / self.cv(full[0], r), T)
        return torch.where(e > emax, self.tmax - (emax - e) / self.cv(full[1], r), T)


_EPS = 2.220446049250313e-16


def _cut(a, d, o, n, t=None, to=0):
    """The points at offset o from the n[d] + 1 faces along axis d (0 x, 1 y, 2 z) of a ghosted
    array (..., Tz, Ty, Tx), interior along the other axes, shifted by `to` along axis t."""
    sl = [Ellipsis, None, None, None]
    for ax in range(3):
        lo, ln = NG + (o if ax == d else 0) + (to if ax == t else 0), n[ax] + (1 if ax == d else 0)
        sl[3 - ax] = slice(lo, lo + ln)
    return a[tuple(sl)]


def _weno(v):
    s = [13 / 12 * (v[0] - 2 * v[1] + v[2]) ** 2 + (v[0] - 4 * v[1] + 3 * v[2]) ** 2 / 4,
         13 / 12 * (v[1] - 2 * v[2] + v[3]) ** 2 + (v[1] - v[3]) ** 2 / 4,
         13 / 12 * (v[2] - 2 * v[3] + v[4]) ** 2 + (3 * v[2] - 4 * v[3] + v[4]) ** 2 / 4]
    tau = (s[0] - s[2]).abs()
    a = [c * (1 + (tau / (1e-26 + b)) ** 2) for c, b in zip((1, 6, 3), s)]
    return (a[0] * (2 * v[0] - 7 * v[1] + 11 * v[2]) + a[1] * (-v[1] + 5 * v[2] + 2 * v[3])
            + a[2] * (2 * v[2] + 5 * v[3] - v[4])) / (6 * (a[0] + a[1] + a[2]))


def _minmod(a, b):
    return torch.where(a * b > 0, torch.where(a.abs() > b.abs(), b, a), torch.zeros_like(a))


def _hybrid(p, m, phi):
    """The face flux from F+ and F- at the six points around the face."""
    c = (17 / 600, -23 / 120, 22 / 30, 0.5, -0.075, 0.005)
    up = sum(c[k] * (p[k] + m[5 - k]) for k in range(6))
    wz = _weno(p[:5]) + _weno(m[:0:-1])
    mm = p[2] + 0.5 * _minmod(p[3] - p[2], p[2] - p[1]) + m[3] - 0.5 * _minmod(m[4] - m[3], m[3] - m[2])
    return torch.where(phi < 1e-3, up, torch.where(phi < 0.1, wz, mm))


def _transport(th, tr, Q, rhoi, Y):
    """mu, lambda and D of every species."""
    T, p, rho = Q[5], Q[4], Q[0].clamp_min(_EPS)
    one = torch.ones_like(T)
    if tr.law == 0:
        return tr.mu_ref * one, tr.lambda_ref * one, (tr.D_ref * one).expand(th.ns, *T.shape)
    if tr.law == 1:
        cp = (th.cp_species(T) * Y / th.mw).sum(0) * th.Ru
        mu = tr.mu_ref * (T / tr.T_ref) ** tr.exponent
        lam = cp * mu / tr.Pr
        return mu, lam, (lam / (rho * cp)).expand(th.ns, *T.shape)
    ns = th.ns
    poly = torch.tensor(tr.poly, dtype=torch.float64, device=T.device)
    lt = torch.log(T)
    fit = lambda c: c[0] + lt * (c[1] + lt * (c[2] + lt * (c[3] + lt * c[4])))  # noqa: E731
    X = Y / th.mw
    X = X / X.sum(0)
    mw = [float(x) for x in th.mw.flatten()]
    vis, con, bnd = poly[:5 * ns].view(ns, 5), poly[5 * ns:10 * ns].view(ns, 5), poly[10 * ns:].view(ns, ns, 5)
    k = [torch.sqrt(T) * fit(con[n]) for n in range(ns)]
    lam = 0.5 * (sum(X[n] * k[n] for n in range(ns)) + 1 / sum(X[n] / k[n] for n in range(ns)))
    mus = [(T ** 0.25 * fit(vis[n])) ** 2 for n in range(ns)]
    mu = torch.zeros_like(T)
    for n in range(ns):
        row = torch.zeros_like(T)
        for q in range(ns):
            if q == n:
                row = row + X[q]
                continue
            # Wilke's factor of the pair: formed for the later species over the earlier one
            a, b = max(n, q), min(n, q)
            wr, vr = mw[b] / mw[a], mus[a] / mus[b]
            w = (1 + torch.sqrt(vr * math.sqrt(wr))) ** 2 / math.sqrt(8 + 8 / wr)
            row = row + X[q] * (w if n == a else w / (vr * wr))
        mu = mu + X[n] * mus[n] / row
    D = []
    for n in range(ns):
        s = torch.zeros_like(T)
        for q in range(ns):
            if q != n:
                s = s + X[q] / (T ** 1.5 * fit(bnd[min(n, q), max(n, q)]))
        D.append((1 - X[n]) / (s * p + _EPS))
    return mu, lam, torch.stack(D)


def _rhs(th, tr, m, Q, rhoi, n):
    """Flux differences of the 5 + ns conserved fields over the interior (before J dt)."""
    ns = th.ns
    Y = (rhoi / Q[0].clamp_min(_EPS)).clamp_min(0.0)
    mu, lam, D = _transport(th, tr, Q, rhoi, Y)
    P = Q[4]
    phi = torch.zeros_like(P)
    c = P[1:-1, 1:-1, 1:-1]
    for lo, hi in ((P[1:-1, 1:-1, :-2], P[1:-1, 1:-1, 2:]), (P[1:-1, :-2, 1:-1], P[1:-1, 2:, 1:-1]),
                   (P[:-2, 1:-1, 1:-1], P[2:, 1:-1, 1:-1])):
        phi[1:-1, 1:-1, 1:-1] += (-lo + 2 * c - hi).abs() / (lo + 2 * c + hi)
    rho, u, v, w, p, T, e = Q
    gam = p / e + 1
    a = torch.sqrt(gam * p / rho)
    total = torch.zeros((5 + ns, n[2], n[1], n[0]), dtype=torch.float64, device=Q.device)
    for d in range(3):
        A = m[3 * d:3 * d + 3]
        ss = torch.sqrt(A[0] ** 2 + A[1] ** 2 + A[2] ** 2)
        un = A[0] * u + A[1] * v + A[2] * w
        B = [x / ss for x in A]
        fs = []
        for sgn in (1, -1):
            lam_ = [0.5 * (x + sgn * x.abs()) for x in (un, un - a * ss, un + a * ss)]
            g2 = 2 * (gam - 1)
            vel = (u, v, w)
            um, up = ([q - s * a * b for q, b in zip(vel, B)] for s in (1, -1))
            sq = lambda x: x[0] ** 2 + x[1] ** 2 + x[2] ** 2  # noqa: E731
            f = [g2 * lam_[0] + lam_[1] + lam_[2]]
            f += [g2 * lam_[0] * vel[k] + lam_[1] * um[k] + lam_[2] * up[k] for k in range(3)]
            f.append(lam_[0] * (gam - 1) * sq(vel) + lam_[1] * sq(um) / 2 + lam_[2] * sq(up) / 2
                     + (3 - gam) / (2 * (gam - 1)) * a ** 2 * (lam_[1] + lam_[2]))
            fs.append(torch.cat([torch.stack(f) * rho / (2 * gam), lam_[0] * rhoi]))
        at = lambda x, o, t=None, to=0: _cut(x, d, o, n, t, to)  # noqa: E731
        pf = torch.maximum(at(phi, -1), at(phi, 0))
        F = torch.stack([_hybrid([at(fs[0][k], o) for o in range(-3, 3)],
                                 [at(fs[1][k], o) for o in range(-3, 3)], pf) for k in range(5 + ns)])
        del fs
        avg = lambda x: (at(x, -1) + at(x, 0)) / 2  # noqa: E731
        mf = [avg(x) for x in m]

        def gradient(q, wide):
            g = [None] * 3
            g[d] = 1.25 * (at(q, 0) - at(q, -1)) - (at(q, 1) - at(q, -2)) / 12
            for t in range(3):
                if t != d:
                    d1 = at(q, 0, t, 1) + at(q, -1, t, 1) - at(q, 0, t, -1) - at(q, -1, t, -1)
                    if wide:
                        d2 = at(q, 0, t, 2) + at(q, -1, t, 2) - at(q, 0, t, -2) - at(q, -1, t, -2)
                        g[t] = (2 / 3 * d1 - d2 / 12) / 2
                    else:
                        g[t] = d1 / 4
            return [(g[0] * mf[x] + g[1] * mf[3 + x] + g[2] * mf[6 + x]) * mf[9] for x in range(3)]

        # species diffusion with the correction velocity (rho D without the half, as the scheme has it)
        rf, Tf = avg(rho), avg(T)
        V = [[x * (at(D[k], -1) + at(D[k], 0)) * rf for x in gradient(Y[k], False)] for k in range(ns)]
        sums = [sum(V[k][x] for k in range(ns)) for x in range(3)]
        h = th.h_species(Tf)
        fh = [torch.zeros_like(rf) for _ in range(3)]
        md = mf[3 * d:3 * d + 3]
        for k in range(ns):
            Vc = [V[k][x] - sums[x] * avg(Y[k]) for x in range(3)]
            F[5 + k] -= sum(Vc[x] * md[x] for x in range(3))
            fh = [fh[x] + Vc[x] * h[k] for x in range(3)]
        del V
        G = [gradient(Q[k], True) for k in (1, 2, 3, 5)]
        div = G[0][0] + G[1][1] + G[2][2]
        muf = avg(mu)
        tau = [[muf * (G[x][y] + G[y][x]) - (2 / 3 * muf * div if x == y else 0) for y in range(3)]
               for x in range(3)]
        vf = [avg(x) for x in (u, v, w)]
        for x in range(3):
            F[1 + x] -= sum(md[y] * tau[x][y] for y in range(3))
            F[4] -= md[x] * (sum(vf[y] * tau[x][y] for y in range(3)) + avg(lam) * G[3][x] + fh[x])
        k = n[d]
        total += F.narrow(3 - d, 0, k) - F.narrow(3 - d, 1, k)
    return total


def _fills(Q, U, r, th, c):
    """The reference's ghost fills (fillGhost, then fillSpec): inflow at x low and z low."""
    f = c.inflow
    nx, ny, nz = c.nx, c.ny, c.nz
    Yin = torch.tensor([f.Y[k] for k in range(th.ns)], dtype=torch.float64, device=Q.device).reshape(-1, 1, 1, 1)
    rho = f.P / (th.Ru * f.T * (Yin / th.mw).sum(0))
    e = th.energy(torch.full_like(rho, f.T), rho * Yin)

    def inflow(dim):
        sl = (slice(None),) + tuple(slice(0, NG + 1) if k == dim else slice(None) for k in range(3))
        Q[sl] = torch.stack([rho] + [torch.full_like(rho, x) for x in (f.u, f.v, f.w, f.P, f.T)] + [e])
        U[sl] = torch.stack([rho, rho * f.u, rho * f.v, rho * f.w,
                             e + 0.5 * rho * (f.u ** 2 + f.v ** 2 + f.w ** 2)])
        r[sl] = rho * Yin

    def outlet(dim, n, *arrays, low=False):
        for a in arrays:
            a.narrow(dim + 1, n + NG - 1, NG + 1).copy_(
                a.narrow(dim + 1, n + NG - 2, 1).clone().expand_as(a.narrow(dim + 1, n + NG - 1, NG + 1)))
            if low:
                a.narrow(dim + 1, 0, NG + 1).copy_(
                    a.narrow(dim + 1, NG + 1, 1).clone().expand_as(a.narrow(dim + 1, 0, NG + 1)))

    inflow(2)
    outlet(2, nx, Q, U, r)
    outlet(1, ny, Q, U, low=True)
    inflow(0)
    outlet(0, nz, Q, U)
    outlet(1, ny, r, low=True)
    outlet(0, nz, r)


def _exact_step(c):
    """One RK3 step of `c` (a `Case` on the GPU) in 64-bit torch operations."""
    th = _Thermo(c.thermo)
    n = (c.nx, c.ny, c.nz)
    names = [a + b for a in ("dxi", "deta", "dzeta") for b in ("dx", "dy", "dz")] + ["J"]
    m = [c.metrics[k].double() for k in names]
    s = (slice(None),) + _inside(*n)
    J = m[9][_inside(*n)]
    Q, r = c.Q.double().clone(), c.rhoi.double().clone()
    U = torch.stack([Q[0], Q[1] * Q[0], Q[2] * Q[0], Q[3] * Q[0],
                     Q[6] + 0.5 * Q[0] * (Q[1] ** 2 + Q[2] ** 2 + Q[3] ** 2)])
    if c.inflow is not None:
        _fills(Q, U, r, th, c)
    Un, rn = U[s].clone(), r[s].clone()
    for a, b in ((1.0, 0.0), (0.25, 0.75), (2 / 3, 1 / 3)):
        dF = _rhs(th, c.transport, m, Q, r, n) * (J * c.dt)
        Ui = (U[s] + dF[:5]) * a + Un * b
        ri = ((r[s] + dF[5:]) * a + rn * b).clamp_min(0.0)
        U[s] = Ui
        rho = Ui[0].clamp_min(_EPS)
        ri = ri * (rho / ri.sum(0))
        vel = Ui[1:4] / rho
        e = (Ui[4] - 0.5 * rho * (vel ** 2).sum(0)).clamp_min(_EPS)
        T = th.temperature(e, ri).clamp_min(_EPS)
        p = (th.Ru * T * (ri / th.mw).sum(0)).clamp_min(_EPS)
        Qi = torch.stack([rho, vel[0], vel[1], vel[2], p, T, e])
        if c.inflow is None:
            Q, r = _pad(Qi, *n, True), _pad(ri, *n, True)
        else:
            Q[s], r[s] = Qi, ri
            _fills(Q, U, r, th, c)
    return {"U": U, "Q": Q, "rhoi": r}


def _exact_chemistry(case, seed):
    mech, U, Q, r = _chemistry_inputs(case, seed)
    th = _Thermo(mech.thermo)
    ns, dt = th.ns, _DT[case["stiff"]]
    s = _inside(case["nx"], case["ny"], case["nz"])
    hot = Q[5][s] > _TCRIT
    T, rho, ein = (Q[k][s][hot] for k in (5, 0, 6))
    ri = torch.stack([r[k][s][hot] for k in range(ns)])
    mw = th.mw.reshape(-1, 1)
    lo = [x.reshape(-1, 1) for x in th.lo]
    sc = ri / mw * 1e-6
    lt, inv = torch.log(T), 1 / T
    gibbs = (lo[0] * (1 - lt) - lo[1] * T / 2 - lo[2] * T ** 2 / 6 - lo[3] * T ** 3 / 12
             - lo[4] * T ** 4 / 20 + lo[5] * inv - lo[6])
    w = torch.zeros_like(sc)
    A = torch.zeros((T.numel(), ns, ns), dtype=torch.float64, device=T.device)
    arr = lambda a: float(a[0]) * torch.exp(float(a[1]) * lt - float(a[2]) * inv)  # noqa: E731
    for k in range(mech.nreacs):
        nu = [int(x) for x in mech.vr[k] - mech.vf[k]]
        kf = arr(mech.Arr[k])
        Kc = (th.Ru / mech.atm * 1e6 * T) ** int(mech.sgm[k]) * torch.exp(-sum(nu[j] * gibbs[j] for j in range(ns)))
        qf, qr = kf.clone(), kf / Kc
        for j in range(ns):
            qf = qf * sc[j] ** int(mech.vf[k, j])
            qr = qr * sc[j] ** int(mech.vr[k, j])
        if mech.reaction_type[k] >= 2:
            mix = sum(float(mech.ef[k, j]) * sc[j] for j in range(ns))
            if mech.reaction_type[k] == 2:
                f = mix
            else:
                tr = [float(x) for x in mech.Troe[k]]
                red = mix / kf * arr(mech.loP[k])
                lp = torch.log10(red)
                fc = torch.log10((1 - tr[0]) * torch.exp(-T / tr[1]) + tr[0] * torch.exp(-T / tr[2])
                                 + torch.exp(-tr[3] * inv))
                x = (-0.4 - 0.67 * fc + lp) / (0.75 - 1.27 * fc - 0.14 * (-0.4 - 0.67 * fc + lp))
                f = red / (1 + red) * 10 ** (fc / (1 + x * x))
            qf, qr = qf * f, qr * f
        for j in range(ns):
            w[j] += (qf - qr) * nu[j]
            dj = (int(mech.vf[k, j]) * qf - int(mech.vr[k, j]) * qr) / (sc[j] + _EPS)
            for q in range(ns):
                if nu[q]:
                    A[:, q, j] += dj * nu[q]
    d = w * mw * 1e6 * dt
    if case["stiff"]:
        ratio = (mw / mw.reshape(1, -1)) * dt
        M = torch.eye(ns, dtype=torch.float64, device=T.device) - A * ratio
        d = torch.linalg.solve(M, d.T.unsqueeze(-1)).squeeze(-1).T
    de = (-lo[5] * d * th.Ru / mw).sum(0)
    ri = (ri + d).clamp_min(0.0)
    ri = ri * (rho.clamp_min(_EPS) / ri.sum(0))
    ein = ein + de
    col = lambda x: x.reshape(x.shape[:-1] + (1, 1, -1))  # noqa: E731
    Tn = th.temperature(col(ein), col(ri)).flatten().clamp_min(_EPS)
    p = (th.Ru * Tn * (ri / mw).sum(0)).clamp_min(_EPS)
    for a, x in ((U[4], U[4][s][hot] + de), (Q[4], p), (Q[5], Tn), (Q[6], ein)):
        a[s] = a[s].masked_scatter(hot, x)
    for k in range(ns):
        r[k][s] = r[k][s].masked_scatter(hot, ri[k])
    return {"U": U, "Q": Q, "rhoi": r}


def exact(case, seed):
    kind = case["kind"]
    if kind == "chemistry":
        return _exact_chemistry(case, seed)
    if kind == "batch":
        return [_exact_step(_make_member(n, ns, 1000 * seed + i))
                for i, (n, ns) in enumerate(_members(case))]
    r = _exact_step(_make(case["field"], case["nx"], case["ny"], case["nz"], case["ns"], case["law"], seed))
    return {"Q": r["Q"], "rhoi": r["rhoi"]} if kind == "host" else r
