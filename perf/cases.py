"""The work that users of this library have it do, as cases that can be measured.

Every case is one call sequence of an application through the package's public entry points, on
meshes and states made from a seed:

  rhs        one allocation-free right-hand side on the caller's own device arrays
  run        a device-resident run: init, a number of SSPRK3 steps, the result
  host       one SSPRK3 step from pinned host memory and back
  batch      many instances of uneven size and order advanced together
  gradient   an objective's forward and backward (lift over alpha, vortex error over beta)
  dropin     the OP2 loops of the airfoil application
  advection  the scalar advection application

exact() restates each of them in plain torch FP64 (dense operators, the textbook Roe flux from
each side, autograd for the gradients).
"""
import ctypes
import functools
import importlib
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_NAME = "airfoil_op2_fem_gb300"
_GAM = 1.4


def _pkg():
    if _NAME not in sys.modules:
        folder = os.path.join(_ROOT, "airfoil-op2-fem_gb300")
        spec = importlib.util.spec_from_file_location(_NAME, os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[_NAME] = mod
        spec.loader.exec_module(mod)
    return sys.modules[_NAME]


# ------------------------------------------------------------------------------- the cases
def listed():
    return [
        # The smallest call: one right-hand side for a caller that owns the arrays (an implicit
        # or coupled time integrator evaluating the residual), on a small mesh.
        {"name": "rhs-small", "kind": "rhs", "order": 3, "n_theta": 64, "n_r": 16},
        # A small vortex run, 2048 triangles at order 3: launches and latency.
        {"name": "vortex-small", "kind": "run", "app": "vortex", "order": 3, "n": 32, "steps": 40},
        # The ordinary production run: NACA 0012 O-grid, 32768 triangles, order 3.
        {"name": "airfoil", "kind": "run", "app": "airfoil", "order": 3, "n_theta": 256, "n_r": 64, "steps": 40},
        # A high-order run on an odd mesh size.
        {"name": "airfoil-high-order", "kind": "run", "app": "airfoil", "order": 5, "n_theta": 211, "n_r": 45,
         "steps": 12},
        # The largest run: 524288 triangles at the reference's order 4.
        {"name": "vortex-large", "kind": "run", "app": "vortex", "order": 4, "n": 512, "steps": 6},
        # One step per call from and to pinned host memory (a host code that owns the state).
        {"name": "airfoil-host", "kind": "host", "app": "airfoil", "order": 3, "n_theta": 256, "n_r": 64},
        # A parameter sweep: instances of uneven size, orders 3 and 4 mixed, launch shape autotuned.
        {"name": "sweep", "kind": "batch", "count": 12, "order_lo": 3, "order_hi": 4, "nt_lo": 128, "nt_hi": 384,
         "nr_lo": 32, "nr_hi": 96, "tune": True, "steps": 6},
        # A sweep of many small instances with the default launch shape.
        {"name": "sweep-small", "kind": "batch", "count": 48, "order_lo": 3, "order_hi": 4, "nt_lo": 32, "nt_hi": 64,
         "nr_lo": 8, "nr_hi": 16, "tune": False, "steps": 40},
        # The lift gradient over alpha and the initial state: forward and backward, checkpointed.
        {"name": "lift-gradient", "kind": "gradient", "app": "airfoil", "order": 3, "n_theta": 256, "n_r": 64,
         "steps": 40, "navg": 4, "every": 20, "count": 1},
        # Vortex-strength gradients of several instances in one batched call.
        {"name": "vortex-gradient", "kind": "gradient", "app": "vortex", "order": 2, "n": 256, "steps": 28,
         "navg": 1, "every": 14, "count": 2},
        # The OP2 application's own loops (the drop-in), the reference's boundary types.
        {"name": "dropin", "kind": "dropin", "order": 3, "n_theta": 256, "n_r": 64, "steps": 5},
        # The scalar advection application on a large square.
        {"name": "advection", "kind": "advection", "order": 4, "n": 512, "steps": 6},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _np(order):
    return (order + 1) * (order + 2) // 2


def draw(rng):
    kind = rng.choice(["rhs", "run", "run", "run", "host", "batch", "gradient", "dropin", "advection"])
    order = rng.choice([1, 2, 3, 3, 3, 4, 4, 5, 6])
    app = rng.choice(["airfoil", "vortex"])
    ogrid = {"n_theta": _log(rng, 32, 384), "n_r": _log(rng, 8, 96)}
    if kind == "rhs":  # the scratch of this entry point holds at most 32 MiB of face fluxes
        n_theta = _log(rng, 32, 256)
        return {"kind": kind, "order": order, "n_theta": n_theta, "n_r": _log(rng, 8, min(64, 100000 // (order + 1) // n_theta))}
    if kind in ("run", "host"):
        c = {"kind": kind, "app": app, "order": order}
        if app == "vortex":
            c["n"] = _log(rng, 16, 512 if order <= 4 else 320)
            cells = 2 * c["n"] ** 2
        else:
            c.update(ogrid)
            cells = 2 * c["n_theta"] * c["n_r"]
        if kind == "run":
            c["steps"] = max(2, min(48, 28_000_000 // (cells * _np(order)))) + rng.randrange(2)
        return c
    if kind == "batch":
        tune = rng.random() < 0.5
        lo = _log(rng, 32, 128)
        hi = lo + rng.randrange(1, 2 * lo)
        count = rng.randrange(5, 13)
        steps = max(2, min(20, 28_000_000 // (count * (lo + hi) ** 2 // 8 * 12))) + rng.randrange(2)
        return {"kind": kind, "count": count, "order_lo": rng.choice([1, 2, 3]),
                "order_hi": rng.choice([3, 4]), "nt_lo": lo, "nt_hi": hi, "nr_lo": max(8, lo // 4),
                "nr_hi": max(9, hi // 4), "tune": tune, "steps": steps}
    if kind == "gradient":
        order = rng.choice([1, 2, 3, 3, 4])
        c = {"kind": kind, "app": app, "order": order, "every": rng.randrange(5, 20), "navg": rng.randrange(1, 5),
             "count": rng.randrange(1, 4)}
        if app == "vortex":
            c["n"] = _log(rng, 16, 192)
            cells = 2 * c["n"] ** 2
        else:
            c.update(n_theta=_log(rng, 32, 256), n_r=_log(rng, 8, 64))
            cells = 2 * c["n_theta"] * c["n_r"]
        c["steps"] = max(5, min(30, 28_000_000 // (c["count"] * cells * _np(order)))) + rng.randrange(3)
        return c
    if kind == "dropin":
        return {"kind": kind, "order": rng.choice([3, 4, 4]), "n_theta": _log(rng, 48, 256), "n_r": _log(rng, 12, 64),
                "steps": rng.randrange(2, 7)}
    return {"kind": "advection", "order": order, "n": _log(rng, 24, 512 if order <= 4 else 360), "steps": rng.randrange(4, 9)}


# ------------------------------------------------------------------------------- meshes
def _square(n, lo, hi, seed):
    """[lo, hi]^2 in 2 n^2 triangles, each square cut along a diagonal drawn from the seed."""
    rng = np.random.default_rng(seed)
    w = n + 1
    x = lo + (hi - lo) * np.arange(w) / n
    coords = np.stack([np.tile(x, w), np.repeat(x, w)], axis=1)
    i, j = np.meshgrid(np.arange(n), np.arange(n))
    a = (j * w + i).ravel()
    b, c, d = a + 1, a + w, a + w + 1
    cut = rng.integers(0, 2, n * n)[:, None, None] == 0
    cells = np.where(cut, np.stack([np.stack([a, b, d], 1), np.stack([a, d, c], 1)], 1),
                     np.stack([np.stack([a, b, c], 1), np.stack([b, d, c], 1)], 1)).reshape(-1, 3)
    return coords, cells.astype(np.int32), None


def _ogrid(n_theta, n_r, far, turn=0.0):
    """NACA 0012 O-grid out to 20 chords (rings stretched by 1.1), turned by `turn` radians.
    Returns a function of boundary edges (vertex pairs) to boundary types: the wall 2, the outer
    ring 3 (characteristic) or inflow / outflow by the sign of x."""
    phi = 2.0 * np.pi * np.arange(n_theta) / n_theta
    xs = 0.5 * (1.0 + np.cos(phi))
    t = 0.594689181 * (0.298222773 * np.sqrt(xs) - 0.127125232 * xs - 0.357907906 * xs ** 2 + 0.291984971 * xs ** 3 -
                       0.105174696 * xs ** 4)
    ys = np.maximum(t, 0.0) * np.where(np.arange(n_theta) <= n_theta // 2, 1.0, -1.0)
    xf, yf = 0.5 + 20.0 * np.cos(phi), 20.0 * np.sin(phi)
    g = ((1.1 ** np.arange(n_r + 1) - 1.0) / (1.1 ** n_r - 1.0))[:, None]
    x, y = (xs + (xf - xs) * g).ravel(), (ys + (yf - ys) * g).ravel()
    coords = np.stack([math.cos(turn) * x - math.sin(turn) * y, math.sin(turn) * x + math.cos(turn) * y], axis=1)
    k, j = np.meshgrid(np.arange(n_theta), np.arange(n_r))
    k, j = k.ravel(), j.ravel()
    k1 = (k + 1) % n_theta
    a, b, c, d = j * n_theta + k, j * n_theta + k1, (j + 1) * n_theta + k, (j + 1) * n_theta + k1
    cells = np.stack([np.stack([a, c, b], 1), np.stack([b, c, d], 1)], 1).reshape(-1, 3)

    def types(pairs):
        wall = (pairs < n_theta).all(axis=1)
        xm = 0.5 * (coords[pairs[:, 0], 0] + coords[pairs[:, 1], 0])
        outer = np.where(xm < 0.0, 0, 1) if far == "reference" else np.full(len(pairs), 3)
        return np.where(wall, 2, outer).astype(np.int32)
    return coords, cells.astype(np.int32), types


def _mesh(tables):
    coords, cells, types = tables
    m = _pkg().Mesh.from_cells(coords, cells, device=True)
    if types is not None:
        m.set_bedge_type(types(m.arrays()["bedge2nodes"]))
    return m


def _flow(seed, k=0):
    """Angle of attack (degrees) and Mach number of instance k."""
    rng = np.random.default_rng([seed, k])
    return float(rng.uniform(-4.0, 8.0)), float(rng.uniform(0.3, 0.6))


def _vortex(seed, k=0):
    """Strength and centre of instance k's vortex."""
    rng = np.random.default_rng([seed, k, 1])
    return float(rng.uniform(3.0, 7.0)), float(rng.uniform(-1.0, 1.0)), float(rng.uniform(-1.0, 1.0))


def _instance(case, seed, k=0):
    """Mesh tables and configuration (a dict) of one run."""
    if case.get("app") == "vortex":
        beta, x0, y0 = _vortex(seed, k)
        # the gradient holds the initial dt over the run
        return _square(case["n"], -5.0, 5.0, seed), dict(
            N=case["order"], app=1, dt_mode=1 if case["kind"] == "gradient" else 0, cfl=0.5, vortex_x0=x0, vortex_y0=y0,
            vortex_beta=beta)
    alpha, mach = _flow(seed, k)
    return _ogrid(case["n_theta"], case["n_r"], "characteristic"), dict(N=case["order"], app=0, cfl=0.5, mach=mach,
                                                                       alpha_deg=alpha)


def _sweep(case, seed):
    """(mesh tables, configuration) of every instance of a batch."""
    out = []
    for k in range(case["count"]):
        f = k / (case["count"] - 1)
        alpha, mach = _flow(seed, k)
        nt = int(round(case["nt_lo"] + f * (case["nt_hi"] - case["nt_lo"])))
        nr = int(round(case["nr_lo"] + f * (case["nr_hi"] - case["nr_lo"])))
        out.append((_ogrid(nt, nr, "characteristic"),
                    dict(N=case["order_hi"] if k % 2 else case["order_lo"], app=0, cfl=0.5, mach=mach, alpha_deg=alpha)))
    return out


def _disturbed(tables, order, mach, alpha, seed):
    """A smooth disturbed flow at the nodes with small jumps between cells, [K][Np][4] on the GPU."""
    coords, cells, _ = tables
    r, s = _operators(order)["rs"]
    v = torch.as_tensor(coords[cells], device="cuda")  # [K][3][2]
    r, s = torch.as_tensor(r, device="cuda"), torch.as_tensor(s, device="cuda")
    x = 0.5 * (-(r + s) * v[:, :1, 0] + (1 + r) * v[:, 1:2, 0] + (1 + s) * v[:, 2:3, 0])
    y = 0.5 * (-(r + s) * v[:, :1, 1] + (1 + r) * v[:, 1:2, 1] + (1 + s) * v[:, 2:3, 1])
    g = torch.Generator(device="cuda").manual_seed(seed)
    p = torch.rand(8, generator=g, device="cuda", dtype=torch.float64)
    e = torch.exp(-0.05 * (x * x + y * y))
    rho = 1.0 + 0.1 * e * torch.sin(2 * x + 6 * p[0]) + 0.02 * torch.cos(y + 6 * p[1])
    speed = mach * math.sqrt(_GAM)
    u = speed * math.cos(math.radians(alpha)) + 0.1 * e * torch.cos(3 * y + 6 * p[2])
    w = speed * math.sin(math.radians(alpha)) + 0.1 * e * torch.sin(x - y + 6 * p[3])
    pr = rho ** _GAM * (1.0 + 0.02 * torch.sin(x + 6 * p[4]))
    q = torch.stack([rho, rho * u, rho * w, pr / (_GAM - 1) + 0.5 * rho * (u * u + w * w)], dim=2)
    return (q * (1.0 + 1e-4 * (torch.rand(q.shape, generator=g, device="cuda", dtype=torch.float64) - 0.5))).contiguous()


# ------------------------------------------------------------------------------- prepare and run
class _DeviceArray:
    """A device array of the library as torch sees it (no copy)."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 3}


class _HostArray:
    """A view of pinned host memory that keeps it allocated."""

    def __init__(self, n):
        self.owner = _pkg().PinnedArray(n)
        self.__array_interface__ = dict(self.owner.array.__array_interface__)


def _view(solver):
    ptr = _pkg().lib().dg_solver_device_ptr(solver.h, b"q")
    return torch.as_tensor(_DeviceArray(ptr, (solver.K, solver.Np, 4), solver), device="cuda")


_HOST_START = 20  # steps behind the state that the host case steps from
_EULER_RHS_DATS = ("rx", "ry", "sx", "sy", "fscale", "nx", "ny")
_op2_started = False


class _DropIn:
    """The airfoil application's declarations and loops on the OP2 interface."""

    def __init__(self, tables, order, mach):
        global _op2_started
        o = self.o = importlib.import_module(_pkg().__name__ + ".op2")
        if not _op2_started:  # one application per process: its constants are global
            o.op_init(0)
            _op2_started = True
        m = _mesh(tables)
        a = m.arrays()
        ops = _pkg().operators(order)
        np_, nfp = _np(order), order + 1
        self.K = K = len(a["cell2nodes"])
        nodes, cells = o.op_decl_set(len(a["coords"]), "nodes"), o.op_decl_set(K, "cells")
        edges, bedges = o.op_decl_set(len(a["edge2cells"]), "edges"), o.op_decl_set(len(a["bedge2cell"]), "bedges")
        c2n = o.op_decl_map(cells, nodes, 3, a["cell2nodes"], "cell2nodes")
        e2c = o.op_decl_map(edges, cells, 2, a["edge2cells"], "edge2cells")
        b2c = o.op_decl_map(bedges, cells, 1, a["bedge2cell"], "bedge2cells")
        xy = o.op_decl_dat(nodes, 2, "double", a["coords"], "node_coords")
        dims = {"nodeX": 3, "nodeY": 3, "q": 4 * np_, "workingQ": 4 * np_, "rk1": 4 * np_, "rk2": 4 * np_,
                "rk3": 4 * np_, "exteriorQ": 12 * nfp}
        dims.update({k: np_ for k in ("x", "y", "xr", "yr", "xs", "ys", "rx", "ry", "sx", "sy")})
        dims.update({k: 3 * nfp for k in ("nx", "ny", "fscale")})
        self.d = d = {k: o.op_decl_dat(cells, v, "double", np.zeros(K * v), k) for k, v in dims.items()}
        btype = o.op_decl_dat(bedges, 1, "int", a["bedge_type"], "bedge_type")
        enum = o.op_decl_dat(edges, 2, "int", a["edgeNum"], "edgeNum")
        bnum = o.op_decl_dat(bedges, 1, "int", a["bedgeNum"], "bedgeNum")
        u = mach * math.sqrt(_GAM)
        for k, v in dict(gam=_GAM, bc_mach=mach, bc_alpha=0.0, bc_p=1.0, bc_r=1.0, bc_u=u, bc_v=0.0,
                         bc_e=1.0 / (_GAM - 1.0) + 0.5 * u * u).items():
            o.op_decl_const2(k, 1, "double", v)
        o.op_decl_const2("ones", np_, "double", np.ones(np_))
        for k in ("r", "s", "Dr", "Ds", "Drw", "Dsw", "LIFT"):
            o.op_decl_const2(k, ops[k].size, "double", ops[k].ravel())
        o.op_decl_const2("FMASK", 3 * nfp, "int", ops["FMASK"])

        def A(name, acc, idx=-1, mp=None):
            return o.op_arg_dat(d[name], idx, mp, dims[name], "double", acc)
        R, W = o.OP_READ, o.OP_WRITE
        o.op_par_loop_init_grid("init_grid", cells, *[o.op_arg_dat(xy, k, c2n, 2, "double", R) for k in range(3)],
                                *[A(n, W) for n in ("nodeX", "nodeY", "x", "y", "xr", "yr", "xs", "ys", "rx", "ry", "sx",
                                                    "sy", "nx", "ny", "fscale")])
        self.dt, self.dt1 = np.zeros(1), np.zeros(1)
        stage = [np.array([j], dtype=np.int32) for j in range(2)]
        # the loops of a step with their arguments, as the application's source spells them out
        ic = (o.op_par_loop_set_ic, "set_ic", cells, A("q", W), A("workingQ", W))
        zero = (o.op_par_loop_neighbour_zero, "neighbour_zero", cells, A("exteriorQ", W))
        self.calc = (o.op_par_loop_calc_dt, "calc_dt", cells, A("q", R), A("fscale", R),
                     o.op_arg_gbl(self.dt1, 1, "double", o.OP_MAX))
        self.start = [ic, zero]
        self.step = []
        for j in range(3):
            self.step.append((o.op_par_loop_get_neighbour_q, "get_neighbour_q", edges, o.op_arg_dat(enum, -1, None, 2, "int", R),
                              A("nodeX", R, 0, e2c), A("nodeY", R, 0, e2c), A("nodeX", R, 1, e2c), A("nodeY", R, 1, e2c),
                              A("workingQ", R, 0, e2c), A("workingQ", R, 1, e2c), A("exteriorQ", o.OP_INC, 0, e2c),
                              A("exteriorQ", o.OP_INC, 1, e2c)))
            self.step.append((o.op_par_loop_get_bedge_q, "get_bedge_q", bedges, o.op_arg_dat(btype, -1, None, 1, "int", R),
                              o.op_arg_dat(bnum, -1, None, 1, "int", R), A("nx", R, 0, b2c), A("ny", R, 0, b2c),
                              A("workingQ", R, 0, b2c), A("exteriorQ", o.OP_INC, 0, b2c)))
            self.step.append((o.op_par_loop_euler_rhs, "euler_rhs", cells, A("workingQ", R), A("exteriorQ", o.OP_RW),
                              *[A(n, R) for n in _EULER_RHS_DATS], A("rk%d" % (j + 1), W)))
            if j < 2:
                self.step.append((o.op_par_loop_set_workingQ, "set_workingQ", cells, o.op_arg_gbl(self.dt, 1, "double", R),
                                  o.op_arg_gbl(stage[j], 1, "int", R), A("q", R), A("rk1", R), A("rk2", R),
                                  A("workingQ", W)))
        self.step.append((o.op_par_loop_update_Q, "update_Q", cells, o.op_arg_gbl(self.dt, 1, "double", R),
                          A("q", o.OP_RW), A("rk1", R), A("rk2", R), A("rk3", R), A("workingQ", W)))
        self.out = np.empty(K * 4 * np_)

    def new_dt(self):
        self.dt1[0] = 0.0
        self.calc[0](*self.calc[1:])
        self.dt[0] = 1.0 / self.dt1[0]

    def run(self, steps):
        for loop in self.start:
            loop[0](*loop[1:])
        self.new_dt()
        for _ in range(steps):
            for loop in self.step:
                loop[0](*loop[1:])
            self.new_dt()
        self.o.op_fetch_data(self.d["q"], self.out)
        return self.out, self.dt


def _advection_instance(case, seed):
    rng = np.random.default_rng(seed)
    ang = float(rng.uniform(0.2, 1.3))
    n = case["n"]
    return _square(n, 0.0, 10.0, seed), (math.sqrt(2.0) * math.cos(ang), math.sqrt(2.0) * math.sin(ang)), \
        0.2 * (10.0 / n) / (case["order"] + 1) ** 2


def prepare(case, seed):
    P = _pkg()
    kind = case["kind"]
    if kind == "rhs":
        alpha, mach = _flow(seed)
        tables = _ogrid(case["n_theta"], case["n_r"], "characteristic")
        m = _mesh(tables)
        cfg = P.config(N=case["order"], mach=mach, alpha_deg=alpha)
        a = m.arrays()
        K = len(a["cell2nodes"])
        # the entry point's documented edge records; every edge is seen in opposite directions
        # by its two (counter-clockwise) cells
        e = np.zeros((len(a["edge2cells"]), 4), dtype=np.int32)
        e[:, :2] = a["edge2cells"]
        e[:, 2] = a["edgeNum"][:, 0] | (a["edgeNum"][:, 1] << 2) | (1 << 4)
        b = np.zeros((len(a["bedge2cell"]), 4), dtype=np.int32)
        b[:, 0], b[:, 1], b[:, 2] = a["bedge2cell"], a["bedgeNum"], a["bedge_type"]
        W = _disturbed(tables, case["order"], mach, alpha, seed)
        f = P.lib().dg_rhs_noalloc
        f.restype = ctypes.c_int
        f.argtypes = [ctypes.c_void_p] + [ctypes.c_int] * 3 + [ctypes.c_void_p] * 6
        geo = P.Solver(m, cfg).get("geo").reshape(K, 16)
        return {"kind": kind, "call": f, "cfg": cfg, "W": W, "geo": torch.as_tensor(geo, device="cuda"),
                "edges": torch.as_tensor(e, device="cuda"), "bedges": torch.as_tensor(b, device="cuda"),
                "out": torch.empty_like(W)}
    if kind in ("run", "host"):
        tables, cfg = _instance(case, seed)
        s = P.Solver(_mesh(tables), P.config(**cfg)).init()
        if kind == "run":
            return {"kind": kind, "solver": s, "steps": case["steps"], "q": _view(s)}
        n = s.K * s.Np * 4
        st = {"kind": kind, "solver": s, "in": np.asarray(_HostArray(n)), "out": np.asarray(_HostArray(n))}
        s.run(_HOST_START)  # a flow that has begun to develop
        s.sync()
        st["in"][:] = s.get("q")
        return st
    if kind == "batch":
        inst = _sweep(case, seed)
        b = P.Batch([_mesh(t) for t, _ in inst], [P.config(**c) for _, c in inst]).init()
        if case["tune"]:
            b.autotune(2)
        return {"kind": kind, "batch": b, "steps": case["steps"], "count": case["count"]}
    if kind == "gradient":
        objs = []
        mesh = None
        for k in range(case["count"]):
            tables, cfg = _instance(case, seed, k)
            mesh = mesh or _mesh(tables)
            objs.append(P.LiftObjective(mesh, P.config(**cfg), case["steps"], case["navg"], case["every"]))
        return {"kind": kind, "objs": objs}
    if kind == "dropin":
        turn = float(np.random.default_rng(seed).uniform(-0.1, 0.1))
        app = _DropIn(_ogrid(case["n_theta"], case["n_r"], "reference", turn), case["order"], 0.4)
        return {"kind": kind, "app": app, "steps": case["steps"]}
    tables, vel, dt = _advection_instance(case, seed)
    a = P.Advection(_mesh(tables), case["order"], vel[0], vel[1], dt).init()
    return {"kind": kind, "advection": a, "steps": case["steps"]}


def run(st):
    P = _pkg()
    kind = st["kind"]
    if kind == "rhs":
        rc = st["call"](ctypes.byref(st["cfg"]), st["W"].shape[0], st["edges"].shape[0], st["bedges"].shape[0],
                        st["W"].data_ptr(), st["geo"].data_ptr(), st["edges"].data_ptr(), st["bedges"].data_ptr(),
                        st["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError("dg_rhs_noalloc: %d" % rc)
        return st["out"]
    if kind == "run":
        s = st["solver"]
        s.init()
        s.run(st["steps"])
        t, dt, _ = s.time()
        return st["q"], np.array([t, dt])
    if kind == "host":
        st["solver"].step_host(st["in"], 1, st["out"])
        return st["out"]
    if kind == "batch":
        b = st["batch"]
        b.init()
        b.run(st["steps"])
        b.sync()
        return [b.get(k) for k in range(st["count"])], np.array([b.time(k)[1] for k in range(st["count"])])
    if kind == "gradient":
        objs = st["objs"]
        if len(objs) == 1:
            J = objs[0].forward()
            g, gq = objs[0].backward(1.0, want_q0=True)
            return np.array([J, g]), [gq]
        J = P.adjoint_batch_forward(objs)
        g, gq = P.adjoint_batch_backward(objs, 1.0, want_q0=True)
        return np.concatenate([J, g]), gq
    if kind == "dropin":
        return st["app"].run(st["steps"])
    a = st["advection"]
    a.init()
    a.run(st["steps"])
    a.sync()
    return a.get("q")


# ------------------------------------------------------------------------------- work
def _work_of(cells, face_nodes, order, evaluations, per_face, variables=4):
    """Operations of right-hand sides: the dense [Drw | Dsw | -LIFT] product on the metric-combined
    fluxes, the nodal fluxes and stage updates, the numerical flux once per face node."""
    n, nfp = _np(order), order + 1
    per_cell = 2 * variables * n * (2 * n + 3 * nfp) + (40 if variables == 4 else 8) * n
    return evaluations * (cells * per_cell + face_nodes * per_face)


def work(case):
    kind, N = case["kind"], case.get("order", 0)
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for k in range(case["count"]):
            f = k / (case["count"] - 1)
            w = work({"kind": "run", "app": "airfoil", "order": case["order_hi"] if k % 2 else case["order_lo"],
                      "n_theta": int(round(case["nt_lo"] + f * (case["nt_hi"] - case["nt_lo"]))),
                      "n_r": int(round(case["nr_lo"] + f * (case["nr_hi"] - case["nr_lo"]))), "steps": case["steps"]})
            total = {k2: total[k2] + w[k2] for k2 in total}
        return total
    if "n" in case:
        cells, faces, nodes = 2 * case["n"] ** 2, 3 * case["n"] ** 2 + 2 * case["n"], (case["n"] + 1) ** 2
    else:
        t, r = case["n_theta"], case["n_r"]
        cells, faces, nodes = 2 * t * r, t * (3 * r + 1), t * (r + 1)
    state = 8.0 * cells * _np(N) * (1 if kind == "advection" else 4)
    mesh = 16.0 * nodes + 12.0 * cells + 16.0 * faces
    fn = faces * (N + 1)
    if kind == "rhs":
        return {"bytes": 2 * state + 128.0 * cells + 16.0 * faces, "flops": _work_of(cells, fn, N, 1, 150)}
    if kind == "advection":
        return {"bytes": state + mesh, "flops": _work_of(cells, fn, N, 4 * case["steps"], 12, 1)}
    steps = case.get("steps", 1)
    if kind == "gradient":  # forward, recomputation, and a transposed right-hand side per stage
        m = case["count"]
        return {"bytes": m * 2 * state + mesh, "flops": m * (2 * _work_of(cells, fn, N, 3 * steps, 150) +
                                                               _work_of(cells, fn, N, 3 * steps, 400))}
    return {"bytes": (2 if kind == "host" else 1) * state + mesh, "flops": _work_of(cells, fn, N, 3 * steps, 150)}


# ------------------------------------------------------------------------------- exact
def _jacobi(x, a, b, n):
    """Orthonormal Jacobi polynomial (Hesthaven & Warburton, appendix A)."""
    g0 = 2 ** (a + b + 1) / (a + b + 1) * math.gamma(a + 1) * math.gamma(b + 1) / math.gamma(a + b + 1)
    p0 = np.full_like(x, 1.0 / math.sqrt(g0))
    if n == 0:
        return p0
    g1 = (a + 1) * (b + 1) / (a + b + 3) * g0
    p1 = ((a + b + 2) * x / 2 + (a - b) / 2) / math.sqrt(g1)
    old = 2 / (2 + a + b) * math.sqrt((a + 1) * (b + 1) / (a + b + 3))
    for i in range(1, n):
        h = 2 * i + a + b
        new = 2 / (h + 2) * math.sqrt((i + 1) * (i + 1 + a + b) * (i + 1 + a) * (i + 1 + b) / (h + 1) / (h + 3))
        p0, p1 = p1, (-old * p0 + (x + (a * a - b * b) / h / (h + 2)) * p1) / new
        old = new
    return p1


def _djacobi(x, a, b, n):
    return np.zeros_like(x) if n == 0 else math.sqrt(n * (n + a + b + 1)) * _jacobi(x, a + 1, b + 1, n - 1)


def _warp(n, out):
    """Warp of equidistant to Legendre-Gauss-Lobatto nodes along an edge."""
    req = np.linspace(-1, 1, n + 1)
    lgl = np.sort(np.concatenate([[-1.0], np.polynomial.legendre.Legendre.basis(n).deriv().roots().real, [1.0]]))
    v = np.stack([_jacobi(req, 0, 0, j) for j in range(n + 1)], axis=1)
    p = np.stack([_jacobi(out, 0, 0, j) for j in range(n + 1)])
    w = np.linalg.solve(v.T, p).T @ (lgl - req)
    inner = np.abs(out) < 1.0 - 1e-10
    return w / (1.0 - (inner * out) ** 2) + w * (inner - 1.0)


@functools.lru_cache(maxsize=None)
def _operators(n):
    """Nodes and nodal operators of order n (Hesthaven & Warburton, chapter 6: warp and blend)."""
    alpha = [0.0, 0.0, 1.4152, 0.1001, 0.2751, 0.98][n - 1]
    l1 = np.array([i / n for i in range(n + 1) for j in range(n + 1 - i)])
    l3 = np.array([j / n for i in range(n + 1) for j in range(n + 1 - i)])
    l2 = 1.0 - l1 - l3
    x, y = -l2 + l3, (-l2 - l3 + 2 * l1) / math.sqrt(3.0)
    for k, (la, lb, lc) in enumerate(((l1, l2, l3), (l2, l3, l1), (l3, l1, l2))):
        w = 4 * lb * lc * _warp(n, lc - lb) * (1 + (alpha * la) ** 2)
        x = x + math.cos(2 * math.pi * k / 3) * w
        y = y + math.sin(2 * math.pi * k / 3) * w
    m1 = (math.sqrt(3.0) * y + 1.0) / 3.0
    m2 = (-3.0 * x - math.sqrt(3.0) * y + 2.0) / 6.0
    m3 = (3.0 * x - math.sqrt(3.0) * y + 2.0) / 6.0
    r, s = -m2 + m3 - m1, -m2 - m3 + m1
    top = np.abs(1 - s) < 1e-13
    a = np.where(top, -1.0, 2 * (1 + r) / np.where(top, 1.0, 1 - s) - 1)
    V, Vr, Vs = [], [], []
    for i in range(n + 1):
        for j in range(n + 1 - i):
            fa, dfa, gb, dgb = _jacobi(a, 0, 0, i), _djacobi(a, 0, 0, i), _jacobi(s, 2 * i + 1, 0, j), _djacobi(s, 2 * i + 1, 0, j)
            h = 0.5 * (1 - s)
            V.append(math.sqrt(2.0) * fa * gb * (1 - s) ** i)
            low = h ** (i - 1) if i > 0 else np.ones_like(s)
            Vr.append(2 ** (i + 0.5) * dfa * gb * low)
            tmp = dgb * h ** i - (0.5 * i * gb * low if i > 0 else 0.0)
            Vs.append(2 ** (i + 0.5) * (dfa * gb * 0.5 * (1 + a) * low + fa * tmp))
    V, Vr, Vs = (np.stack(c, axis=1) for c in (V, Vr, Vs))
    mass = np.linalg.inv(V @ V.T)
    face = [np.nonzero(np.abs(s + 1) < 1e-10)[0], np.nonzero(np.abs(r + s) < 1e-10)[0],
            np.nonzero(np.abs(r + 1) < 1e-10)[0][::-1]]
    E, wq = np.zeros((len(r), 3 * (n + 1))), None
    for f, (idx, c) in enumerate(zip(face, (r, r, s))):
        v1 = np.stack([_jacobi(c[idx], 0, 0, j) for j in range(n + 1)], axis=1)
        m = np.linalg.inv(v1 @ v1.T)
        E[idx, f * (n + 1):(f + 1) * (n + 1)] = m
        wq = m.sum(axis=1) if f == 0 else wq
    return {"rs": (r, s), "Drw": V @ Vr.T @ mass, "Dsw": V @ Vs.T @ mass, "LIFT": V @ (V.T @ E),
            "fmask": np.concatenate(face), "wq": wq}


class _Plain:
    """The discretisation on one mesh in torch FP64: dense operators, gathered face traces."""

    def __init__(self, tables, order):
        coords, cells, types = tables
        T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
        o = _operators(order)
        self.N, self.K, self.Np, self.nfp = order, len(cells), _np(order), order + 1
        self.A = T(np.concatenate([o["Drw"], o["Dsw"], -o["LIFT"]], axis=1))
        self.fmask, self.wq = T(o["fmask"]), T(o["wq"])
        r, s = (T(v) for v in o["rs"])
        v = T(coords[cells])
        self.x = 0.5 * (-(r + s) * v[:, :1, 0] + (1 + r) * v[:, 1:2, 0] + (1 + s) * v[:, 2:3, 0])
        self.y = 0.5 * (-(r + s) * v[:, :1, 1] + (1 + r) * v[:, 1:2, 1] + (1 + s) * v[:, 2:3, 1])
        e1, e2 = 0.5 * (v[:, 1] - v[:, 0]), 0.5 * (v[:, 2] - v[:, 0])
        xr, yr, xs, ys = e1[:, 0], e1[:, 1], e2[:, 0], e2[:, 1]
        J = xr * ys - xs * yr
        self.met = [(m / J)[:, None] for m in (ys, -xs, -yr, xr)]  # rx, ry, sx, sy
        nx, ny = torch.stack([yr, ys - yr, -ys], 1), torch.stack([-xr, xr - xs, xs], 1)
        sj = torch.sqrt(nx * nx + ny * ny)
        rep = lambda a: a.repeat_interleave(self.nfp, dim=1)  # noqa: E731
        self.nx, self.ny, self.fs, self.sj = rep(nx / sj), rep(ny / sj), rep(sj / J[:, None]), rep(sj)
        # the face's fscale that the time-step estimate multiplies a face point's speed with
        idx = o["fmask"] // self.nfp if self.Np <= 3 * self.nfp else np.arange(3 * self.nfp) // self.nfp
        self.dtfs = (sj / J[:, None])[:, T(idx)]
        # neighbours: the two cells of an edge walk it in opposite directions
        a, b = cells, cells[:, [1, 2, 0]]
        key = (np.minimum(a, b).astype(np.int64) * len(coords) + np.maximum(a, b)).ravel()
        order_ = np.argsort(key, kind="stable")
        same = np.nonzero(key[order_][1:] == key[order_][:-1])[0]
        other = np.full(key.size, -1, dtype=np.int64)
        p, q = order_[same], order_[same + 1]
        other[p], other[q] = q, p
        edge = np.nonzero(other < 0)[0]
        nb = np.where(other < 0, np.arange(key.size), other).reshape(-1, 3)
        node = o["fmask"].reshape(3, self.nfp)[:, ::-1]
        gather = (nb // 3)[:, :, None] * self.Np + node[nb % 3]
        self.gather = T(gather.reshape(self.K, -1))
        c, f = edge // 3, edge % 3
        self.bc, self.bj = T(np.repeat(c, self.nfp)), T((f[:, None] * self.nfp + np.arange(self.nfp)).ravel())
        pairs = np.stack([cells[c, f], cells[c, (f + 1) % 3]], axis=1)
        self.btype = T(np.repeat(types(pairs) if types is not None else np.zeros(len(pairs), np.int32), self.nfp))
        self.bnode = self.fmask[self.bj]

    def traces(self, q):
        return q[:, self.fmask], q.reshape(self.K * self.Np, -1)[self.gather]


def _euler_flux(q):
    rho, mu, mv, e = q.unbind(-1)
    u, v = mu / rho, mv / rho
    p = (_GAM - 1) * (e - 0.5 * (mu * u + mv * v))
    return rho, u, v, p, torch.stack([mu, mu * u + p, mv * u, u * (e + p)], -1), \
        torch.stack([mv, mu * v, mv * v + p, v * (e + p)], -1)


def _roe(qm, qp, nx, ny):
    def turn(q):
        return torch.stack([q[..., 0], nx * q[..., 1] + ny * q[..., 2], nx * q[..., 2] - ny * q[..., 1], q[..., 3]], -1)
    qm, qp = turn(qm), turn(qp)
    rl, ul, vl, pl, fl, _ = _euler_flux(qm)
    rr, ur, vr, pr, fr, _ = _euler_flux(qp)
    hl, hr = (qm[..., 3] + pl) / rl, (qp[..., 3] + pr) / rr
    sl, sr = torch.sqrt(rl), torch.sqrt(rr)
    rho, t = sl * sr, sl + sr
    u, v, h = (sl * ul + sr * ur) / t, (sl * vl + sr * vr) / t, (sl * hl + sr * hr) / t
    c2 = (_GAM - 1) * (h - 0.5 * (u * u + v * v))
    c = torch.sqrt(c2)
    w1 = torch.abs(u - c) * (0.5 * (pr - pl) / c2 - 0.5 * rho * (ur - ul) / c)
    w4 = torch.abs(u + c) * (0.5 * (pr - pl) / c2 + 0.5 * rho * (ur - ul) / c)
    w2 = torch.abs(u) * ((rr - rl) - (pr - pl) / c2)
    w3 = torch.abs(u) * rho * (vr - vl)
    d = torch.stack([w1 + w2 + w4, w1 * (u - c) + w2 * u + w4 * (u + c), (w1 + w2 + w4) * v + w3,
                     w1 * (h - u * c) + w2 * (u * u + v * v) + w3 * v + w4 * (h + u * c)], -1)
    f = 0.5 * (fl + fr - d)
    return torch.stack([f[..., 0], nx * f[..., 1] - ny * f[..., 2], ny * f[..., 1] + nx * f[..., 2], f[..., 3]], -1)


def _vortex_state(x, y, t, beta, x0, y0):
    e = torch.exp(1.0 - ((x - t - x0) ** 2 + (y - y0) ** 2))
    u, v = 1.0 - beta * e * (y - y0) / (2 * math.pi), beta * e * (x - x0) / (2 * math.pi)
    rho = (1.0 - (_GAM - 1) / (16 * _GAM * math.pi ** 2) * beta ** 2 * e * e) ** (1.0 / (_GAM - 1))
    return torch.stack([rho, rho * u, rho * v, rho ** _GAM / (_GAM - 1) + 0.5 * rho * (u * u + v * v)], -1)


class _Freestream:
    def __init__(self, mach, alpha):
        """alpha in degrees, a number or a tensor"""
        alpha = torch.as_tensor(alpha, dtype=torch.float64, device="cuda") * (math.pi / 180.0)
        V = math.sqrt(_GAM) * mach
        self.u, self.v, self.speed, self.alpha = V * torch.cos(alpha), V * torch.sin(alpha), V, alpha
        self.state = torch.stack([torch.ones_like(self.u), self.u, self.v,
                                  torch.ones_like(self.u) * (1.0 / (_GAM - 1) + 0.5 * V * V)])

    def ghost(self, kind, q, nx, ny):
        inf = self.state.expand_as(q)
        rho, u, v, p, _, _ = _euler_flux(q)
        c = torch.sqrt(_GAM * p / rho)
        vn, cinf = u * nx + v * ny, math.sqrt(_GAM)
        vinf = self.u * nx + self.v * ny
        rp, rm = vn + 2 * c / (_GAM - 1), vinf - 2 * cinf / (_GAM - 1)
        vb, cb = 0.5 * (rp + rm), 0.25 * (_GAM - 1) * (rp - rm)
        out = vb > 0
        ent = torch.where(out, p / rho ** _GAM, torch.ones_like(p))
        ut, vt = torch.where(out, u - vn * nx, self.u - vinf * nx), torch.where(out, v - vn * ny, self.v - vinf * ny)
        rb = (cb * cb / (_GAM * ent)) ** (1.0 / (_GAM - 1))
        pb, ub, wb = rb * cb * cb / _GAM, ut + vb * nx, vt + vb * ny
        far = torch.stack([rb, rb * ub, rb * wb, pb / (_GAM - 1) + 0.5 * rb * (ub * ub + wb * wb)], -1)
        far = torch.where((vn <= -c)[:, None], inf, torch.where((vn >= c)[:, None], q, far))
        mn = 2 * (nx * q[:, 1] + ny * q[:, 2])
        wall = torch.stack([q[:, 0], q[:, 1] - mn * nx, q[:, 2] - mn * ny, q[:, 3]], -1)
        outflow = torch.cat([inf[:, :3], q[:, 3:]], -1)
        k = kind[:, None]
        return torch.where(k == 0, inf, torch.where(k == 1, outflow, torch.where(k == 2, wall, far)))


def _rhs(P, q, ghost):
    """ghost(q at the boundary face nodes) -> the exterior states there"""
    rx, ry, sx, sy = (m[..., None] for m in P.met)
    _, _, _, _, F, G = _euler_flux(q)
    qm, qp = P.traces(q)
    qp = qp.index_put((P.bc, P.bj), ghost(q[P.bc, P.bnode]))
    flux = _roe(qm, qp, P.nx, P.ny) * P.fs[..., None]
    return torch.matmul(P.A, torch.cat([rx * F + ry * G, sx * F + sy * G, flux], dim=1))


def _dt(P, q, cfl):
    rho, u, v, p, _, _ = _euler_flux(q[:, P.fmask])
    speed = torch.sqrt(u * u + v * v) + torch.sqrt(_GAM * p / rho)
    return float(cfl / (0.5 * (P.N + 1) ** 2 * P.dtfs * speed).max())


def _step(P, q, dt, t, ghost):
    """One SSPRK3 step; ghost(boundary states, time)"""
    w = q + dt * _rhs(P, q, lambda b: ghost(b, t))
    w = 0.75 * q + 0.25 * (w + dt * _rhs(P, w, lambda b: ghost(b, t + dt)))
    return q / 3.0 + 2.0 / 3.0 * (w + dt * _rhs(P, w, lambda b: ghost(b, t + 0.5 * dt)))


def _ghosts(P, cfg):
    if cfg["app"] == 1:
        bx, by = P.x[P.bc, P.bnode], P.y[P.bc, P.bnode]
        return lambda b, t: _vortex_state(bx, by, t, cfg["vortex_beta"], cfg["vortex_x0"], cfg["vortex_y0"])
    fs = cfg["freestream"]
    bnx, bny = P.nx[P.bc, P.bj], P.ny[P.bc, P.bj]
    return lambda b, t: fs.ghost(P.btype, b, bnx, bny)


def _initial(P, cfg):
    if cfg["app"] == 1:
        return _vortex_state(P.x, P.y, 0.0, cfg["vortex_beta"], cfg["vortex_x0"], cfg["vortex_y0"])
    return cfg["freestream"].state.expand(P.K, P.Np, 4)


def _plain_run(tables, cfg, steps):
    """q, t and the next dt after the steps"""
    P = _Plain(tables, cfg["N"])
    cfg = dict(cfg)
    if cfg["app"] == 0:
        cfg["freestream"] = _Freestream(cfg["mach"], cfg["alpha_deg"])
    q, t = _initial(P, cfg).contiguous(), 0.0
    ghost = _ghosts(P, cfg)
    dt = _dt(P, q, cfg["cfl"])
    for _ in range(steps):
        q = _step(P, q, dt, t, ghost)
        t += dt
        dt = _dt(P, q, cfg["cfl"])
    return q, t, dt


def _plain_gradient(tables, cfg, case):
    """J, dJ/dparameter and dJ/dq0 with the dt sequence held, by autograd (a step at a time)"""
    from torch.utils.checkpoint import checkpoint
    P = _Plain(tables, cfg["N"])
    cfg = dict(cfg)
    vortex = cfg["app"] == 1
    par = torch.tensor(cfg["vortex_beta"] if vortex else cfg["alpha_deg"], dtype=torch.float64, device="cuda",
                       requires_grad=True)
    if vortex:
        cfg["vortex_beta"] = par
    else:
        cfg["freestream"] = _Freestream(cfg["mach"], par)
    q0 = _initial(P, cfg) + 0.0
    q0.retain_grad()
    ghost = _ghosts(P, cfg)
    wall = torch.nonzero(P.btype == 2)[:, 0]
    wc, wj, wn = P.bc[wall], P.bj[wall], P.bnode[wall]

    def lift(q):
        fs = cfg["freestream"]
        _, _, _, p, _, _ = _euler_flux(q[wc, wn])
        n = -P.nx[wc, wj] * torch.sin(fs.alpha) + P.ny[wc, wj] * torch.cos(fs.alpha)
        return (P.wq[wj % P.nfp] * P.sj[wc, wj] * p * n).sum() / (0.5 * fs.speed ** 2)

    q, t, J = q0, 0.0, 0.0
    with torch.no_grad():
        dt = _dt(P, q, cfg["cfl"])
    for k in range(case["steps"]):
        q = checkpoint(lambda a, dt=dt, t=t: _step(P, a, dt, t, ghost), q, use_reentrant=False)
        t += dt
        if not vortex:
            if k + 1 > case["steps"] - case["navg"]:
                J = J + lift(q) / case["navg"]
            with torch.no_grad():
                dt = _dt(P, q, cfg["cfl"])
    if vortex:
        J = ((q - _vortex_state(P.x, P.y, t, par, cfg["vortex_x0"], cfg["vortex_y0"])) ** 2).sum()
    J.backward()
    return float(J.detach()), float(par.grad), q0.grad.reshape(-1)


def _plain_advection(tables, order, vel, dt, steps):
    P = _Plain(tables, order)
    q = torch.exp(-40.0 * (P.x - 0.5) ** 2) * torch.exp(-40.0 * (P.y - 0.5) ** 2)
    rx, ry, sx, sy = P.met
    speed, vn = math.hypot(*vel), vel[0] * P.nx + vel[1] * P.ny

    def rhs(w):
        wm, wp = P.traces(w[..., None])
        wm, wp = wm[..., 0], wp[..., 0].index_put((P.bc, P.bj), torch.tensor(4.5e-5, dtype=torch.float64, device="cuda"))
        flux = 0.5 * (vn * (wm + wp) + speed * (wm - wp)) * P.fs
        return torch.matmul(torch.cat([(vel[0] * rx + vel[1] * ry) * w, (vel[0] * sx + vel[1] * sy) * w, flux], dim=1), P.A.T)
    for _ in range(steps):
        k1 = rhs(q)
        k2 = rhs(q + 0.5 * dt * k1)
        k3 = rhs(q + 0.5 * dt * k2)
        k4 = rhs(q + dt * k3)
        q = q + dt / 6.0 * (k1 + 2 * k2 + 2 * k3 + k4)
    return q


def exact(case, seed):
    kind = case["kind"]
    if kind == "rhs":
        alpha, mach = _flow(seed)
        tables = _ogrid(case["n_theta"], case["n_r"], "characteristic")
        P = _Plain(tables, case["order"])
        ghost = _ghosts(P, {"app": 0, "freestream": _Freestream(mach, alpha)})
        return _rhs(P, _disturbed(tables, case["order"], mach, alpha, seed), lambda b: ghost(b, 0.0))
    if kind in ("run", "host"):
        tables, cfg = _instance(case, seed)
        q, t, dt = _plain_run(tables, cfg, case["steps"] if kind == "run" else _HOST_START + 1)
        return (q, np.array([t, dt])) if kind == "run" else q.reshape(-1)
    if kind == "batch":
        got = [_plain_run(t, c, case["steps"]) for t, c in _sweep(case, seed)]
        return [q.reshape(-1) for q, _, _ in got], np.array([dt for _, _, dt in got])
    if kind == "gradient":
        got = [_plain_gradient(*_instance(case, seed, k), case) for k in range(case["count"])]
        return np.array([g[0] for g in got] + [g[1] for g in got]), [g[2] for g in got]
    if kind == "dropin":
        turn = float(np.random.default_rng(seed).uniform(-0.1, 0.1))
        tables = _ogrid(case["n_theta"], case["n_r"], "reference", turn)
        q, _, dt = _plain_run(tables, dict(N=case["order"], app=0, cfl=1.0, mach=0.4, alpha_deg=0.0), case["steps"])
        return q.reshape(-1), np.array([dt])
    tables, vel, dt = _advection_instance(case, seed)
    return _plain_advection(tables, case["order"], vel, dt, case["steps"]).reshape(-1)
