"""What a user of the library has it do, as cases that can be timed.

A host code keeps its octree state in (pinned) host memory or in a device
table of EOS points, hands it to the library, advances it and takes the
result back, as the reference's drivers do through the C ABI:

  euler   gas dynamics on an octree of 8^3 bricks, no gravity: whole RK3
          steps through hydro_step (with its regrid check), or call by call
          through sub_step or fused_sub_step
  star    the self-gravitating n = 1.5 polytrope: RK3 steps with a multigrid
          solve in every substep, in the plain, graph and persistent forms
  solve   one Poisson solve of that star from a zero potential
  binary  the ZTWD binary (13 fields, PPM, Helmholtz EOS, rotating frame):
          BinaryDriver steps on 12^3 or 8^3 bricks
  eos     the batched Helmholtz EOS on device arrays: (rho, T) -> (p, e, cs)
          and the Newton inversion for T

The tree cases upload the state they start from, advance it and download it
in every pass, so each pass does the same work.  Returned states are the
interiors of the bricks: edge and corner ghosts are never written, and face
ghosts are copies of interiors.
"""

import ctypes
import importlib.util
import json
import math
import os
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "3d-eulerian-amr_b200")


def _module(name):
    spec = importlib.util.spec_from_file_location("perf_" + name, os.path.join(PKG, name + ".py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


amr = _module("amr")
initial = _module("initial")
helm = _module("helm")
helm_table = _module("helm_table")

DYNAMIC_RANGE = 1.0e6
MAXDTINC = 1.25
GAMMA = 5.0 / 3.0


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a first look at a small problem: 5 steps of a two-level moving bump,
        # the tree adapting as it goes; a handful of bricks, so every launch,
        # synchronisation and the host's octree work count
        dict(name="hydro-adaptive-small", kind="euler", field="bump", level=2, cut=3.0, recon="minmod",
             prec="fp64", call="hydro_step", adapt=True, steps=5),
        # a production-like gas run with the PPM build's bricks (BW 3)
        dict(name="hydro-ppm", kind="euler", field="bump", level=4, cut=2.0, recon="ppm", prec="fp64",
             call="hydro_step", adapt=False, steps=16),
        # an uneven octree of a turbulent density field, call by call, as a
        # driver that keeps the reference's own sequence does
        dict(name="hydro-substeps", kind="euler", field="modes", level=3, cut=3.6, recon="minmod", prec="fp64",
             call="sub_step", adapt=False, steps=20),
        # the same kind of field at scale through the fused substep, FP64
        dict(name="fused-large", kind="euler", field="modes", level=5, cut=5.0, recon="minmod", prec="fp64",
             call="fused", adapt=False, steps=24),
        # ... and a mid-sized one with the FP32 reconstruction and flux
        dict(name="fused-mixed", kind="euler", field="modes", level=4, cut=4.5, recon="minmod", prec="mixed",
             call="fused", adapt=False, steps=32),
        # the default configuration on a small star: FP64, host-driven loops
        dict(name="star-plain-small", kind="star", level=2, form="plain", prec="fp64", steps=1),
        # the four-level star in the fastest form
        dict(name="star-mixed", kind="star", level=4, form="persistent", prec="mixed", steps=6),
        # a cold FP64 solve of that star to a tight tolerance
        dict(name="solve-fp64", kind="solve", level=4, form="persistent", prec="fp64", tol=1.0e-8),
        # the five-level white-dwarf binary on the BINARY build's 12^3 bricks
        dict(name="binary-mixed", kind="binary", nx=12, level=5, form="persistent", prec="mixed_solve", steps=1),
        # a coarser binary in the reference-order FP64 form
        dict(name="binary-plain", kind="binary", nx=12, level=3, form="plain", prec="fp64", steps=1),
        # EOS post-processing of a large particle or cell set
        dict(name="eos-forward", kind="eos", call="forward", n=1 << 24, units="cgs"),
        # temperatures of an odd-sized set from its energies
        dict(name="eos-newton", kind="eos", call="newton", n=3000001, units="cgs"),
    ]


def draw(rng):
    """One more case of the ranges above: tree sizes from a few bricks to
    about ten thousand, point counts from a thousand to 2^24."""
    kind = rng.choice(["euler", "euler", "euler", "star", "solve", "binary", "eos", "eos"])
    if kind == "euler":
        recon = rng.choice(["minmod", "minmod", "ppm"])
        call = "hydro_step" if recon == "ppm" else rng.choice(["hydro_step", "sub_step", "fused"])
        field = rng.choice(["bump", "modes"])
        level = rng.randint(1, 4)
        cut = round(rng.uniform(1.7, 5.0), 3)
        adapt = call == "hydro_step" and field == "bump" and level <= 3 and rng.random() < 0.5
        return dict(kind="euler", field=field, level=level, cut=cut, recon=recon,
                    prec="mixed" if rng.random() < 0.3 else "fp64", call=call, adapt=adapt,
                    steps=rng.randint(3, 12))
    if kind == "star":
        form = rng.choice(["plain", "graph", "persistent"])
        return dict(kind="star", level=rng.randint(1, 3 if form == "plain" else 4), form=form,
                    prec="fp64" if form == "plain" else rng.choice(["fp64", "mixed", "mixed_solve"]),
                    steps=rng.randint(1, 2 if form == "plain" else 4))
    if kind == "solve":
        return dict(kind="solve", level=rng.randint(2, 4), form=rng.choice(["graph", "persistent"]),
                    prec=rng.choice(["fp64", "mixed"]), tol=float("%.3g" % 10.0 ** rng.uniform(-7.0, -5.0)))
    if kind == "binary":
        form = rng.choice(["plain", "persistent", "persistent"])
        return dict(kind="binary", nx=rng.choice([8, 12]), level=rng.randint(2, 3 if form == "plain" else 4),
                    form=form, prec="fp64" if form == "plain" else rng.choice(["fp64", "mixed", "mixed_solve"]),
                    steps=rng.randint(1, 2))
    call = rng.choice(["forward", "newton"])
    top = 24.0 if call == "forward" else 22.0
    return dict(kind="eos", call=call, n=int(2.0 ** rng.uniform(10.0, top)) | 1, units=rng.choice(["cgs", "code"]))


# ---------------------------------------------------------------------------
# trees and states
# ---------------------------------------------------------------------------
PREC = {"fp64": 0, "mixed": 1, "mixed_solve": 2}
FIXED = 1 << 30  # min_grid_life of a fixed tree: no brick ever gets old enough to go


def _config(case):
    kind = case["kind"]
    prec = PREC[case["prec"]]
    pers = 2 if case.get("form") == "persistent" else 0
    if kind == "euler":
        cfg = dict(physics=amr.PHYSICS_EULER, max_refine_level=case["level"], grid_dim=0.5, z_reflect=0,
                   precision=prec)
        if case["recon"] == "ppm":
            cfg.update(bw=3, reconstruction=amr.RECON_PPM)
        if not case["adapt"]:
            cfg.update(min_grid_life=FIXED)
        return cfg
    if kind in ("star", "solve"):
        return dict(physics=amr.PHYSICS_EULER_GRAVITY, max_refine_level=case["level"], grid_dim=0.5, z_reflect=0,
                    precision=prec, persistent_solve=pers, min_grid_life=FIXED)
    return dict(physics=amr.PHYSICS_ZTWD, nf=13, bw=3, nx=case["nx"], reconstruction=amr.RECON_PPM, grid_dim=1.0,
                z_reflect=1, mirror_refine_y=1, max_refine_level=case["level"],
                rho_floor=initial.BINARY["rho_floor"], cfl=0.3, maxdtinc=MAXDTINC, precision=prec,
                persistent_solve=pers, min_grid_life=FIXED)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _centres(tree, nx, grid_dim, z_reflect):
    """Cell centres of the interiors: three broadcastable [n, nx, nx, nx] tensors."""
    dev = _device()
    h = torch.from_numpy(tree["h"]).to(dev)[:, None]
    off = torch.from_numpy(tree["offset"].astype(np.float64)).to(dev)
    i = torch.arange(nx, dtype=torch.float64, device=dev)[None, :]
    out = []
    for d in range(3):
        x = (off[:, d:d + 1] + i + 0.5) * h - (0.0 if d == 2 and z_reflect else grid_dim)
        shape = [x.shape[0], 1, 1, 1]
        shape[3 - d] = nx
        out.append(x.reshape(shape))
    return out


def _modes(seed, count, kmax, slope, X):
    """A sum of plane waves with amplitudes falling as a power of the
    wavenumber, scaled to unit variance."""
    rs = np.random.RandomState(seed)
    total, power = 0.0, 0.0
    for _ in range(count):
        k = rs.randint(-kmax, kmax + 1, 3)
        kk = max(1.0, math.sqrt(float((k * k).sum())))
        a, p = kk ** slope, rs.uniform(0.0, 2.0 * math.pi)
        total = total + a * torch.cos(2.0 * math.pi * (k[0] * X[0] + k[1] * X[1] + k[2] * X[2]) + p)
        power += 0.5 * a * a
    return total / math.sqrt(power)


def _euler_density(case, X):
    if case["field"] == "bump":  # the moving bump: a Gaussian off the centre
        r2 = (X[0] - 0.08) ** 2 + (X[1] + 0.05) ** 2 + (X[2] - 0.06) ** 2
        return 1.0 + 9.0 * torch.exp(-r2 / (0.15 * 0.15))
    return torch.exp(_modes(20261203, 40, 8, -1.5, X))  # log-normal, sigma 1


def _octant_flags(rho, cut):
    n, nx = rho.shape[0], rho.shape[1]
    h = nx // 2
    dense = (rho > cut).reshape(n, 2, h, 2, h, 2, h).permute(0, 1, 3, 5, 2, 4, 6).reshape(n, 8, -1).any(2)
    return dense.to(torch.uint8).cpu().numpy()  # octant = x | y << 1 | z << 2


_BASES = {}


def _base(case):
    """Tree (and, where the library's initial data give it, the state) that a
    case's inputs of every seed start from."""
    key = json.dumps({k: v for k, v in case.items() if k not in ("name", "steps", "call", "prec", "form", "tol")},
                     sort_keys=True) + ("solve" if case["kind"] == "solve" else "")
    if key in _BASES:
        return _BASES[key]
    cfg = _config(case)
    host = amr.AMR(max_bricks=0, **cfg)
    base = {}
    if case["kind"] == "euler":
        host.init()
        host.set_time(0.0)
        for _ in range(case["level"]):
            rho = _euler_density(case, _centres(host.get_tree(), host.nx, 0.5, 0))
            host.refine_from_flags(_octant_flags(rho, case["cut"]), True)
    elif case["kind"] in ("star", "solve"):
        _, U = initial.build_tree(host, "polytrope", 1.0e-6, 0.5, 0, case["level"], device=False, ghosts=False)
        base["U"] = np.ascontiguousarray(U[:, :, 2:-2, 2:-2, 2:-2])
    else:
        host.init()
        U = initial.evaluate("binary", host.get_tree(), 3, case["nx"], 1.0, 1, case["level"], ghosts=False)
        _, U = initial.build_tree(host, "binary", float(U[:, 0].max()) / DYNAMIC_RANGE, 1.0, 1, case["level"],
                                  device=False, ghosts=False)
        base["U"] = np.ascontiguousarray(U[:, :, 3:-3, 3:-3, 3:-3])
    base["tree"] = host.get_tree()
    host.close()
    if len(_BASES) >= 4:
        _BASES.pop(next(iter(_BASES)))
    _BASES[key] = base
    return base


def _interior(case, base, seed):
    """Interior state of every brick for one seed: the base density with a
    smooth few-per-cent perturbation of that seed, and its motion."""
    tree, dev = base["tree"], _device()
    if case["kind"] == "euler":
        X = _centres(tree, 8, 0.5, 0)
        f = 1.0 + 0.03 * _modes(seed % (1 << 31), 6, 4, -1.0, X).clamp(-3.0, 3.0)
        rho = _euler_density(case, X)
        if not case["adapt"]:  # an adaptive tree follows the same density whatever the seed
            rho = rho * f
        gen = torch.Generator(device=dev).manual_seed(seed)
        if case["field"] == "bump":
            v = [torch.full_like(rho, 0.4), torch.full_like(rho, 0.25),
                 (-0.15 + 0.1 * torch.sin(2.0 * math.pi * X[0])).expand_as(rho)]
            ei = torch.full_like(rho, 0.6 / (GAMMA - 1.0)) * f
        else:  # cell-wise random velocities
            v = [0.1 * torch.randn(rho.shape, generator=gen, dtype=torch.float64, device=dev) for _ in range(3)]
            ei = rho ** GAMMA / (GAMMA - 1.0)
        ek = 0.5 * rho * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2])
        return torch.stack([rho, rho * v[0], rho * v[1], rho * v[2], ei + ek, ei ** (1.0 / GAMMA)], 1)
    U = torch.from_numpy(base["U"]).to(dev)
    zt = case["kind"] == "binary"
    X = _centres(tree, U.shape[-1], 1.0 if zt else 0.5, 1 if zt else 0)
    f = 1.0 + 0.03 * _modes(seed % (1 << 31), 6, 3, -1.0, X).clamp(-3.0, 3.0)
    if zt:
        for l in (0, 1, 2, 4, 10, 11, 12):  # densities, and lz at the same rotation
            U[:, l] *= f
        return U
    U[:, :5] *= f[:, None]
    U[:, 5] *= f ** (1.0 / GAMMA)
    return U


def _pinned(count):
    return torch.empty(count, dtype=torch.float64, pin_memory=True)


def _ptr(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


class _Run:
    """A context with its tree, and the host's copies of state and potential."""

    def __init__(self, case, seed):
        self.case = case
        base = _base(case)
        t = base["tree"]
        room = 4 * t["level"].size + 64 if case["kind"] == "euler" and case["adapt"] else t["level"].size + 8
        self.a = a = amr.AMR(max_bricks=room, **_config(case))
        if case["kind"] == "binary":
            P = initial.binary_params()
            a.ztwd_set_eos(_helm("binary"))
            a.ztwd_set_frame(P["omega"], P["omega"], 0.0, 0.0)
        a.load_tree(t["level"], t["loc"], np.zeros(t["level"].size, np.int32))
        a.set_time(1.0)
        if case["kind"] == "binary" and case["form"] == "persistent" and case["nx"] == 12:
            a.set_solve_layout(1, 1)  # what the library's autotuner keeps for these bricks
        g, b = a.gnx, a.bw
        full = torch.zeros((a.nbricks, a.nf, g, g, g), dtype=torch.float64, device="cuda")
        full[:, :, b:-b, b:-b, b:-b] = _interior(case, base, seed)
        a.upload_state(full.cpu().numpy())
        del full
        a.inject_from_children()
        a.enforce_boundaries()
        self.P = self.oP = None
        if case["kind"] in ("star", "binary"):
            self.step(0, 1.0)  # the first step, with its cold solve; no cell asks for a new brick
        self.tree = a.get_tree()
        n = a.nbricks
        cap = room if case["kind"] == "euler" and case["adapt"] else n
        self.U, self.oU = _pinned(n * a.nf * g ** 3), _pinned(cap * a.nf * g ** 3)
        a._check(a.lib.amr_download_state(a.ctx, _ptr(self.U)))
        if case["kind"] != "euler":
            self.P, self.oP = _pinned(8 * n * a.pnx ** 3), _pinned(8 * n * a.pnx ** 3)
            if case["kind"] == "solve":
                self.P.zero_()
            else:
                a._check(a.lib.amr_download_poisson(a.ctx, _ptr(self.P)))

    def step(self, index, dynamic_range=DYNAMIC_RANGE):
        a, c = self.a, self.case
        if c["kind"] == "star":
            if c["form"] == "plain":
                dt = a.max_dt()
                a.grav_step(dt, 1.0e-6, dynamic_range, index)
                return dt
            return a.graph_grav_step(1.0e-6, dynamic_range, index)
        return a.ztwd_step(a.max_dt(), 1.0e-7, dynamic_range, index)

    def hydro(self):
        a, c = self.a, self.case
        last, dts = 0.0, []
        for s in range(c["steps"]):
            dt = a.max_dt()
            last = dt if s == 0 else min(MAXDTINC * last, dt)
            dts.append(last)
            if c["call"] == "hydro_step":
                # a fixed tree asks for no new brick; an adaptive one follows the density
                a.hydro_step(last, c["cut"] if c["adapt"] else 1.0e30)
                continue
            a.store()
            for beta in (1.0, 0.25, 2.0 / 3.0):
                if c["call"] == "fused":
                    a.fused_sub_step(last, beta)
                else:
                    a.sub_step(last, beta)
                a.inject_from_children()
            a.enforce_boundaries()
        return dts

    def one(self):
        a, c = self.a, self.case
        if c["kind"] == "euler" and c["adapt"]:
            a.load_tree(self.tree["level"], self.tree["loc"], self.tree["age"])
            a.set_time(1.0)
        if c["kind"] != "solve":
            a._check(a.lib.amr_upload_state(a.ctx, _ptr(self.U)))
        if self.P is not None:
            a._check(a.lib.amr_upload_poisson(a.ctx, _ptr(self.P)))
        out = {}
        if c["kind"] == "solve":
            out["err"], out["cycles"] = a.graph_solve(c["tol"], 10000)
        elif c["kind"] == "euler":
            out["dt"] = np.array(self.hydro())
        else:
            out["dt"] = np.array([self.step(s) for s in range(1, c["steps"] + 1)])
        n, g, b = a.nbricks, a.gnx, a.bw
        if c["kind"] != "solve":
            a._check(a.lib.amr_download_state(a.ctx, _ptr(self.oU)))
            U = self.oU[:n * a.nf * g ** 3].view(n, a.nf, g, g, g)
            out["U"] = U[:, :, b:-b, b:-b, b:-b]
        if self.P is not None:
            a._check(a.lib.amr_download_poisson(a.ctx, _ptr(self.oP)))
            out["phi"] = self.oP.view(8, n, a.pnx, a.pnx, a.pnx)[0, :, 1:-1, 1:-1, 1:-1]
        return out


# ---------------------------------------------------------------------------
# the EOS
# ---------------------------------------------------------------------------
_HELMS = {}
# code units of the "code" cases: cm, g, s, K of one code unit
CODE_UNITS = (6.0e9, 2.0e31, 10.0, 1.0)


def _helm(units):
    """The EOS handle a program keeps: the table in cgs, in code units, or in
    the binary's units."""
    if units not in _HELMS:
        folder = os.path.join(tempfile.gettempdir(), "helm_table_%d" % os.getuid())
        h = helm.Helm(helm_table.ensure_table(folder))
        if units == "code":
            h.set_cgs_units(*CODE_UNITS)
        elif units == "binary":
            P = initial.binary_params()
            h.set_cgs_units(P["cm"], P["g"], P["s"], 1.0)
        _HELMS[units] = h
    return _HELMS[units]


def _points(case, seed):
    """rho log-uniform in [1e-2, 1e9] g/cm^3, T in [1e4, 1e9] K, abar uniform
    in [12, 16], zbar = abar / 2; and a guess for T within half a decade."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = lambda lo, hi: lo + (hi - lo) * torch.rand(case["n"], dtype=torch.float64, device="cuda", generator=g)
    rho, T, abar = torch.pow(10.0, u(-2.0, 9.0)), torch.pow(10.0, u(4.0, 9.0)), u(12.0, 16.0)
    guess = T * torch.pow(10.0, u(-0.5, 0.5))
    if case["units"] == "code":
        cm, gr, _, K = CODE_UNITS
        rho, T, guess = rho / (gr / cm ** 3), T / K, guess / K
    return rho, T, abar, abar / 2.0, guess


class _Eos:
    def __init__(self, case, seed):
        self.case, self.h = case, _helm(case["units"])
        self.rho, T, self.abar, self.zbar, self.guess = _points(case, seed)
        new = lambda: torch.empty_like(self.rho)
        self.p, self.e, self.cs = new(), new(), new()
        self.status = torch.empty(case["n"], dtype=torch.int32, device="cuda")
        self.T = T
        if case["call"] == "newton":
            self.h.eos_device(self.rho, T, self.abar, self.zbar, self.p, self.e, self.cs, self.status,
                              stream=torch.cuda.current_stream().cuda_stream)
            self.T, self.iters = new(), torch.empty_like(self.status)

    def one(self):
        stream = torch.cuda.current_stream().cuda_stream
        if self.case["call"] == "forward":
            self.h.eos_device(self.rho, self.T, self.abar, self.zbar, self.p, self.e, self.cs, self.status,
                              stream=stream)
            return {"p": self.p, "e": self.e, "cs": self.cs, "status": self.status}
        self.T.copy_(self.guess)
        self.h.invert_T_device(self.rho, self.e, self.abar, self.zbar, self.T, self.status, iters=self.iters,
                               stream=stream)
        return {"T": self.T, "iters": self.iters, "status": self.status}


def prepare(case, seed):
    return (_Eos if case["kind"] == "eos" else _Run)(case, int(seed))


def run(state):
    return state.one()


# ---------------------------------------------------------------------------
# the work of a pass
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: the state (and potential) read once and written once per pass,
    interiors only.  Operations: per cell and substep about 3 faces of two
    flux evaluations, three with the EOS for the binary; a solve's smoothing
    as 10 V-cycles of 20 seven-point sweeps.  EOS: 56 bytes and about 1000
    operations a point, five evaluations for an inversion."""
    if case["kind"] == "eos":
        each = 1.0 if case["call"] == "forward" else 5.0
        return {"bytes": (56.0 if case["call"] == "forward" else 56.0 + 4.0) * case["n"],
                "flops": 1000.0 * each * case["n"]}
    n = _base(case)["tree"]["level"].size
    nx, nf = case.get("nx", 8), 13 if case["kind"] == "binary" else 6
    cells = float(n * nx ** 3)
    if case["kind"] == "solve":
        return {"bytes": 16.0 * cells, "flops": cells * 10 * 20 * 10}
    hydro = 3 * case["steps"] * cells * (6000.0 if case["kind"] == "binary" else 400.0)
    solve = 0.0 if case["kind"] == "euler" else 3 * case["steps"] * cells * 10 * 20 * 10
    return {"bytes": 16.0 * nf * cells + (16.0 * cells if case["kind"] != "euler" else 0.0), "flops": hydro + solve}


# ---------------------------------------------------------------------------
# what a pass returns, in plain torch
# ---------------------------------------------------------------------------
def _psi(z):
    """Quintic Hermite basis functions of value, slope and curvature at one
    end of [0, 1], with their first and second derivatives."""
    p = [1.0 + z ** 3 * (-10.0 + z * (15.0 - 6.0 * z)), z + z ** 3 * (-6.0 + z * (8.0 - 3.0 * z)),
         0.5 * z * z * (1.0 + z * (-3.0 + z * (3.0 - z)))]
    d = [z * z * (-30.0 + z * (60.0 - 30.0 * z)), 1.0 + z * z * (-18.0 + z * (32.0 - 15.0 * z)),
         0.5 * z * (2.0 + z * (-9.0 + z * (12.0 - 5.0 * z)))]
    e = [z * (-60.0 + z * (180.0 - 120.0 * z)), z * (-36.0 + z * (96.0 - 60.0 * z)),
         0.5 * (2.0 + z * (-18.0 + z * (36.0 - 20.0 * z)))]
    return p, d, e


def _weights(x, h):
    """w[derivative][order][side] of an interval of width h at fraction x."""
    lo, hi = _psi(x), _psi(1.0 - x)
    return [[(lo[q][o] * h ** (o - q), (-1.0) ** (o + q) * hi[q][o] * h ** (o - q)) for o in range(3)]
            for q in range(3)]


def _eos_exact(rho, T, abar, zbar):
    """p, e, cs (cgs) of ions plus the biquintic interpolant of the tabulated
    free energy F = A d^(2/3) - B T^2 d^(-2/3)."""
    avo, kerg = 6.0221417930e23, 1.380650424e-16
    A, B = 1.5 * 1.0036e13, 1.0e4
    dev = rho.device
    dn = torch.from_numpy(10.0 ** (-12.0 + np.arange(1081) * (27.0 / 1080.0))).to(dev)
    tn = torch.from_numpy(10.0 ** (3.0 + np.arange(401) * (10.0 / 400.0))).to(dev)
    ye = zbar / abar
    din = ye * rho
    i = ((torch.log10(din) + 12.0) * (1080.0 / 27.0)).long().clamp(0, 1079)
    j = ((torch.log10(T) - 3.0) * (400.0 / 10.0)).long().clamp(0, 399)
    hd, ht = dn[i + 1] - dn[i], tn[j + 1] - tn[j]
    wd, wt = _weights((din - dn[i]) / hd, hd), _weights((T - tn[j]) / ht, ht)
    # derivative (a, b) of F in (d, T) at a node: F is a sum of two products
    c1 = [1.0, 2.0 / 3.0, -2.0 / 9.0]
    c2 = [1.0, -2.0 / 3.0, 10.0 / 9.0]
    want = {(0, 0): 0.0, (1, 0): 0.0, (0, 1): 0.0, (2, 0): 0.0, (0, 2): 0.0, (1, 1): 0.0}
    for sd in range(2):
        d = dn[i + sd]
        for st in range(2):
            t = tn[j + st]
            for od in range(3):
                cold = A * c1[od] * d ** (2.0 / 3.0 - od)
                warm = B * c2[od] * d ** (-2.0 / 3.0 - od)
                for ot, f in enumerate((cold - warm * t * t, -2.0 * warm * t, -2.0 * warm)):
                    for q, r in want:
                        want[q, r] = want[q, r] + f * wd[q][od][sd] * wt[r][ot][st]
    pion = avo / abar * rho * kerg * T
    p = din * din * want[1, 0] + pion
    e = ye * (want[0, 0] - T * want[0, 1]) + 1.5 * pion / rho
    cv = 1.5 * avo / abar * kerg - T * ye * want[0, 2]
    dpdd = avo / abar * kerg * T + ye * (din * din * want[2, 0] + 2.0 * din * want[1, 0])
    dpdt = avo / abar * rho * kerg + din * din * want[1, 1]
    return p, e, torch.sqrt(p / rho ** 2 * dpdt / cv + dpdd)


def exact(case, seed):
    """The forward EOS.  A step of the hydro or of a solve has no value free
    of the method (limiters, stopping tests); a Newton temperature is the
    iterate at which it stops."""
    if case["kind"] != "eos" or case["call"] != "forward":
        return None
    rho, T, abar, zbar, _ = _points(case, int(seed))
    cm, gr, s, K = CODE_UNITS if case["units"] == "code" else (1.0, 1.0, 1.0, 1.0)
    p, e, cs = [torch.empty_like(rho) for _ in range(3)]
    for a in range(0, case["n"], 1 << 20):
        z = slice(a, a + (1 << 20))
        p[z], e[z], cs[z] = _eos_exact(rho[z] * (gr / cm ** 3), T[z] * K, abar[z], zbar[z])
    return {"p": p / (gr / cm / s ** 2), "e": e / (cm / s) ** 2, "cs": cs / (cm / s), "status": None}
