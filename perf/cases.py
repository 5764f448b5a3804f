"""Performance cases of the framework: what its users have it do, through its
public entry points, on the puncture configurations, grids and options the
repository runs.

  main_c    main.c's loop through the drop-in functions: residual_all_points,
            L2_norm_of_gf and MoL_step_forward_in_time, one call each per step
  relax     nrpyell_relax: one configuration from the zero guess, FP64
  mixed     nrpyell_relax_mixed: the same with FP32 correction stretches
  batch     nrpyell_relax_batch: a sweep of configurations in one call
  batch_mixed  nrpyell_relax_batch_mixed: a sweep in the FP32 correction form
  train     nrpyell_mlp_train: epochs of the learned guess's network
  guess     nrpyell_mlp_predict and nrpyell_pod_guess: one learned guess
  export    nrpyell_interpolate_solution: ADM quantities at Cartesian points

exact() restates each path in torch and numpy, in 64 bits and without this
repository's code.
"""
import ctypes as C
import math
import random
from fractions import Fraction

import numpy as np
import torch

from nrpyelliptic_b200 import _lib, abi
from nrpyelliptic_b200.problem import Config, Problem, Punctures

NG = 5
AMAX, SINHWAA, ETA, R_L2 = 1.0e6, 0.07, 20.0, 100.0
FEATURES = 13


def listed():
    return [
        # smallest calls: the drop-in functions on the shipped grid, one short call after the other
        {"name": "main_c_64x64x8", "kind": "main_c", "n0": 64, "n1": 64, "n2": 8, "steps": 16},
        # a whole solve on the shipped grid
        {"name": "relax_64x64x8", "kind": "relax", "n0": 64, "n1": 64, "n2": 8, "tol": -10.0, "steps": 4000},
        # a whole solve on a grid that fills no tile, to a looser tolerance
        {"name": "relax_90x75x10", "kind": "relax", "n0": 90, "n1": 75, "n2": 10, "tol": -8.0, "steps": 4000},
        # a whole solve at the production size (bench.py's workload)
        {"name": "relax_128x128x16", "kind": "relax", "n0": 128, "n1": 128, "n2": 16, "tol": -10.0, "steps": 8000},
        # the largest grid: a bounded stretch of its tens of thousands of steps
        {"name": "relax_256x256x32", "kind": "relax", "n0": 256, "n1": 256, "n2": 32, "tol": -10.0, "steps": 500},
        # mixed precision on the small grid: FP32 to 1e-6, then FP64
        {"name": "mixed_64x64x8", "kind": "mixed", "n0": 64, "n1": 64, "n2": 8, "tol": -10.0, "switch": -6.0,
         "fold": 256, "steps": 4000},
        # mixed precision on the largest grid, every step FP32
        {"name": "mixed_256x256x32", "kind": "mixed", "n0": 256, "n1": 256, "n2": 32, "tol": -10.0, "switch": -10.0,
         "fold": 256, "steps": 512},
        # the seeded sweep: configurations on its three grids in one call
        {"name": "batch_sweep_12", "kind": "batch", "n": 12, "g0": 96, "g1": 128, "g2": 192, "tol": -10.0,
         "steps": 256},
        # training solves of the learned guess in the FP32 correction form
        {"name": "batch_mixed_16", "kind": "batch_mixed", "n": 16, "g0": 128, "g1": 128, "g2": 128, "tol": -10.0,
         "steps": 512},
        # two epochs of the learned guess's network at its own sizes
        {"name": "train_4096x256", "kind": "train", "rows": 4096, "width": 512, "depth": 4, "modes": 256,
         "batch": 256, "epochs": 2},
        # one learned guess: network evaluation and POD reconstruction
        {"name": "guess_128x128x16", "kind": "guess", "n0": 128, "n1": 128, "n2": 16, "modes": 256, "width": 512,
         "depth": 4},
        # a solution handed to an evolution code: ADM quantities at a Cartesian grid's points
        {"name": "export_200k", "kind": "export", "n0": 128, "n1": 128, "n2": 16, "points": 200000, "order": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["main_c", "relax", "relax", "relax", "mixed", "mixed", "batch", "batch_mixed", "train", "guess",
                       "export"])
    # grids from 48 to 256 columns with their usual proportions, odd sizes among them; i2 is even
    n0 = _log_int(rng, 48, 256)
    n1 = max(40, min(256, int(n0 * rng.uniform(0.75, 1.1))))
    n2 = max(6, 2 * int(round(n0 / 16.0 * rng.uniform(0.85, 1.15))))
    grid = {"n0": n0, "n1": n1, "n2": min(n2, 32)}
    points = grid["n0"] * grid["n1"] * grid["n2"]
    cap = max(64, min(6000, int(8.0e8 / points)))  # RK4 steps, so that a pass stays below the largest listed one
    if kind == "main_c":
        return {"kind": kind, **grid, "steps": rng.randint(4, 24)}
    if kind == "relax":
        return {"kind": kind, **grid, "tol": rng.choice([-8.0, -9.0, -10.0]), "steps": cap}
    if kind == "mixed":
        return {"kind": kind, **grid, "tol": -10.0, "switch": rng.choice([-6.0, -10.0]),
                "fold": rng.choice([64, 128, 256]), "steps": min(cap, 2000)}
    if kind in ("batch", "batch_mixed"):
        g = sorted(rng.choice([48, 64, 80, 96, 112, 128, 144]) for _ in range(3))
        n = rng.randint(3, 16)
        mean = sum(x ** 3 / 8 for x in g) / 3
        return {"kind": kind, "n": n, "g0": g[0], "g1": g[1], "g2": g[2], "tol": -10.0,
                "steps": max(64, min(1024, int(6.0e8 / (mean * n))))}
    if kind == "train":
        batch = rng.choice([64, 128, 256])
        return {"kind": kind, "rows": batch * rng.randint(4, 16), "width": 8 * rng.randint(16, 64),
                "depth": rng.randint(2, 4), "modes": rng.randint(24, 256), "batch": batch, "epochs": rng.randint(1, 2)}
    if kind == "guess":
        n0, n1 = rng.randint(48, 128), rng.randint(48, 128)
        return {"kind": kind, "n0": n0, "n1": n1, "n2": 2 * rng.randint(4, 8), "modes": _log_int(rng, 24, 256),
                "width": 8 * rng.randint(16, 64), "depth": rng.randint(2, 4)}
    return {"kind": kind, "n0": rng.randint(48, 128), "n1": rng.randint(48, 128), "n2": 2 * rng.randint(4, 8),
            "points": _log_int(rng, 1000, 200000), "order": rng.randint(2, 8)}


# ------------------------------------------------------------------ inputs

def _punctures(rng):
    """A draw of the sweep's distribution: total bare mass 1, separation 4 to
    20 along z, momenta up to 0.15 in the xy-plane, dimensionless spins up to
    0.8 in random directions.  Returns (punctures, bScale)."""
    q = math.exp(rng.uniform(0.0, math.log(10.0)))
    m0, m1 = q / (1 + q), 1 / (1 + q)
    d, p, ang = rng.uniform(4.0, 20.0), rng.uniform(0.02, 0.15), rng.uniform(0.0, 2 * math.pi)
    P0 = (p * math.cos(ang), p * math.sin(ang), 0.0)
    spins = []
    for m in (m0, m1):
        chi, v = rng.uniform(0.0, 0.8), [rng.gauss(0, 1) for _ in range(3)]
        r = math.sqrt(sum(x * x for x in v))
        spins.append(tuple(chi * m * m * x / r for x in v))
    return Punctures(m0, m1, (0.0, 0.0, d / 2), (0.0, 0.0, -d / 2), P0, tuple(-x for x in P0), *spins), d / 2


def _config(nxx, rng):
    pu, b = _punctures(rng)
    return Config("case", tuple(nxx), pu, bScale=b, AMAX=AMAX, SINHWAA=SINHWAA, eta=ETA, R_L2=R_L2)


def _configs(case, seed):
    rng = random.Random("%s %d" % (case["kind"], seed))
    if "g0" not in case:
        return [_config((case["n0"], case["n1"], case["n2"]), rng)]
    out = []
    for i in range(case["n"]):
        g = case["g%d" % (i % 3)]
        out.append(_config((g, g, max(6, 2 * round(g / 16))), rng))
    return out


class _Grid:
    """One configuration set up on the GPU (tables and auxevol built there),
    its gridfunctions in torch memory."""

    def __init__(self, cfg, lib):
        self.lib, self.cfg = lib, cfg
        self.prob = p = Problem(cfg, lib=lib, host_aux=False, device_tables=True)
        n = p.Ntot
        self.gf = {k: torch.zeros(m * n, dtype=torch.float64, device="cuda")
                   for k, m in (("y_n", 2), ("acc", 2), ("k_odd", 2), ("k_even", 2), ("aux", 3))}
        torch.cuda.synchronize()
        ptr = {k: t.data_ptr() for k, t in self.gf.items()}
        lib.nrpyell_auxevol_device(C.byref(p.params), p.xx, cfg.CFL, p.dt, C.cast(ptr["aux"], abi.PREAL))
        p.set_wavespeed_at_OB(float(self.gf["aux"][abi.WAVESPEEDGF * n + p.wavespeed_OB_index()]))
        self.g = p.griddata(ptr)
        lib.nrpyell_setup_tables_device(C.byref(p.params), p.xx, C.byref(self.g.rfmstruct), C.byref(self.g.bcstruct))
        _lib.check(lib)

    def zero_guess(self):
        y = self.gf["y_n"]
        self.lib.nrpyell_memset(y.data_ptr(), 0, 8 * y.numel())

    @property
    def y(self):
        return self.gf["y_n"].view(2, *self.prob.N[::-1])


class _Network:
    def __init__(self, lib, case, seed, batch):
        self.lib = lib
        self.handle = lib.nrpyell_mlp_create(FEATURES, case["width"], case["depth"], case["modes"], batch, 1)
        _lib.check(lib)
        self.params = _weights(case, seed)
        lib.nrpyell_mlp_set_params(self.handle, self.params.ctypes.data)
        _lib.check(lib)

    def __del__(self):
        self.lib.nrpyell_mlp_destroy(self.handle)


def _dims(case):
    return [FEATURES] + [case["width"]] * case["depth"] + [case["modes"]]


def _weights(case, seed):
    """Glorot-uniform weights and small biases, in the library's layout."""
    rng = np.random.default_rng([seed, 7])
    out, dims = [], _dims(case)
    for i, o in zip(dims[:-1], dims[1:]):
        a = math.sqrt(6.0 / (i + o))
        out += [rng.uniform(-a, a, i * o), rng.uniform(-0.05, 0.05, o)]
    return np.concatenate(out).astype(np.float32)


def _training_set(case, seed):
    """Standardised features and coefficients that are smooth functions of
    them, with the fast decay of POD modes."""
    rng = np.random.default_rng([seed, 8])
    x = rng.normal(size=(case["rows"], FEATURES)).astype(np.float32)
    a = rng.normal(size=(FEATURES, case["modes"])) / 4
    t = np.sin(x @ a) * (1.0 / np.arange(1, case["modes"] + 1)) ** 0.7
    return x, (t / t.std()).astype(np.float32)


def _pod(case, seed):
    """Mean and basis of a POD reconstruction (float32, on the GPU)."""
    g = torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)
    n = (case["n0"] + 2 * NG) * (case["n1"] + 2 * NG) * (case["n2"] + 2 * NG)
    mean = 0.02 * torch.rand(n, generator=g, device="cuda")
    basis = torch.randn(case["modes"], n, generator=g, device="cuda") / math.sqrt(n)
    return mean, basis


def _features(case, seed):
    return np.random.default_rng([seed, 9]).normal(size=(1, FEATURES)).astype(np.float32)


def _points(case, seed):
    """Cartesian points around the punctures, out to r ~ 50."""
    rng = np.random.default_rng([seed, 10])
    r = np.exp(rng.uniform(math.log(0.3), math.log(50.0), case["points"]))
    v = rng.normal(size=(case["points"], 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True) * r[:, None]


def _field(case, seed, b):
    """A solution-like uu on the whole grid: a bump of the size of the
    punctures' correction with an angular dependence, regular on the axis."""
    rng = random.Random("field %d" % seed)
    amp, a1, ph = rng.uniform(0.01, 0.05), rng.uniform(-0.2, 0.2), rng.uniform(0, 2 * math.pi)
    gm = _Geometry((case["n0"], case["n1"], case["n2"]), b)
    rad = torch.sqrt(9.0 + gm.r ** 2)
    u = amp / rad * (1.0 + a1 * (gm.A * gm.s / rad) * torch.cos(gm.x2 - ph))
    return torch.stack([u, ETA * u]).reshape(-1).contiguous()


# ------------------------------------------------------------------- passes

def prepare(case, seed):
    lib = _lib.load()
    kind = case["kind"]
    st = {"case": case, "lib": lib}
    if kind in ("main_c", "relax", "mixed", "batch", "batch_mixed", "export"):
        st["grids"] = gs = [_Grid(c, lib) for c in _configs(case, seed)]
        st["dt"] = np.array([g.prob.dt for g in gs])
    if kind.startswith("batch"):
        st["array"] = (abi.griddata_struct * len(gs))(*[g.g for g in gs])
    if kind == "train":
        st["net"] = _Network(lib, case, seed, case["batch"])
        st["x"], st["t"] = (torch.from_numpy(a).cuda() for a in _training_set(case, seed))
    if kind == "guess":
        st["net"] = _Network(lib, case, seed, 256)
        st["mean"], st["basis"] = _pod(case, seed)
        st["x"] = torch.from_numpy(_features(case, seed)).cuda()
        st["c"] = torch.empty(1, case["modes"], device="cuda")
        st["y"] = torch.empty(2, st["mean"].numel(), dtype=torch.float64, device="cuda")
    if kind == "export":
        gs[0].gf["y_n"].copy_(_field(case, seed, gs[0].cfg.bScale))
        st["xyz"] = _points(case, seed)
    torch.cuda.synchronize()
    return st


def _dptr(a):
    return a.ctypes.data_as(abi.PREAL)


def run(st):
    case, lib, kind = st["case"], st["lib"], st["case"]["kind"]
    if kind == "main_c":
        out = _run_main_c(st)
    elif kind in ("relax", "mixed"):
        out = _run_relax(st)
    elif kind in ("batch", "batch_mixed"):
        out = _run_batch(st)
    elif kind == "train":
        lib.nrpyell_mlp_train(st["net"].handle, st["x"].data_ptr(), st["t"].data_ptr(), case["rows"], case["batch"],
                              case["epochs"], 1e-3, 2, None)
        p = np.empty_like(st["net"].params)
        lib.nrpyell_mlp_get_params(st["net"].handle, p.ctypes.data)
        out = {"params": p}
    elif kind == "guess":
        lib.nrpyell_mlp_predict(st["net"].handle, st["x"].data_ptr(), 1, st["c"].data_ptr())
        lib.nrpyell_pod_guess(st["mean"].data_ptr(), st["basis"].data_ptr(), case["modes"], st["mean"].numel(),
                              st["c"].data_ptr(), ETA, st["y"].data_ptr())
        out = {"c": st["c"], "y": st["y"]}
    else:
        g, n = st["grids"][0], case["points"]
        out = {"uu": np.empty(n), "psi": np.empty(n), "gamma": np.empty((n, 6)), "K": np.empty((n, 6))}
        lib.nrpyell_interpolate_solution(C.byref(g.prob.params), g.prob.xx, g.g.gridfuncs.y_n_gfs, n, _dptr(st["xyz"]),
                                         case["order"], *[_dptr(a) for a in out.values()])
    _lib.check(lib)
    return out


def _run_main_c(st):
    g, lib = st["grids"][0], st["lib"]
    f, p = g.g.gridfuncs, g.g.params
    g.zero_guess()
    l2 = []
    for _ in range(st["case"]["steps"]):
        lib.residual_all_points(C.byref(p), C.byref(g.g.rfmstruct), f.auxevol_gfs, f.y_n_gfs, f.diagnostic_output_gfs)
        l2.append(lib.L2_norm_of_gf(C.byref(p), abi.UUGF, R_L2, g.prob.xx, f.diagnostic_output_gfs))
        lib.MoL_step_forward_in_time(C.byref(g.g), g.prob.dt)
    return {"y": g.y, "l2": np.array(l2)}


def _run_relax(st):
    case, g, lib = st["case"], st["grids"][0], st["lib"]
    n32, n64, fin = C.c_int(0), C.c_int(0), C.c_double(0)
    g.zero_guess()
    if case["kind"] == "relax":
        lib.nrpyell_relax(C.byref(g.g), g.prob.dt, case["tol"], case["steps"], R_L2, C.byref(n64), C.byref(fin), None)
    else:
        lib.nrpyell_relax_mixed(C.byref(g.g), g.prob.dt, case["tol"], case["switch"], case["fold"], case["steps"], R_L2,
                                C.byref(n32), C.byref(n64), C.byref(fin), None)
    return {"y": g.y, "l2": fin.value, "steps": n32.value + n64.value}


def _run_batch(st):
    case, gs, lib = st["case"], st["grids"], st["lib"]
    n = len(gs)
    for g in gs:
        g.zero_guess()
    fin, n32, n64 = np.zeros(n), np.zeros(n, np.int32), np.zeros(n, np.int32)
    pi = C.POINTER(C.c_int)
    i32, i64 = n32.ctypes.data_as(pi), n64.ctypes.data_as(pi)
    if case["kind"] == "batch":
        lib.nrpyell_relax_batch(n, st["array"], _dptr(st["dt"]), case["tol"], case["steps"], R_L2, i64, _dptr(fin))
    else:
        lib.nrpyell_relax_batch_mixed(n, st["array"], _dptr(st["dt"]), case["tol"], case["tol"], 256, case["steps"],
                                      R_L2, i32, i64, _dptr(fin))
    return {"y": [g.y for g in gs], "l2": fin, "steps": n32 + n64}


def work(case):
    """Inputs read and outputs written once, and the arithmetic of the path."""
    kind = case["kind"]
    if kind == "train":
        d = _dims(case)
        prods = sum(a * b for a, b in zip(d[:-1], d[1:]))
        rows = case["rows"] // case["batch"] * case["batch"] * case["epochs"]
        n_par = prods + sum(d[1:])
        return {"bytes": 4.0 * rows * (FEATURES + case["modes"]) + 8.0 * n_par, "flops": 6.0 * rows * prods}
    if kind == "guess":
        n = (case["n0"] + 2 * NG) * (case["n1"] + 2 * NG) * (case["n2"] + 2 * NG)
        d = _dims(case)
        return {"bytes": 4.0 * n * (case["modes"] + 1) + 16.0 * n + 4.0 * sum(a * b for a, b in zip(d[:-1], d[1:])),
                "flops": 2.0 * n * case["modes"]}
    if kind == "export":
        return {"bytes": 17 * 8.0 * case["points"], "flops": case["points"] * (2.0 * (case["order"] + 1) ** 3 + 300)}
    grids = [case["g%d" % (i % 3)] for i in range(case["n"])] if "g0" in case else None
    pts = float(sum(g * g * max(6, 2 * round(g / 16)) for g in grids) if grids else case["n0"] * case["n1"] * case["n2"])
    # three auxevol fields in, two gridfunctions out; about 90 operations per
    # point and RHS, four of these per RK4 step (a solve takes about 9 steps
    # per column of the grid, at most the number asked for)
    side = case["g1"] if grids else case["n0"]
    steps = case["steps"] if kind == "main_c" else min(case["steps"], 30 * side)
    return {"bytes": 40.0 * pts, "flops": 4 * 90.0 * pts * steps}


# -------------------------------------------------- the paths in 64 bits

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(a, dtype=torch.float64, device=_dev())


class _Geometry:
    """Coordinates and metric factors of the SinhSymTP grid, shape [N2, N1, N0]."""

    def __init__(self, nxx, b):
        self.nxx, self.b = nxx, b
        lo, hi = (0.0, 0.0, -math.pi), (1.0, math.pi, math.pi)
        self.dx = [(hi[i] - lo[i]) / nxx[i] for i in range(3)]
        self.N = [n + 2 * NG for n in nxx]
        x = [_t(lo[i] + (np.arange(self.N[i]) - NG + 0.5) * self.dx[i]) for i in range(3)]
        self.x0, self.x1, self.x2 = x[0][None, None, :], x[1][None, :, None], x[2][:, None, None]
        k = AMAX / math.sinh(1.0 / SINHWAA)
        self.A = k * torch.sinh(self.x0 / SINHWAA)
        self.A1 = k / SINHWAA * torch.cosh(self.x0 / SINHWAA)
        self.A2 = self.A / SINHWAA ** 2
        self.s, self.c = torch.sin(self.x1), torch.cos(self.x1)
        self.B = torch.sqrt(self.A ** 2 + b * b)
        self.F = self.A ** 2 + (b * self.s) ** 2
        self.r = torch.sqrt((self.A * self.s) ** 2 + (self.B * self.c) ** 2)

    def cartesian(self):
        rho = self.A * self.s
        return torch.broadcast_tensors(rho * torch.cos(self.x2), rho * torch.sin(self.x2), self.B * self.c)


def _bowen_york(pu, X):
    """Conformal extrinsic curvature A_ij (six components xx xy xz yy yz zz) and psi_BL at X."""
    eps = {(0, 1, 2): 1, (1, 2, 0): 1, (2, 0, 1): 1, (0, 2, 1): -1, (2, 1, 0): -1, (1, 0, 2): -1}
    A, psi = [0.0] * 6, 1.0
    for m, pos, P, S in ((pu.m0, pu.pos0, pu.P0, pu.S0), (pu.m1, pu.pos1, pu.P1, pu.S1)):
        d = [X[i] - pos[i] for i in range(3)]
        r = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
        n = [v / r for v in d]
        Pn = sum(P[i] * n[i] for i in range(3))
        Sn = [sum(e * S[k] * n[l] for (i_, k, l), e in eps.items() if i_ == i) for i in range(3)]
        for c, (i, j) in enumerate(((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))):
            A[c] = A[c] + 1.5 / r ** 2 * (P[i] * n[j] + P[j] * n[i] - (float(i == j) - n[i] * n[j]) * Pn)
            A[c] = A[c] + 3.0 / r ** 3 * (Sn[i] * n[j] + Sn[j] * n[i])
        psi = psi + m / (2.0 * r)
    return A, psi


def _first_weights(off):
    """d/dx at node 0 on the eleven nodes off-5 .. off+5."""
    x = [off - 5 + j for j in range(11)]
    w = []
    for j, xj in enumerate(x):
        if xj == 0:
            w.append(Fraction(0))
            continue
        num = math.prod(Fraction(-xm) for xm in x if xm not in (xj, 0))
        w.append(num / math.prod(Fraction(xj - xm) for xm in x if xm != xj))
    w[x.index(0)] = -sum(w)
    return [float(v) for v in w]


def _band(n, dx, second):
    """[n x (n + 10)] matrix of the centred tenth-order first or second derivative."""
    d1 = [5 / 6, -5 / 21, 5 / 84, -5 / 504, 1 / 1260]
    d2 = [5 / 3, -5 / 21, 5 / 126, -5 / 1008, 1 / 3150]
    M = np.zeros((n, n + 2 * NG))
    for i in range(n):
        for k in range(1, 6):
            M[i, i + NG + k] = d2[k - 1] if second else d1[k - 1]
            M[i, i + NG - k] = d2[k - 1] if second else -d1[k - 1]
        if second:
            M[i, i + NG] = -5269 / 1800
    return _t(M / (dx * dx if second else dx))


class _Relaxation:
    """The hyperbolic relaxation of one configuration."""

    def __init__(self, cfg):
        n0, n1, n2 = self.nxx = cfg.Nxx
        gm = _Geometry(cfg.Nxx, cfg.bScale)
        self.N = N0, N1, N2 = gm.N
        X = gm.cartesian()
        a, psi = _bowen_york(cfg.punctures, X)
        I = self.I = (slice(NG, NG + n2), slice(NG, NG + n1), slice(NG, NG + n0))
        aa = a[0] ** 2 + a[3] ** 2 + a[5] ** 2 + 2 * (a[1] ** 2 + a[2] ** 2 + a[4] ** 2)
        self.S8, self.psi = (aa[I] / 8).contiguous(), psi[I].contiguous()
        rows = (slice(None), I[1], slice(None))
        cols = (slice(None), slice(None), I[2])
        A, A1, A2, B = (v[cols] for v in (gm.A, gm.A1, gm.A2, gm.B))
        s, c, F = gm.s[rows], gm.c[rows], gm.F[:, I[1], I[2]]
        self.c00 = B ** 2 / (A1 ** 2 * F)
        self.c0 = B * (B + A ** 2 / B - A * B * A2 / A1 ** 2) / (A1 * F * A)
        self.c11, self.c1, self.c22 = 1 / F, c / (s * F), 1 / (A * s) ** 2
        dx = gm.dx
        ds = [dx[0] * A1 * torch.sqrt(F) / B, dx[1] * torch.sqrt(F), dx[2] * A * s]
        ds = torch.minimum(torch.minimum(ds[0], ds[1]), ds[2])
        self.dt = float(ds.min())
        ws = cfg.CFL * ds / self.dt
        self.ws2 = ws ** 2
        self.cob = float(ws[0, 0, -1])
        dV = A1 * F * A * s / B * dx[0] * dx[1] * dx[2] * (gm.r[:, I[1], I[2]] < R_L2)
        self.dV, self.volume = dV, float(dV.sum()) * n2
        self.M0, self.M00 = _band(n0, dx[0], False).T, _band(n0, dx[0], True).T
        self.M1, self.M11, self.M22 = _band(n1, dx[1], False), _band(n1, dx[1], True), _band(n2, dx[2], True)
        # radiation condition: radial derivative at the last interior plane and the five outer ones
        o = (slice(None), I[1], slice(N0 - 6, N0))
        Ao, A1o, Bo, Fo, ro = gm.A[..., N0 - 6:], gm.A1[..., N0 - 6:], gm.B[..., N0 - 6:], gm.F[o], gm.r[o]
        self.ro = ro
        self.dx0dr = Ao * Bo ** 2 / (ro * A1o * Fo)
        self.dx1dr = -cfg.bScale ** 2 * s * c / (ro * Fo)
        R = np.zeros((17, 6))
        for j in range(6):
            off = -1 if j <= 1 else -j
            for m, w in enumerate(_first_weights(off)):
                R[11 + j + off - 5 + m, j] = w / dx[0]
        self.R0 = _t(R)
        # ghost points read from their images: across xx0 = 0 and the axis half a turn on
        i2, i1, i0 = np.meshgrid(np.arange(N2), np.arange(N1), np.arange(N0), indexing="ij")
        turn = np.zeros_like(i0)
        turn += i0 < NG
        i0 = np.where(i0 < NG, 2 * NG - 1 - i0, i0)
        turn += (i1 < NG) | (i1 >= NG + n1)
        i1 = np.where(i1 < NG, 2 * NG - 1 - i1, np.where(i1 >= NG + n1, 2 * (NG + n1) - 1 - i1, i1))
        i2 = NG + (i2 - NG + (turn % 2) * (n2 // 2)) % n2
        self.src = torch.as_tensor((i0 + N0 * (i1 + N1 * i2)).reshape(-1), device=_dev())
        self.eta = cfg.eta

    def ghosts(self, y):
        return y.reshape(2, -1).index_select(1, self.src).reshape(y.shape)

    def rhs(self, y):
        """(RHS on the interior and the outer layers, the residual); y has its ghost zones."""
        I, u = self.I, y[0]
        ui = u[I]
        row, plane = u[I[0], I[1], :], u[I[0], :, I[2]]
        lap = self.c00 * (row @ self.M00) + self.c0 * (row @ self.M0)
        lap += self.c11 * (self.M11 @ plane) + self.c1 * (self.M1 @ plane)
        lap += self.c22 * torch.tensordot(self.M22, u[:, I[1], I[2]], 1)
        res = lap + self.S8 / (self.psi + ui) ** 7
        k = torch.zeros_like(y)
        k[(0, *I)] = y[(1, *I)] - self.eta * ui
        k[(1, *I)] = self.ws2 * res
        N0 = self.N[0]
        d0 = y[:, I[0], I[1], N0 - 17:] @ self.R0
        d1 = self.M1 @ y[:, I[0], :, N0 - 6:]
        f = y[:, I[0], I[1], N0 - 6:]
        out = -self.cob * (self.dx0dr * d0 + self.dx1dr * d1 + f / self.ro)
        kp = k[:, I[0], I[1], N0 - 6]
        for j in range(1, 6):
            kp = out[..., j] + (kp - out[..., j - 1]) * (self.ro[..., j - 1] / self.ro[..., j]) ** 3
            k[:, I[0], I[1], N0 - 6 + j] = kp
        return k, res

    def solve(self, tol, steps):
        """(y, log10 L2 before each step, steps taken) from the zero guess."""
        y = torch.zeros(2, *self.N[::-1], dtype=torch.float64, device=_dev())
        dt, hist = self.dt, []
        for n in range(steps + 1):
            k1, res = self.rhs(y)
            hist.append(math.log10(1e-16 + math.sqrt(float((res ** 2 * self.dV).sum()) / self.volume)))
            if n == steps or hist[-1] <= tol:
                return y, hist, n
            k2, _ = self.rhs(self.ghosts(y + 0.5 * dt * k1))
            k3, _ = self.rhs(self.ghosts(y + 0.5 * dt * k2))
            k4, _ = self.rhs(self.ghosts(y + dt * k3))
            y = self.ghosts(y + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4))


def _layers(case, p):
    out, o, d = [], 0, _dims(case)
    for a, b in zip(d[:-1], d[1:]):
        out.append((p[o:o + a * b].view(a, b), p[o + a * b:o + a * b + b]))
        o += a * b + b
    return out


def _forward(layers, x):
    for k, (W, b) in enumerate(layers):
        x = x @ W + b
        x = torch.tanh(x) if k + 1 < len(layers) else x
    return x


def _train(case, seed):
    """Adam over shuffled minibatches, as nrpyell_mlp_train documents it."""
    x, t = (_t(a) for a in _training_set(case, seed))
    p = _t(_weights(case, seed)).requires_grad_(True)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    n, batch = case["rows"], case["batch"]
    s, mask, perm, it = 0xD1B54A32D192ED03 ^ 2, (1 << 64) - 1, list(range(n)), 0
    total = n // batch * case["epochs"]
    for _ in range(case["epochs"]):
        for i in range(n - 1, 0, -1):
            s = (s * 6364136223846793005 + 1442695040888963407) & mask
            j = (s >> 33) % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        for b in range(n // batch):
            idx = torch.as_tensor(perm[b * batch:(b + 1) * batch], device=x.device)
            loss = ((_forward(_layers(case, p), x[idx]) - t[idx]) ** 2).mean()
            g, = torch.autograd.grad(loss, p)
            lr = 1e-3 * (0.01 + 0.99 * 0.5 * (1 + math.cos(math.pi * it / total)))
            it += 1
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            step = lr * (m / (1 - 0.9 ** it)) / (torch.sqrt(v / (1 - 0.999 ** it)) + 1e-8)
            p = (p - step).detach().requires_grad_(True)
    return p.detach()


def _interpolate(case, seed):
    """Lagrange interpolation of uu and the ADM quantities at the points."""
    cfg, order = _configs(case, seed)[0], case["order"]
    u, X, b = _field(case, seed, cfg.bScale), _t(_points(case, seed)).T, cfg.bScale
    gm = _Geometry(cfg.Nxx, b)
    u = u[:gm.N[0] * gm.N[1] * gm.N[2]]
    rho2 = X[0] ** 2 + X[1] ** 2
    q = rho2 + X[2] ** 2 - b * b
    A2 = 0.5 * (q + torch.sqrt(q * q + 4 * b * b * rho2))
    xx = [SINHWAA * torch.asinh(torch.sqrt(A2) * math.sinh(1 / SINHWAA) / AMAX),
          torch.acos((X[2] / torch.sqrt(A2 + b * b)).clamp(-1, 1)), torch.atan2(X[1], X[0])]
    start, weight = [], []
    for d, lo in enumerate((0.0, 0.0, -math.pi)):
        t = (xx[d] - lo) / gm.dx[d] + NG - 0.5
        s = torch.floor(t + 0.5) - order // 2 if order % 2 == 0 else torch.floor(t) - (order - 1) // 2
        s = s.clamp(0, gm.N[d] - (order + 1))
        w = []
        for j in range(order + 1):
            l = torch.ones_like(t)
            for k in range(order + 1):
                if k != j:
                    l = l * (t - (s + k)) / (j - k)
            w.append(l)
        start.append(s.long())
        weight.append(w)
    uu = torch.zeros_like(X[0])
    for k in range(order + 1):
        for j in range(order + 1):
            for i in range(order + 1):
                at = (start[0] + i) + gm.N[0] * ((start[1] + j) + gm.N[1] * (start[2] + k))
                uu += weight[0][i] * weight[1][j] * weight[2][k] * u[at]
    a, psi = _bowen_york(cfg.punctures, X)
    psi = psi + uu
    gamma = torch.zeros(len(uu), 6, dtype=torch.float64, device=uu.device)
    gamma[:, [0, 3, 5]] = (psi ** 4)[:, None]
    return {"uu": uu, "psi": psi, "gamma": gamma, "K": torch.stack(a, 1) / psi[:, None] ** 2}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return {"params": _train(case, seed)}
    if kind == "guess":
        mean, basis = _pod(case, seed)
        c = _forward(_layers(case, _t(_weights(case, seed))), _t(_features(case, seed)))
        u = mean.double()
        for k in range(case["modes"]):
            u = u + c[0, k] * basis[k].double()
        return {"c": c, "y": torch.stack([u, ETA * u])}
    if kind == "export":
        return _interpolate(case, seed)
    tol = -math.inf if kind == "main_c" else case["tol"]
    got = [_Relaxation(c).solve(tol, case["steps"]) for c in _configs(case, seed)]
    if kind == "main_c":
        return {"y": got[0][0], "l2": np.array(got[0][1][:-1])}
    if kind in ("relax", "mixed"):
        return {"y": got[0][0], "l2": got[0][1][-1], "steps": None}
    return {"y": [g[0] for g in got], "l2": np.array([g[1][-1] for g in got]), "steps": None}
