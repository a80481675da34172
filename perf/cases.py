"""The work this framework is used for, as cases that can be timed one by one.

Each case is one pass through the public entry points (`abi.Engine`,
`adjoint.Rollout`, `sph_density_noalloc`) the way a program calls them:

  steps      a time loop continued from a saved state: the table's moving
             columns written from device memory, k leapfrog steps, the new
             state read back into device memory
  diffusion  the same with super-time-stepping of an anisotropic diffusion run
  density    the density and smoothing lengths of a new snapshot (positions
             and starting h handed over in device memory, no lists kept)
  noalloc    the density of another program's device arrays
  gradient   a differentiable rollout: forward steps and their adjoint
  roundtrip  one step on a table that lives on the host

The inputs are periodic particle sets: lattices with every particle moved a
little (what a settled particle set looks like), at the resolutions of the
repository's configurations and at odd ones.
"""
import ctypes
import math

import numpy as np
import torch

from sph_playground_b200 import abi, adjoint, consts, ic

KRAD = {"m4": 2.0, "m6": 3.0}
NORM = {"m4": (2.0 / 3.0, 10.0 / (7.0 * math.pi), 1.0 / math.pi),
        "m6": (1.0 / 120.0, 7.0 / (478.0 * math.pi), 1.0 / (120.0 * math.pi))}
FW = {"m4": (6.0, 6.3226, 6.66400), "m6": (4.0, 9.31505 / 2.25, 9.6429 / 2.25)}
CN_HYDRO = {"m4": 0.1, "m6": 0.3}
CN_DIFF = {"m4": {"fab": 0.15, "n2w": 0.2, "2nw-+": 0.96},
           "m6": {"fab": 0.2, "n2w": 0.4, "2nw-+": 1.1}}
PREC = {"fp64": abi.PREC_FP64, "fp32": abi.PREC_FP32_COMP}
HFAC, GAMMA, FAR = 1.2, 5.0 / 3.0, 1.0e6

MOVING = ["rx", "ry", "rz", "vx", "vy", "vz", "ax", "ay", "az", "h", "dh", "u", "du", "den", "c"]
FIELD = ["bx", "by", "bz", "dbx", "dby", "dbz"]
HEAT = ["t", "ddt"]


def listed():
    return [
        # an interactive run or a convergence study's coarse end: a thousand
        # particles, where launches and host round trips count
        {"name": "steps2d_32_fp64", "kind": "steps", "flow": "shear", "dim": 2, "n": 32, "prec": "fp64",
         "kernel": "m6", "skin": 0.1, "steps": 4},
        # a 2D MHD run of ordinary size, odd resolution
        {"name": "mhd2d_201_fp64", "kind": "steps", "flow": "mhd", "dim": 2, "n": 201, "prec": "fp64",
         "kernel": "m6", "skin": 0.1, "steps": 4},
        # the small and the large instance of the diffusion sweep
        {"name": "diffusion2d_64_fp64", "kind": "diffusion", "ddw": "fab", "n": 64, "prec": "fp64",
         "kernel": "m6", "stages": 8},
        {"name": "diffusion2d_256_fp32", "kind": "diffusion", "ddw": "2nw-+", "n": 256, "prec": "fp32",
         "kernel": "m6", "stages": 8},
        # density of a snapshot: a mid-size set in double precision, and the
        # repository's density configuration in its fast precision
        {"name": "density3d_51_fp64", "kind": "density", "dim": 3, "n": 51, "prec": "fp64", "kernel": "m6"},
        {"name": "density3d_128_fp32", "kind": "density", "dim": 3, "n": 128, "prec": "fp32", "kernel": "m6"},
        # the headline blast wave, in both precisions, early in the run where
        # the neighbour lists are kept between steps
        {"name": "blast3d_128_fp32", "kind": "steps", "flow": "blast", "dim": 3, "n": 128, "prec": "fp32",
         "kernel": "m6", "skin": 0.1, "steps": 4},
        {"name": "blast3d_96_fp64", "kind": "steps", "flow": "blast", "dim": 3, "n": 96, "prec": "fp64",
         "kernel": "m6", "skin": 0.1, "steps": 4},
        # the same with a search every step, as late in a run or in fast flows
        {"name": "blast3d_99_fp32_search", "kind": "steps", "flow": "blast", "dim": 3, "n": 99, "prec": "fp32",
         "kernel": "m6", "skin": 0.0, "steps": 4},
        # an in-situ hook inside another program's memory budget, at its limit
        {"name": "noalloc3d_262144", "kind": "noalloc", "dim": 3, "n": 262144, "kernel": "m6"},
        # one gradient of a shear-flow misfit
        {"name": "gradient2d_128", "kind": "gradient", "n": 128, "steps": 10, "every": 5, "kernel": "m6"},
        # a host program that owns the particle table
        {"name": "roundtrip3d_64_fp64", "kind": "roundtrip", "flow": "shear", "dim": 3, "n": 64, "prec": "fp64",
         "kernel": "m6", "skin": 0.1, "steps": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps2d", "steps3d", "steps3d", "density", "density", "diffusion", "noalloc",
                       "gradient", "roundtrip"])
    kernel = rng.choice(["m6", "m6", "m4"])
    prec = rng.choice(["fp64", "fp32"])
    if kind == "steps2d":
        return {"kind": "steps", "flow": rng.choice(["shear", "mhd"]), "dim": 2, "n": _log(rng, 24, 320),
                "prec": prec, "kernel": kernel, "skin": rng.choice([0.0, 0.1]), "steps": rng.randint(2, 6)}
    if kind == "steps3d":
        return {"kind": "steps", "flow": rng.choice(["blast", "shear", "mhd"]), "dim": 3,
                "n": _log(rng, 16, 112 if prec == "fp32" else 72), "prec": prec, "kernel": kernel,
                "skin": rng.choice([0.0, 0.1]), "steps": rng.randint(2, 4)}
    if kind == "density":
        dim = rng.choice([1, 2, 3, 3])
        n = {1: _log(rng, 100, 100000), 2: _log(rng, 24, 900), 3: _log(rng, 16, 120)}[dim]
        return {"kind": "density", "dim": dim, "n": n, "prec": prec, "kernel": kernel}
    if kind == "diffusion":
        return {"kind": "diffusion", "ddw": rng.choice(["fab", "n2w", "2nw-+"]), "n": _log(rng, 24, 256),
                "prec": prec, "kernel": kernel, "stages": rng.randint(3, 10)}
    if kind == "noalloc":
        return {"kind": "noalloc", "dim": rng.choice([1, 2, 3, 3]), "n": _log(rng, 300, 262144),
                "kernel": kernel}
    if kind == "gradient":
        return {"kind": "gradient", "n": _log(rng, 24, 144), "steps": rng.randint(3, 10),
                "every": rng.randint(2, 5), "kernel": kernel}
    return {"kind": "roundtrip", "flow": "shear", "dim": 3, "n": _log(rng, 16, 72), "prec": "fp64",
            "kernel": kernel, "skin": 0.1, "steps": rng.randint(1, 3)}


# ---- inputs -------------------------------------------------------------------
def _lattice(n, dim):
    ax = (np.arange(n) + 0.5) / n
    return np.stack([g.ravel() for g in np.meshgrid(*([ax] * dim), indexing="ij")], axis=1)


def _inputs(case, seed):
    """The particle set of a case as named numpy columns, from the seed alone."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "noalloc":
        n, dim = case["n"], case["dim"]
        h = HFAC * n ** (-1.0 / dim) * rng.uniform(0.9, 1.1, n)
        return {"r": rng.uniform(0.0, 1.0, (n, dim)), "h": h, "m": rng.uniform(0.8, 1.2, n) / n}
    dim, n = case.get("dim", 2), case["n"]
    r = _lattice(n, dim)
    N = r.shape[0]
    flow = case.get("flow")
    amp = {"density": 0.1, "diffusion": 0.05, "gradient": 0.1}.get(kind, 0.02 if flow == "blast" else 0.05)
    pos = np.zeros((N, 3))
    pos[:, :dim] = np.mod(r + rng.uniform(-amp, amp, (N, dim)) / n, 1.0)
    P = 2.5 if flow or kind == "gradient" else 1.0
    col = {"r": pos, "v": np.zeros((N, 3)), "b": np.zeros((N, 3)), "t": np.zeros(N),
           "m": np.full(N, 1.0 / N), "h": np.full(N, HFAC / n), "u": np.full(N, P / (GAMMA - 1.0))}
    tau = 2.0 * math.pi
    x, y, z = pos[:, 0], pos[:, 1], pos[:, 2]
    if kind == "diffusion":
        th = math.radians(rng.uniform(20.0, 40.0))
        col["t"] = np.sin(tau * x) * np.sin(tau * y)
        col["b"][:, 0], col["b"][:, 1] = math.cos(th), math.sin(th)
        col["u"][:] = 1.0 / (GAMMA * (GAMMA - 1.0))
    elif kind == "gradient" or flow in ("shear", "mhd"):
        col["v"][:, 0] = 0.1 * np.sin(tau * y) + rng.normal(0.0, 1e-3, N)
        if dim > 1:
            col["v"][:, 1] = 0.05 * np.sin(tau * x + 0.3) + rng.normal(0.0, 1e-3, N)
        if dim > 2:
            col["v"][:, 2] = 0.05 * np.sin(tau * (x + y)) + rng.normal(0.0, 1e-3, N)
        if flow:
            col["u"] *= 1.0 + 0.1 * np.sin(tau * (x - y)) + rng.normal(0.0, 1e-3, N)
        if flow == "mhd":
            col["b"][:, 0] = 0.3 + 0.1 * np.sin(tau * y)
            col["b"][:, 1] = 0.2 * np.sin(2 * tau * x)
            col["b"][:, 2] = 0.1 * np.cos(tau * (x + z))
    elif flow == "blast":
        # energy 1 laid on the particles within two smoothing lengths of the
        # centre, background pressure 1e-5
        col["u"][:] = 1e-5 / (GAMMA - 1.0) * (1.0 + rng.uniform(-0.05, 0.05, N))
        d = np.sqrt(((pos[:, :dim] - 0.5) ** 2).sum(1)) * n / HFAC
        sel = d < 2.0
        w = np.clip(3 - d[sel], 0, None) ** 5 - 6 * np.clip(2 - d[sel], 0, None) ** 5 \
            + 15 * np.clip(1 - d[sel], 0, None) ** 5
        col["u"][sel] += w / w.sum() * N
    return col


def _engine(case, seed):
    col = _inputs(case, seed)
    kind, dim, n = case["kind"], case.get("dim", 2), case["n"]
    N = col["m"].shape[0]
    diff = kind == "diffusion"
    eqs = "manual" if diff else ("magnetohydro" if case.get("flow") == "mhd" else "hydro")
    au = 1.0 if case.get("flow") else 0.0
    st = ic.make_state(dim, equations=eqs, ddw=case.get("ddw", "fab"), hfac=HFAC, tfinish=FAR, npics=1,
                       resolution=n, spacing=1.0 / n, au=au, artts="no" if diff else "yes",
                       disotropic="no" if diff else "yes",
                       ymax=1.0 if dim > 1 else 0.0, zmax=1.0 if dim > 2 else 0.0)
    for k, v in (("bordsize", (int(KRAD[case["kernel"]] * HFAC) + 1) / n), ("padding", 0.5 / n), ("fixedpn", 0),
                 ("realpn", N), ("gamma", GAMMA), ("dcondconst", 1.0), ("muzero", 1.0), ("dtprint", FAR),
                 ("time", 0.0)):
        ic.set_state(st, k, v)
    if diff:
        for k, v in (("eqonhydro", 0.0), ("eqondiff", 1.0), ("eqonfluxlim", 0.0), ("eqonradexch", 0.0),
                     ("eqonsts", 1.0), ("ststype", consts.ests["fixeds"]), ("stsfixeds", case["stages"])):
            ic.set_state(st, k, v)
    store = np.zeros((N, consts.ES_TOTAL))
    for k, name in enumerate(("rx", "ry", "rz")):
        store[:, ic.col(name)] = col["r"][:, k]
    for k, ax in enumerate("xyz"):
        store[:, ic.col("v" + ax)] = col["v"][:, k]
        store[:, ic.col("b" + ax)] = col["b"][:, k]
    for name in ("m", "h", "u", "t"):
        store[:, ic.col(name)] = col[name]
    store[:, ic.col("den")] = store[:, ic.col("om")] = 1.0
    store[:, ic.col("p")] = (GAMMA - 1.0) * col["u"]
    store[:, ic.col("c")] = np.sqrt(GAMMA * (GAMMA - 1.0) * col["u"])
    store[:, ic.col("kappa")] = 1.0 if diff else 0.0
    store[:, ic.col("type")] = consts.ept["real"]
    return st, store


class State:
    def __init__(self, **kw):
        self.__dict__.update(kw)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "noalloc":
        col = _inputs(case, seed)
        dev = torch.device("cuda")
        r = torch.tensor(np.ascontiguousarray(col["r"].T), device=dev)
        lib = abi.load()
        f = lib.sph_density_noalloc
        f.argtypes = [ctypes.c_void_p] * 5 + [ctypes.c_int64, ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 2
        f.restype = ctypes.c_int
        s = State(kind=kind, f=f, r=r, h=torch.tensor(col["h"], device=dev), m=torch.tensor(col["m"], device=dev),
                  rho=torch.zeros(case["n"], dtype=torch.float64, device=dev), n=case["n"], dim=case["dim"],
                  kernel=consts.KERNELS[case["kernel"]])
        torch.cuda.synchronize()
        return s
    st, store = _engine(case, seed)
    if kind == "gradient":
        v0 = torch.tensor(np.ascontiguousarray(store[:, 3:6]), device="cuda", requires_grad=True)
        ab = [torch.tensor(x, dtype=torch.float64, requires_grad=True) for x in (1.0, 2.0)]
        target = torch.tensor(1.2 * store[:, 3:6], device="cuda")
        setup = adjoint.RolloutSetup(st, store, nsteps=case["steps"], every=case["every"],
                                     dt=0.1 / case["n"], kernel=case["kernel"])
        return State(kind=kind, v0=v0, ab=ab, target=target, setup=setup)
    e = abi.Engine(st, store, case["kernel"], precision=PREC[case["prec"]])
    s = State(kind=kind, e=e, fast=case["prec"] == "fp32", steps=case.get("steps", 1))
    if kind == "density":
        e.set_param(abi.P_SKIN, 0.0)
        s.put, s.get = ["rx", "ry", "rz", "h"], ["den", "h", "om"]
        s.groups = [("den", 1), ("h", 1), ("om", 1)]
    elif kind == "roundtrip":
        e.set_param(abi.P_SKIN, case["skin"])
        e.step(0)
        s.host_in = torch.empty((e.n_rows, consts.ES_TOTAL), dtype=torch.float64, pin_memory=True)
        s.host_out = torch.empty_like(s.host_in).pin_memory()
        e.get_store(s.host_in.numpy())
        return s
    else:
        if kind == "steps":
            e.set_param(abi.P_SKIN, case["skin"])
        e.step(0)  # the force evaluation a run starts with
        extra = HEAT if kind == "diffusion" else (FIELD if case["flow"] == "mhd" else [])
        s.put = MOVING + extra
        if kind == "diffusion":
            s.get, s.groups = ["t", "ddt", "h", "den"], [("t", 1), ("ddt", 1), ("h", 1), ("den", 1)]
        else:
            s.get = ["rx", "ry", "rz", "vx", "vy", "vz", "ax", "ay", "az", "u", "du", "h", "den"] + extra
            s.groups = [("r", 3), ("v", 3), ("a", 3), ("u", 1), ("du", 1), ("h", 1), ("den", 1)]
            s.groups += [("b", 3), ("db", 3)] if extra else []
    s.saved = torch.empty((len(s.put), e.n_rows), dtype=torch.float64, device="cuda")
    s.out = torch.empty((len(s.get), e.n_rows), dtype=torch.float64, device="cuda")
    s.out32 = torch.empty(s.out.shape, dtype=torch.float32, device="cuda") if s.fast else None
    torch.cuda.synchronize()
    e.get_columns(s.put, s.saved.data_ptr())
    return s


# ---- one pass -------------------------------------------------------------------
def run(s):
    if s.kind == "noalloc":
        ptr = [s.r[k].data_ptr() for k in range(s.dim)] + [None] * (3 - s.dim)
        rc = s.f(*ptr, s.m.data_ptr(), s.h.data_ptr(), s.n, s.dim, s.kernel, s.rho.data_ptr(),
                 torch.cuda.current_stream().cuda_stream or None)
        if rc:
            raise RuntimeError("sph_density_noalloc: %d" % rc)
        return s.rho
    if s.kind == "gradient":
        vT = adjoint.Rollout.apply(s.v0, s.ab[0], s.ab[1], s.setup)
        g = torch.autograd.grad(((vT - s.target) ** 2).sum(), [s.v0] + s.ab)
        return {"v": vT.detach(), "g_v0": g[0], "g_alpha": g[1], "g_beta": g[2]}
    e = s.e
    if s.kind == "roundtrip":
        e.set_store(s.host_in.numpy())
        e.step(s.steps)
        return e.get_store(s.host_out.numpy())
    e.set_columns(s.put, s.saved.data_ptr())
    if s.kind == "density":
        e.density()
    else:
        e.step(s.steps)
    e.get_columns(s.get, s.out.data_ptr())
    out = s.out
    if s.fast:  # pair sums in single precision: handed on as such
        out = s.out32.copy_(s.out)
        torch.cuda.current_stream().synchronize()  # s.out belongs to the engine's stream
    res, k = {}, 0
    for name, w in s.groups:
        res[name] = out[k:k + w]
        k += w
    return res


# ---- the work a pass cannot do without ---------------------------------------------
def work(case):
    kind, dim, kr = case["kind"], case.get("dim", 2), KRAD[case["kernel"]] * HFAC
    N = case["n"] if kind == "noalloc" else case["n"] ** dim
    pairs = N * {1: 2 * kr, 2: math.pi * kr ** 2, 3: 4.0 / 3.0 * math.pi * kr ** 3}[dim]
    if kind == "noalloc":
        return {"bytes": 8 * N * (dim + 3), "flops": 30 * pairs}
    if kind == "density":  # two Newton sweeps: one update and the sweep that confirms it
        return {"bytes": 8 * N * (dim + 2 + 3), "flops": 2 * 50 * pairs}
    if kind == "diffusion":
        return {"bytes": 8 * N * (dim * 2 + 12), "flops": (case["stages"] + 1) * (50 + 80) * pairs}
    if kind == "gradient":
        return {"bytes": 8 * N * 30 * case["steps"], "flops": (200 + 600) * pairs * (case["steps"] + 1)}
    f = 200 + (60 if case["flow"] == "mhd" else 0)
    if kind == "roundtrip":
        return {"bytes": 2 * 8 * 32 * N, "flops": case["steps"] * f * pairs}
    cols = len(MOVING) + 13 + (2 * len(FIELD) if case["flow"] == "mhd" else 0)
    return {"bytes": 8 * N * cols, "flops": case["steps"] * f * pairs}


# ---- the same in plain torch, 64 bits ----------------------------------------------
def _shape(q, kernel):
    """f, f', f'' of the kernel's shape."""
    t = lambda k: (k - q).clamp(min=0.0)  # noqa: E731
    if kernel == "m6":
        a, b, c = t(3.0), t(2.0), t(1.0)
        return (a ** 5 - 6 * b ** 5 + 15 * c ** 5, -5 * a ** 4 + 30 * b ** 4 - 75 * c ** 4,
                20 * a ** 3 - 120 * b ** 3 + 300 * c ** 3)
    a, b = t(2.0), t(1.0)
    return 0.25 * a ** 3 - b ** 3, -0.75 * a ** 2 + 3 * b ** 2, 1.5 * a - 6 * b


class Plain:
    """A periodic set whose particles stay near their lattice points: the
    neighbours of all particles at once are shifted copies of the arrays."""

    def __init__(self, case, seed):
        col = _inputs(case, seed)
        self.case, self.kernel = case, case["kernel"]
        self.dim, self.n = case.get("dim", 2), case["n"]
        self.box = (self.n,) * self.dim
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        T = lambda a: torch.tensor(a, dtype=torch.float64, device=self.dev)  # noqa: E731
        vec = lambda a, w: T(np.ascontiguousarray(a.T)).reshape((w,) + self.box)  # noqa: E731
        self.home = vec(_lattice(self.n, self.dim), self.dim)
        self.r = vec(col["r"], 3)[:self.dim]
        self.rest = vec(col["r"], 3)[self.dim:]
        self.v, self.b = vec(col["v"], 3), vec(col["b"], 3)
        self.m, self.h, self.u, self.t = (T(col[k]).reshape(self.box) for k in ("m", "h", "u", "t"))
        z = torch.zeros_like
        self.a, self.db, self.du, self.dh, self.ddt = z(self.v), z(self.b), z(self.u), z(self.u), z(self.u)
        self.norm, self.krad = NORM[self.kernel][self.dim - 1], KRAD[self.kernel]
        self.tol, self.flow = 1e-8, case.get("flow")
        self.alpha, self.beta, self.au = 1.0, 2.0, 1.0 if self.flow else 0.0

    def offsets(self, h):
        with torch.no_grad():
            d = self.r - self.home
            d = d - torch.round(d)
            far = float((d ** 2).sum(0).max().sqrt())
            reach = (self.krad * float(h.max()) + 2 * far) * self.n + 1e-6
        k = min(int(reach), (self.n - 1) // 2)
        ax = [range(-k, k + 1)] * self.dim
        grid = np.stack([g.ravel() for g in np.meshgrid(*ax, indexing="ij")], axis=1)
        d2 = (grid ** 2).sum(1)
        return [tuple(int(x) for x in o) for o in grid[(d2 > 0) & (d2 <= reach ** 2)]]

    def near(self, o, *fields):
        dims = tuple(range(-self.dim, 0))
        got = [torch.roll(f, tuple(-x for x in o), dims) for f in (self.r,) + fields]
        d = self.r - got[0]
        d = d - torch.round(d)
        r2 = (d ** 2).sum(0)
        # the list's distance counts every axis, those beyond the dimension too
        self.list_r2 = r2.detach()
        if self.dim < 3:
            self.list_r2 = self.list_r2 + ((self.rest - torch.roll(self.rest, tuple(-x for x in o), dims)) ** 2).sum(0)
        return d, r2, got[1:]

    def listed(self, m):
        """m where the last shift's pair is on the neighbour list, made with the h a pass starts from."""
        return torch.where(self.list_r2 <= (self.krad * self.h_list) ** 2, m, torch.zeros_like(m))

    def sums(self, h):
        """rho and its derivative in h."""
        f0 = float(_shape(torch.zeros(1, dtype=torch.float64), self.kernel)[0])
        w, q_ = self.m * f0, self.m * f0 * self.dim
        for o in self.offsets(h):
            _, r2, (mj,) = self.near(o, self.m)
            mj = self.listed(mj)
            q = r2.sqrt() / h
            f, df, _ = _shape(q, self.kernel)
            w = w + mj * f
            q_ = q_ + mj * (self.dim * f + q * df)
        return self.norm * w / h ** self.dim, -self.norm * q_ / h ** (self.dim + 1)

    def newton(self, h, rho, slope):
        om = 1.0 + slope * h / (self.dim * rho)
        return om, h + (self.m * (HFAC / h) ** self.dim - rho) * h / (self.dim * rho * om)

    def density(self):
        h0, h = self.h, self.h.clone()
        self.h_list = h0
        rho, om, hn = h * 0, h * 0, h.clone()
        live = torch.ones_like(h, dtype=torch.bool)
        for _ in range(100):
            r_, s_ = self.sums(h)
            o_, n_ = self.newton(h, r_, s_)
            rho, om, hn = torch.where(live, r_, rho), torch.where(live, o_, om), torch.where(live, n_, hn)
            live = live & ((hn - h).abs() / h0 > self.tol)
            h = torch.where(live, hn, h)
            if not bool(live.any()):
                break
        self.finish(hn, rho, om)

    def density_smooth(self):
        """At convergence, with h a function of the positions (implicit)."""
        self.h_list = self.h.detach()
        with torch.no_grad():
            h = self.h
            for _ in range(100):
                rho, s_ = self.sums(h)
                hn = self.newton(h, rho, s_)[1]
                done = float(((hn - h).abs() / h).max()) < 1e-13
                h = hn
                if done:
                    break
            rho, s_ = self.sums(h)
            om = self.newton(h, rho, s_)[0]
        rho, _ = self.sums(h)
        h = h + (self.m * (HFAC / h) ** self.dim - rho) * (h / (self.dim * rho * om)).detach()
        rho, s_ = self.sums(h)
        self.finish(h, rho, self.newton(h, rho, s_)[0])

    def finish(self, h, rho, om):
        self.h, self.rho, self.om = h, rho, om
        self.P = (GAMMA - 1.0) * rho * self.u
        self.c = (GAMMA * self.P / rho).sqrt()

    def forces(self):
        D = self.dim
        h, rho, om, P, c = self.h, self.rho, self.om, self.P, self.c
        Pi = 1.0 / (rho * rho * om)
        K = self.norm / h ** (D + 1)
        mhd = self.flow == "mhd"
        a, du, drho = [0.0] * 3, 0.0, 0.0
        db = [0.0] * 3
        for o in self.offsets(h):
            x, r2, (m_, h_, rho_, Pi_, K_, P_, c_, u_, v_) = self.near(o, self.m, h, rho, Pi, K, P, c, self.u, self.v)
            r = r2.sqrt()
            m_ = self.listed(m_)
            ga = K * _shape(r / h, self.kernel)[1] / r
            gb = K_ * _shape(r / h_, self.kernel)[1] / r
            v = self.v - v_
            w = (v[:D] * x).sum(0)
            drho = drho + m_ * ga * w
            s = (w / r).clamp(max=0.0)
            qa = -0.5 * rho * (self.alpha * c - self.beta * s) * s
            qb = -0.5 * rho_ * (self.alpha * c_ - self.beta * s) * s
            F = (qa + P) * ga * Pi + (qb + P_) * gb * Pi_
            du = du + m_ * ga * w * Pi * (qa * rho + P)
            if self.au:
                vs = ((P - P_).abs() / (0.5 * (rho + rho_))).sqrt()
                du = du + m_ * self.au * vs * (self.u - u_) * 0.5 * r * (ga * rho * Pi + gb * rho_ * Pi_)
            for k in range(D):
                a[k] = a[k] - m_ * F * x[k]
            if mhd:
                B, (B_,) = self.b, self.near(o, self.b)[2]
                Br, B_r = (B[:D] * x).sum(0), (B_[:D] * x).sum(0)
                e, e_ = 0.5 * (B ** 2).sum(0), 0.5 * (B_ ** 2).sum(0)
                for k in range(3):
                    xk = x[k] if k < D else 0.0
                    a[k] = a[k] - m_ * (ga * Pi * (e * xk - B[k] * Br) + gb * Pi_ * (e_ * xk - B_[k] * B_r))
                    db[k] = db[k] - m_ * rho * Pi * ga * (v[k] * Br - B_[k] * w)
        z = torch.zeros_like(h)
        self.a = torch.stack([k + z for k in a])
        self.db = torch.stack([k + z for k in db])
        self.du, self.dh = du, -D * h * rho * Pi * drho

    def dt(self):
        dt = CN_HYDRO[self.kernel] * self.h.min() / self.c.max()
        if self.flow == "mhd":
            dt = torch.minimum(dt, 0.1 * self.h.min() / self.c.max() / self.b.max())
        return dt

    def step(self, dt, density):
        D, a, du, dh, db = self.dim, self.a, self.du, self.dh, self.db
        r = self.r + dt * self.v[:D] + 0.5 * dt * dt * a[:D]
        self.r = r - torch.floor(r)
        self.rest = (self.rest + dt * self.v[D:] + 0.5 * dt * dt * a[D:]).detach()
        self.v, self.u, self.h = self.v + dt * a, self.u + dt * du, self.h + dt * dh
        self.b = self.b + dt * db
        density()
        self.forces()
        self.v = self.v + 0.5 * dt * (self.a - a)
        self.u = self.u + 0.5 * dt * (self.du - du)
        self.h = self.h + 0.5 * dt * (self.dh - dh)
        self.b = self.b + 0.5 * dt * (self.db - db)

    # ---- diffusion at rest ----
    def heat(self, T):
        """dT/dt of the anisotropic diffusion term (diagonal tensor b_x^2, b_y^2)."""
        D, ddw = self.dim, self.case["ddw"]
        h, rho, om = self.h, self.rho, self.om
        Pi, K = 1.0 / (rho * rho * om), self.norm / h ** (D + 1)
        kk = self.b[:D] ** 2 / (self.b ** 2).sum(0)
        out, mask = 0.0, self.listed
        if ddw == "2nw-+":
            g = [0.0] * D
            for o in self.offsets(h):
                x, r2, (m_, rho_, T_) = self.near(o, self.m, rho, T)
                r = r2.sqrt()
                w = mask(m_) / rho / om * (T_ * rho_ - T * rho) * K * _shape(r / h, self.kernel)[1] / r
                g = [g[k] + w * x[k] for k in range(D)]
            flux = torch.stack(g) * kk
            for o in self.offsets(h):
                x, r2, (m_, h_, K_, Pi_, f_) = self.near(o, self.m, h, K, Pi, flux)
                r = r2.sqrt()
                ga, gb = K * _shape(r / h, self.kernel)[1] / r, K_ * _shape(r / h_, self.kernel)[1] / r
                out = out + mask(m_) * (ga * Pi * (flux * x).sum(0) + gb * Pi_ * (f_ * x).sum(0))
            return out
        for o in self.offsets(h):
            x, r2, (m_, rho_, T_, k_) = self.near(o, self.m, rho, T, kk)
            r = r2.sqrt()
            f, df, ddf = _shape(r / h, self.kernel)
            kb = 0.5 * (kk + k_)
            tr, rr, ga = kb.sum(0), (kb * x * x).sum(0) / r2, K * df / r
            if ddw == "n2w":
                c = K / h * ddf * rr + ga * (tr - rr)
            else:
                c = -ga * ((D + 2) * rr - tr)
            out = out + mask(m_) / (rho * rho_) * (T_ * rho_ - T * rho) * c
        return out

    def sts(self, s):
        """One step of the s-stage Runge-Kutta-Legendre scheme."""
        b = lambda j: 1.0 / 3.0 if j <= 2 else (j * j + j - 2.0) / (2.0 * j * (j + 1.0))  # noqa: E731
        w = 4.0 / (s * s + s - 2.0)
        dt = (s * s + s - 2.0) * 0.25 * CN_DIFF[self.kernel][self.case["ddw"]] * self.rho.min() * self.c.min() \
            * self.h.min() ** 2
        # the leapfrog part leaves T alone; the stages move it
        y0, d0 = self.t, self.heat(self.t)
        y2, y1 = y0, y0 + b(1) * w * dt * d0
        d1 = d0
        for j in range(2, s + 1):
            mu = (2.0 * j - 1.0) / j * b(j) / b(j - 1)
            nu = -(j - 1.0) / j * b(j) / b(j - 2)
            d1 = self.heat(y1)
            y = mu * y1 + nu * y2 + (1.0 - mu - nu) * y0 + mu * w * dt * d1 - (1.0 - b(j - 1)) * mu * w * dt * d0
            y2, y1 = y1, y
        self.t, self.ddt = y1, d1


def _exact_noalloc(case, seed):
    col = _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    r, h, m = (torch.tensor(col[k], device=dev) for k in ("r", "h", "m"))
    order = torch.argsort(r[:, 0])
    r, h, m = r[order].contiguous(), h[order], m[order]
    kr, D, kernel = KRAD[case["kernel"]], case["dim"], case["kernel"]
    x, rho = r[:, 0].contiguous(), torch.zeros_like(h)
    reach = kr * h.max()
    for i in range(0, r.shape[0], 1024):
        ri, hi = r[i:i + 1024], h[i:i + 1024]
        lo = int(torch.searchsorted(x, ri[0, 0] - reach))
        hi_ = int(torch.searchsorted(x, ri[-1, 0] + reach, right=True))
        for a in range(lo, hi_, 1 << 15):
            e = min(hi_, a + (1 << 15))
            r2 = torch.zeros((ri.shape[0], e - a), dtype=torch.float64, device=dev)
            for k in range(D):
                r2 += (ri[:, k, None] - r[None, a:e, k]) ** 2
            f = _shape(r2.sqrt() / hi[:, None], kernel)[0]
            rho[i:i + 1024] += f @ m[a:e]
    rho *= NORM[kernel][D - 1] / h ** D
    out = torch.empty_like(rho)
    out[order] = rho
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "noalloc":
        return _exact_noalloc(case, seed)
    p = Plain(case, seed)
    if kind == "gradient":
        v0 = p.v.clone().requires_grad_(True)
        ab = [torch.tensor(x, dtype=torch.float64, requires_grad=True) for x in (1.0, 2.0)]
        dt = 0.1 / case["n"]
        target = 1.2 * p.v
        p.v, (p.alpha, p.beta) = v0, ab
        p.density_smooth()
        p.forces()
        for _ in range(case["steps"]):
            p.step(dt, p.density_smooth)
        g = torch.autograd.grad(((p.v - target) ** 2).sum(), [v0] + ab)
        row = lambda t: t.detach().reshape(3, -1).T.contiguous()  # noqa: E731
        return {"v": row(p.v), "g_v0": row(g[0]), "g_alpha": g[1], "g_beta": g[2]}
    flat = lambda t: t.reshape((-1, p.n ** p.dim))  # noqa: E731
    with torch.no_grad():
        p.density()
        if kind == "density":
            return {"den": flat(p.rho), "h": flat(p.h), "om": flat(p.om)}
        if kind == "diffusion":
            p.density()
            p.sts(case["stages"])
            return {"t": flat(p.t), "ddt": flat(p.ddt), "h": flat(p.h), "den": flat(p.rho)}
        p.forces()
        for _ in range(case["steps"]):
            p.step(p.dt(), p.density)
        if kind == "roundtrip":
            tab = torch.zeros((p.n ** p.dim, consts.ES_TOTAL), dtype=torch.float64, device=p.dev)
            r3 = torch.cat([p.r, p.rest])
            for k, ax in enumerate("xyz"):
                for name, f in (("r", r3), ("v", p.v), ("a", p.a)):
                    tab[:, ic.col(name + ax)] = f[k].reshape(-1)
            for name, f in (("m", p.m), ("den", p.rho), ("h", p.h), ("dh", p.dh), ("p", p.P), ("u", p.u),
                            ("du", p.du), ("c", p.c), ("om", p.om)):
                tab[:, ic.col(name)] = f.reshape(-1)
            tab[:, ic.col("type")] = 1.0
            return tab.cpu().numpy()
        r3 = torch.cat([p.r, p.rest])
        out = {"r": flat(r3), "v": flat(p.v), "a": flat(p.a), "u": flat(p.u), "du": flat(p.du), "h": flat(p.h),
               "den": flat(p.rho)}
        if case["flow"] == "mhd":
            out.update(b=flat(p.b), db=flat(p.db))
        return out
