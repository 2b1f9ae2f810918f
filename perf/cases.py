"""The workloads whose time is watched, each through the package's public entry points.

A case is a dict of plain values: what is run ("kind"), on which node set
("problem", "nx", "ny", "nz", "shuffle"; equal spacings, unless "cube"), in which form ("hydro",
"precision", "xsph") and for how many RK2 steps.  Kinds:

  evaluate   one derivative evaluation of the hydro package on a new state:
             set_state, ghosts + ConnectivityMap, initialize,
             evaluateDerivatives, dt, and the derivative fields to the host
  steps      a run between two dumps: new state, (start-up H relaxation,)
             ConnectivityMap, evaluateDerivatives, `steps`
             CheapSynchronousRK2 steps in one call, the state to the host
  host_step  the drop-in under a host integrator: one step_host call on
             pinned host arrays
  batch      an ensemble of Sod-type tubes of uneven sizes stepped together
  serve      a burst of requests through the server until all are fetched

Node sets are the package's benchmark shapes: lattices with a seeded jitter
of +-0.01 spacings, a Sod-type shock tube (B-spline, nPerh 1.51, fixed dt
1e-4) and the Kelvin-Helmholtz cube (Wendland C4, nPerh 1.35, Courant dt).

exact() is the same physics written out in torch, FP64, over an explicit
list of directed pairs.
"""
import ctypes
import importlib
import math
import random

import numpy as np
import torch

pkg = importlib.import_module("llnl-spheral_b200")

JITTER = 0.01
WIDEST = 2.1e6           # nodes of the largest single problem
EXACT_MOST = 3.0e9       # directed pairs x evaluations that exact() takes on


def listed():
    def case(name, kind, problem, nx, ny, nz, steps=1, hydro="sph", precision="fp64", xsph=False, shuffle=False,
             relax=False, cube=False):
        return dict(name=name, kind=kind, problem=problem, nx=nx, ny=ny, nz=nz, steps=steps, hydro=hydro,
                    precision=precision, xsph=xsph, shuffle=shuffle, relax=relax, cube=cube)

    return [
        # the smoke-test tube: one evaluation of a problem too small to fill the GPU, bound by launches
        case("eval_sod_2k", "evaluate", "sod", 32, 8, 8),
        # the Sod configuration's one evaluateDerivatives: 115 neighbors per node, FP64
        case("eval_sod_262k", "evaluate", "sod", 256, 32, 32),
        # the smallest tube of the ensemble, mixed form, alone
        case("steps_sod_4k_mixed", "steps", "sod", 64, 8, 8, steps=20, precision="mixed"),
        # the Sod configuration between two dumps
        case("steps_sod_262k", "steps", "sod", 256, 32, 32, steps=10),
        # Kelvin-Helmholtz of a served request's size, no axis a multiple of a warp, XSPH, nodes in no order
        case("steps_kh_odd_mixed", "steps", "kh", 47, 53, 50, steps=20, precision="mixed", xsph=True, shuffle=True),
        # the headline configuration, plain FP64, with the controller's start-up relaxation of H
        case("steps_kh_2m", "steps", "kh", 128, 128, 128, steps=20, relax=True),
        # the same in the mixed form
        case("steps_kh_2m_mixed", "steps", "kh", 128, 128, 128, steps=20, precision="mixed", relax=True),
        # the drop-in under the host's integrator: state in, one step, state out
        case("host_step_kh_262k", "host_step", "kh", 64, 64, 64),
        # the CRKSPH configuration, plain FP64: the unit cube, dz = 2 dx
        case("steps_crk_1m", "steps", "kh", 128, 128, 64, steps=10, hydro="crk", cube=True),
        # CRKSPH in the mixed form at a ragged size
        case("steps_crk_odd_mixed", "steps", "kh", 61, 43, 37, steps=10, hydro="crk", precision="mixed"),
        # the ensemble: tubes of 4,096 to 262,144 nodes (8k x k x k), gamma and density ratio of their own
        dict(name="batch_tubes_mixed", kind="batch", members=24, kmin=8, kmax=32, sizes=7, steps=5,
             precision="mixed"),
        # a burst of served requests, half Kelvin-Helmholtz, half tubes, plain FP64
        dict(name="serve_mix", kind="serve", members=8, nmin=8192, nmax=131072, sizes=11, steps=10,
             precision="fp64"),
    ]


def draw(rng):
    def size(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["evaluate", "steps", "steps", "steps", "host_step", "batch", "serve"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "batch":
        return dict(kind=kind, members=rng.randint(4, 14), kmin=8, kmax=rng.randint(10, 32),
                    sizes=rng.randrange(1 << 20), steps=rng.randint(2, 5), precision=precision)
    if kind == "serve":
        return dict(kind=kind, members=rng.randint(3, 8), nmin=8192, nmax=int(size(16384, 131072)),
                    sizes=rng.randrange(1 << 20), steps=rng.randint(4, 10), precision=precision)
    hydro = rng.choice(["sph", "sph", "crk"])
    problem = "kh" if hydro == "crk" else rng.choice(["sod", "kh"])
    if problem == "sod":
        k = size(2048, 190000) ** (1.0 / 3.0) / 2.0
        nx, ny, nz = int(8 * k * rng.uniform(0.8, 1.2)), max(8, int(k * rng.uniform(0.9, 1.1))), max(8, int(k))
        steps = 1 if kind != "steps" else rng.randint(2, 10)
    else:
        m = size(4096, 0.3 * WIDEST if hydro == "crk" else 0.6 * WIDEST) ** (1.0 / 3.0)
        nx, ny, nz = (max(12, int(m * rng.uniform(0.9, 1.1))) for _ in range(3))
        steps = 1 if kind != "steps" else rng.randint(2, 10 if hydro == "crk" else 20)
    return dict(kind=kind, problem=problem, nx=nx, ny=ny, nz=nz, steps=steps, hydro=hydro, precision=precision,
                xsph=hydro == "sph" and rng.random() < 0.3, shuffle=rng.random() < 0.3,
                relax=kind == "steps" and hydro == "sph" and rng.random() < 0.3, cube=False)


# ------------------------------------------------------------------ node sets
def one_problem(case):
    """(problem, nx, ny, nz) of each member of a case, from the case alone."""
    if case["kind"] == "batch":
        r = random.Random(case["sizes"])
        ks = [int(round(math.exp(r.uniform(math.log(case["kmin"]), math.log(case["kmax"]))))) for _ in range(case["members"])]
        return [("sod", 8 * k, k, k) for k in ks]
    if case["kind"] == "serve":
        r = random.Random(case["sizes"])
        out = []
        for q in range(case["members"]):
            n = math.exp(r.uniform(math.log(case["nmin"]), math.log(case["nmax"])))
            m, k = max(8, int(round(n ** (1.0 / 3.0)))), max(4, int(round((n / 8.0) ** (1.0 / 3.0))))
            out.append(("kh", m, m, m) if q % 2 == 0 else ("sod", 8 * k, k, k))
        return out
    return [(case["problem"], case["nx"], case["ny"], case["nz"])]


def nodes_of(case, seed, at=0):
    """Inputs and parameters of one member: AoS tensors on the GPU, in lattice order and in the caller's."""
    problem, nx, ny, nz = one_problem(case)[at]
    g = torch.Generator(device="cuda").manual_seed(seed * 1009 + at)
    n = nx * ny * nz
    ens = random.Random(seed * 31 + at) if case["kind"] == "batch" else None
    gamma = ens.uniform(1.3, 1.67) if ens else 5.0 / 3.0
    L = (1.0, 1.0, 1.0) if case.get("cube") else (1.0, ny / nx, nz / nx)
    if problem == "sod":
        nPerh, kernel = 1.51, pkg.abi.KERNEL_BSPLINE
    else:
        nPerh, kernel = 1.35, pkg.abi.KERNEL_WENDLANDC4
    d = torch.tensor([L[0] / nx, L[1] / ny, L[2] / nz], dtype=torch.float64, device="cuda")
    ig = torch.arange(n, device="cuda")
    idx = torch.stack([ig % nx, (ig // nx) % ny, ig // (nx * ny)], 1)
    lat = (idx + 0.5) * d
    pos = lat + (torch.rand(n, 3, dtype=torch.float64, device="cuda", generator=g) * 2 - 1) * JITTER * d
    vel = torch.zeros_like(pos)
    if problem == "sod":
        left = lat[:, 0] < 0.5
        rho = torch.where(left, 1.0, 1.0 / ens.uniform(2.0, 8.0) if ens else 0.25).double()
        P = torch.where(left, 1.0, 0.1795).double()
        # shortly after the membrane broke: gas moving around it, and the lattice noise of a run
        vel[:, 0] = 0.1 * torch.exp(-((lat[:, 0] - 0.5) / 0.1) ** 2)
        vel += (torch.rand(n, 3, dtype=torch.float64, device="cuda", generator=g) * 2 - 1) * 1.0e-3
    else:
        y = lat[:, 1] / L[1]
        inside = (y - 0.5).abs() < 0.25
        rho = torch.where(inside, 2.0, 1.0).double()
        P = torch.full_like(rho, 2.5)
        vel[:, 0] = torch.where(inside, 0.5, -0.5)
        env = torch.exp(-((y - 0.25) ** 2) / 0.005) + torch.exp(-((y - 0.75) ** 2) / 0.005)
        vel[:, 1] = 0.01 * torch.sin(4.0 * math.pi * lat[:, 0]) * env
    H = torch.zeros(n, 6, dtype=torch.float64, device="cuda")
    for c, a in ((0, 0), (3, 1), (5, 2)):
        H[:, c] = 1.0 / (nPerh * d[a])
    perm = torch.randperm(n, device="cuda", generator=g) if case.get("shuffle") else None
    return dict(n=n, dims=(nx, ny, nz), L=L, d=d, lat=lat, perm=perm, nPerh=nPerh, kernel=kernel, gamma=gamma,
                dtMin=1.0e-4 if problem == "sod" else 0.0, dtMax=1.0e-4 if problem == "sod" else 0.1,
                arrays=[pos, vel, rho * d.prod(), rho, P / ((gamma - 1.0) * rho), H])


def config_of(case, p):
    return pkg.abi.make_config(
        kernel=p["kernel"], nPerh=p["nPerh"], gamma=p["gamma"], xmin=(0.0, 0.0, 0.0), xmax=p["L"],
        dtMin=p["dtMin"], dtMax=p["dtMax"], XSPH=int(case.get("xsph", False)),
        hydro=pkg.abi.HYDRO_CRKSPH if case.get("hydro") == "crk" else pkg.abi.HYDRO_SPH,
        precision=pkg.abi.PRECISION_MIXED if case["precision"] == "mixed" else pkg.abi.PRECISION_FP64)


def callers_order(p):
    return [a if p["perm"] is None else a[p["perm"]].contiguous() for a in p["arrays"]]


STATE = (("position", 3), ("velocity", 3), ("mass", 1), ("mass density", 1), ("specific thermal energy", 1), ("H", 6))
DERIVS = ("delta velocity hydro", "delta specific thermal energy", "delta mass density", "velocity gradient", "new H",
          "max viscous pressure")


def pinned(n, comps):
    return torch.empty(n, comps, dtype=torch.float64, pin_memory=True) if comps > 1 else \
        torch.empty(n, dtype=torch.float64, pin_memory=True)


class Nodes:
    """Host AoS arrays of a request, under the names the package reads."""

    def __init__(self, arrays):
        self.pos, self.vel, self.mass, self.rho, self.eps, self.H = (a.cpu().numpy() for a in arrays)
        self.n = self.mass.shape[0]


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        reqs = []
        for q in range(case["members"]):
            p = nodes_of(case, seed, q)
            reqs.append((config_of(case, p), Nodes(p["arrays"])))
        return dict(case=case, server=pkg.serving.Server(100e9), reqs=reqs)
    members = []
    for q in range(len(one_problem(case))):
        p = nodes_of(case, seed, q)
        members.append((pkg.SPHHydro(config_of(case, p), n=p["n"]), callers_order(p)))
    n = sum(h.n for h, _ in members)
    state = dict(case=case, members=members)
    if kind == "evaluate":
        state["out"] = {k: pinned(n, pkg.hydro.FIELD_COMPONENTS[k]) for k in DERIVS}
    else:
        state["out"] = {k: pinned(n, c) for k, c in STATE}
    if kind == "batch":
        state["batch"] = pkg.SPHBatch([h for h, _ in members])
    torch.cuda.synchronize()
    if kind == "host_step":
        h, arrays = members[0]
        state["in"] = [pinned(*(a.shape if a.dim() > 1 else (a.shape[0], 1))).copy_(a) for a in arrays]
        torch.cuda.synchronize()
        # the program's start: derivatives at t = 0 feed the first predictor
        h.set_state_device([a.data_ptr() for a in arrays])
        h.build_neighbors()
        h.initialize()
        h.evaluateDerivatives()
        h.synchronize()
    return state


def get_state(h, out, at):
    ptrs = [ctypes.c_void_p(out[k].data_ptr() + 8 * c * at) for k, c in STATE]
    pkg.abi.check(h.lib.sphgpu_get_state(h.h, *ptrs), h.lib)


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "serve":
        return serve(state)
    out = state["out"]
    if kind == "host_step":
        h = state["members"][0][0]
        h.step_host([a.numpy() for a in state["in"]], [out[k].numpy() for k, _ in STATE])
        return out
    for h, arrays in state["members"]:
        h.set_state_device([a.data_ptr() for a in arrays])
    if kind == "batch":
        b = state["batch"]
        b.build_neighbors()
        b.evaluateDerivatives()
        b.step(case["steps"])
        at = 0
        for h, _ in state["members"]:
            get_state(h, out, at)
            at += h.n
        return out
    h = state["members"][0][0]
    if case["relax"]:
        h.iterateIdealH()
    h.build_neighbors()
    h.initialize()
    h.evaluateDerivatives()
    if kind == "evaluate":
        dt = h.dt()
        for k, v in out.items():
            pkg.abi.check(h.lib.sphgpu_get_field(h.h, k.encode(), ctypes.c_void_p(v.data_ptr()), v.numel()), h.lib)
        return dict(out, dt=dt, pairs=h.num_pairs())
    h.step(case["steps"])
    get_state(h, out, 0)
    return out


def serve(state):
    s = state["server"]
    ids = [s.submit(cfg, nodes, state["case"]["steps"]) for cfg, nodes in state["reqs"]]
    while True:
        running, queued = s.tick()
        if not running and not queued:
            break
    s.finished()
    got = [s.fetch(i) for i in ids]
    return {k: np.concatenate([g[k] for g in got]) for k, _ in STATE}


# ------------------------------------------------------------------ work
def work(case):
    """Per step and node: the state read and written (15 doubles), the 54 StateDerivatives doubles written and the
    16 the update needs read, the ConnectivityMap written and read (4-byte entries); plus the pass's inputs and
    outputs.  Operations per directed pair: about 250 for the derivatives, 70 for the summed density, the compatible
    energy and the dt vote; CRKSPH 600 with its moments."""
    bytes_, flops = 0.0, 0.0
    for problem, nx, ny, nz in one_problem(case):
        n = nx * ny * nz
        reach = 2 * 1.51 if problem == "sod" else 1.35
        entries = n * 4.0 / 3.0 * math.pi * reach ** 3
        pair = 600 if case.get("hydro") == "crk" else 320
        if case["kind"] == "evaluate":
            bytes_ += n * (120 + 432 + 8 * 21) + 8 * entries
            flops += entries * 260
            continue
        first = 0 if case["kind"] in ("serve", "host_step") else 1
        steps = case["steps"]
        bytes_ += n * 240 + steps * (n * (240 + 432 + 128) + 8 * entries) + first * (n * (120 + 432) + 8 * entries)
        flops += entries * (steps * pair + first * 260)
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------------------ the same in torch, 64 bits
class Table:
    """The tabulated kernel: 1000 points over the extent, a parabola through each three, and the lattice sums that
    turn the zeroth moment of the gradient into nodes per smoothing scale."""

    N = 1000

    def __init__(self, kernel):
        bspline = kernel == pkg.abi.KERNEL_BSPLINE
        self.extent = 2.0 if bspline else 1.0
        self.step = self.extent / (self.N - 1)
        x = np.arange(self.N) * self.step
        if bspline:
            w = np.where(x < 1, 1 - 1.5 * x ** 2 + 0.75 * x ** 3, 0.25 * np.maximum(2 - x, 0) ** 3) / math.pi
            g = np.where(x < 1, -(3 - 2.25 * x) * x, -0.75 * np.maximum(2 - x, 0) ** 2) / math.pi
        else:
            c = 495.0 / (32.0 * math.pi)
            w = c * (1 - x) ** 6 * (1 + 6 * x + 35.0 / 3.0 * x ** 2) * (x < 1)
            g = c * 56.0 / 3.0 * (x - 1) ** 5 * x * (5 * x + 1) * (x < 1)
        self.w, self.g = (torch.tensor(self.parabolas(t), device="cuda") for t in (w, g))
        nperh = 0.25 + np.arange(self.N) * (9.75 / (self.N - 1))
        wsum = np.empty(self.N)
        for i, p in enumerate(nperh):
            e = np.cumsum(np.concatenate([[0.0], np.full(int(self.extent * p) + 2, 1.0 / p)]))
            e = e[e < self.extent]
            k = np.where(e > 0, 2.0, 1.0)
            r = np.sqrt(e[:, None, None] ** 2 + e[None, :, None] ** 2 + e[None, None, :] ** 2)
            s = np.abs(self.lookup_np(r)) * k[:, None, None] * k[None, :, None] * k[None, None, :]
            s[0, 0, 0] = 0.0
            wsum[i] = s.sum() ** (1.0 / 3.0)
        self.nperh, self.wsum = torch.tensor(nperh, device="cuda"), torch.tensor(wsum, device="cuda")

    def parabolas(self, t):
        c = np.zeros((self.N - 2, 3))
        c[:, 0], c[:, 1] = t[:-2], -1.5 * t[:-2] + 2 * t[1:-1] - 0.5 * t[2:]
        c[:, 2] = 0.5 * t[:-2] - t[1:-1] + 0.5 * t[2:]
        return c

    def lookup_np(self, eta):
        c = self.g.cpu().numpy() if not hasattr(self, "gn") else self.gn
        self.gn = c
        q = eta / self.step
        i = np.minimum(q.astype(np.int64), self.N - 3)
        x = q - i
        return np.where(eta < self.extent, c[i, 0] + x * (c[i, 1] + x * c[i, 2]), 0.0)

    def __call__(self, eta, det):
        q = eta / self.step
        i = q.long().clamp(max=self.N - 3)
        x = q - i
        inside = eta < self.extent

        def look(c):
            return torch.where(inside, det * (c[:, 0][i] + x * (c[:, 1][i] + x * c[:, 2][i])), 0.0)

        return look(self.w), look(self.g)

    def nodes_per_scale(self, w, nPerh):
        j = (torch.searchsorted(self.wsum, w.contiguous(), right=True) - 1).clamp(0, self.N - 2)
        a, b = self.wsum[j], self.wsum[j + 1]
        t = ((w - a) / (b - a)).clamp(0.0, 1.0)
        return torch.where(w < 1.0e-15, 0.5 * nPerh, self.nperh[j] + t * (self.nperh[j + 1] - self.nperh[j]))


TABLES = {}


def full(h):
    """(n, 6) symmetric records to (n, 3, 3)."""
    return h[:, [0, 1, 2, 1, 3, 4, 2, 4, 5]].reshape(-1, 3, 3)


def mv(m, v):
    return (m * v[:, None, :]).sum(2)


def dot(a, b):
    return (a * b).sum(1)


class Exact:
    """One problem: state tensors in lattice order, H as (n, 3, 3)."""

    def __init__(self, case, p):
        self.p, self.crk, self.xsph = p, case.get("hydro") == "crk", case.get("xsph", False)
        if p["kernel"] not in TABLES:
            TABLES[p["kernel"]] = Table(p["kernel"])
        self.T = TABLES[p["kernel"]]
        self.L = torch.tensor(p["L"], dtype=torch.float64, device="cuda")
        x, v, m, rho, eps, H = p["arrays"]
        self.x, self.v, self.m, self.rho, self.eps, self.H = x, v, m, rho, eps, full(H)
        self.zero = torch.zeros(p["n"], dtype=torch.float64, device="cuda")
        self.lastDt = 1.0e-5
        self.D = None
        self.vol = None
        self.pressure()

    def pressure(self):
        g1 = self.p["gamma"] - 1.0
        self.P = g1 * self.rho * self.eps
        self.cs = torch.sqrt((self.p["gamma"] * g1 * self.eps).clamp(min=0.0))

    def add(self, what):
        """Sums over the pairs of each node."""
        return torch.zeros((self.p["n"],) + what.shape[1:], dtype=torch.float64, device="cuda").index_add_(0, self.i, what)

    def largest(self, what):
        return torch.zeros_like(self.zero).scatter_reduce_(0, self.i, what, "amax", include_self=True)

    def connect(self):
        """Directed pairs (i, j, image shift): |H_i r| or |H_j r| within the kernel extent."""
        p, lat = self.p, self.p["lat"]
        moved = self.x - lat
        x = self.x = lat + moved - self.L * torch.round(moved / self.L)
        stray = (x - lat).abs().amax(0).tolist()
        reach = self.T.extent / float(self.eigenvalues().min())
        d = p["d"].tolist()
        win = [math.ceil((reach + 2 * stray[a]) / d[a]) for a in range(3)]
        ig = torch.arange(p["n"], device="cuda")
        nx, ny, nz = p["dims"]
        ix, iy, iz = ig % nx, (ig // nx) % ny, ig // (nx * ny)
        I, J, S = [], [], []
        for oz in range(-win[2], win[2] + 1):
            for oy in range(-win[1], win[1] + 1):
                for ox in range(-win[0], win[0] + 1):
                    least = sum(max(0.0, abs(o) * d[a] - 2 * stray[a]) ** 2 for a, o in enumerate((ox, oy, oz)))
                    if (ox == oy == oz == 0) or least > reach * reach:
                        continue
                    j = ((iz + oz) % nz * ny + (iy + oy) % ny) * nx + (ix + ox) % nx
                    s = torch.stack([(ix + ox) // nx, (iy + oy) // ny, (iz + oz) // nz], 1) * self.L
                    r = x - (x[j] + s)
                    Hj = self.H[j]
                    near = torch.minimum((mv(self.H, r) ** 2).sum(1), (mv(Hj, r) ** 2).sum(1)) <= self.T.extent ** 2
                    I.append(ig[near])
                    J.append(j[near])
                    S.append(s[near])
        self.i, self.j, self.s = torch.cat(I), torch.cat(J), torch.cat(S)
        self.count = torch.bincount(self.i, minlength=p["n"])

    def pairs(self):
        """A pair of two nodes counts once, a pair with a periodic image at the node that has it."""
        image = int((self.s != 0).any(1).sum())
        return (self.i.numel() - image) // 2 + image

    def eigenvalues(self):
        """H is diagonal throughout: the lattice's along the axes, the ideal one a multiple of one."""
        return self.H.diagonal(dim1=1, dim2=2)

    def sides(self):
        """Kernel and gradient of each pair with either node's H."""
        i, j = self.i, self.j
        self.det = torch.linalg.det(self.H)
        r = self.x[i] - (self.x[j] + self.s)
        out = [r]
        for k in (i, j):
            eta = mv(self.H[k], r)
            mag = torch.sqrt((eta ** 2).sum(1))
            W, gW = self.T(mag, self.det[k])
            out += [eta, W, gW, mv(self.H[k], eta / mag[:, None]) * gW[:, None]]
        return out

    def ideal_h(self, moment):
        p = self.p
        s = (p["nPerh"] / (self.T.nodes_per_scale(moment, p["nPerh"]) + 1.0e-30)).clamp(0.25, 4.0)
        a = torch.where(s < 1.0, 0.4 * (1.0 + s * s), 0.4 * (1.0 + 1.0 / s ** 3))
        h = (1.0 / self.H[:, 0, 0] * (1.0 - a + a * s)).clamp(1.0e-20, 1.0e20)
        return torch.eye(3, dtype=torch.float64, device="cuda") / h[:, None, None]

    def relax(self):
        """Start-up: H replaced by the ideal H until no node changes by more than 1e-4."""
        moving = torch.ones(self.p["n"], dtype=torch.bool, device="cuda")
        for _ in range(50):
            self.connect()
            eta = mv(self.H[self.i], self.x[self.i] - (self.x[self.j] + self.s))
            _, gW = self.T(torch.sqrt((eta ** 2).sum(1)), torch.ones_like(eta[:, 0]))
            H1 = self.ideal_h(self.add(gW.abs()) ** (1.0 / 3.0))
            change = (H1[:, 0, 0, None] / self.eigenvalues() - 1.0).abs().amax(1)
            self.H = torch.where(moving[:, None, None], H1, self.H)
            moving = moving & (change > 1.0e-4)
            if not bool(moving.any()):
                return

    def volumes(self):
        """Kernel-sum volumes of the CRKSPH form."""
        r, _, W, *_ = self.sides()
        W0 = self.T(self.zero, self.det)[0]
        top = (0.5 * self.T.extent) ** 3 * 4.0 / 3.0 * math.pi
        self.vol = torch.minimum(top / self.det, 1.0 / (self.add(W) + W0))

    def corrections(self):
        """Linear corrections A, B and their gradients from the moments."""
        r, _, Wi, _, Gi, _, Wj, _, Gj = self.sides()
        W, G, vj = 0.5 * (Wi + Wj), 0.5 * (Gi + Gj), self.vol[self.j]
        ww, eye = vj * W, torch.eye(3, dtype=torch.float64, device="cuda")
        vG, wr = vj[:, None] * G, ww[:, None] * r
        m0 = self.add(ww) + self.vol * self.T(self.zero, self.det)[0]
        m1, gm0 = self.add(wr), self.add(vG)
        m2 = self.add(wr[:, :, None] * r[:, None, :])
        gm1 = self.add(r[:, :, None] * vG[:, None, :]) + m0[:, None, None] * eye
        gm2 = self.add((r[:, :, None] * r[:, None, :]).reshape(-1, 9)[:, :, None] * vG[:, None, :]).reshape(-1, 3, 3, 3)
        gm2 = gm2 + m1[:, :, None, None] * eye[None, None] + m1[:, None, :, None] * eye[None, :, None, :]
        # too few neighbors to span the space: no first-order correction
        spans = (torch.linalg.det(m2).abs() > 1.0e-5 / self.det ** 2)[:, None, None]
        inv = torch.where(spans, torch.linalg.inv(torch.where(spans, m2, eye)), 0.0)
        C = mv(inv, m1)
        A = 1.0 / (m0 - dot(C, m1))
        gA = -(A * A)[:, None] * (gm0 - 2 * torch.einsum("nj,nji->ni", C, gm1) + torch.einsum("nk,nkli,nl->ni", C, gm2, C))
        gB = -inv @ gm1 + torch.einsum("nik,nklj,nl->nij", inv, gm2, C)
        return A, -C, gA, gB

    def evaluate(self):
        """Derivatives at the current state on the current pairs."""
        i, j, p = self.i, self.j, self.p
        r, ei, Wi, gWi, Gi, ej, Wj, gWj, Gj = self.sides()
        m, v, rho = self.m, self.v, self.rho
        vij = v[i] - v[j]

        def q(k, eta):
            mu = (dot(vij, eta) / (dot(eta, eta) + 1.0e-2)).clamp(max=0.0)
            return (-self.cs[k] * mu + mu * mu) / rho[k]

        qi, qj = q(i, ei), q(j, ej)
        D = {}
        if self.crk:
            A, B, gA, gB = self.corrections()
            W, G = 0.5 * (Wi + Wj), 0.5 * (Gi + Gj)

            def corrected(k, sign):
                rk = sign * r
                f = 1.0 + dot(B[k], rk)
                grad = (A[k] * f)[:, None] * (sign * G) + (A[k] * W)[:, None] * (B[k] + mv(gB[k].transpose(1, 2), rk)) \
                    + (f * W)[:, None] * gA[k]
                return A[k] * f * W, grad

            Wci, gci = corrected(i, 1.0)
            _, gcj = corrected(j, -1.0)
            dg = gci - gcj
            vi, vj = self.vol[i], self.vol[j]
            f = 0.5 * vi * vj
            force = (f * (self.P[i] + self.P[j] + qi * rho[i] ** 2 + qj * rho[j] ** 2))[:, None] * dg
            dd = force / (m[i] * m[j])[:, None]
            work = rho[j] ** 2 * qj * dot(vij, dg)
            D["eps"] = self.add(f * (self.P[j] * dot(vij, dg) + work) / m[i])
            D["maxvp"] = self.largest(4.0 * rho[i] ** 2 * qi.abs())
            grad = -self.add(vj[:, None, None] * vij[:, :, None] * gci[:, None, :])
            moment = self.add((0.5 * (gWi + gWj)).abs())
            D["x"] = v - self.add((vj * Wci)[:, None] * vij) if self.xsph else v
        else:
            Qi, Qj = 0.5 * qi[:, None] * Gi, 0.5 * qj[:, None] * Gj
            Pr = self.P / rho ** 2
            dd = Pr[i][:, None] * Gi + Pr[j][:, None] * Gj + Qi + Qj
            D["eps"] = self.add(m[j] * (Pr[i] * dot(vij, Gi) + dot(vij, Qi)))
            D["maxvp"] = self.largest(rho[i] ** 2 * qi.abs())
            mG = m[j][:, None] * Gi
            grad = -self.add(vij[:, :, None] * mG[:, None, :])
            M = -self.add(r[:, :, None] * mG[:, None, :])
            good = (torch.linalg.det(M).abs() > 1.0e-10) & (self.count > 8)
            inv = torch.linalg.inv(torch.where(good[:, None, None], M, torch.eye(3, dtype=torch.float64, device="cuda")))
            grad = torch.where(good[:, None, None], grad @ inv, grad / rho[:, None, None])
            moment = self.add(gWi.abs())
            D["x"] = v
            if self.xsph:
                w = 0.5 * ((m / rho)[i] * Wi + (m / rho)[j] * Wj)
                own = self.det * m / rho * self.T(self.zero, torch.ones_like(self.zero))[0]
                D["x"] = v - self.add(w[:, None] * vij) / (self.add(w) + own)[:, None]
        D["v"] = -self.add(m[j][:, None] * dd)
        D["grad"] = grad
        trace = grad.diagonal(dim1=1, dim2=2).sum(1)
        D["rho"] = -rho * trace
        D["H"] = -self.H / 3.0 * trace[:, None, None]
        D["ideal"] = self.ideal_h((moment / self.det).clamp(min=0.0) ** (1.0 / 3.0))
        D["dd"] = dd
        self.D = D

    def vote(self):
        D, v = self.D, self.v
        scale = 1.0 / self.eigenvalues().amax(1) / self.p["nPerh"]
        tiny = 1.17549435082228750797e-38
        vij = v[self.i] - v[self.j]
        fast = torch.sqrt(self.largest(dot(vij, vij)))
        trace = D["grad"].diagonal(dim1=1, dim2=2).sum(1)
        votes = [scale / (self.cs + tiny), scale / (torch.sqrt(D["maxvp"] / self.rho) + tiny),
                 1.0 / (trace.abs() + tiny), scale / fast.clamp(min=1.0e-30),
                 torch.sqrt(scale / (torch.sqrt(dot(D["v"], D["v"])) + tiny))]
        return 0.25 * min(float(t.min()) for t in votes)

    def step(self):
        p, old = self.p, self.D
        dt = min(p["dtMax"], self.vote(), 2.0 * self.lastDt)
        dt = min(p["dtMax"], max(p["dtMin"], dt))
        start = self.x, self.v, self.rho, self.eps, self.H, self.vol

        def advance(D, h, eps_rate, H):
            x, v, rho, eps, _, vol = start
            self.x, self.v, self.eps = x + h * D["x"], v + h * D["v"], eps + h * eps_rate
            self.rho, self.H = (rho + h * D["rho"]).clamp(1.0e-10, 1.0e10), H
            if self.crk:
                low, top = 0.5 * self.m / self.rho, 4.0 * math.pi / (3.0 * torch.linalg.det(H))
                self.vol = torch.maximum(low, torch.minimum(top, vol - h * self.m / self.rho ** 2 * D["rho"]))
            self.pressure()

        advance(old, 0.5 * dt, old["eps"], start[4] + 0.5 * dt * old["H"])
        self.evaluate()
        D, i, j = self.D, self.i, self.j
        half = start[1] + 0.5 * dt * D["v"]
        weight = D["eps"].abs() + 2.220446049250313e-16
        rate = self.add(weight[i] / (weight[i] + weight[j]) * self.m[j] * dot(half[i] - half[j], D["dd"]))
        advance(D, dt, rate, D["ideal"])
        self.lastDt = dt
        # the summed density at the new state, then the periodic wrap
        if self.crk:
            self.volumes()
        r, _, _, _, _, _, Wj, _, _ = self.sides()
        W0 = self.T(self.zero, self.det)[0]
        if self.crk:
            vj, vol = self.vol[j], self.vol
            ws = self.add(vj * Wj) + vol * W0
            v1 = (self.add(vj * vj * Wj) + vol * vol * W0) / ws
            top = (self.add(self.m[j] * vj * Wj) + self.m * vol * W0) / (ws * v1)
            self.rho = torch.maximum(0.1 * self.m * self.det, top)
        else:
            self.rho = self.add(self.m[j] * Wj) + self.m * W0
        self.x = self.x - self.L * torch.floor(self.x / self.L)

    def still(self):
        """Derivatives before any evaluation."""
        n, z = self.p["n"], self.zero
        m33 = torch.zeros(n, 3, 3, dtype=torch.float64, device="cuda")
        self.D = dict(x=m33[:, 0], v=m33[:, 0], rho=z, eps=z, H=m33, grad=m33, maxvp=z)


def exact_member(case, seed, at):
    p = nodes_of(case, seed, at)
    e = Exact(case, p)
    if case["kind"] == "serve":
        e.still()
    else:
        if case.get("relax"):
            e.relax()
        e.connect()
        if e.crk:
            e.volumes()
        e.evaluate()
    order = (lambda a: a) if p["perm"] is None else (lambda a: a[p["perm"]])
    sym = (lambda H: H.reshape(-1, 9)[:, [0, 1, 2, 4, 5, 8]])
    if case["kind"] == "evaluate":
        D = e.D
        fields = [D["v"], D["eps"], D["rho"], D["grad"].reshape(-1, 9), sym(D["ideal"]), D["maxvp"]]
        return dict(zip(DERIVS, (order(f) for f in fields)), dt=e.vote(), pairs=e.pairs())
    for _ in range(case["steps"]):
        e.connect()
        if e.crk and e.vol is None:
            e.volumes()
        e.step()
    fields = [e.x, e.v, e.m, e.rho, e.eps, sym(e.H)]
    return dict(zip([k for k, _ in STATE], (order(f) for f in fields)))


def exact(case, seed):
    pairs = 0.0
    for problem, nx, ny, nz in one_problem(case):
        pairs += nx * ny * nz * (118.0 if problem == "sod" else 14.0) * (3.0 if case.get("hydro") == "crk" else 1.0)
    if pairs * (case["steps"] + 1) > EXACT_MOST:
        return None
    got = [exact_member(case, seed, q) for q in range(len(one_problem(case)))]
    return got[0] if len(got) == 1 else {k: torch.cat([g[k] for g in got]) for k in got[0]}
