"""The work a user of this library has it do, as cases that can be timed.

Every case goes through the public Python entry points (Solver, Batch and the
C ABI's adjoint calls); the field is read through the solver's device pointer,
as a program that keeps its data on the GPU does.  Lengths are in um, times in
min; the coefficients are the ranges of the library's own workloads (D
log-uniform in [1e3, 1e5], decay uniform in [0.01, 1], dt 0.01, 10 um voxels,
cells of 2494 um^3 with uptake in [0, 10] and secretion in [0, 1]).

Kinds:
  step      n whole steps (bulk, cells, LOD_3D) in one Solver.step call
  calls     one step as the reference's drivers make it: the three
            simulate_* calls one after another
  plane     one LOD_2D step
  exchange  one step of a coupled program: the agents' voxels and constants
            go up from host memory, one step, the agents' densities come back
  batch     several independent microenvironments of uneven sizes, n steps
            of all of them in one Batch.step call
  adjoint   n recorded steps from an initial field, then the gradients of a
            misfit's seed with respect to the coefficients and agents
  gradient  compute_all_gradient_vectors on the whole field
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.utils.checkpoint

from biofvm_b200 import Batch, Solver, _abi

DT = 0.01
CELL_VOLUME = 2494.0
PRECISION = {"fp64": _abi.FP64, "fp32": _abi.FP32, "mixed": _abi.FP32_FP64MATH}


def _case(name, kind, nx, ny, nz, S, agents=0, radius=0.0, dirichlet="none", precision="fp64",
          steps=1, members=1, every=0, dx=10.0):
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "S": S, "agents": agents,
         "radius": radius, "dirichlet": dirichlet, "precision": precision, "steps": steps,
         "members": members, "every": every, "dx": dx}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small tissue with a fixed boundary, stepped one step per call by
        # a program that moves its cells between steps
        _case("small_one_step", "step", 50, 50, 50, 1, agents=1000, dirichlet="boundary", dx=20.0),
        # the same domain left to run for a hundred steps in one call
        _case("small_100_steps", "step", 50, 50, 50, 1, agents=1000, dirichlet="boundary",
              steps=100, dx=20.0),
        # a domain whose sides are whatever the tissue measured: odd rows,
        # three substrates, scattered fixed nodes (vessels) and a supply region
        _case("odd_domain", "step", 161, 97, 123, 3, agents=20_000, radius=300.0,
              dirichlet="scattered"),
        # the ordinary size: oxygen, glucose and two factors on 128^3, driven
        # as the reference's example programs drive it
        _case("medium_calls", "calls", 128, 128, 128, 4, agents=20_000, radius=500.0),
        # the headline workload: ten substrates on 256^3
        _case("large_10", "step", 256, 256, 256, 10, agents=100_000, radius=500.0),
        # single precision at the largest size
        _case("largest_fp32", "step", 512, 512, 512, 8, agents=1_000_000, radius=500.0,
              precision="fp32"),
        # an FP32 field with FP64 arithmetic, the option for long runs in half the memory
        _case("large_mixed", "step", 256, 256, 256, 4, agents=50_000, radius=500.0,
              precision="mixed"),
        # a thin culture: the 2-D solver on a plane of 1000 x 1000 voxels
        _case("plane_16", "plane", 1000, 1000, 1, 16, dirichlet="boundary"),
        # a step of a coupled program with its agents in host memory
        _case("agent_exchange", "exchange", 128, 128, 128, 4, agents=50_000, radius=500.0),
        # an ensemble: independent domains of uneven sizes, run for 20 steps
        _case("ensemble", "batch", 128, 128, 128, 8, agents=10_000, radius=150.0, steps=20,
              members=12),
        # calibration: the gradient of a misfit through 40 steps
        _case("adjoint", "adjoint", 128, 128, 128, 4, agents=20_000, radius=300.0, steps=40,
              every=20),
        # chemotaxis: every substrate's gradient in every voxel
        _case("gradients", "gradient", 256, 256, 256, 4),
    ]


def _spread(rng, lo, hi):
    """An integer between lo and hi, spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _domain(rng, most, lo, hi, S):
    """Three side lengths in [lo, hi] with at most `most` voxel-densities."""
    while True:
        n = [_spread(rng, lo, hi) for _ in range(3)]
        if n[0] * n[1] * n[2] * S <= most:
            return n


def draw(rng):
    kind = rng.choice(["step", "step", "step", "small", "small", "single", "calls", "plane",
                       "exchange", "batch", "adjoint", "gradient"])
    agents = _spread(rng, 100, 100_000)
    radius = rng.choice([0.0, 150.0, 300.0, 500.0])
    dirichlet = rng.choice(["none", "boundary", "scattered"])
    if kind == "small":
        S = rng.randint(1, 3)
        n = _domain(rng, 1 << 19, 16, 64, S)
        return _case(None, "step", *n, S, agents=_spread(rng, 100, 5000), radius=radius,
                     dirichlet=dirichlet, steps=rng.choice([1, 10, 100]), dx=20.0)
    if kind == "single":
        S = rng.randint(1, 10)
        n = _domain(rng, 400_000_000, 48, 512, S)
        return _case(None, "step", *n, S, agents=agents, radius=radius, dirichlet="none",
                     precision=rng.choice(["fp32", "mixed"]))
    if kind == "plane":
        S = rng.randint(1, 16)
        return _case(None, "plane", _spread(rng, 100, 1024), _spread(rng, 100, 1024), 1, S,
                     dirichlet=dirichlet)
    if kind == "batch":
        S = rng.randint(1, 8)
        return _case(None, "batch", *[rng.randint(40, 128) for _ in range(3)], S,
                     agents=_spread(rng, 100, 10_000), radius=150.0, steps=rng.randint(5, 20),
                     members=rng.randint(3, 12))
    if kind == "adjoint":
        S = rng.randint(1, 4)
        n = _domain(rng, 128 ** 3 * 4, 24, 160, S)
        every = rng.randint(4, 20)
        return _case(None, "adjoint", *n, S, agents=_spread(rng, 100, 20_000), radius=300.0,
                     dirichlet=dirichlet, steps=rng.randint(8, 40), every=every)
    if kind == "gradient":
        S = rng.randint(1, 8)
        return _case(None, "gradient", *_domain(rng, 256 ** 3 * 4, 32, 320, S), S)
    S = rng.randint(1, 12)
    most = 128 ** 3 * 4 if kind == "exchange" else 150_000_000
    n = _domain(rng, most, 32, 320, S)
    if kind == "calls" or (dirichlet == "boundary" and max(n) > 96):
        dirichlet = "none"  # a fixed boundary is a small domain's; large ones have vessels
    return _case(None, kind, *n, S, agents=agents, radius=radius, dirichlet=dirichlet)


# ---- inputs, from the seed alone ---------------------------------------------


def _shapes(case):
    """(nx, ny, nz, S, agents) of every member."""
    if case["kind"] != "batch":
        return [(case["nx"], case["ny"], case["nz"], case["S"], case["agents"])]
    out = []
    # an ensemble's sizes belong to the case, not to the seed: the same work for every seed
    sizes = np.random.default_rng([case["members"], case["nx"], case["ny"], case["nz"]])
    for _ in range(case["members"]):
        n = [int(sizes.integers(min(32, v), v + 1)) for v in (case["nx"], case["ny"], case["nz"])]
        out.append((*n, int(sizes.integers(1, case["S"] + 1)),
                    int(sizes.integers(0, case["agents"] + 1))))
    return out


def _sphere(nx, ny, nz, dx, radius):
    """Voxels whose centre lies within `radius` of the domain's centre, ascending."""
    def near(n):
        x = (np.arange(n) + 0.5) * dx - 0.5 * n * dx
        k = np.flatnonzero(np.abs(x) <= radius)
        return k, x[k]
    (i, x), (j, y), (k, z) = near(nx), near(ny), near(nz)
    inside = x[None, None, :] ** 2 + y[None, :, None] ** 2 + z[:, None, None] ** 2 <= radius ** 2
    kk, jj, ii = np.nonzero(inside)
    return ((k[kk].astype(np.int64) * ny + j[jj]) * nx + i[ii]).astype(np.int64)


def _boundary(nx, ny, nz):
    on = np.zeros((nz, ny, nx), bool)
    on[:, :, 0] = on[:, :, -1] = on[:, 0] = on[:, -1] = True
    if nz > 1:
        on[0] = on[-1] = True
    return np.flatnonzero(on.ravel()).astype(np.int64)


def _inputs(case, seed):
    """Every member's inputs: host arrays, and a maker of the initial field on the GPU."""
    rng = np.random.default_rng(seed)
    out = []
    for b, (nx, ny, nz, S, agents) in enumerate(_shapes(case)):
        N, dx = nx * ny * nz, case["dx"]
        m = {"shape": (nx, ny, nz), "S": S, "N": N, "dx": dx, "gseed": int(seed) * 1000 + b}
        m["D"] = np.exp(rng.uniform(math.log(1e3), math.log(1e5), S))
        m["decay"] = rng.uniform(0.01, 1.0, S)
        m["bulk"] = _sphere(nx, ny, nz, dx, case["radius"]) if case["radius"] else \
            np.zeros(0, np.int64)
        m["supply"], m["target"] = 0.5, 1.0
        if case["dirichlet"] == "boundary":
            m["nodes"] = _boundary(nx, ny, nz)
            m["node_values"] = np.ones((m["nodes"].size, S))
        elif case["dirichlet"] == "scattered":
            m["nodes"] = np.sort(rng.choice(N, min(2000, N // 50), replace=False))
            m["node_values"] = rng.uniform(0.5, 5.0, (m["nodes"].size, S))
        else:
            m["nodes"], m["node_values"] = np.zeros(0, np.int64), np.zeros((0, S))
        pos = rng.random((agents, 3))
        ijk = np.minimum((pos * (nx, ny, nz)).astype(np.int64), np.array([nx, ny, nz]) - 1)
        m["agents"] = np.ascontiguousarray((ijk[:, 2] * ny + ijk[:, 1]) * nx + ijk[:, 0])
        c = DT * CELL_VOLUME / dx ** 3
        uptake, secretion = rng.uniform(0, 10.0, (agents, S)), rng.uniform(0, 1.0, (agents, S))
        m["temp1"] = secretion * c
        m["temp2"] = 1.0 + c * secretion + c * uptake
        out.append(m)
    return out


def _field(m, dtype=torch.float64, salt=0):
    """[N, S] densities between 0.5 and 1.5 on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(m["gseed"] * 2 + salt)
    return torch.rand((m["N"], m["S"]), generator=g, device="cuda", dtype=dtype) + 0.5


class _View:
    """Device memory of a solver as torch sees it; the tensor keeps this object, and so the
    solver, alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr,
                                         "data": (ptr, False), "version": 3, "strides": None}


def _view(owner, ptr, shape, fp64=True):
    t = torch.as_tensor(_View(owner, ptr, tuple(shape), "<f8" if fp64 else "<f4"), device="cuda")
    t.owner = owner
    return t


def _solver(case, m):
    sv = Solver(0)
    nx, ny, nz = m["shape"]
    S, dx = m["S"], m["dx"]
    sv.resize_densities(S)
    sv.resize_space(0.0, nx * dx, 0.0, ny * dx, 0.0, nz * dx, dx)
    sv.set_coefficients(m["D"], m["decay"])
    precision = PRECISION[case["precision"]]
    if precision != _abi.FP64:
        sv.set_precision(precision)
    fp64 = precision == _abi.FP64
    field = _view(sv, sv.device_pointer(), (m["N"], S), fp64)
    sv.synchronize()
    field.copy_(_field(m, torch.float64 if fp64 else torch.float32))
    if m["bulk"].size:
        E = m["bulk"].size
        sv.set_bulk_rates_sparse(m["bulk"], np.full((E, S), m["supply"]),
                                 np.full((E, S), m["target"]), np.zeros((E, S)))
    if m["nodes"].size:
        sv.add_dirichlet_nodes(m["nodes"], m["node_values"])
    if m["agents"].size and case["kind"] != "exchange":
        sv.set_agents(m["agents"], m["temp1"], m["temp2"])
    torch.cuda.synchronize()
    return sv, field


def prepare(case, seed):
    members = _inputs(case, seed)
    made = [_solver(case, m) for m in members]
    state = {"case": case, "solvers": [sv for sv, _ in made], "fields": [f for _, f in made]}
    sv, m = state["solvers"][0], members[0]
    if case["kind"] == "batch":
        batch = Batch(0)
        for s in state["solvers"]:
            batch.add(s)
        batch.set_mode(_abi.BATCH_BRANCHES)
        state["batch"] = batch
    elif case["kind"] == "exchange":
        # page-locked, as a program that copies every step keeps its arrays
        pin = lambda a: torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()  # noqa: E731
        state["agents"] = (pin(m["agents"]), pin(m["temp1"]), pin(m["temp2"]))
        state["read"] = pin(np.zeros((m["agents"].size, m["S"])))
    elif case["kind"] == "adjoint":
        A, S = m["agents"].size, m["S"]
        state["p0"] = state["fields"][0].clone()
        state["target"] = _field(m, salt=1)
        state["seed"] = torch.empty_like(state["p0"])
        state["grads"] = (np.zeros(S), np.zeros(S), np.zeros((A, S)), np.zeros((A, S)))
        state["stream"] = torch.cuda.ExternalStream(sv.stream)
    elif case["kind"] == "gradient":
        p = _abi.c_void_p()
        _abi.call("bfvm_device_gradients", sv.handle, _abi.ctypes.byref(p))
        state["gradients"] = _view(sv, p.value, (m["N"], m["S"], 3))
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    kind, sv, field = case["kind"], state["solvers"][0], state["fields"][0]
    if kind == "step":
        sv.step(DT, case["steps"])
        return field
    if kind == "calls":
        sv.simulate_bulk_sources_and_sinks(DT)
        sv.simulate_cell_sources_and_sinks(DT)
        sv.simulate_diffusion_decay(DT)
        return field
    if kind == "plane":
        sv.simulate_diffusion_decay_2d(DT)
        return field
    if kind == "exchange":
        sv.set_agents(*state["agents"])
        sv.step(DT, 1)
        sv.get_agent_densities(state["read"])
        return {"field": field, "read": state["read"]}
    if kind == "batch":
        state["batch"].step(DT, case["steps"])
        return state["fields"]
    if kind == "gradient":
        sv.compute_all_gradient_vectors()
        return state["gradients"]
    # adjoint: the loss is half the squared distance of the final field from the target
    with torch.cuda.stream(state["stream"]):
        field.copy_(state["p0"])
        _abi.call("bfvm_adjoint_forward", sv.handle, DT, case["steps"], _abi.STEP_ALL,
                  case["every"])
        torch.sub(field, state["target"], out=state["seed"])
        gD, gdecay, g1, g2 = state["grads"]
        agents = g1.shape[0] > 0
        _abi.call("bfvm_adjoint_backward", sv.handle, _abi.c_void_p(state["seed"].data_ptr()), 1,
                  _abi.dptr(gD), _abi.dptr(gdecay), _abi.dptr(g1) if agents else None,
                  _abi.dptr(g2) if agents else None, None)
    return {"field": field, "D": gD, "decay": gdecay, "temp1": g1, "temp2": g2}


# ---- what a pass cannot do without ---------------------------------------------


def work(case):
    es = 8 if case["precision"] == "fp64" else 4
    kind = case["kind"]
    bytes_, flops = 0.0, 0.0
    for nx, ny, nz, S, agents in _shapes(case):
        NS = nx * ny * nz * S
        lists = 16.0 * S * agents + 8.0 * agents
        if kind == "gradient":
            bytes_ += 8.0 * NS + 24.0 * NS
            flops += 6.0 * NS
        elif kind == "adjoint":
            # initial field, target and seed in, the final field out; the agents' gradients out
            bytes_ += 4 * 8.0 * NS + 2 * lists
            flops += 3 * 20.0 * NS * case["steps"]
        else:
            # the field in and out, the agents in (an exchange also returns their densities)
            bytes_ += 2.0 * es * NS + lists + (8.0 * S * agents if kind == "exchange" else 0.0)
            flops += (10.0 if kind == "plane" else 15.0) * NS * case["steps"]
    return {"bytes": bytes_, "flops": flops}


# ---- the same in 64 bits ---------------------------------------------------------


def _inverse(n, c1, c2):
    """(1 + c2) I + c1 L inverted, L the second difference with closed ends (zero for one point)."""
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    if n == 1:
        return eye / (1.0 + c2)
    off = torch.diag(torch.ones(n - 1, dtype=torch.float64, device="cuda"), 1)
    d = torch.full((n,), 2.0, dtype=torch.float64, device="cuda")
    d[0] = d[-1] = 1.0
    return torch.linalg.inv((1.0 + c2) * eye + c1 * (torch.diag(d) - off - off.T))


def _ranks(vox):
    """Agents as layers in which no voxel repeats, list order kept within a voxel."""
    order = np.argsort(vox, kind="stable")
    v = vox[order]
    first = np.flatnonzero(np.r_[True, v[1:] != v[:-1]])
    rank = np.arange(v.size) - np.repeat(first, np.diff(np.r_[first, v.size]))
    return [order[rank == r] for r in range(int(rank.max()) + 1)] if v.size else []


class _Exact:
    """One microenvironment in plain torch operations on FP64 tensors."""

    def __init__(self, m, dims=3):
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        self.m, self.dims = m, dims
        self.D, self.decay = up(m["D"]), up(m["decay"])
        self.bulk, self.nodes, self.values = up(m["bulk"]), up(m["nodes"]), up(m["node_values"])
        self.t1, self.t2 = up(m["temp1"]), up(m["temp2"])
        self.layers = [(up(k), up(m["agents"][k])) for k in _ranks(m["agents"])]

    def matrices(self):
        nx, ny, nz = self.m["shape"]
        c1 = DT * self.D / self.m["dx"] ** 2
        c2 = DT * self.decay / self.dims
        one = {n: [_inverse(n, c1[s], c2[s]) for s in range(self.m["S"])] for n in {nx, ny, nz}}
        return one[nx], one[ny], one[nz]

    def sources(self, p):
        if self.bulk.numel():
            su, st = self.m["supply"], self.m["supply"] * self.m["target"]
            p = p.index_copy(0, self.bulk, (p[self.bulk] + DT * st) / (su * DT + 1.0))
        for who, where in self.layers:
            p = p.index_copy(0, where, (p[where] + self.t1[who]) / self.t2[who])
        return p

    def fixed(self, p):
        return p.index_copy(0, self.nodes, self.values) if self.nodes.numel() else p

    def sweep(self, p, axis, inv):
        nx, ny, nz = self.m["shape"]
        planes = 1 if self.dims == 2 else nz
        q = p.view(nz, ny, nx, -1)[:planes]
        out = []
        for s, A in enumerate(inv):
            f = q[..., s]
            if axis == 0:
                f = f @ A.T
            elif axis == 1:
                f = A @ f
            else:
                f = (A @ f.reshape(nz, ny * nx)).view(nz, ny, nx)
            out.append(f)
        return torch.stack(out, dim=-1).view(planes * ny * nx, -1)

    def step(self, p, inverses):
        p = self.sources(p)
        for axis in range(3):
            p = self.sweep(self.fixed(p), axis, inverses[axis])
        return p


def _exact_adjoint(case, m):
    e = _Exact(m)
    for t in (e.D, e.decay, e.t1, e.t2):
        t.requires_grad_(True)
    inverses = e.matrices()
    p = _field(m)
    for _ in range(case["steps"]):
        p = torch.utils.checkpoint.checkpoint(e.step, p, inverses, use_reentrant=False)
    loss = 0.5 * ((p - _field(m, salt=1)) ** 2).sum()
    g = torch.autograd.grad(loss, (e.D, e.decay, e.t1, e.t2), allow_unused=True)
    g = [torch.zeros_like(t) if v is None else v for v, t in zip(g, (e.D, e.decay, e.t1, e.t2))]
    return {"field": p.detach(), "D": g[0], "decay": g[1], "temp1": g[2], "temp2": g[3]}


def _exact_gradient(m):
    nx, ny, nz = m["shape"]
    p = _field(m).view(nz, ny, nx, m["S"])
    g = torch.zeros((nz, ny, nx, m["S"], 3), dtype=torch.float64, device="cuda")
    d = 2.0 * m["dx"]
    g[:, :, 1:-1, :, 0] = (p[:, :, 2:] - p[:, :, :-2]) / d
    g[:, 1:-1, :, :, 1] = (p[:, 2:] - p[:, :-2]) / d
    g[1:-1, :, :, :, 2] = (p[2:] - p[:-2]) / d
    return g.view(m["N"], m["S"], 3)


def exact(case, seed):
    members = _inputs(case, seed)
    kind, m = case["kind"], members[0]
    if kind == "adjoint":
        return _exact_adjoint(case, m)
    if kind == "gradient":
        return _exact_gradient(m)
    dtype = torch.float64 if case["precision"] == "fp64" else torch.float32
    out = []
    with torch.no_grad():
        for m in members:
            e = _Exact(m, 2 if kind == "plane" else 3)
            inverses = e.matrices()
            p = _field(m, dtype).double()
            if kind == "plane":
                for axis in range(2):
                    p = e.sweep(e.fixed(p), axis, inverses[axis])
            else:
                for _ in range(case["steps"]):
                    p = e.step(p, inverses)
            out.append(p)
    if kind == "batch":
        return out
    if kind == "exchange":
        where = torch.from_numpy(m["agents"]).cuda()
        return {"field": out[0], "read": out[0][where]}
    return out[0]
