"""Timed cases of the framework: time marching through plfbs.capi.Solver and
the warm-start network through plfbs.gnn.GraphNet.

A marching pass is what a solver program repeats between two outputs: run a
chunk of time steps, then read the fields (and the nodes of an immersed body)
back into page-locked host arrays. The state carries on from pass to pass,
except on tetrahedra, where a pass starts from the given field (the method
loses its stability there after some hundreds of steps). A `create` pass is the whole drop-in call of a program that solves once: create
the context from the host mesh, set the state, march, read back, free. A
network pass is one inference or one loss-and-gradient evaluation on host
arrays.

Sizes are the repository's own (the 32^3 cavity, the sphere channels of 64, 128
and 256 cells length, the 64^3 tetrahedra, the warm-start network's graph),
ragged ones of the same kinds, and draw() spreads over the range between.
Passes march steps_of(cells) steps, so that small meshes are timed over many
steps and large ones over few, as their output intervals are.
"""

from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "3d-plfbs-gpu_b200"))

from plfbs import capi, cases, gnn  # noqa: E402

FP64, FP32 = "fp64", "fp32"


def steps_of(cells):
    """Time steps of one pass."""
    return int(min(200, max(20, 1e8 / cells)))


def listed():
    out = []

    def add(name, **kw):
        out.append(dict(kw, name=name))

    # the smallest call: a channel of 360 cells (parabolic inlet, body force,
    # 32 nodes), where launches and their latency are all there is
    add("channel_10_fp64", kind="channel", nx=10, ny=6, nz=6, fp=FP64, body=True, inlet="parabolic",
        create=False, steps=10)
    # the lid-driven cavity of the plain-method configuration
    add("cavity_32_fp64", kind="cavity", nx=32, ny=32, nz=32, fp=FP64, body=False, inlet="uniform",
        create=False, steps=200)
    # the small sphere channel that is marched to a residual of 1e-6, in both precisions
    add("channel_64_fp64", kind="channel", nx=64, ny=32, nz=32, fp=FP64, body=True,
        inlet="uniform", create=False, steps=200)
    add("channel_64_fp32", kind="channel", nx=64, ny=32, nz=32, fp=FP32, body=True,
        inlet="uniform", create=False, steps=200)
    # the whole drop-in call on the middle sphere channel: create, set, march, read, free
    add("solve_128_fp64", kind="channel", nx=128, ny=64, nz=64, fp=FP64, body=True,
        inlet="uniform", create=True, steps=40)
    # the largest channel, the headline configuration, in both precisions
    add("channel_256_fp64", kind="channel", nx=256, ny=128, nz=128, fp=FP64, body=True,
        inlet="uniform", create=False, steps=24)
    add("channel_256_fp32", kind="channel", nx=256, ny=128, nz=128, fp=FP32, body=True,
        inlet="uniform", create=False, steps=48)
    # ragged graded hexes: every face record differs, hybrid gradient weights, gamma 1.3
    add("graded_odd_fp64", kind="graded", nx=89, ny=61, nz=47, fp=FP64, body=False,
        inlet="uniform", create=False, steps=200)
    # the unstructured stress mesh (64^3 jittered hexes, six tetrahedra each)
    add("tets_64_fp64", kind="tets", nx=64, ny=64, nz=64, fp=FP64, body=False, inlet="uniform",
        create=False, steps=40)
    # the CPU Solver's reconstruction and boundary rules on tetrahedra
    add("tets_23_cpu_fp64", kind="cpu_tets", nx=23, ny=23, nz=23, fp=FP64, body=False,
        inlet="uniform", create=False, steps=100)
    # the warm-start network on the small channel's graph: inference, and the
    # loss with its gradient (a training step's forward and backward)
    add("network_64_forward", kind="network", nx=64, ny=32, nz=32, layers=8, grad=False)
    add("network_64_gradient", kind="network", nx=64, ny=32, nz=32, layers=8, grad=True)
    return out


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["channel", "channel", "channel", "cavity", "graded", "tets", "cpu_tets",
                       "network"])
    if kind == "network":
        return dict(kind=kind, nx=_log_int(rng, 12, 64), ny=_log_int(rng, 8, 32),
                    nz=_log_int(rng, 8, 32), layers=rng.choice([4, 8]),
                    grad=rng.choice([False, True]))
    if kind in ("tets", "cpu_tets"):
        nx = ny = nz = _log_int(rng, 6, 60 if kind == "tets" else 32)
        cells = 6 * nx ** 3
    else:
        top = {"channel": 1.0, "cavity": 0.5, "graded": 0.5}[kind]
        nx = _log_int(rng, 8, 250 * top)
        ny, nz = (_log_int(rng, 6, 125 * top) for _ in range(2))
        cells = nx * ny * nz
    body = kind == "channel" and min(ny, nz) >= 16 and nx >= 24 and rng.random() < 0.7
    return dict(kind=kind, nx=nx, ny=ny, nz=nz,
                fp=FP64 if kind == "cpu_tets" else rng.choice([FP64, FP32]), body=body,
                inlet=rng.choice(["uniform", "parabolic"]) if kind == "channel" else "uniform",
                create=cells < 600000 and rng.random() < 0.25, steps=steps_of(cells))


# ---------------------------------------------------------------------------
# the solver's inputs
# ---------------------------------------------------------------------------
def _graded(n, ratio):
    return np.concatenate([[0.0], np.cumsum(ratio ** np.arange(n))])


@functools.lru_cache(maxsize=3)
def _problem(kind, nx, ny, nz, fp, body, inlet):
    """(mesh arrays, boundary types and values, solver configuration, immersed
    body or None) of a case: what the program has read or built before it
    calls the solver."""
    U, precision, gamma, fneq, mode, flavour = 0.05, capi.FP64, 1.0, 0.0, capi.GRAD_LS, 0
    pressure, origin, ibm = 0.0, (0.0, 0.0, 0.0), None
    lengths = (float(nx), float(ny), float(nz))
    sides = ["inlet", "outlet", "side", "side", "side", "side"]
    bcs = [cases.BC("inlet", 1, 1, 0, 0, "dirichlet", "neumann"),
           cases.BC("outlet", 1, 0, 0, 0, "neumann", "dirichlet"),
           cases.BC("side", 1, 0, 0, 0, "neumann", "neumann")]
    if kind == "channel":
        # sphere of a quarter of the channel, four nodes per unit area, Re 100
        ref, re, dt = max(2.0, min(ny, nz) / 4.0), 100.0, 0.2
        if inlet == "parabolic":  # no-slip walls and the profile about the centre line
            origin, pressure = (0.0, -ny / 2.0, -nz / 2.0), 1e-6
            bcs[0] = cases.BC("inlet", 1, 1, 0, 0, "parabolic", "neumann")
            bcs[2] = cases.BC("side", 1, 0, 0, 0, "dirichlet", "neumann")
        pm = cases.uniform_box(nx, ny, nz, origin=origin, patch_types=sides)
    elif kind == "cavity":
        ref, re, dt, U = float(nx), 100.0, 0.18, 0.1
        pm = cases.uniform_box(nx, ny, nz, patch_types=["wall"] * 3 + ["lid"] + ["wall"] * 2)
        bcs = [cases.BC("wall", 1, 0, 0, 0, "dirichlet", "neumann"),
               cases.BC("lid", 1, 1, 0, 0, "dirichlet", "neumann")]
    elif kind == "graded":
        xs, ys, zs = _graded(nx, 1.01), _graded(ny, 1.015), _graded(nz, 1.02)
        ref, re, dt, gamma, fneq, mode = 20.0, 50.0, 0.1, 1.3, 0.05, capi.GRAD_HYBRID
        lengths = (float(xs[-1]), float(ys[-1]), float(zs[-1]))
        pm = cases.hex_box(xs, ys, zs, patch_types=sides)
    else:
        ref, re, dt = float(nx), 400.0, 0.05
        pm = cases.jittered_tet_box(nx, jitter=0.1, seed=11, patch_types=["wall"] * 6)
        bcs = [cases.BC("wall", 1, 0, 0, 0, "dirichlet", "neumann")]
        if kind == "tets":
            mode = capi.GRAD_LS | capi.GRAD_EXACT_INVERSE
        else:
            mode, flavour = capi.GRAD_GREEN_GAUSS, capi.FLAVOUR_CPU_SOLVER
    if fp == FP32:
        precision = capi.FP32_DEVIATION
    c = cases.Case(mesh_dir="", X=lengths[0], Y=lengths[1], Z=lengths[2], dt=dt, mach=U,
                   reynolds=re, ref_length=ref, bcs=bcs)
    ma = capi.polymesh_geometry(pm, c.visc, gamma, fneq)
    rt, vt, val = cases.bc_arrays(ma, c)
    cfg = dict(visc=c.visc, gamma=gamma, dt=dt, domain_dt=0.5, max_velocity=U, ref_rho=1.0,
               tolerance=0.0, pressure_gradient=pressure, channel_height=lengths[1],
               origin=origin, lengths=lengths, gradient_mode=mode, precision=precision,
               renumber=0, flavour=flavour)
    if body:
        centre = (origin[0] + min(nx / 2.0, ny / 2.0), origin[1] + ny / 2.0, origin[2] + nz / 2.0)
        nodes = cases.fibonacci_sphere(int(round(4 * math.pi * ref * ref)), ref / 2, centre)
        ibm = dict(node_ref=nodes, stiffness=0.5, radius=ref / 2, depth=ref,
                   object_nodes=len(nodes))
    return ma, rt, vt, val, cfg, ibm


def _initial(case, seed):
    """The start field [C + B] x (rho, u, v, w) on the GPU: the case's mean flow
    (uniform, at rest, or a Taylor-Green field) and seeded long waves of a few
    percent on it, the kind of field a restart finds."""
    ma, _, _, _, cfg, _ = _mesh_of(case)
    g = torch.Generator().manual_seed(seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.from_numpy(np.asarray(ma.cell_centroid).reshape(-1, 3)).to(dev)
    U, L = cfg["max_velocity"], cfg["lengths"]
    out = []
    for amp in (2e-4, 0.03 * U, 0.03 * U, 0.03 * U):
        f = torch.zeros(x.shape[0], dtype=torch.float64, device=dev)
        for _ in range(3):
            k = torch.randint(1, 4, (3,), generator=g).tolist()
            p = (2 * math.pi * torch.rand(1, generator=g, dtype=torch.float64)).item()
            a = torch.randn(1, generator=g, dtype=torch.float64).item()
            arg = sum(2 * math.pi * k[d] / L[d] * x[:, d] for d in range(3))
            f += amp * a * torch.sin(arg + p)
        out.append(f)
    out[0] += 1.0
    if case["kind"] in ("channel", "graded"):
        out[1] += U
    elif case["kind"] in ("tets", "cpu_tets"):
        s = [2 * math.pi / L[d] * x[:, d] for d in range(3)]
        out[1] += U * torch.sin(s[0]) * torch.cos(s[1]) * torch.cos(s[2])
        out[2] -= U * torch.cos(s[0]) * torch.sin(s[1]) * torch.cos(s[2])
    return out


def _mesh_of(case):
    return _problem(*(case[k] for k in ("kind", "nx", "ny", "nz", "fp", "body", "inlet")))


# ---------------------------------------------------------------------------
# the network's inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _graph(nx, ny, nz):
    ma = cases.mesh_arrays(cases.uniform_box(nx, ny, nz), 0.008, 1.0, 0.0)
    return (ma,) + gnn.mesh_graph(ma)


def _network_inputs(case, seed):
    ma, src, dst, ef = _graph(case["nx"], case["ny"], case["nz"])
    rng = np.random.Generator(np.random.PCG64(seed))
    D = case["ny"] / 4.0
    centre = np.array([case["nx"] * 0.375, case["ny"] / 2, case["nz"] / 2]) + rng.uniform(-D, D, 3)
    x = gnn.node_features(ma, (case["nx"], case["ny"], case["nz"]), centre, D,
                          float(rng.uniform(20, 200)))
    t = np.stack([np.exp(-x[:, 3] ** 2), x[:, 4] * x[:, 6], x[:, 4] * x[:, 7], x[:, 4]], axis=1)
    t = ((t - t.mean(0)) / (t.std(0) + 1e-6) + 0.05 * rng.standard_normal(t.shape))
    p = gnn.init_params(x.shape[1], ef.shape[1], case["layers"], 4, seed=seed)
    return src, dst, ef, x, t.astype(np.float32), p


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
class _Marching:
    """The context (unless a pass creates its own), the start field and the
    arrays that the results are read into, in page-locked memory."""

    def __init__(self, case, seed):
        self.case = case
        self.problem = _mesh_of(case)
        T = self.problem[0].total_cells

        def pinned():
            return torch.empty(T, dtype=torch.float64,
                               pin_memory=torch.cuda.is_available()).numpy()

        self.start = []
        for f in _initial(case, seed):
            a = pinned()
            a[:] = f.cpu().numpy()
            self.start.append(a)
        self.out = [pinned() for _ in range(4)]
        # a single-precision run's fields are kept in single precision
        self.single = [torch.empty(T) for _ in range(4)] if case["fp"] == FP32 else None
        self.solver = None if case["create"] else self.create()

    def create(self):
        ma, rt, vt, val, cfg, ibm = self.problem
        s = capi.Solver(ma, rt, vt, val, cfg, ibm=ibm)
        s.set_fields(*self.start)
        return s


def prepare(case, seed):
    if case["kind"] == "network":
        src, dst, ef, x, t, p = _network_inputs(case, seed)
        net = gnn.GraphNet(src, dst, ef, x.shape[0], x.shape[1], case["layers"], t.shape[1])
        net.set_params(p)
        return dict(case=case, net=net, x=x, t=t)
    return _Marching(case, seed)


def run(state):
    if isinstance(state, dict):
        if state["case"]["grad"]:
            loss, grad = state["net"].gradients(state["x"], state["t"])
            return dict(loss=np.float32(loss), grad=grad)
        return dict(y=state["net"].forward(state["x"]))
    case, single = state.case, state.single
    s = state.solver or state.create()
    if state.solver is not None and case["kind"] in ("tets", "cpu_tets"):
        s.set_fields(*state.start)
    # the residual history of a single-precision run is not an output: its
    # last digits are rounding
    stats, hist = s.run(case["steps"], history=single is None)
    if stats["rc"]:
        raise RuntimeError("the solve diverged after %d steps" % stats["steps_done"])
    s.get_fields(*state.out)
    nodes = s.nodes() if s.N else ()
    if state.solver is None:
        s.close()
    if single is not None:
        for a, b in zip(state.out, single):
            b.copy_(torch.from_numpy(a))
        return dict(fields=list(single), nodes=[np.float32(a) for a in nodes])
    return dict(fields=list(state.out), history=hist, nodes=list(nodes))


def work(case):
    if case["kind"] == "network":
        n = case["nx"] * case["ny"] * case["nz"]
        e = 2 * (3 * n - case["nx"] * case["ny"] - case["ny"] * case["nz"] - case["nx"] * case["nz"])
        L, h = case["layers"], 64
        mac = (n * (9 * h + h * h) + e * (4 * h + h * h) + n * (h * h + h * 4)
               + L * (e * 4 * h * h + n * 3 * h * h))
        # node and edge states of each layer written once and read once by the
        # next; the gradient reads them (and the pre-activations) again and
        # moves the states' gradients the same way
        states = 4.0 * h * (L + 1) * (n + e)
        return {"bytes": (6 if case["grad"] else 2) * states, "flops": (6.0 if case["grad"] else 2.0) * mac}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["kind"] in ("tets", "cpu_tets"):
        c, b = 6 * nx ** 3, 12 * nx * nx
        f = 12 * nx ** 3 + b // 2
    else:
        c, b = nx * ny * nz, 2 * (nx * ny + ny * nz + nx * nz)
        f = 3 * c + b // 2
    v = 4 if case["fp"] == FP32 else 8
    # one RK stage: the state read and written, the step's start read, the
    # accumulator read and written, the connectivity; where geometry does not
    # repeat also 9 reals a face and 3 a gradient weight
    stage = 20 * v * c + 8 * f
    if case["kind"] not in ("channel", "cavity"):
        stage += 9 * v * f + 3 * v * (2 * f - b)
    steps = case["steps"]
    more = 8.0 * 4 * (c + b)  # the fields read back
    if case["kind"] in ("tets", "cpu_tets"):
        more *= 2  # and set
    if case["create"]:
        more += 8.0 * 4 * (c + b) + 76.0 * f + 40.0 * c + 8.0 * (2 * f - b)
    # per face: reconstruction, 15 equilibria and their moments; per cell:
    # gradient and update
    return {"bytes": 4.0 * steps * stage + more, "flops": 4.0 * steps * (420.0 * f + 250.0 * c)}


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _exact_network(case, seed):
    src, dst, ef, x, t, p = _network_inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    src, dst, ef, x, t = (torch.as_tensor(a).to(dev) for a in (src, dst, ef, x, t))
    src, dst, ef, x, t = src.long(), dst.long(), ef.double(), x.double(), t.double()
    params = torch.tensor(p, dtype=torch.float64, device=dev, requires_grad=case["grad"])
    H, at = 64, [0]

    def mlp(v, k, o):
        w = []
        for shape in ((k, H), (H,), (H, o), (o,)):
            n = math.prod(shape)
            w.append(params[at[0]:at[0] + n].view(shape))
            at[0] += n
        return torch.relu(v @ w[0] + w[1]) @ w[2] + w[3]

    with torch.set_grad_enabled(case["grad"]):
        h = mlp(x, x.shape[1], H)
        e = mlp(ef, ef.shape[1], H)
        for _ in range(case["layers"]):
            e = e + mlp(torch.cat([e, h[src], h[dst]], 1), 3 * H, H)
            h = h + mlp(torch.cat([h, torch.zeros_like(h).index_add(0, dst, e)], 1), 2 * H, H)
        y = mlp(h, H, t.shape[1])
        if not case["grad"]:
            return dict(y=y.cpu().numpy())
        loss = ((y - t) ** 2).mean()
        loss.backward()
    return dict(loss=float(loss), grad=params.grad.cpu().numpy())


_PAIRS = ((1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 1), (1, 1, -1), (1, -1, 1), (-1, 1, 1))
_IDX = (3, 0, 1, 2)  # state column of each field rho, u, v, w


class _Exact:
    """The time step on the whole mesh with torch's own operations: states
    (u, v, w, rho) [T, 4], gradients [T, 4 fields, 3]."""

    def __init__(self, case):
        ma, rt, vt, val, cfg, ibm = _mesh_of(case)
        self.dev = dev = "cuda" if torch.cuda.is_available() else "cpu"

        def t(a, dtype=torch.float64):
            return torch.as_tensor(np.asarray(a)).to(dev, dtype)

        self.cfg, self.ibm = cfg, ibm
        self.cpu_rules = cfg["flavour"] == capi.FLAVOUR_CPU_SOLVER
        self.C, self.F, self.Fi = ma.n_cells, ma.n_faces, ma.n_internal
        self.o, self.nb = t(ma.owner, torch.int64), t(ma.neighbour, torch.int64)
        self.n, self.A, self.dts = t(ma.face_normal), t(ma.face_area), t(ma.streaming_dt)
        xf, cc = t(ma.face_centroid), t(ma.cell_centroid)
        self.vol = t(ma.cell_volume)[: self.C]
        self.t1, self.t2 = cc[self.o] - xf, cc[self.nb] - xf
        self.rt, self.vt, self.val = t(rt, torch.int64), t(vt, torch.int64), t(val)
        bo = self.o[self.Fi:]
        d = cc[self.C:] - cc[bo]
        self.dmag = d.norm(dim=1)
        self.dhat = self.n[self.Fi:] if self.cpu_rules else d / self.dmag[:, None]
        nb_n = self.n[self.Fi:]
        self.keep = 1 - (nb_n if self.cpu_rules else nb_n.abs())
        self.target = self.val.clone()
        if not self.cpu_rules:
            Hh = cfg["channel_height"]
            y, z = cc[self.C:, 1], cc[self.C:, 2]
            prof = 16 * self.val[:, 0] * (Hh / 2 + y) * (Hh / 2 - y) * (Hh / 2 + z) * (Hh / 2 - z) / Hh ** 4
            self.target[:, 0] = torch.where(self.vt == 9, prof, self.target[:, 0])
        self._weights(cc, xf)

    def _weights(self, cc, xf):
        """Gradient weights of each face for its owner and its neighbour."""
        C, o, nb, inner = self.C, self.o, self.nb, self.nb[: self.Fi]
        d = cc[nb] - cc[o]
        disp = d.norm(dim=1)
        amax, dmax = (torch.zeros(C, dtype=torch.float64, device=self.dev) for _ in range(2))
        for acc, v in ((amax, self.A), (dmax, disp)):
            acc.scatter_reduce_(0, o, v, "amax")
            acc.scatter_reduce_(0, inner, v[: self.Fi], "amax")
        mode = self.cfg["gradient_mode"] & 0xff
        if mode == capi.GRAD_HYBRID:
            beta = (2 / (2 * dmax * amax / self.vol)).clamp(max=1.0)
        else:
            beta = torch.full((C,), 1.0 if mode == capi.GRAD_LS else 0.0, dtype=torch.float64,
                              device=self.dev)
        L = torch.zeros(C, 3, 3, dtype=torch.float64, device=self.dev)
        L += (2 * (1 - beta) * self.vol)[:, None, None] * torch.eye(3, device=self.dev, dtype=torch.float64)
        rhs = []
        for cell, sel, sgn in ((o, slice(None), 1.0), (inner, slice(0, self.Fi), -1.0)):
            dd, n, A = sgn * d[sel], self.n[sel], self.A[sel]
            ln = ((xf[sel] - cc[cell]) * n).sum(1)
            w = (2 * ln / (dd * n).sum(1)) ** 2 * A / disp[sel]
            b = beta[cell]
            L.index_add_(0, cell, (b * w)[:, None, None] * dd[:, :, None] * dd[:, None, :])
            rhs.append((b * w)[:, None] * dd + ((1 - b) * sgn * A)[:, None] * n)
        a, b, c, d_, e, f, g, h, k = (L[:, i, j] for i in range(3) for j in range(3))
        if self.cfg["gradient_mode"] & capi.GRAD_EXACT_INVERSE:
            det = a * (e * k - f * h) - b * (d_ * k - f * g) + c * (d_ * h - e * g)
        else:  # the reference's determinant as written, gradients.cpp:282-284
            det = a * (e * k - f * h) + b * (d_ * k - f - g) + c * (d_ * h - e * g)
        adj = torch.stack([e * k - f * h, c * h - b * k, b * f - c * e, f * g - d_ * k, a * k - c * g,
                           c * d_ - a * f, d_ * h - e * g, b * g - a * h, a * e - b * d_], 1)
        inv = (adj / det[:, None]).view(C, 3, 3)
        self.Go = torch.einsum("fij,fj->fi", inv[o], rhs[0])
        self.Gn = torch.einsum("fij,fj->fi", inv[inner], rhs[1])

    def ghosts(self, q):
        s, rt, vt, v = q[self.o[self.Fi:]], self.rt, self.vt, self.target
        g = q[self.C:]
        mirror = 2 * v - s
        if self.cpu_rules:
            g[:, 3] = torch.where(rt == 1, mirror[:, 3], torch.where(rt == 2, s[:, 3], v[:, 3]))
            flip = s[:, :3] * torch.tensor([1.0, -1.0, 1.0], device=self.dev, dtype=torch.float64)
            vel = torch.where((vt == 1)[:, None], mirror[:, :3], v[:, :3])
            vel = torch.where((vt == 2)[:, None], s[:, :3], vel)
            g[:, :3] = torch.where((vt == 8)[:, None], flip, vel)
        else:
            g[:, 3] = torch.where(rt == 1, mirror[:, 3], s[:, 3])
            g[:, :3] = torch.where((vt == 2)[:, None], s[:, :3], mirror[:, :3])

    def gradients(self, q):
        grad = torch.zeros(q.shape[0], 4, 3, dtype=torch.float64, device=self.dev)
        dq = (q[self.nb] - q[self.o])[:, _IDX]
        grad.index_add_(0, self.o, dq[:, :, None] * self.Go[:, None, :])
        grad.index_add_(0, self.nb[: self.Fi], -dq[: self.Fi, :, None] * self.Gn[:, None, :])
        bo = self.o[self.Fi:]
        jump = 2 * (self.val - q[bo])[:, _IDX]
        fixed = (jump / self.dmag[:, None])[:, :, None] * self.dhat[:, None, :]
        free = grad[bo] * self.keep[:, None, :]
        types = torch.stack([self.rt, self.vt, self.vt, self.vt], 1)
        if self.cpu_rules:
            velocity = torch.arange(4, device=self.dev) > 0
            dirichlet = (types == 1) | ((types == 8) & velocity)
            gb = torch.where((types == 2)[:, :, None], free, torch.zeros_like(free))
            gb = torch.where((types == 7)[:, :, None], grad[bo], gb)
            grad[self.C:] = torch.where(dirichlet[:, :, None], fixed, gb)
        else:
            grad[self.C:] = torch.where((types == 2)[:, :, None], free, fixed)
        return grad

    def fluxes(self, q, grad):
        pg, dt, n = 1.0 / self.cfg["gamma"], self.dts[:, None], self.n
        g1, g2 = grad[self.o], grad[self.nb]
        si = q[self.o][:, _IDX] - (self.t1[:, None, :] * g1).sum(2)
        sn = q[self.nb][:, _IDX] - (self.t2[:, None, :] * g2).sum(2)
        sc = 0.5 * (si + sn)
        # boundary faces; the reference's strict test leaves its first ghost
        # to the interior branch (LBFS.cu:356)
        b = slice(self.Fi + 1, None)
        owner = q[self.o[b]][:, _IDX]
        v = owner - (self.t1[b][:, None, :] * g2[b]).sum(2)
        rt, vt, val = self.rt[1:], self.vt[1:], self.val[1:]
        v[:, 0] = torch.where(rt == 1, val[:, 3], v[:, 0])
        fixed = vt == 1 if self.cpu_rules else vt != 2
        v[:, 1:] = torch.where(fixed[:, None], val[:, :3], v[:, 1:])
        if self.cpu_rules:
            sym = owner[:, 1:] * torch.tensor([1.0, 0.0, 1.0], device=self.dev, dtype=torch.float64)
            v[:, 1:] = torch.where((vt == 8)[:, None], sym, v[:, 1:])
        else:
            g1[b] = g2[b]
        si[b] = sn[b] = sc[b] = v

        def feq(w, lat, e):
            u = lat[:, 1:]
            eu = sum(e[k] * u[:, k] for k in range(3) if e[k]) if any(e) else 0.0 * u[:, 0]
            return w * lat[:, 0] * (1 + 3 * eu + 4.5 * eu * eu * pg - 1.5 * (u * u).sum(1) * pg)

        rho = feq(2 / 9, sc, (0, 0, 0))
        m = [torch.zeros_like(rho) for _ in range(3)]
        P = [[torch.zeros_like(rho) for _ in range(3)] for _ in range(3)]
        band = torch.zeros_like(rho) if self.cpu_rules else 0.001 * self.dts
        for e in _PAIRS:
            s = sum(e[k] * n[:, k] for k in range(3) if e[k])
            up, down = (s > band)[:, None], (s < -band)[:, None]
            e1 = sum(e[k] * g1[:, :, k] for k in range(3) if e[k])
            e2 = sum(e[k] * g2[:, :, k] for k in range(3) if e[k])
            mid = (si, e1) if self.cpu_rules else (sc, 0.5 * (e1 + e2))
            qa = torch.where(up, si - e1 * dt, torch.where(down, sn - e2 * dt, mid[0] - mid[1] * dt))
            qb = torch.where(up, sn + e2 * dt, torch.where(down, si + e1 * dt, mid[0] + mid[1] * dt))
            w = 1 / 9 if sum(map(abs, e)) == 1 else 1 / 72
            fa, fb = feq(w, qa, e), feq(w, qb, tuple(-k for k in e))
            rho = rho + fa + fb
            for i in range(3):
                if e[i]:
                    m[i] = m[i] + e[i] * (fa - fb)
                    for j in range(3):
                        if e[j]:
                            P[i][j] = P[i][j] + e[i] * e[j] * (fa + fb)
        tau = 3 * self.cfg["visc"] / self.dts * pg
        mn = sum(m[k] * n[:, k] for k in range(3))
        out = torch.empty(self.F, 4, dtype=torch.float64, device=self.dev)
        for a in range(3):
            eq = rho / 3 * n[:, a] + m[a] * mn / rho * pg
            out[:, a] = ((1 - tau) * eq + tau * sum(P[a][k] * n[:, k] for k in range(3))) * self.A
        out[:, 3] = mn * self.A
        return out

    def stencil(self, x):
        """Cells and weights of the nodes' 2 x 2 x 2 stencils [N, 8]."""
        h = self.cfg["domain_dt"] * 2
        xc, yc = int(self.cfg["lengths"][0] / h), int(self.cfg["lengths"][1] / h)
        org = torch.tensor(self.cfg["origin"], device=self.dev, dtype=torch.float64)
        r = (x - org) / h
        r = torch.stack([r[:, 0], r[:, 1].abs(), r[:, 2].abs()], 1)
        lo = torch.trunc(r + torch.copysign(torch.full_like(r, 0.5), r)) - 1
        off = torch.tensor([[i, j, k] for i in (0, 1) for j in (0, 1) for k in (0, 1)], device=self.dev)
        at = lo[:, None, :] + off
        w = (1 - (at + 0.5 - r[:, None, :]).abs()).prod(2) / h ** 3
        cell = (at[:, :, 0] + at[:, :, 1] * xc + at[:, :, 2] * xc * yc).long()
        ok = (cell >= 0) & (cell < self.C)
        return torch.where(ok, cell, 0), torch.where(ok, w, 0.0)

    def march(self, fields, steps):
        cfg = self.cfg
        q = torch.stack([fields[1], fields[2], fields[3], fields[0]], 1).to(self.dev)
        t1, hist, nodes = q[: self.C].clone(), [], []
        pressure = -cfg["pressure_gradient"] if self.cpu_rules else cfg["pressure_gradient"]
        if self.ibm:
            ref = torch.as_tensor(self.ibm["node_ref"]).to(self.dev)
            x = ref.clone()
            stiff = self.ibm["stiffness"] * (2 * math.pi * self.ibm["radius"]
                                             / self.ibm["object_nodes"] * self.ibm["depth"])
        mom = cfg["ref_rho"] * cfg["max_velocity"]
        for step in range(steps):
            t0 = t1.clone()
            force = torch.zeros(self.C, 4, dtype=torch.float64, device=self.dev)
            force[:, 0] = pressure
            if self.ibm:
                cell, w = self.stencil(x)
                vel = (q[cell][:, :, :3] * w[:, :, None]).sum(1)
                x = x + vel * cfg["dt"]
                fn = -stiff * (x - ref)
                cell, w = self.stencil(x)
                force[:, :3].index_add_(0, cell.reshape(-1), (fn[:, None, :] * w[:, :, None]).reshape(-1, 3))
                nodes = [x, vel, fn]
            for rk, (al, be) in enumerate(((1.0, 1 / 6), (0.5, 1 / 3), (0.5, 1 / 3), (1.0, 1 / 6))):
                self.ghosts(q)
                flux = self.fluxes(q, self.gradients(q))
                R = torch.zeros(self.C, 4, dtype=torch.float64, device=self.dev)
                R.index_add_(0, self.o, -flux)
                R.index_add_(0, self.nb[: self.Fi], flux[: self.Fi])
                R = R / self.vol[:, None] + force
                f = t0 + al * cfg["dt"] * R
                t1 = t1 + be * cfg["dt"] * R
                new = t1 if rk == 3 else f
                q[: self.C, :3], q[: self.C, 3] = new[:, :3] / new[:, 3:], new[:, 3]
            rms = (R ** 2).mean(0).sqrt()
            u, v, w, rho = (rms / rms.new_tensor([mom, mom, mom, cfg["ref_rho"]])).tolist()
            hist.append([float(step), max(u, v, w), rho, u, v, w])
        return q, hist, nodes


def exact(case, seed):
    if case["kind"] == "network":
        return _exact_network(case, seed)
    e = _Exact(case)
    q, hist, nodes = e.march(_initial(case, seed), case["steps"])
    out = dict(fields=[q[:, k].cpu().numpy() for k in (3, 0, 1, 2)],
               nodes=[a.cpu().numpy() for a in nodes])
    if case["fp"] == FP64:
        out["history"] = np.array(hist)
    return out
