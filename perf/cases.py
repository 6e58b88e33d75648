"""Performance cases of the framework's public entry points, over the range users run them at.

A case is a dict of plain values. `kind` names the entry point:

  steps     EulerDevice.upload, .step, .download: explicit steps on one mesh, the state taken from
            and returned to pinned host memory (a restart, some steps, a checkpoint)
  march     EulerDevice.upload, .march, .download: a steady march to the convergence rule
  batch     many steady channels as one union mesh: .upload, .march_cases, .download
  residual  EulerDevice.residual: R(U) of a host state into a host residual
  train     warmstart.MLP.set_parameters, .train, .parameters: the warm start's training
  gradient  warmstart.MLP.gradient: loss and gradient of one set of rows
  predict   warmstart.MLP.predict: the warm start's prediction of every cell
  wall      warmstart.wall_distance: the exact wall distance of every cell of several channels

`tuned` steppers run their autotuner when they are prepared, as the steady drivers and the benchmark
do; the others step with the launch choices a new handle has. Meshes do not depend on the seed
(generators with a fixed jitter) and are kept between preparations; states, parameters and training
rows come from the seed."""

from __future__ import annotations

import functools
from dataclasses import replace

import numpy as np
import torch

from autan_b200 import cases as C
from autan_b200 import mesh as M
from autan_b200.euler import ROUND_OFF_FLOOR, EulerDevice, residual_scales
from autan_b200.warmstart import MLP, wall_distance, wall_triangles

GAMMA = 1.4
# 600 steps of training with the FP32 sums of every GEMM in another order: 6e-4 of the parameters
TRAIN = {"rel": 3e-3, "max": 3e-2}


def listed() -> list[dict]:
    return [
        # the smallest solver call: the first-order vortex on the 64 x 64 x 2 periodic box, FP64,
        # classical RK4 with a global CFL step; twelve or so small launches a step
        dict(name="hex-8k-rk4-fp64", kind="steps", mesh="hex", nx=64, ny=64, nz=2, order="none",
             flux="roe", precision="fp64", second=False, rk=4, cfl=0.5, steps=10, tuned=False),
        # a coarse-grid start in reverse Cuthill-McKee order, odd sizes, another flux, untuned
        dict(name="channel-5k-hllc-rcm", kind="steps", mesh="channel", nx=37, ny=13, nz=9,
             order="rcm", flux="hllc", precision="fp32+acc64", second=True, rk=3, cfl=1.5, steps=20,
             tuned=False),
        # a single steady case of the size of the warm start's smaller channels, marched
        dict(name="channel-31k-march", kind="march", mesh="channel", nx=78, ny=27, nz=13,
             order="morton", flux="ausm", precision="fp32+acc64", second=True, rk=3, cfl=1.5,
             steps=30, tuned=True),
        # the steady production size class: AUSM+-up, local steps, mesh far beyond the caches
        dict(name="channel-2M-ausm", kind="steps", mesh="channel", nx=300, ny=94, nz=62,
             order="morton", flux="ausm", precision="fp32+acc64", second=True, rk=3, cfl=1.5, steps=20,
             tuned=True),
        # the unsteady tetrahedral vortex (2 073 600 cells), global CFL step, untuned
        dict(name="tets-2M-hllc", kind="steps", mesh="tets", nx=240, ny=240, nz=6, order="morton",
             flux="hllc", precision="fp32+acc64", second=True, rk=3, cfl=0.8, steps=20, tuned=False),
        # the same in FP64 at a medium odd size (accuracy checks and the FP64 force checks)
        dict(name="tets-136k-fp64", kind="steps", mesh="tets", nx=61, ny=53, nz=7, order="morton",
             flux="hllc", precision="fp64", second=True, rk=3, cfl=0.8, steps=10, tuned=False),
        # many steady channels of different sizes, Mach numbers and angles in one batch
        dict(name="batch-24-roe", kind="batch", cases=24, low=8000, high=60000, draw_seed=0,
             flux="roe", precision="fp32+acc64", steps=20, tuned=True),
        # one residual of a host state on warped hexahedra in the generator's order: the call a
        # host-side solver makes
        dict(name="residual-31k-warped", kind="residual", mesh="warped", nx=57, ny=49, nz=11,
             order="none", flux="roe", precision="fp32+acc64", second=True),
        # an epoch's worth of minibatches of the warm start's training
        dict(name="train-256k", kind="train", rows=262144, batch=8192, epochs=2),
        # one forward and backward pass of an odd number of rows
        dict(name="gradient-5k", kind="gradient", rows=5003),
        # the prediction of every cell of a large test set
        dict(name="predict-1M", kind="predict", rows=1048576),
        # the wall distance of every cell of a few channels
        dict(name="wall-4x60k", kind="wall", cases=4, low=30000, high=90000, draw_seed=5),
    ]


def draw(rng) -> dict:
    def log(lo, hi):
        return float(np.exp(rng.uniform(np.log(lo), np.log(hi))))

    kind = rng.choice(["steps"] * 6 + ["march", "batch", "residual", "train", "gradient", "predict",
                                       "wall"])  # fmt: skip
    flux = rng.choice(["roe", "hllc", "ausm"])
    precision = rng.choice(["fp32+acc64", "fp32+acc64", "fp64"])
    order = rng.choice(["morton", "morton", "rcm", "none"])
    tuned = rng.random() < 0.5
    if kind in ("steps", "march", "residual"):
        family = "channel" if kind == "march" else rng.choice(["hex", "channel", "tets", "warped"])
        cells = log(4e3, 1.2e6 if kind == "steps" else 2e5)
        if family == "channel":
            a = (cells / (1.111 * 12.0)) ** (1.0 / 3.0)
            n = [6 * a, 2 * a, a]
            n = [max(9, round(v * rng.uniform(0.85, 1.15))) for v in n]
        else:
            per = 6.0 if family == "tets" else 1.0
            nz = rng.randint(4, 9)
            side = (cells / (per * nz)) ** 0.5
            n = [max(9, round(side * rng.uniform(0.8, 1.25))), max(9, round(side)), nz]
        second = family != "hex" or rng.random() < 0.5
        out = dict(kind=kind, mesh=family, nx=n[0], ny=n[1], nz=n[2], order=order, flux=flux,
                   precision=precision, second=second)  # fmt: skip
        if kind == "residual":
            return out
        rk = 3 if kind == "march" else rng.choice([3, 3, 4])
        cfl = 1.2 if family == "channel" else 0.5
        return dict(out, rk=rk, cfl=cfl, steps=rng.randint(6, 20), tuned=tuned)
    if kind == "batch":
        return dict(kind=kind, cases=rng.randint(4, 20), low=4000, high=rng.randint(8000, 50000),
                    draw_seed=rng.randrange(1000), flux=flux, precision=precision,
                    steps=rng.randint(8, 20), tuned=tuned)  # fmt: skip
    if kind == "train":
        return dict(kind=kind, rows=int(log(3e4, 3e5)), batch=128 * rng.randint(4, 96), epochs=1)
    if kind == "gradient":
        return dict(kind=kind, rows=int(log(500, 200000)))
    if kind == "predict":
        return dict(kind=kind, rows=int(log(2000, 1.5e6)))
    return dict(kind=kind, cases=rng.randint(2, 5), low=4000, high=rng.randint(8000, 60000),
                draw_seed=rng.randrange(1000))  # fmt: skip


# ---------------------------------------------------------------- inputs


@functools.lru_cache(maxsize=2)
def solver_case(family, nx, ny, nz, order, flux, precision, second):
    """The mesh, scheme and boundary data of a case, and its LSQ weights."""
    if family == "channel":
        case = C.bump_channel(nx, ny, nz, precision=precision, order=order)
    elif family == "tets":
        case = C.vortex_tets(nx, ny, nz, precision=precision, rcm=order)
    elif family == "hex":
        h = 10.0 / nx
        mesh = M.periodic_box_hex(nx, ny, nz, extent=(10.0, h * ny, h * nz), rcm=order)
        case = vortex_case(mesh, precision)
    else:  # warped hexahedra: the periodic box with jittered nodes
        h = 10.0 / 240
        extent = (nx * h, ny * h, nz * h)
        mesh = M.lattice("hexa", (nx, ny, nz), (0.0, 0.0, 0.0), extent, (True, True, False),
                         displacement=M.vortex_jitter((nx, ny, nz), extent), rcm=order)  # fmt: skip
        case = vortex_case(mesh, precision)
    scheme = replace(case.scheme, flux=flux, second_order=second, limiter=second)
    weights = case.mesh.gradient_weights(case.bc_kind)
    return replace(case, scheme=scheme), weights


def vortex_case(mesh, precision):
    speed = float(np.hypot(C.FREESTREAM[1], C.FREESTREAM[2]))
    scheme = C.Scheme(flux="roe", second_order=True, limiter=True, venkat_k=5.0, length=1.0,
                      scale=(C.FREESTREAM[0], speed, speed, speed, C.FREESTREAM[4]),
                      reference=C.freestream_reference(), precision=precision,
                      planar=bool(mesh.all_planar))  # fmt: skip
    kind = np.full(mesh.n_boundary_faces, M.BC_SLIP, dtype=np.uint8)
    return C.Case("vortex", mesh, scheme, kind, np.zeros((5, mesh.n_boundary_faces)),
                  np.zeros((5, mesh.n_cells)), rk=3, cfl=0.8, steps=1)  # fmt: skip


def solver_args(case):
    return (case["mesh"], case["nx"], case["ny"], case["nz"], case["order"], case["flux"],
            case["precision"], case["second"])  # fmt: skip


def smooth(x, rng, periods):
    """A smooth field over the points x (3 x n), in [-1, 1]: three products of sines and cosines
    with whole periods in x and y."""
    out = np.zeros(x.shape[1])
    lo, size = x.min(axis=1), np.maximum(np.ptp(x, axis=1), 1e-30)
    size = np.where(periods > 0, periods, size)
    for _ in range(3):
        k = rng.integers(1, 4, size=2)
        ph = rng.uniform(0, 2 * np.pi, size=2)
        out += np.sin(2 * np.pi * k[0] * (x[0] - lo[0]) / size[0] + ph[0]) * np.cos(
            2 * np.pi * k[1] * (x[1] - lo[1]) / size[1] + ph[1]
        )
    return out / 3.0


def start_state(case, sc, seed):
    """The conserved start (5 x n_cells): a developing flow, the freestream (channels) or a vortex
    with smooth perturbations of 2 per cent drawn from the seed."""
    rng = np.random.default_rng(seed)
    m = sc.mesh
    x = m.cell_centroid
    if case["mesh"] == "channel":
        w = np.array([1.0, 0.5, 0.0, 0.0, 1.0 / GAMMA])[:, None] * np.ones(m.n_cells)
        periods = np.zeros(3)
    else:
        size = np.array([case["nx"], case["ny"], case["nz"]]) * (
            10.0 / case["nx"] if case["mesh"] == "hex" else 10.0 / 240
        )
        scale = 10.0 / size[0]  # the vortex fills the box whatever its size
        centre = size[:2] * rng.uniform(0.4, 0.6, size=2)
        beta = rng.uniform(3.0, 5.0)
        dx, dy = (x[0] - centre[0]) * scale, (x[1] - centre[1]) * scale
        r2 = dx * dx + dy * dy
        f = beta / (2 * np.pi) * np.exp(0.5 * (1.0 - r2))
        t = 1.0 - (GAMMA - 1.0) * beta**2 / (8 * GAMMA * np.pi**2) * np.exp(1.0 - r2)
        rho = t ** (1.0 / (GAMMA - 1.0))
        w = np.stack([rho, 1.0 - f * dy, 1.0 + f * dx, np.zeros_like(rho), rho * t])
        periods = np.array([size[0], size[1], 0.0])
    for k, unit in ((0, 1.0), (1, 0.5), (2, 0.5), (4, 1.0 / GAMMA)):
        w[k] += 0.02 * unit * smooth(x, rng, periods)
    u = C.conserved(*w, GAMMA)
    if m.n_cells > m.n_owned_cells:
        u[:, m.n_owned_cells :] = u[:, m.ghost_owner]
    return np.ascontiguousarray(u)


def pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


@functools.lru_cache(maxsize=2)
def batch_case(n, low, high, draw_seed, flux, precision):
    return C.bump_batch(n, seed=draw_seed, cells=(low, high), flux=flux, precision=precision)


@functools.lru_cache(maxsize=2)
def wall_case(n, low, high, draw_seed):
    tri, pts = [], []
    for p in C.batch_parameters(n, draw_seed, (low, high)):
        m = M.bump_channel(*p["boxes"], bump=p["bump"])
        tri.append(wall_triangles(m, M.ZONE_BUMP))
        pts.append(m.cell_centroid[:, : m.n_owned_cells].copy())
        m.close()
    return tri, pts


def training_rows(rows, seed):
    """Features as the warm start's (a cell's position and wall distance, its case's Mach number,
    angle and bump height) and a smooth target of them with a little noise."""
    rng = np.random.default_rng(seed)
    x = np.column_stack([rng.uniform(0, 3, rows), rng.uniform(0, 1, rows), rng.uniform(0, 0.5, rows),
                         rng.uniform(0, 1, rows) ** 2, rng.uniform(0.3, 0.75, rows),
                         rng.uniform(-4, 4, rows), rng.uniform(0.02, 0.1, rows)])  # fmt: skip
    b = x[:, 6] * np.exp(-25.0 * (x[:, 0] - 1.5) ** 2) * np.exp(-3.0 * x[:, 3])
    a = np.radians(x[:, 5])
    y = np.column_stack([b * x[:, 4] ** 2, b * x[:, 4], a * np.tanh(5 * x[:, 3]), 0.01 * x[:, 2] * b,
                         2.5 * b * x[:, 4] ** 2 + 0.01 * a])  # fmt: skip
    y += 0.002 * rng.standard_normal(y.shape)
    return x.astype(np.float32), y.astype(np.float32)


def scaling(x, y):
    return [v.astype(np.float32) for v in (x.mean(0), np.maximum(x.std(0), 1e-6), y.mean(0),
                                           np.maximum(y.std(0), 1e-9))]  # fmt: skip


def network(case, seed):
    x, y = training_rows(case["rows"], seed)
    net = MLP(seed=seed % 1000003)
    net.set_scaling(*scaling(x, y))
    return net, x, y


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("steps", "march", "residual"):
        sc, weights = solver_case(*solver_args(case))
        dev = EulerDevice(sc.mesh, sc.scheme, sc.bc_kind, sc.bc_data, weights=weights)
        u = pinned((5, sc.mesh.n_cells))
        u[:] = start_state(case, sc, seed)
        s = dict(case=case, dev=dev, u=u)
        if kind != "residual":
            s["out"] = pinned(u.shape)
            if case["tuned"]:
                dev.upload(u)
                dev.autotune(cfl=case["cfl"], rk=case["rk"], local=local(case))
        if kind == "march":
            s["floors"] = ROUND_OFF_FLOOR * residual_scales(sc.mesh, 1.0, 1.0 / GAMMA, 0.5)
        return s
    if kind == "batch":
        b = batch_case(case["cases"], case["low"], case["high"], case["draw_seed"], case["flux"],
                       case["precision"])  # fmt: skip
        dev = b.open()
        u = pinned(b.u0.shape)
        u[:] = batch_state(b, seed)
        if case["tuned"]:
            dev.upload(u)
            dev.autotune(cfl=b.cfl, rk=b.rk, local=True)
        floors = np.stack([ROUND_OFF_FLOOR * p["phi"] for p in b.params])
        return dict(case=case, dev=dev, u=u, out=pinned(u.shape), floors=floors, cfl=b.cfl, rk=b.rk)
    if kind == "wall":
        tri, pts = wall_case(case["cases"], case["low"], case["high"], case["draw_seed"])
        rng = np.random.default_rng(seed)
        # another wall height and other points of the same channels
        s = rng.uniform(0.9, 1.1)
        pts = [p * (1.0 + 1e-3 * rng.uniform(-1, 1, size=p.shape)) for p in pts]
        tri = [t * np.tile([1.0, s, 1.0], 3) for t in tri]
        return dict(case=case, tri=tri, pts=pts)
    net, x, y = network(case, seed)
    s = dict(case=case, net=net, x=x, y=y)
    if kind == "train":
        net.set_data(x, y)
        s["p0"] = net.parameters()
    return s


def batch_state(b, seed):
    rng = np.random.default_rng(seed)
    u = b.u0.copy()
    off = b.cell_offsets
    for k in range(len(b.params)):
        at = slice(int(off[k]), int(off[k + 1]))
        x = b.mesh["cell_centroid"][:, at]
        for c in (0, 1, 4):
            u[c, at] *= 1.0 + 0.02 * smooth(x, rng, np.zeros(3))
    return u


def local(case):
    return case["mesh"] == "channel"


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "steps":
        dev = s["dev"]
        dev.upload(s["u"])
        r = dev.step(cfl=case["cfl"], rk=case["rk"], local=local(case), n_steps=case["steps"])
        return dict(u=dev.download(s["out"]), rms=r.residuals, dt=r.time_step)
    if kind == "march":
        dev = s["dev"]
        dev.upload(s["u"])
        r = dev.march(cfl=case["cfl"], rk=case["rk"], local=True, max_steps=case["steps"],
                      batch=max(1, case["steps"] // 2), orders=8.0, floors=s["floors"])  # fmt: skip
        return dict(u=dev.download(s["out"]), first=r["first"], last=r["last"], dt=r["time_step"],
                    iterations=r["iterations"])  # fmt: skip
    if kind == "batch":
        dev = s["dev"]
        dev.upload(s["u"])
        r = dev.march_cases(cfl=s["cfl"], rk=s["rk"], local=True, max_steps=case["steps"],
                            batch=max(1, case["steps"] // 2), orders=8.0, floors=s["floors"])  # fmt: skip
        return dict(u=dev.download(s["out"]), first=r["first"], iterations=r["iterations"])
    if kind == "residual":
        return s["dev"].residual(s["u"])
    if kind == "train":
        s["net"].set_parameters(s["p0"])
        loss = s["net"].train(epochs=case["epochs"], batch=case["batch"], lr=1e-3, seed=12)
        return dict(loss=loss, parameters=s["net"].parameters())
    if kind == "gradient":
        loss, g = s["net"].gradient(s["x"], s["y"])
        return dict(loss=loss, grad=g)
    if kind == "predict":
        return s["net"].predict(s["x"])
    return wall_distance(s["tri"], s["pts"])


# ---------------------------------------------------------------- work, tolerance


def solver_sizes(case):
    """(cells, faces, stencil entries) of a solver case from its boxes."""
    if case["kind"] in ("batch", "wall"):
        n = sum(1.111 * np.prod(p["boxes"]) for p in
                C.batch_parameters(case["cases"], case["draw_seed"], (case["low"], case["high"])))  # fmt: skip
        return n, 3.1 * n, 23.0 * n
    n = case["nx"] * case["ny"] * case["nz"]
    if case["mesh"] == "channel":
        return 1.111 * n, 3.4 * n, 25.5 * n
    if case["mesh"] == "tets":
        return 6.0 * n, 12.2 * n, 83.0 * n
    return n, 3.1 * n, 24.0 * n


def work(case):
    kind = case["kind"]
    if kind in ("steps", "march", "batch", "residual"):
        n, f, e = solver_sizes(case)
        w = 8.0 if case["precision"] == "fp64" else 4.0
        second = case.get("second", True)
        # per evaluation: the stencil's weights and cells, the faces' normals, areas, offsets and
        # cells, the cells' primitives; per stage the FP64 state read and written and the stage read
        stencil = e * (3 * w + 4) if second else 0.0
        face = f * (4 * w + (6 * w if second else 0) + 8)
        per_eval = stencil + face + n * (5 * w + 8)
        flops_eval = (e * 35.0 + f * 90.0 if second else 0.0) + f * 250.0
        if kind == "residual":
            return dict(bytes=per_eval + 80.0 * n, flops=flops_eval)
        stages = case.get("rk", 3) * case["steps"]
        return dict(bytes=stages * (per_eval + 120.0 * n) + 80.0 * n,
                    flops=stages * (flops_eval + 40.0 * n))  # fmt: skip
    macs = 7 * 128 + 3 * 128 * 128 + 128 * 5
    if kind == "wall":
        n, _, _ = solver_sizes(case)
        return dict(bytes=32.0 * n, flops=n * 60.0 * 16)
    rows = case["rows"]
    if kind == "predict":
        return dict(bytes=rows * 48.0, flops=2.0 * macs * rows)
    if kind == "gradient":
        return dict(bytes=rows * 48.0 + macs * 8.0, flops=6.0 * macs * rows)
    return dict(bytes=case["epochs"] * (rows * 52.0 + (rows // case["batch"]) * macs * 28.0),
                flops=6.0 * macs * case["epochs"] * (rows // case["batch"]) * case["batch"])  # fmt: skip


def tolerance(case):
    kind = case["kind"]
    if kind in ("steps", "march", "batch", "residual"):
        if case["precision"] == "fp64":
            return {"rel": 1e-12, "max": 1e-10}
        # a host state's residual is a small difference of its fluxes: up to 5e-5 off FP64; a state
        # after some steps, its norms and steps: 2e-7 off
        return {"rel": 2e-4, "max": 5e-3} if kind == "residual" else {"rel": 1e-6, "max": 2e-5}
    if kind == "wall":
        return {"rel": 1e-14, "max": 1e-13}
    # BF16 operands: the gradient is 3.5e-3 off FP64, the prediction 1.7e-3
    return TRAIN if kind == "train" else {"rel": 1e-2, "max": 0.3}


# ---------------------------------------------------------------- the same in 64 bits


def exact(case, seed):
    kind = case["kind"]
    if kind in ("steps", "march", "residual"):
        n, _, e = solver_sizes(case)
        evals = 1 if kind == "residual" else case["rk"] * case["steps"]
        if evals * (e if case["second"] else 6 * n) > 6e7:
            return None
        sc, weights = solver_case(*solver_args(case))
        solver = Reference(sc, weights, case["flux"])
        u = start_state(case, sc, seed)
        if kind == "residual":
            r = np.zeros_like(u)
            r[:, : solver.no] = solver.residual(u[:, : solver.no])
            return r
        v = u[:, : solver.no].copy()
        rms = []
        for _ in range(case["steps"]):
            v, norm, dt = solver.step(v, case["cfl"], local(case), case["rk"])
            rms.append(norm)
        u[:, : solver.no] = v
        u[:, solver.no :] = v[:, sc.mesh.ghost_owner]
        if kind == "march":
            return dict(u=u, first=rms[0], last=rms[-1], dt=dt, iterations=None)
        return dict(u=u, rms=rms[-1], dt=dt)
    if kind == "wall":
        s = prepare(case, seed)
        if sum(t.shape[0] * p.shape[1] for t, p in zip(s["tri"], s["pts"])) > 3e8:
            return None
        return [exact_distance(t, p) for t, p in zip(s["tri"], s["pts"])]
    if kind in ("gradient", "predict"):
        net, x, y = network(case, seed)
        loss, grad, pred = exact_network(net.parameters(), x, y, scaling(x, y), kind == "gradient")
        return dict(loss=loss, grad=grad) if kind == "gradient" else pred
    return None


def exact_network(p, x, y, sc, backward):
    """The 7 -> 4 x 128 (GELU) -> 5 network's loss, gradient and prediction."""
    im, isd, om, osd = (torch.from_numpy(v.astype(np.float64)) for v in sc)
    q = torch.from_numpy(p.astype(np.float64)).requires_grad_(backward)
    a = (torch.from_numpy(x.astype(np.float64)) - im) / isd
    t = (torch.from_numpy(y.astype(np.float64)) - om) / osd
    at = 0
    for i, o in ((7, 128), (128, 128), (128, 128), (128, 128), (128, 5)):
        z = a @ q[at : at + i * o].reshape(o, i).T + q[at + i * o : at + i * o + o]
        at += i * o + o
        a = torch.nn.functional.gelu(z) if o == 128 else z
    loss = ((a - t) ** 2).mean()
    if backward:
        loss.backward()
        return float(loss.detach()), q.grad.numpy(), None
    return float(loss), None, (a * osd + om).numpy()


def exact_distance(tri, pts):
    """Each point's least distance to the triangles: inside a triangle's prism its plane's, else the
    least of its edges'."""
    a, b, c = (torch.from_numpy(tri[:, 3 * k : 3 * k + 3].copy()) for k in range(3))
    x = torch.from_numpy(np.ascontiguousarray(pts.T))
    out = torch.empty(x.shape[0], dtype=torch.float64)
    n = torch.linalg.cross(b - a, c - a)
    nn = (n * n).sum(1)
    step = max(1, 2_000_000 // max(1, a.shape[0]))
    for i in range(0, x.shape[0], step):
        p = x[i : i + step, None, :]
        best = None
        inside = None
        for s, e in ((a, b), (b, c), (c, a)):
            d = e - s
            w = p - s
            h = ((w * d).sum(2) / (d * d).sum(1)).clamp(0.0, 1.0)
            r = w - h[..., None] * d
            r2 = (r * r).sum(2)
            best = r2 if best is None else torch.minimum(best, r2)
            side = (torch.linalg.cross(d.expand_as(w), w) * n).sum(2) >= 0
            inside = side if inside is None else inside & side
        plane = ((p - a) * n).sum(2) ** 2 / nn
        best = torch.where(inside, torch.minimum(best, plane), best)
        out[i : i + step] = best.min(dim=1).values.sqrt()
    return out.numpy()


class Reference:
    """The explicit Euler residual and its Runge-Kutta steps in FP64 numpy: least-squares face2
    gradients with the given weights, the Venkatakrishnan limiter, MUSCL reconstruction, Roe (with
    Harten's fix), HLLC or AUSM+-up fluxes, warped-face terms, boundary states."""

    def __init__(self, case, weights, flux):
        m, s = case.mesh, case.scheme
        self.s, self.flux, self.second = s, flux, s.second_order
        self.g, self.rgas = s.gamma, s.gas_constant
        self.no, self.ni, self.nif = m.n_owned_cells, m.n_interior_faces, m.n_owned_interior_faces
        self.val = np.concatenate([np.arange(self.no), np.asarray(m.ghost_owner, dtype=np.int64)])
        r = s.reference
        self.pref = (self.g - 1) * (r[4] - 0.5 * (r[1] ** 2 + r[2] ** 2 + r[3] ** 2) / r[0])
        self.n, self.area = m.face_normal, m.face_area_magnitude
        own = m.owner.astype(np.int64)
        nei = m.neighbour.astype(np.int64)
        xc, xf = m.cell_centroid, m.face_centroid
        f = np.arange(self.nif)
        self.l, self.r = own[f], nei[f]
        self.rl, self.rr = xf[:, f] - xc[:, self.l], xf[:, f] - xc[:, self.r]
        self.bo = own[self.ni :]
        self.rb = xf[:, self.ni :] - xc[:, self.bo]
        self.kind, self.data = case.bc_kind, case.bc_data
        self.volume = m.cell_volume[: self.no]
        end = int(m.stencil_offsets[self.no])
        st = m.stencil[:end].astype(np.int64)
        nb = self.bo.size
        self.sidx = np.where(st >= 0, self.val[np.maximum(st, 0)], self.no + (-st - 1 - self.ni))
        assert nb == 0 or self.sidx.max() < self.no + nb
        self.soff = np.asarray(m.stencil_offsets[: self.no], dtype=np.int64)
        self.scell = np.repeat(np.arange(self.no), np.diff(m.stencil_offsets[: self.no + 1]))
        self.w = np.asarray(weights).reshape(3, -1)[:, :end]
        ce = int(m.cell_face_offsets[self.no])
        self.cf = m.cell_faces[:ce].astype(np.int64)
        self.coff = np.asarray(m.cell_face_offsets[: self.no], dtype=np.int64)
        self.ccell = np.repeat(np.arange(self.no), np.diff(m.cell_face_offsets[: self.no + 1]))
        self.crel = xf[:, self.cf] - xc[:, self.ccell]
        inside = self.cf < self.ni
        side = own[self.cf] == self.ccell
        other = np.where(inside, np.where(side, nei[np.minimum(self.cf, self.ni - 1)], own[self.cf]), 0)
        self.cother = np.where(inside, self.val[other], self.no + self.cf - self.ni)
        self.csign = np.where(side, 1.0, -1.0)
        self.moment = None if s.planar else m.face_moment

    def prim(self, u):
        rho, v = u[0], u[1:4] / u[0]
        p = (self.g - 1) * (u[4] - 0.5 * (u[1:4] * v).sum(0))
        return np.concatenate([rho[None], v, p[None] - self.pref])

    def boundary(self, wg):
        """The boundary state (gauge) of every boundary face from interior values wg (gauge)."""
        g, out = self.g, wg.copy()
        n = self.n[:, self.ni :]
        w = wg.copy()
        w[4] += self.pref
        vn = (w[1:4] * n).sum(0)
        with np.errstate(invalid="ignore"):
            c = np.sqrt(g * w[4] / w[0])
        for kind in np.unique(self.kind):
            k = self.kind == kind
            d, wi, nk = self.data[:, k], w[:, k], n[:, k]
            o = wi.copy()
            if kind == M.BC_STATE:
                o = d.copy()
            elif kind == M.BC_SLIP:
                o[1:4] -= 2 * vn[k] * nk
            elif kind == M.BC_OUTLET:
                dp = wi[4] - d[4]
                sub = vn[k] < c[k]
                q = np.concatenate([(wi[0] - dp / c[k] ** 2)[None], wi[1:4] + dp / (wi[0] * c[k]) * nk,
                                    d[4][None]])  # fmt: skip
                o = np.where(sub, q, wi)
            elif kind == M.BC_INLET:
                gm = g - 1
                rr = vn[k] + 2 * c[k] / gm
                h0 = g * self.rgas * d[1] / gm
                disc = np.maximum((gm + 2) * h0 - 0.5 * gm * rr * rr, 0)
                cb = gm * (rr + np.sqrt(disc)) / (gm + 2)
                vb = np.minimum(rr - 2 * cb / gm, 0)
                tb = d[1] - 0.5 * gm * vb * vb / (g * self.rgas)
                pb = d[0] * (tb / d[1]) ** (g / gm)
                o = np.concatenate([(pb / (self.rgas * tb))[None], vb * nk, pb[None]])
            elif kind == M.BC_FARFIELD:
                vf = (d[1:4] * nk).sum(0)
                cf = np.sqrt(g * d[4] / d[0])
                rp, rm = vn[k] + 2 * c[k] / (g - 1), vf - 2 * cf / (g - 1)
                vb, cb = 0.5 * (rp + rm), 0.25 * (g - 1) * (rp - rm)
                ws = np.where(vb < 0, d, wi)
                vs = np.where(vb < 0, vf, vn[k])
                rb = (cb * cb / (g * ws[4] / ws[0] ** g)) ** (1 / (g - 1))
                o = np.concatenate([rb[None], ws[1:4] + (vb - vs) * nk, (rb * cb * cb / g)[None]])
                o = np.where(vn[k] >= c[k], wi, np.where(vf <= -cf, d, o))
            else:  # no-slip wall at rest
                o[0] = np.where(d[0] > 0, wi[4] / (self.rgas * np.where(d[0] > 0, d[0], 1)), wi[0])
                o[1:4] = 0
            out[:, k] = o
            out[4, k] -= self.pref
        return out

    def physical(self, w, n):
        g = self.g
        p = w[4] + self.pref
        vn = (w[1:4] * n).sum(0)
        h = g / (g - 1) * p / w[0] + 0.5 * (w[1:4] ** 2).sum(0)
        m = w[0] * vn
        return np.concatenate([m[None], m * w[1:4] + w[4] * n, (m * h)[None]]), vn, p, h

    def numerical(self, a, b, n):
        g = self.g
        fl, vl, pl, hl = self.physical(a, n)
        fr, vr, pr, hr = self.physical(b, n)
        rl, rr = a[0], b[0]
        if self.flux == "ausm":
            minf = self.s.mach_ref
            csl, csr = (np.sqrt(2 * (g - 1) / (g + 1) * h) for h in (hl, hr))
            c = np.minimum(csl**2 / np.maximum(csl, vl), csr**2 / np.maximum(csr, -vr))
            ml, mr = vl / c, vr / c
            mb = 0.5 * (vl**2 + vr**2) / c**2
            mo = np.sqrt(np.minimum(1, np.maximum(mb, minf**2)))
            fa = mo * (2 - mo)
            al = 3 / 16 * (-4 + 5 * fa * fa)
            rho = 0.5 * (rl + rr)
            mp = -0.25 / fa * np.maximum(1 - mb, 0) * (pr - pl) / (rho * c * c)

            def m2(m):
                return 0.25 * (m + 1) ** 2, -0.25 * (m - 1) ** 2

            lp, lm = m2(ml)
            rp, rm = m2(mr)
            big_l, big_r = np.abs(ml) >= 1, np.abs(mr) >= 1
            m = (np.where(big_l, 0.5 * (ml + np.abs(ml)), lp * (1 - 2 * lm))
                 + np.where(big_r, 0.5 * (mr - np.abs(mr)), rm * (1 + 2 * rp)) + mp)  # fmt: skip
            pp = np.where(big_l, (ml > 0) * 1.0, lp * ((2 - ml) - 16 * al * ml * lm))
            pm = np.where(big_r, (mr < 0) * 1.0, rm * ((-2 - mr) + 16 * al * mr * rp))
            p = pp * a[4] + pm * b[4] - 0.75 * pp * pm * (rl + rr) * fa * c * (vr - vl)
            p = p + (pp + pm - 1) * self.pref
            up = m > 0
            md = c * m * np.where(up, rl, rr)
            w, h = np.where(up, a, b), np.where(up, hl, hr)
            return np.concatenate([md[None], md * w[1:4] + p * n, (md * h)[None]])
        s = np.sqrt(rr / rl)
        v = (a[1:4] + s * b[1:4]) / (1 + s)
        h = (hl + s * hr) / (1 + s)
        q2 = (v * v).sum(0)
        c = np.sqrt((g - 1) * (h - 0.5 * q2))
        vn = (v * n).sum(0)
        if self.flux == "roe":
            dv, dp, dr = b[1:4] - a[1:4], b[4] - a[4], rr - rl
            dvn, rho = vr - vl, s * rl

            def fix(lam):
                d = 0.1 * c
                return np.where(np.abs(lam) < d, (lam**2 + d**2) / (2 * d), np.abs(lam))

            l1, l2, l5 = fix(vn - c), np.abs(vn), fix(vn + c)
            a1, a5 = l1 * (dp - rho * c * dvn) / (2 * c * c), l5 * (dp + rho * c * dvn) / (2 * c * c)
            a2, lr = l2 * (dr - dp / (c * c)), l2 * rho
            d = np.concatenate([
                (a1 + a2 + a5)[None],
                a1 * (v - c * n) + a2 * v + lr * (dv - dvn * n) + a5 * (v + c * n),
                (a1 * (h - c * vn) + a2 * 0.5 * q2 + lr * ((v * dv).sum(0) - vn * dvn)
                 + a5 * (h + c * vn))[None]])  # fmt: skip
            return 0.5 * (fl + fr) - 0.5 * d
        cl, cr = np.sqrt(g * pl / rl), np.sqrt(g * pr / rr)
        sl, sr = np.minimum(vl - cl, vn - c), np.maximum(vr + cr, vn + c)
        sm = (pr - pl + rl * vl * (sl - vl) - rr * vr * (sr - vr)) / (rl * (sl - vl) - rr * (sr - vr))

        def star(w, f, vk, p, sk):
            rs = w[0] * (sk - vk) / (sk - sm)
            q = (w[1:4] ** 2).sum(0)
            e = p / ((g - 1) * w[0]) + 0.5 * q
            st = np.concatenate([rs[None], rs * (w[1:4] + (sm - vk) * n),
                                 (rs * (e + (sm - vk) * (sm + p / (w[0] * (sk - vk)))))[None]])  # fmt: skip
            cs = np.concatenate([w[:1], w[0] * w[1:4], (w[0] * e)[None]])
            return f + sk * (st - cs)

        return np.where(sl >= 0, fl, np.where(sm >= 0, star(a, fl, vl, pl, sl),
                                              np.where(sr > 0, star(b, fr, vr, pr, sr), fr)))  # fmt: skip

    def evaluate(self, u):
        """Primitives, boundary states, gradients (5 x 3 x n) and limiter (5 x n)."""
        w = self.prim(u)
        wb = self.boundary(w[:, self.val[self.bo]])
        if not self.second:
            return w, wb, None, None
        allw = np.concatenate([w, wb], axis=1)
        grad = np.empty((5, 3, self.no))
        phi = np.empty((5, self.no))
        k3 = (self.s.venkat_k / self.s.length) ** 3
        for k in range(5):
            v = allw[k, self.sidx]
            dw = v - w[k, self.scell]
            for a in range(3):
                grad[k, a] = np.add.reduceat(dw * self.w[a], self.soff)
            hi = np.maximum(np.maximum.reduceat(v, self.soff), w[k]) - w[k]
            lo = np.minimum(np.minimum.reduceat(v, self.soff), w[k]) - w[k]
            d = (grad[k][:, self.ccell] * self.crel).sum(0)
            dp = np.where(d > 0, hi[self.ccell], lo[self.ccell])
            e2 = (k3 * self.s.scale[k] ** 2 * self.volume)[self.ccell]
            lim = (dp * dp + e2 + 2 * d * dp) / (dp * dp + 2 * d * d + d * dp + e2)
            phi[k] = np.minimum(np.minimum.reduceat(lim, self.coff), 1.0)
        return w, wb, grad, phi

    def reconstruct(self, w, grad, phi, cell, rel):
        if grad is None:
            return w[:, cell]
        t = w[:, cell] + phi[:, cell] * (grad[:, :, cell] * rel[None]).sum(1)
        ok = (t[0] > 0) & (t[4] + self.pref > 0)
        return np.where(ok, t, w[:, cell])

    def increment(self, w, dw, axis):
        """The physical flux's increment along one axis."""
        g = self.g
        ve, dve = w[1 + axis], dw[1 + axis]
        vv = (w[1:4] ** 2).sum(0)
        rh = g / (g - 1) * (w[4] + self.pref) + 0.5 * w[0] * vv
        drh = g / (g - 1) * dw[4] + 0.5 * dw[0] * vv + w[0] * (w[1:4] * dw[1:4]).sum(0)
        dm = dw[0] * ve + w[0] * dve
        out = np.concatenate([dm[None], dm * w[1:4] + w[0] * ve * dw[1:4], (drh * ve + rh * dve)[None]])
        out[1 + axis] += dw[4]
        return out

    def residual(self, u, ev=None):
        w, wb, grad, phi = ev if ev is not None else self.evaluate(u)
        l, r = self.val[self.l], self.val[self.r]
        a = self.reconstruct(w, grad, phi, l, self.rl)
        b = self.reconstruct(w, grad, phi, r, self.rr)
        f = self.area[: self.nif] * self.numerical(a, b, self.n[:, : self.nif])
        if self.moment is not None and grad is not None:
            m = self.moment[:, : self.nif].reshape(3, 3, -1)
            for j in range(3):
                d = 0.5 * sum(phi[:, c] * (grad[:, :, c] * m[None, :, j]).sum(1) for c in (l, r))
                f = f + self.increment(0.5 * (a + b), d, j)
        o = self.val[self.bo]
        wi = self.reconstruct(w, grad, phi, o, self.rb)
        n = self.n[:, self.ni :]
        fb = self.numerical(wi, self.boundary(wi), n)
        wall = self.kind == M.BC_SLIP
        if self.moment is not None:
            wall = wall | (self.kind == M.BC_WALL)
        fb = np.where(wall, np.concatenate([0 * wi[:1], wi[4] * n, 0 * wi[:1]]), fb)
        fb = self.area[self.ni :] * fb
        if self.moment is not None and grad is not None:
            m = self.moment[:, self.ni :].reshape(3, 3, -1)
            fb[1:4] += wall * phi[4, o] * (grad[4][:, None, o] * m).sum(0)
        if self.nif < self.ni:  # faces between ghosts, which no owned cell reads
            f = np.concatenate([f, np.zeros((5, self.ni - self.nif))], axis=1)
        allf = np.concatenate([f, fb], axis=1)
        return np.stack([np.add.reduceat(self.csign * allf[k, self.cf], self.coff) for k in range(5)])

    def time_step(self, w, wb, cfl):
        allw = np.concatenate([w, wb], axis=1)
        c = np.sqrt(self.g * (allw[4] + self.pref) / allw[0])
        n = self.n[:, self.cf]
        speed = [np.abs((allw[1:4, i] * n).sum(0)) + c[i] for i in (self.ccell, self.cother)]
        lam = np.add.reduceat(np.maximum(*speed) * self.area[self.cf], self.coff)
        return cfl * self.volume / lam

    def step(self, u, cfl, local_steps, rk):
        ev = self.evaluate(u)
        dt = self.time_step(ev[0], ev[1], cfl)
        least = dt.min()
        h = (dt if local_steps else least) / self.volume
        r = self.residual(u, ev)
        norm = np.sqrt((r * r).sum(1) / self.no)
        if rk == 3:
            s1 = u - h * r
            s2 = 0.75 * u + 0.25 * (s1 - h * self.residual(s1))
            return u / 3.0 + 2.0 / 3.0 * (s2 - h * self.residual(s2)), norm, least
        acc = r
        for c, b in ((0.5, 2.0), (0.5, 2.0), (1.0, 1.0)):
            r = self.residual(u - c * h * r)
            acc = acc + b * r
        return u - h / 6.0 * acc, norm, least
