"""Workloads of the library's main entry points, for timing and comparison.

Each case is a dict of plain values.  ``prepare(case, seed)`` builds what a
program holds before the call (a Solver, Batch or MLP handle and host data made
from the seed), ``run(state)`` makes one pass through the public entry points,
``exact(case, seed)`` evaluates the same quantities in plain float64 tensor
operations, written here from the scheme's equations without the library.

Kinds of case:
  integrate  state in from pinned host memory, a run of Runge-Kutta steps,
             state back out (a host program between two of its saves)
  residual   one compute_residual with gradient and limiter read back into
             ordinary host arrays (a host code that keeps its own integrator)
  sweep      a batch of first-order airfoil cases advanced together
  dc         the batch's defect-correction phase from a half-converged state
  train      epochs of the warm-start network
  predict    its evaluation over the cells of a sweep
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from fvs2d_gb300 import Options, Solver, meshgen
from fvs2d_gb300.batch import Batch
from fvs2d_gb300.mlp import MLP

GAMMA = 1.4
PREC = {"fp64": 1, "mixed": 2, "df": 3}
GRAD = {"ggcell": 1, "ggnode": 2, "lsq-fn": 3, "lsq-nn": 3}
BC = {"freestream": 1, "slip_wall": 2, "dirichlet": 4}
MACH_VORTEX = 0.5
KAPPA_REF = 5.0


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed() -> list:
    return [
        # a host code with its own time integrator calls the residual of a
        # small box once per stage: the smallest call, all latency
        dict(name="residual-box-2k", kind="residual", mesh="box", nx=36, ny=30, prec="fp64", grad="lsq-nn", limiter=0),
        # unit-test and teaching size in the fast mode: a Dirichlet box under
        # classic RK4, time-dependent boundary values
        dict(name="box-7k-mixed-rk4", kind="integrate", mesh="box", nx=61, ny=59, prec="mixed", grad="lsq-nn",
             limiter=0, recon=2, kappa=0.0, rk="rk4", cfl=0.6, steps=60),
        # the small benchmark box, 8,192 triangles and 200 steps, in FP64
        dict(name="vortex-8k-fp64", kind="integrate", mesh="periodic", nx=64, ny=64, prec="fp64", grad="lsq-fn",
             limiter=0, recon=2, kappa=0.0, rk="ssprk3", cfl=0.8, steps=200),
        # the headline mesh, 1,048,576 triangles, in the drop-in's FP64
        dict(name="vortex-1m-fp64", kind="integrate", mesh="periodic", nx=1024, ny=512, prec="fp64", grad="lsq-fn",
             limiter=0, recon=2, kappa=0.0, rk="ssprk3", cfl=0.8, steps=10),
        # the same mesh in mixed precision
        dict(name="vortex-1m-mixed", kind="integrate", mesh="periodic", nx=1024, ny=512, prec="mixed", grad="lsq-fn",
             limiter=0, recon=2, kappa=0.0, rk="ssprk3", cfl=0.8, steps=50),
        # double-float on a mixed triangle/quad mesh with the GG-cell gradient
        dict(name="mixedmesh-218k-df", kind="integrate", mesh="periodic-mixed", nx=363, ny=360, prec="df",
             grad="ggcell", limiter=0, recon=3, kappa=1.0 / 3.0, rk="ssprk3", cfl=0.8, steps=20),
        # the GG-node gradient, the widest stencil, at a large odd size
        dict(name="vortex-525k-mixed-ggnode", kind="integrate", mesh="periodic", nx=719, ny=365, prec="mixed",
             grad="ggnode", limiter=0, recon=2, kappa=0.0, rk="ssprk3", cfl=0.8, steps=20),
        # a transonic O-grid of 65,024 quadrilaterals, node-neighbour LSQ with
        # the Venkatakrishnan limiter, steady local time steps
        dict(name="ogrid-65k-fp64-limited", kind="integrate", mesh="ogrid-quad", nx=512, ny=128, prec="fp64",
             grad="lsq-nn", limiter=1, recon=2, kappa=0.0, rk="ssprk42", cfl=0.5, mach=0.8, aoa=1.25, steps=15),
        # a reduced airfoil sweep in mixed precision: eight first-order cases
        dict(name="sweep-8-mixed", kind="sweep", ncases=8, wmin=64, wmax=192, rmin=32, rmax=96, mesh_seed=6,
             prec="mixed", steps=100),
        # the tail of such a sweep: defect correction with its shape trials
        dict(name="sweep-6-dc", kind="dc", ncases=6, wmin=64, wmax=128, rmin=24, rmax=64, mesh_seed=5, steps=400,
             chunk=50),
        # one epoch of the warm-start network over the samples of a few cases
        dict(name="mlp-train-131k", kind="train", n=131072, n_in=5, width=256, depth=4, n_out=4, batch=4096, epochs=1),
        # its prediction for every cell of a full-size airfoil
        dict(name="mlp-predict-261k", kind="predict", n=261120, n_in=5, width=256, depth=4, n_out=4),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choices(["integrate", "residual", "sweep", "dc", "train", "predict"], [12, 3, 3, 1, 2, 2])[0]
    prec = rng.choice(["fp64", "mixed", "df"])
    if kind == "integrate":
        mesh = rng.choice(["periodic", "periodic", "periodic-mixed", "box", "ogrid-quad", "ogrid-tri"])
        small = mesh in ("box", "ogrid-quad", "ogrid-tri")
        grad = rng.choice(["lsq-fn", "lsq-fn", "lsq-nn", "ggcell", "ggnode"])
        if small and grad == "lsq-fn":
            grad = "lsq-nn"
        limiter = rng.choice([0, 1]) if grad.startswith("lsq") else 0
        recon = rng.choice([1, 2, 2, 3])
        cells = _logint(rng, 600, 90000 if small else 500000)
        aspect = math.exp(rng.uniform(-0.7, 0.7))
        per = 1 if mesh == "ogrid-quad" else 2
        nx = max(16, int(math.sqrt(cells / per * aspect)))
        c = dict(kind=kind, mesh=mesh, prec=prec, grad=grad, limiter=limiter, recon=recon,
                 kappa=rng.choice([-1.0, 0.0, 1.0 / 3.0]) if recon == 3 else 0.0)
        if mesh.startswith("ogrid"):
            nx = max(32, nx + nx % 2)
            c.update(rk="ssprk42", cfl=0.5, mach=round(rng.uniform(0.3, 0.85), 3), aoa=round(rng.uniform(-2, 4), 3))
        else:
            c.update(rk=rng.choice(["ssprk3", "rk4", "ssprk42"]), cfl=0.6)
        ny = max(14, cells // (per * nx))
        c.update(nx=nx, ny=ny, steps=max(1, min(200, int((3e6 if prec == "fp64" else 6e6) / (per * nx * ny)))))
        return c
    if kind == "residual":
        mesh = rng.choice(["periodic", "box", "ogrid-quad"])
        grad = rng.choice(["lsq-nn", "lsq-nn", "ggcell", "ggnode"])
        nx = _logint(rng, 16, 180)
        return dict(kind=kind, mesh=mesh, nx=max(32, nx + nx % 2) if mesh == "ogrid-quad" else nx,
                    ny=max(14, int(nx * rng.uniform(0.5, 1.5))), prec=prec, grad=grad,
                    limiter=rng.choice([0, 1]) if grad == "lsq-nn" else 0, mach=round(rng.uniform(0.3, 0.85), 3),
                    aoa=round(rng.uniform(-2, 4), 3))
    if kind in ("sweep", "dc"):
        big = kind == "sweep"
        c = dict(kind=kind, ncases=_logint(rng, 1, 12 if big else 6), wmin=64, wmax=192 if big else 128,
                 rmin=24 if not big else 32, rmax=96 if big else 64, mesh_seed=rng.randrange(1, 1000))
        return dict(c, prec=rng.choice(["mixed", "mixed", "fp64"]), steps=rng.randrange(5, 60)) if big else \
            dict(c, steps=rng.randrange(210, 400), chunk=50)
    net = dict(n_in=rng.choice([3, 5, 8]), width=16 * _logint(rng, 2, 16), depth=rng.randrange(1, 5),
               n_out=rng.choice([1, 4]))
    if kind == "train":
        n = _logint(rng, 600, 100000)
        return dict(kind=kind, n=n, batch=min(n, _logint(rng, 200, 4096)), epochs=1, **net) if n < 20000 else \
            dict(kind=kind, n=n, batch=_logint(rng, 2000, 4096), epochs=1, **net)
    return dict(kind=kind, n=_logint(rng, 300, 250000), **net)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _mesh(kind: str, nx: int, ny: int):
    if kind == "periodic":
        return meshgen.periodic_square(nx, ny, jitter=0.2)
    if kind == "periodic-mixed":
        return meshgen.periodic_square(nx, ny, jitter=0.2, quad_every=3)
    if kind == "box":
        return meshgen.dirichlet_square(nx, ny, jitter=0.2)
    return meshgen.naca0012_ogrid(nx, ny, quads=kind == "ogrid-quad")


def _vortex(seed: int) -> dict:
    """Strength and centre of the start's vortex."""
    r = np.random.default_rng([seed, 11])
    return dict(kappa=float(KAPPA_REF * r.uniform(0.8, 1.1)), x=float(r.uniform(-0.5, 0.5)), y=float(r.uniform(-0.5, 0.5)))


def _options(c: dict, seed: int) -> Options:
    o = dict(grad_method=GRAD[c["grad"]], lsq_stencil="nn" if c["grad"] == "lsq-nn" else "fn", limiter=c["limiter"],
             reconst=c.get("recon", 2), umuscl=c.get("kappa", 0.0), precision=PREC[c["prec"]])
    if c["mesh"].startswith("ogrid"):
        o.update(mach_inf=c.get("mach", 0.8), aoa_inf_deg=c.get("aoa", 1.25), steady=True, cfl=c.get("cfl", 0.5),
                 dt=0.01, rk_nstages=4, rk_order=2, ssprk=True)
        return Options(**o)
    v = _vortex(seed)
    rk = {"ssprk3": (3, 3, True), "rk4": (4, 4, False), "ssprk42": (4, 2, True)}[c.get("rk", "ssprk3")]
    return Options(vortex=True, vortex_x=v["x"], vortex_y=v["y"], vortex_kappa=v["kappa"],
                   vortex_inf=(1.0, MACH_VORTEX * math.sqrt(GAMMA), 0.0, 1.0), rk_nstages=rk[0], rk_order=rk[1],
                   ssprk=rk[2], cfl=c.get("cfl", 0.8), dt_from_cfl=True, **o)


def _centroids(m) -> np.ndarray:
    """Cell centroids (vertex means, unwrapped on periodic meshes, not folded back)."""
    out = []
    for nodes in (m.tri_nodes, m.quad_nodes):
        if nodes.shape[0]:
            p = m.node_xy[nodes - 1]
            for a, length in ((0, m.period_x), (1, m.period_y)):
                if length > 0:
                    p[:, :, a] -= length * np.rint((p[:, :, a] - p[:, :1, a]) / length)
            out.append(p.mean(1))
    return np.concatenate(out)


def _vortex_prim(o, x, y, t, lib):
    """Isentropic vortex (rho, u, v, p) at points x, y and time t (lib: numpy or torch)."""
    rho_i, u_i, v_i, p_i = o.vortex_inf
    dx, dy = x - (o.vortex_x + u_i * t), y - (o.vortex_y + v_i * t)
    r2, q = dx * dx + dy * dy, o.vortex_kappa / (2.0 * math.pi)
    e = lib.exp(0.5 * (1.0 - r2))
    temp = p_i / rho_i - q * q * (GAMMA - 1.0) / (2.0 * GAMMA) * e * e
    rho = temp ** (1.0 / (GAMMA - 1.0))
    return rho, u_i - q * dy * e, v_i + q * dx * e, rho ** GAMMA


def _conserved(rho, u, v, p) -> np.ndarray:
    return np.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)], 1)


def _waves(xy, seed, length):
    """Two smooth seeded waves of amplitude about one."""
    r = np.random.default_rng([seed, 7])
    k = 2.0 * math.pi / length * r.integers(1, 4, size=(2, 2))
    ph = r.uniform(0, 2 * math.pi, 2)
    return np.sin(k[0, 0] * xy[:, 0] + ph[0]) * np.cos(k[1, 1] * xy[:, 1] + ph[1]), np.cos(k[1, 0] * xy[:, 0] + k[0, 1] * xy[:, 1])


def _free_stream(mach, aoa):
    a = aoa * math.pi / 180.0
    return 1.0, mach * math.cos(a), mach * math.sin(a), 1.0 / GAMMA


def _start(m, o, seed: int) -> np.ndarray:
    """The start state: the vortex with a 1 % wave on it, or the free stream
    with a smooth 2 % disturbance that fades away from the body."""
    xy = _centroids(m)
    if o.steady:
        w1, w2 = _waves(xy, seed, 4.0)
        f = 0.02 * np.exp(-0.05 * ((xy[:, 0] - 0.5) ** 2 + xy[:, 1] ** 2))
        rho, u, v, p = _free_stream(o.mach_inf, o.aoa_inf_deg)
        return _conserved(rho + f * w1, u + f * w2, v + f * w1, p * (1.0 + f * w2))
    w1, w2 = _waves(xy, seed, 10.0)
    rho, u, v, p = _vortex_prim(o, xy[:, 0], xy[:, 1], 0.0, np)
    return _conserved(rho * (1.0 + 0.01 * w1), u, v, p * (1.0 + 0.01 * w2))


def _sweep_cases(c: dict, seed: int) -> list:
    """(mesh, options) per case: meshes from the case's mesh_seed, flow conditions from the seed."""
    g = np.random.default_rng([c["mesh_seed"], 3])
    r = np.random.default_rng([seed, 5])
    out = []
    for _ in range(c["ncases"]):
        nw, nr = int(g.integers(c["wmin"], c["wmax"] + 1)), int(g.integers(c["rmin"], c["rmax"] + 1))
        o = Options(mach_inf=float(r.uniform(0.3, 0.85)), aoa_inf_deg=float(r.uniform(-2, 4)), steady=True, cfl=1.25,
                    rk_nstages=4, rk_order=2, ssprk=True, grad_method=3, lsq_stencil="fn", limiter=1, reconst=1, dt=0.01,
                    precision=PREC[c.get("prec", "mixed")])
        out.append((meshgen.naca0012_ogrid(nw + nw % 2, nr), o))
    return out


def _samples(c: dict, seed: int):
    r = np.random.default_rng([seed, 9])
    x = r.uniform(-1.0, 1.0, (c["n"], c["n_in"])).astype(np.float32)
    a = r.standard_normal((c["n_in"], c["n_out"])).astype(np.float32)
    y = (0.5 * np.tanh(x @ a) + 0.2 * (x[:, :1] * x[:, 1:2]) ** 2).astype(np.float32)
    return x, y


def _dims(c: dict) -> list:
    return [c["n_in"]] + [c["width"]] * c["depth"] + [c["n_out"]]


def _weights(c: dict, seed: int) -> np.ndarray:
    """Scaled normal weights and small biases, per layer W[out][in] then b[out]."""
    r, d = np.random.default_rng([seed, 13]), _dims(c)
    return np.concatenate([np.concatenate([r.standard_normal(i * j) * math.sqrt(2.0 / i), 0.05 * r.standard_normal(j)])
                           for i, j in zip(d, d[1:])]).astype(np.float32)


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind in ("integrate", "residual"):
        m, o = _mesh(case["mesh"], case["nx"], case["ny"]), _options(case, seed)
        u = _start(m, o, seed)
        s = dict(kind=kind, solver=Solver(m, o))
        if kind == "residual":
            return dict(s, u=u)
        pin = torch.from_numpy(u).pin_memory()
        return dict(s, steps=case["steps"], u=pin, out=torch.empty_like(pin, pin_memory=True))
    if kind in ("sweep", "dc"):
        cs = _sweep_cases(case, seed)
        b = Batch([m for m, _ in cs], [o for _, o in cs])
        starts = [_start(m, o, seed + k) for k, (m, o) in enumerate(cs)]
        for k, u in enumerate(starts):
            b.set_state(k, u)
        b.autotune(3)
        if kind == "dc":
            # the mixed phase that precedes it
            for _ in range(3):
                b.steps(1000)
            starts = [b.get_state(k) for k in range(b.ncases)]
        return dict(kind=kind, batch=b, starts=starts, steps=case["steps"], chunk=case.get("chunk", 50),
                    levels=np.full((b.ncases, 4), 1e-30))
    x, y = _samples(case, seed)
    net = MLP(case["n_in"], case["width"], case["depth"], case["n_out"])
    net.set_params(_weights(case, seed))
    return dict(kind=kind, net=net, x=x, y=y,
                batch=case.get("batch"), epochs=case.get("epochs"), seed=seed % 1000)


def run(state: dict):
    kind = state["kind"]
    if kind == "integrate":
        s = state["solver"]
        s.set_state_ptr(state["u"].data_ptr())
        norms = s.time_integration(0.0, state["steps"])
        s.get_state_ptr(state["out"].data_ptr())
        return dict(state=state["out"], norms=norms)
    if kind == "residual":
        s = state["solver"]
        s.cvar = state["u"]
        resid, ws = s.compute_residual(0.0)
        grad, phi = s.gradient()
        return dict(resid=resid, ws=ws, grad=grad, phi=phi)
    if kind == "sweep":
        b = state["batch"]
        for k, u in enumerate(state["starts"]):
            b.set_state(k, u)
        norms, _ = b.steps(state["steps"])
        return dict(states=[b.get_state(k) for k in range(b.ncases)], norms=norms)
    if kind == "dc":
        b = state["batch"]
        for k, u in enumerate(state["starts"]):
            b.set_state(k, u)
        done, first, last, _ = b.run_to_level(state["steps"], state["levels"], state["chunk"], dc=True)
        return dict(states=[b.get_state(k) for k in range(b.ncases)], done=done, first=first, last=last)
    if kind == "train":
        net = state["net"]
        losses = net.train(state["x"], state["y"], batch=state["batch"], epochs=state["epochs"], lr=1e-3,
                           seed=state["seed"])
        return dict(losses=losses, params=net.get_params())
    return dict(y=state["net"].predict(state["x"]))


# ---------------------------------------------------------------------------
# the work of a pass
# ---------------------------------------------------------------------------
def _shape(c: dict):
    """(cells, edges) of a mesh."""
    nx, ny = c["nx"], c["ny"]
    if c["mesh"] == "ogrid-quad":
        return nx * (ny - 1), nx * (2 * ny - 1)
    if c["mesh"] == "ogrid-tri":
        return 2 * nx * (ny - 1), nx * (3 * ny - 2)
    if c["mesh"] == "periodic-mixed":
        kept = (nx + 2) // 3 * ny
        return 2 * nx * ny - kept, 3 * nx * ny - kept
    return 2 * nx * ny, 3 * nx * ny


def work(case: dict) -> dict:
    """Per evaluation of the residual: the mesh (normals, lengths, face offsets
    and cell ids of the edges; ids and two coefficients per stencil entry;
    volumes), the FP64 state read and written, and the operations of gradient
    (4 per stencil entry and variable plus the differences), flux (about 190)
    and update."""
    kind = case["kind"]
    if kind in ("train", "predict"):
        dims = _dims(case)
        params = sum(a * b + b for a, b in zip(dims, dims[1:]))
        mac = sum(a * b for a, b in zip(dims, dims[1:]))
        if kind == "predict":
            return dict(bytes=4.0 * case["n"] * (case["n_in"] + case["n_out"]) + 4.0 * params, flops=2.0 * case["n"] * mac)
        rows = case["n"] // case["batch"] * case["batch"] * case["epochs"]
        return dict(bytes=4.0 * rows * (case["n_in"] + case["n_out"]) + 28.0 * params * (rows // case["batch"]),
                    flops=6.0 * rows * mac)
    t = 4 if case.get("prec", "mixed") == "mixed" else 8
    if kind in ("sweep", "dc"):
        g = np.random.default_rng([case["mesh_seed"], 3])
        nc = ne = 0
        for _ in range(case["ncases"]):
            nw, nr = int(g.integers(case["wmin"], case["wmax"] + 1)), int(g.integers(case["rmin"], case["rmax"] + 1))
            a, b = _shape(dict(mesh="ogrid-tri", nx=nw + nw % 2, ny=nr))
            nc, ne = nc + a, ne + b
        evals, sten, second = 4 * case["steps"], 0, False
    else:
        nc, ne = _shape(case)
        evals = 1 if kind == "residual" else case["steps"] * (3 if case["rk"] == "ssprk3" else 4)
        second = case.get("recon", 2) != 1
        sten = {"lsq-fn": 3, "ggcell": 3, "lsq-nn": 12 if case["mesh"] != "ogrid-quad" else 8, "ggnode": 18}[case["grad"]]
    per_eval = ne * (8 + (7 if second else 3) * t) + nc * (8 + 64 + (4 + 2 * t) * (sten if second else 0))
    flops = ne * 190.0 + nc * (60.0 + (20.0 * sten if second else 0))
    out = 64.0 * nc + (80.0 * nc if kind == "residual" else 0)
    return dict(bytes=float(evals * per_eval + out), flops=float(evals * flops))


# ---------------------------------------------------------------------------
# the same quantities in plain float64
# ---------------------------------------------------------------------------
class _Exact:
    """The scheme in float64 tensor operations: connectivity and geometry from
    the mesh's nodes, gradients, limiter, reconstruction, Roe flux and boundary
    states as the equations are written."""

    def __init__(self, m, o):
        self.o, self.dev = o, torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.first = o.reconst == 1
        L = np.array([m.period_x, m.period_y])
        nc, nt = m.ncells, m.tri_nodes.shape[0]
        cn = np.full((nc, 4), -1, np.int64)
        cn[:nt, :3] = m.tri_nodes - 1
        cn[nt:] = m.quad_nodes - 1
        nv = np.where(np.arange(nc) < nt, 3, 4)
        xy = m.node_xy

        def img(d):
            d = d.copy()
            for a in range(2):
                if L[a] > 0:
                    d[..., a] -= L[a] * np.rint(d[..., a] / L[a])
            return d
        xc = _centroids(m)
        # directed edges of all cells, outward normals (cells are counter-clockwise)
        cell = np.repeat(np.arange(nc), nv)
        k = np.concatenate([np.arange(3)[None].repeat(nt, 0).ravel(), np.arange(4)[None].repeat(nc - nt, 0).ravel()])
        a = cn[cell, k]
        b = cn[cell, (k + 1) % nv[cell]]
        key = np.minimum(a, b) * m.nnodes + np.maximum(a, b)
        order = np.lexsort((cell, key))
        ks = key[order]
        first = np.concatenate([[True], ks[1:] != ks[:-1]])
        eid_sorted = np.cumsum(first) - 1
        ne = int(eid_sorted[-1]) + 1
        eid = np.empty(len(key), np.int64)
        eid[order] = eid_sorted
        h = order[first]                      # the lower cell's side of each edge
        left = cell[h]
        right = np.full(ne, -1, np.int64)
        second = np.concatenate([~first, [False]])[1:] & first  # an entry followed by its twin
        right[eid_sorted[second]] = cell[order[np.nonzero(second)[0] + 1]]
        pa = xy[a[h]]
        dab = img(xy[b[h]] - pa)
        length = np.hypot(dab[:, 0], dab[:, 1])
        n = np.stack([dab[:, 1], -dab[:, 0]], 1) / length[:, None]
        xf = pa + 0.5 * dab
        dl = img(xf - xc[left])
        dr = img(xf - xc[np.maximum(right, 0)])
        # volumes (shoelace of the unwrapped vertices)
        P = np.stack([xc[:, None] + img(xy[np.maximum(cn[:, j], 0)][:, None] - xc[:, None]) for j in range(4)], 2)[:, 0]
        P[:nt, 3] = P[:nt, 0]
        x, y = P[..., 0] - xc[:, :1], P[..., 1] - xc[:, 1:]
        vol = 0.5 * (x * np.roll(y, -1, 1) - np.roll(x, -1, 1) * y).sum(1)
        # boundary conditions of the edges without a right cell
        bt = np.zeros(ne, np.int64)
        be = np.nonzero(right < 0)[0]
        by_cell = {}
        for t, cells in zip(m.bndry_types, m.bndry_cells):
            for q in np.asarray(cells):
                by_cell[int(q) - 1] = BC[t]
        bt[be] = [by_cell[int(q)] for q in left[be]]
        T = lambda v: torch.as_tensor(np.ascontiguousarray(v), device=self.dev)  # noqa: E731
        inner = np.nonzero(right >= 0)[0]
        eo = np.concatenate([inner, be])
        self.ni, self.nc = len(inner), nc
        self.L_, self.R_ = T(left[eo]), T(right[inner])
        self.n, self.A, self.dl, self.dr, self.xf = T(n[eo]), T(length[eo])[:, None], T(dl[eo]), T(dr[inner]), T(xf[be])
        self.bt, self.vol = T(bt[be]), T(vol)[:, None]
        # gradient operator: a list of (cell, other, coefficient) entries
        self.grad_kind = "lsq" if o.grad_method == 3 else "ggcell" if o.grad_method == 1 else "ggnode"
        if self.first:
            pass  # no gradient is read
        elif self.grad_kind == "lsq":
            if o.lsq_stencil == "fn":  # face neighbours (meshes without boundary only)
                i, j = np.concatenate([left[inner], right[inner]]), np.concatenate([right[inner], left[inner]])
            else:
                i, j = self._around(cn, nv, m.nnodes)
            d = img(xc[j] - xc[i])
            G = np.zeros((nc, 3))
            for q, v in enumerate((d[:, 0] ** 2, d[:, 0] * d[:, 1], d[:, 1] ** 2)):
                G[:, q] = np.bincount(i, v, nc)
            det = G[:, 0] * G[:, 2] - G[:, 1] ** 2
            cx = (G[i, 2] * d[:, 0] - G[i, 1] * d[:, 1]) / det[i]
            cy = (G[i, 0] * d[:, 1] - G[i, 1] * d[:, 0]) / det[i]
            self.si, self.sj, self.cx, self.cy = T(i), T(j), T(cx)[:, None], T(cy)[:, None]
        elif self.grad_kind == "ggcell":
            d0, d1 = np.hypot(*dl.T), np.hypot(*dr.T)
            d1 = np.where(right >= 0, d1, d0)
            self.wl = T((d1 / (d0 + d1))[eo])[:, None]
        elif self.grad_kind == "ggnode":
            dn = img(xc[cell] - xy[a])
            w = 1.0 / np.hypot(dn[:, 0], dn[:, 1])
            tot = np.bincount(a, w, m.nnodes)
            self.nn, self.ncell, self.nnode, self.nw = m.nnodes, T(cell), T(a), T(w / tot[a])[:, None]
            self.ea, self.eb = T(a[h][eo]), T(b[h][eo])
        # limiter: centre-to-face offsets of every (cell, face) pair
        self.fi = T(cell)
        sgn_l = left[eid] == cell
        self.fd = T(np.where(sgn_l[:, None], dl[eid], dr[eid]))
        t = 5.0 * 2.0 * np.sqrt(vol / math.pi)
        self.eps2 = T(t ** 3)[:, None]

    @staticmethod
    def _around(cn, nv, nnodes):
        """Pairs (cell, other) of cells that share a node."""
        nc = len(cn)
        cell = np.repeat(np.arange(nc), nv)
        node = cn[cn >= 0]
        order = np.argsort(node, kind="stable")
        count = np.bincount(node, minlength=nnodes)
        start = np.concatenate([[0], np.cumsum(count)[:-1]])
        rep = count[node]
        i = np.repeat(cell, rep)
        off = np.arange(rep.sum()) - np.repeat(np.cumsum(rep) - rep, rep)
        j = cell[order][np.repeat(start[node], rep) + off]
        u = np.unique(i[i != j] * nc + j[i != j])
        return u // nc, u % nc

    def _add(self, idx, v, n=None):
        return torch.zeros((n or self.nc, v.shape[1]), dtype=torch.float64, device=self.dev).index_add_(0, idx, v)

    def prim(self, U):
        r, u, v = U[:, 0], U[:, 1] / U[:, 0], U[:, 2] / U[:, 0]
        return torch.stack([r, u, v, (GAMMA - 1.0) * (U[:, 3] - 0.5 * r * (u * u + v * v))], 1)

    def gradient(self, p):
        if self.grad_kind == "lsq":
            d = p[self.sj] - p[self.si]
            gx, gy = self._add(self.si, self.cx * d), self._add(self.si, self.cy * d)
        else:
            if self.grad_kind == "ggcell":
                f = self.wl * p[self.L_] + (1.0 - self.wl) * torch.cat([p[self.R_], p[self.L_[self.ni:]]])
            else:
                q = self._add(self.nnode, self.nw * p[self.ncell], self.nn)
                f = 0.5 * (q[self.ea] + q[self.eb])
            fr = f[:self.ni]
            nx, ny = self.n[:, :1] * self.A, self.n[:, 1:] * self.A
            gx = self._add(self.L_, f * nx) - self._add(self.R_, fr * nx[:self.ni])
            gy = self._add(self.L_, f * ny) - self._add(self.R_, fr * ny[:self.ni])
            gx, gy = gx / self.vol, gy / self.vol
        phi = torch.ones((self.nc, 1), dtype=torch.float64, device=self.dev)
        if self.o.limiter == 1:
            lo, hi = p.clone(), p.clone()
            idx = self.si[:, None].expand(-1, 4)
            hi.scatter_reduce_(0, idx, p[self.sj], "amax")
            lo.scatter_reduce_(0, idx, p[self.sj], "amin")
            c = self.fi
            diff = self.fd[:, :1] * gx[c] + self.fd[:, 1:] * gy[c]
            a = torch.where(diff > 0, hi[c] - p[c], lo[c] - p[c])
            e = self.eps2[c]
            v = ((a * a + e) + 2.0 * diff * a) / (a * a + 2.0 * diff * diff + a * diff + e)
            v = torch.where(diff == 0, torch.ones_like(v), v).amin(1, keepdim=True)
            phi.scatter_reduce_(0, c[:, None], v, "amin")
        return gx, gy, phi

    def ghost(self, pf, time):
        n = self.n[self.ni:]
        out = pf.clone()
        un = (pf[:, 1:3] * n).sum(1, keepdim=True)
        wall = (self.bt == 2)[:, None]
        out[:, 1:3] = torch.where(wall, pf[:, 1:3] - 2.0 * un * n, pf[:, 1:3])
        fs = torch.tensor(_free_stream(self.o.mach_inf, self.o.aoa_inf_deg), dtype=torch.float64, device=self.dev)
        out = torch.where((self.bt == 1)[:, None], fs, out)
        if bool((self.bt == 4).any()):
            ex = torch.stack(_vortex_prim(self.o, self.xf[:, 0], self.xf[:, 1], time, torch), 1)
            out = torch.where((self.bt == 4)[:, None], ex, out)
        return out

    def residual(self, U, time):
        """dU/dt, the wave-speed sums, gradient and limiter."""
        p = self.prim(U)
        pl, pr = p[self.L_], p[self.R_]
        ni, grads = self.ni, None
        if self.first:
            fl, fr = pl, pr
        else:
            grads = gx, gy, phi = self.gradient(p)
            k = self.o.umuscl if self.o.reconst == 3 else 0.0
            gl = self.dl[:, :1] * gx[self.L_] + self.dl[:, 1:] * gy[self.L_]
            gr = self.dr[:, :1] * gx[self.R_] + self.dr[:, 1:] * gy[self.R_]
            dc = pr - pl[:ni]
            fl = pl + phi[self.L_] * torch.cat([0.5 * k * dc + (1.0 - k) * gl[:ni], gl[ni:]])
            fr = pr + phi[self.R_] * (-0.5 * k * dc + (1.0 - k) * gr)
        fr = torch.cat([fr, self.ghost(fl[ni:], time)])
        F, w = self.roe(fl, fr)
        F, w = F * self.A, w * self.A
        R = self._add(self.L_, F) - self._add(self.R_, F[:ni])
        ws = self._add(self.L_, w) + self._add(self.R_, w[:ni])
        return -R / self.vol, ws, grads

    def roe(self, a, b):
        nx, ny = self.n[:, 0], self.n[:, 1]
        (rl, ul, vl, ql), (rr, ur, vr, qr) = a.unbind(1), b.unbind(1)
        unl, unr, utl, utr = ul * nx + vl * ny, ur * nx + vr * ny, vl * nx - ul * ny, vr * nx - ur * ny
        g1 = GAMMA - 1.0
        Hl = GAMMA * ql / rl / g1 + 0.5 * (ul * ul + vl * vl)
        Hr = GAMMA * qr / rr / g1 + 0.5 * (ur * ur + vr * vr)
        s = torch.sqrt(rr / rl)
        rho, u, v, H = s * rl, (ul + s * ur) / (1 + s), (vl + s * vr) / (1 + s), (Hl + s * Hr) / (1 + s)
        c = torch.sqrt(g1 * (H - 0.5 * (u * u + v * v)))
        un, ut = u * nx + v * ny, v * nx - u * ny
        dr, dp, dn, dt = rr - rl, qr - ql, unr - unl, utr - utl
        def fix(x):
            x = x.abs()
            return torch.where(x < 0.2, 0.5 * (x * x / 0.2 + 0.2), x)
        w1, w2, w3, w4 = fix(un - c) * (dp - rho * c * dn) / (2 * c * c), un.abs() * rho * dt, \
            un.abs() * (dr - dp / (c * c)), fix(un + c) * (dp + rho * c * dn) / (2 * c * c)
        D = torch.stack([w1 + w3 + w4,
                         w1 * (u - c * nx) - w2 * ny + w3 * u + w4 * (u + c * nx),
                         w1 * (v - c * ny) + w2 * nx + w3 * v + w4 * (v + c * ny),
                         w1 * (H - un * c) + w2 * ut + w3 * 0.5 * (u * u + v * v) + w4 * (H + un * c)], 1)
        F = torch.stack([rl * unl + rr * unr, rl * unl * ul + rr * unr * ur + (ql + qr) * nx,
                         rl * unl * vl + rr * unr * vr + (ql + qr) * ny, rl * unl * Hl + rr * unr * Hr], 1)
        return 0.5 * (F - D), (0.5 * (un.abs() + c))[:, None]

    def steps(self, U, nsteps, rk, cfl):
        """nsteps Runge-Kutta steps from t = 0: the state and the RMS of the increments."""
        norms, dt = [], None
        for it in range(nsteps):
            U0, f = U, 0.0
            if not self.o.steady and dt is None:
                dt = float((cfl * self.vol / (0.5 * self.residual(U, 0.0)[1])).min())
            told = it * dt if dt is not None else 0.0
            for k in range(3 if rk == "ssprk3" else 4):
                if self.o.steady:
                    R, ws, _ = self.residual(U, 0.0)
                    if k == 0:
                        loc = cfl * self.vol / (0.5 * ws)
                    h = loc
                elif rk == "ssprk3":
                    R, h = self.residual(U, told + (0.0, dt, 0.5 * dt)[k])[0], dt
                else:
                    off = (0.0, dt / 3.0, dt * 2.0 / 3.0, dt) if rk == "ssprk42" else (0.0, 0.5 * dt, 0.5 * dt, dt)
                    R, h = self.residual(U, told + off[k])[0], dt
                if rk == "ssprk3":
                    s = U + h * R
                    U = s if k == 0 else 0.75 * U0 + 0.25 * s if k == 1 else U0 / 3.0 + s * (2.0 / 3.0)
                elif rk == "ssprk42":
                    U, f = U0 + h * (0.25 if k == 3 else 1.0 / 3.0) * (R + f), f + R
                else:
                    f = f + (1.0, 2.0, 2.0, 1.0)[k] * R
                    U = U0 + (h / 6.0 * f if k == 3 else h * (1.0 if k == 2 else 0.5) * R)
            norms.append(torch.sqrt(((U - U0) ** 2).mean(0)))
        return U, torch.stack(norms)


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("integrate", "residual"):
        m, o = _mesh(case["mesh"], case["nx"], case["ny"]), _options(case, seed)
        e = _Exact(m, o)
        U = torch.as_tensor(_start(m, o, seed), device=e.dev)
        if kind == "integrate":
            U, norms = e.steps(U, case["steps"], case["rk"], case["cfl"])
            return dict(state=U.cpu(), norms=norms.cpu().numpy())
        R, ws, (gx, gy, phi) = e.residual(U, 0.0)
        return dict(resid=R.cpu().numpy(), ws=ws[:, 0].cpu().numpy(), grad=torch.stack([gx, gy]).cpu().numpy(),
                    phi=phi[:, 0].cpu().numpy())
    if kind == "sweep":
        states, norms = [], []
        for k, (m, o) in enumerate(_sweep_cases(case, seed)):
            e = _Exact(m, o)
            U, n = e.steps(torch.as_tensor(_start(m, o, seed + k), device=e.dev), case["steps"], "ssprk42", o.cfl)
            states.append(U.cpu().numpy())
            norms.append(n.cpu().numpy())
        return dict(states=states, norms=np.stack(norms))
    if kind == "predict":
        x, _ = _samples(case, seed)
        p, dims, dev = _weights(case, seed).astype(np.float64), _dims(case), "cuda" if torch.cuda.is_available() else "cpu"
        a, off = torch.as_tensor(x, device=dev).double(), 0
        for q, (i, j) in enumerate(zip(dims, dims[1:])):
            W = torch.as_tensor(p[off:off + i * j].reshape(j, i), device=dev)
            a = a @ W.T + torch.as_tensor(p[off + i * j:off + i * j + j], device=dev)
            off += i * j + j
            if q < case["depth"]:
                a = torch.nn.functional.gelu(a)
        return dict(y=a.cpu().numpy())
    # defect correction and training: their outputs are those of an iteration
    # (the tangent's path, the library's own shuffle of the samples)
    return None
