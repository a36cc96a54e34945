"""The work a user of flecsale_gb300 has it do, as cases that can be timed and
compared: whole runs of the hydro step in both precisions and both dimensions
(the solver's time loop), the four hydro tasks called one by one on
caller-owned field buffers (the drop-in boundary), a step on a state that
lives in host memory, and a batch of independent problems.

listed() gives the named cases, draw(rng) more of the same ranges, prepare()
what a user's program holds before the call, run() one pass, work() the bytes
and operations a pass cannot do without, exact() the pass in plain FP64 torch.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

import flecsale_gb300.hydro as H

FAR = 1.0e9  # a final time no run reaches


def case(name, kind, dim, n, problem, flux, precision, steps, boundary="wall", jitter=0.0,
         order=2, limiter="barth_jespersen", swap=True, cfl=0.4, split=0, stop=0.0, stream=True,
         autotune=False, problems=1, hi=1.0, waves=False):
    c = {"kind": kind, "dim": dim, "n": "x".join(str(k) for k in n), "problem": problem,
         "flux": flux, "precision": precision, "steps": steps, "boundary": boundary,
         "jitter": jitter, "order": order, "limiter": limiter, "swap": swap, "cfl": cfl,
         "split": split, "stop": stop, "stream": stream, "autotune": autotune,
         "problems": problems, "hi": hi, "waves": waves}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the reference's regression run (apps/hydro/2d): 32x32, HLLE, walls, 20 steps, on the
        # default stream as the command-line driver runs it; latency and launches
        case("shock_box_2d_32", "run", 2, (32, 32), "shock_box", "hlle", "fp64", 20, cfl=0.5,
             stream=False),
        # the CPU-sized Sod tube, first order, run until its final time with the host looking at
        # the solution time every 10 steps
        case("sod_100x10_first_order", "run", 2, (100, 10), "sod", "hllc", "fp64", 400, order=1,
             cfl=0.5, stop=0.2, hi=0.1),
        # a served request's smallest size: a Kelvin-Helmholtz layer in the mixed form
        case("kh_64_mixed", "run", 2, (64, 64), "kelvin_helmholtz", "hllc", "mixed", 50,
             jitter=0.2, swap=False),
        # ordinary unstructured meshes (quads and triangles), odd sizes, both precisions, with waves
        # over the whole domain as a flow has them some time after its start
        case("quad_tri_211x157_fp64", "run", 2, (211, 157), "shock_box", "hlle", "fp64", 10,
             jitter=0.2, split=3, waves=True),
        case("tri_203x149_mixed", "run", 2, (203, 149), "sod", "hllc", "mixed", 20, jitter=0.2,
             split=1, swap=False, waves=True),
        # the 2D headline workload: four-quadrant Riemann problem, jittered 1024x1024 quads
        case("four_quadrant_1024_fp64", "run", 2, (1024, 1024), "four_quadrant", "hllc", "fp64",
             4, boundary="outflow", jitter=0.2),
        case("four_quadrant_1024_mixed", "run", 2, (1024, 1024), "four_quadrant", "hllc", "mixed",
             20, boundary="outflow", jitter=0.2, autotune=True),
        # the 3D shock box with Rusanov fluxes, plain FP64 and mixed
        case("shock_box_3d_80_fp64", "run", 3, (80, 80, 80), "inner_cube", "rusanov", "fp64", 2,
             jitter=0.15, cfl=0.3),
        case("shock_box_3d_128_mixed", "run", 3, (128, 128, 128), "inner_cube", "rusanov",
             "mixed", 8, jitter=0.15, cfl=0.3, autotune=True),
        # the four tasks one by one on the caller's fields, as a task runtime calls them
        case("tasks_2d_401x283", "tasks", 2, (401, 283), "sod", "hllc", "fp64", 1, jitter=0.2,
             waves=True),
        # one step of a state that lives in (pinned) host memory
        case("host_state_640x448", "host", 2, (640, 448), "four_quadrant", "hllc", "fp64", 1,
             boundary="outflow", jitter=0.2, waves=True),
        # a batch of independent problems of uneven sizes advanced together, host to host
        case("batch_40_mixed", "batch", 2, (32, 256), "mix", "hllc", "mixed", 40,
             boundary="outflow", jitter=0.2, swap=False, autotune=True, problems=40),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["run", "run", "run", "run", "tasks", "tasks", "host", "batch"])
    precision = "fp64" if kind == "tasks" else "mixed" if kind == "batch" else rng.choice(["fp64", "mixed"])
    dim = 2 if kind == "batch" else rng.choice([2, 2, 3])
    flux = rng.choice(["hllc", "hlle", "rusanov"])
    if kind == "batch":
        return case(None, kind, 2, (32, log(48, 256)), "mix", flux, "mixed", rng.randint(5, 40),
                    boundary="outflow", jitter=0.2, swap=False, autotune=rng.random() < 0.5,
                    problems=log(2, 40))
    # cells: up to the listed sizes of the kind
    most = {("run", 2, "fp64"): 1 << 20, ("run", 2, "mixed"): 1 << 20, ("run", 3, "fp64"): 512000,
            ("run", 3, "mixed"): 2000000}.get((kind, dim, precision), 260000)
    cells = log(1000, most)
    side = cells ** (1.0 / dim)
    n = [max(7, int(side * rng.uniform(0.7, 1.4))) for _ in range(dim)]
    n[-1] = max(7, int(cells / math.prod(n[:-1])))
    problem = rng.choice(["four_quadrant", "kelvin_helmholtz", "sod", "shock_box"] if dim == 2
                         else ["inner_cube", "sod", "shock_box"])
    smooth = problem == "kelvin_helmholtz"
    zones = min(20, max(2, 8000000 // cells)) if precision == "mixed" else min(20, max(1, 1500000 // cells))
    return case(None, kind, dim, n, problem, flux, precision,
                1 if kind != "run" else rng.randint(max(1, zones // 2), zones),
                boundary="outflow" if problem == "four_quadrant" else "wall",
                jitter=rng.choice([0.0, 0.1, 0.15]) if dim == 3 else rng.choice([0.0, 0.1, 0.2]),
                order=1 if rng.random() < 0.15 else 2,
                limiter="none" if smooth and rng.random() < 0.3 else "barth_jespersen",
                swap=rng.random() < 0.5 and not smooth, cfl=0.3 if dim == 3 else 0.4,
                split=rng.choice([0, 0, 1, 2, 5]) if dim == 2 else 0,
                stream=rng.random() < 0.8,
                autotune=precision == "mixed" and kind == "run" and rng.random() < 0.5,
                waves=kind == "tasks" or rng.random() < 0.6)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def sizes(c):
    return [int(k) for k in c["n"].split("x")]


def batch_sides(c):
    lo, hi = sizes(c)
    r = np.random.default_rng(3)
    return [int(round(math.exp(x))) for x in r.uniform(math.log(lo), math.log(hi), c["problems"])]


def box(c, n, seed):
    D = c["dim"]
    lo, hi = [0.0] * D, [1.0] * D
    hi[-1] = c["hi"]
    if c["problem"] == "shock_box":  # the reference's domain, the shock at its middle
        lo, hi = [-0.5] * D, [0.5] * D
    mesh = H.HostMesh.box(D, n, lo, hi, c["jitter"], seed)
    if not c["split"]:
        return mesh
    # every split-th quad cut into two triangles, diagonals alternating
    a = mesh.arrays()
    q = a["cell_vertices"].reshape(-1, 4)
    k = np.arange(len(q))
    cut, odd = k % c["split"] == 0, k % 2 == 1
    corners = np.full((len(q), 2, 4), -1, np.int32)
    corners[~cut, 0] = q[~cut]
    for rows, first, second in ((cut & odd, (0, 1, 2), (0, 2, 3)), (cut & ~odd, (0, 1, 3), (1, 2, 3))):
        corners[rows, 0, :3] = q[rows][:, first]
        corners[rows, 1, :3] = q[rows][:, second]
    flat = corners.reshape(-1, 4)
    flat = flat[flat[:, 0] >= 0]
    offsets = np.concatenate([[0], np.cumsum((flat >= 0).sum(1))]).astype(np.int32)
    return H.HostMesh.from_cells(2, a["vertex_coord"].T.copy(), offsets, flat[flat >= 0])


def params(c):
    return H.make_params(c["dim"], flux=c["flux"], limiter=c["limiter"], order=c["order"],
                         swap=c["swap"], precision=c["precision"], cfl=c["cfl"],
                         final_time=c["stop"] or FAR, boundary=c["boundary"])


def initial(c, problem, mesh, p, seed):
    """The problem's state, its gas a few percent denser or hotter from one
    seed to the next; with waves, a seeded sound wave along each axis on top."""
    D = c["dim"]
    s = H.initial_state(problem, mesh, p, seed)
    r = np.random.default_rng(seed)
    f = 1.0 + r.uniform(-0.05, 0.05, 2)
    d, v, e = s[0] * f[0], s[1:1 + D], s[2 + D] * f[1]
    if c["waves"]:
        x = mesh.arrays()["cell_centroid"]
        k, at = r.integers(1, 6, D), r.uniform(0.0, 2.0 * np.pi, D)
        w = 0.04 * np.sin(2.0 * np.pi * k[:, None] * x + at[:, None])
        all_w = w.sum(0)
        d, v, e = d * (1.0 + all_w), v + w, e * (1.0 + 1.4 * all_w)
    return H.state_from_dvp(D, d, v, e)


def batch_problem(k):
    return ("kelvin_helmholtz", "four_quadrant", "sod")[k % 3]


class Fields:
    """State planes in the caller's own device memory, as the library takes them."""

    def __init__(self, planes, dim, pad=64):
        nc = planes.shape[1]
        self.all = torch.zeros((5 + dim, -(-nc // pad) * pad), dtype=torch.float64, device="cuda")
        self.planes = self.all[:, :nc]
        self.planes.copy_(torch.from_numpy(planes))
        self.first = self.planes.clone()
        self.dim, self.num_cells = dim, nc
        row = rows(self.all)
        v = self.view = H.StateView()
        v.density = row[0]
        for d in range(dim):
            v.velocity[d] = row[1 + d]
        v.internal_energy, v.pressure, v.temperature, v.sound_speed = row[1 + dim:5 + dim]


def rows(t):
    return [C.cast(C.c_void_p(t[r].data_ptr()), C.POINTER(C.c_double)) for r in range(t.shape[0])]


def prepare(c, seed):
    p = params(c)
    D = c["dim"]
    s = {"case": c, "params": p}
    if c["kind"] == "batch":
        s["stream"] = torch.cuda.Stream()
        s["meshes"] = [box(c, (n, n), seed * 64 + k) for k, n in enumerate(batch_sides(c))]
        s["in"], s["out"] = [], []
        for k, m in enumerate(s["meshes"]):
            planes = torch.from_numpy(initial(c, batch_problem(k), m, p, seed * 64 + k))
            s["in"].append(planes.pin_memory())
            s["out"].append(torch.empty_like(planes).pin_memory())
        b = s["batch"] = H.Batch.for_meshes(p, s["meshes"])
        b.assign(s["meshes"], c["cfl"], FAR, stream=s["stream"])
        for k, planes in enumerate(s["in"]):
            b.set_state(k, planes.numpy(), stream=s["stream"])
        if c["autotune"]:
            b.autotune(3, use_cache=False, stream=s["stream"])
        return s
    mesh = box(c, sizes(c), seed)
    planes = initial(c, c["problem"], mesh, p, seed)
    s["stream"] = torch.cuda.Stream() if c["stream"] else torch.cuda.default_stream()
    s["handle"] = s["stream"] if c["stream"] else None
    dm = s["mesh"] = H.DeviceMesh(mesh)
    f = s["fields"] = Fields(planes, D, 1 if c["kind"] == "tasks" else 64)
    torch.cuda.synchronize()
    if c["kind"] == "tasks":
        def new(*shape):
            return torch.zeros(shape, dtype=torch.float64, device="cuda")

        s["grads"], s["flux"] = new((D + 4) * D, mesh.num_cells), new(D + 2, mesh.num_faces)
        g, fl = rows(s["grads"]), rows(s["flux"])
        s["grad_view"] = H.gradient_view_from(range(len(g)), D, ptr_of=lambda r: g[r])
        s["flux_view"] = H.flux_view_from(range(len(fl)), D, ptr_of=lambda r: fl[r])
        s["time"], s["dt"] = new(1), new(1)
        s["status"] = torch.full((1,), -1, dtype=torch.int64, device="cuda")
        s["work_bytes"] = H.lib().fvh_time_step_workspace_bytes(dm.num_cells)
        s["work"] = torch.zeros(s["work_bytes"], dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        return s
    s["solver"] = H.Solver(dm, p)
    if c["autotune"]:
        s["solver"].autotune(f, 5, stream=s["handle"])
    if c["kind"] == "host":
        s["from"] = torch.from_numpy(planes).pin_memory()
        s["host"] = torch.empty_like(s["from"]).pin_memory()
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    c = s["case"]
    return {"run": run_solver, "tasks": run_tasks, "host": run_host, "batch": run_batch}[c["kind"]](s, c)


def run_solver(s, c):
    """The time loop from the initial state."""
    f = s["fields"]
    with torch.cuda.stream(s["stream"]):
        f.planes.copy_(f.first, non_blocking=True)
    s["solver"].reset(0.0, stream=s["handle"])
    steps = s["solver"].run(f, c["steps"], stop_at_final_time=c["stop"] > 0, check_every=10,
                            stream=s["handle"])
    return {"state": f.planes, "steps": steps}


def run_tasks(s, c):
    """dt, gradients, fluxes and a half-step update, task by task."""
    L, f = H.lib(), s["fields"]
    stream = H.stream_handle(s["handle"])
    m, p, v = C.byref(s["mesh"].view), C.byref(s["params"]), C.byref(f.view)
    g, fl = C.byref(s["grad_view"]), C.byref(s["flux_view"])
    t, dt, st = (C.c_void_p(s[k].data_ptr()) for k in ("time", "dt", "status"))
    with torch.cuda.stream(s["stream"]):
        f.planes.copy_(f.first, non_blocking=True)
        s["time"].zero_()
    H.check(L.fvh_evaluate_time_step(m, v, p, t, dt, C.c_void_p(s["work"].data_ptr()),
                                     s["work_bytes"], st, stream))
    H.check(L.fvh_evaluate_gradients(m, v, g, p, stream))
    H.check(L.fvh_evaluate_fluxes(m, v, g, fl, p, stream))
    H.check(L.fvh_apply_update(m, p, dt, 0.5, fl, v, t, st, stream))
    return {"state": f.planes, "grads": s["grads"], "flux": s["flux"], "dt": s["dt"]}


def run_host(s, c):
    """A step of a state held in host memory, in place."""
    s["host"].copy_(s["from"])
    s["solver"].advance_host(s["fields"], s["host"].numpy(), c["steps"], 0.0, stream=s["handle"])
    return {"state": s["host"]}


def run_batch(s, c):
    """Every problem's state in, one launch of all steps, every state out."""
    b = s["batch"]
    for k, planes in enumerate(s["in"]):
        b.set_state(k, planes.numpy(), stream=s["stream"])
    b.step(c["steps"], stream=s["stream"])
    for k, planes in enumerate(s["out"]):
        H.check(H.lib().fvh_batch_get_state(b._h, k, C.cast(planes.data_ptr(), C.POINTER(C.c_double)),
                                            H.stream_handle(s["stream"])))
    return s["out"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def counts(c, n):
    """(cells, faces, vertices, and per cell: faces, vertices, vertex neighbours)"""
    D, nc = c["dim"], math.prod(n)
    nf = sum((n[d] + 1) * math.prod(n[:d] + n[d + 1:]) for d in range(D))
    nv = math.prod(k + 1 for k in n)
    if not c["split"]:
        return nc, nf, nv, 2 * D, 2 ** D, 3 ** D - 1
    cut = -(-nc // c["split"])
    cells = nc + cut
    share = cut / cells
    return cells, nf + cut, nv, 4 - 2 * share, 4 - 2 * share, 8 + 6 * share


@functools.lru_cache(maxsize=None)
def work_of(items):
    c = dict(items)
    D = c["dim"]
    every = [[k, k] for k in batch_sides(c)] if c["kind"] == "batch" else [sizes(c)]
    steps = c["steps"]
    if c["stop"]:  # steps until the final time: wave speed about 2.2
        steps = int(c["stop"] * 2.2 * max(sizes(c)) / c["cfl"])
    stages = 1 if c["kind"] == "tasks" else 2 * steps
    nbytes = flops = 0.0
    for n in every:
        nc, nf, nv, cf, cv, nb = counts(c, n)
        # per step: the state in (T is not an input) and out, the lists and the FP64 geometry once
        once = 8 * (2 * D + 9) * nc + 4 * (2 * nf + (cf + cv + nb + 3) * nc) \
            + 8 * ((D + 1) * nc + (2 * D + 1) * nf + D * nv)
        if c["kind"] == "tasks":
            once += 8 * (2 * D * (D + 4) * nc + 2 * (D + 2) * nf)  # gradients and fluxes out and in
        nbytes += once * (steps if c["kind"] != "tasks" else 1)
        v = D + 4
        gradients = nb * (v * (1 + 2 * D) + D + D * (D + 1)) + v * D * (2 * D + 1) + cv * v * (2 * D + 1)
        fluxes = nf / nc * ((4 * D * v if c["order"] == 2 else 0) + 60 + 12 * D)
        update = cf * (D + 2) + 12 * D + 20
        dt = cf * (2 * D + 3)
        flops += nc * (stages * ((gradients if c["order"] == 2 else 0) + fluxes + update)
                       + dt * (steps if c["kind"] != "tasks" else 1))
    return {"bytes": nbytes, "flops": flops}


def work(c):
    return work_of(tuple(sorted((k, v) for k, v in c.items() if k != "name")))


# ---------------------------------------------------------------------------
# the same pass in plain FP64 torch
# ---------------------------------------------------------------------------
class Plain:
    """The scheme on one mesh: least-squares gradients over the vertex
    neighbours, the vertex limiter, a Riemann flux per face and the
    conservative update."""

    def __init__(self, mesh, c, p, device):
        a = mesh.arrays()
        D = self.D = mesh.dim

        def t(x):
            return torch.as_tensor(np.ascontiguousarray(x), device=device)

        self.c, self.gamma, self.cv, self.tf = c, p.gamma, p.cv, p.final_time
        self.x, self.vol = t(a["cell_centroid"]), t(a["cell_volume"])
        self.xf, self.nrm, self.area = t(a["face_centroid"]), t(a["face_normal"]), t(a["face_area"])
        self.xv = t(a["vertex_coord"])
        fc = t(a["face_cells"]).long()
        self.l, r = fc[:, 0], fc[:, 1]
        self.inner = r >= 0
        self.r = torch.where(self.inner, r, self.l)
        nc = len(self.vol)
        self.nbr = self.slots(t(a["cell_nbr_offsets"]), t(a["cell_nbrs"]), nc, None)
        self.vtx = self.slots(t(a["cell_vertex_offsets"]), t(a["cell_vertices"]), nc, 0)
        if c["order"] == 2:
            M = torch.zeros((nc, D, D), dtype=torch.float64, device=device)
            for q in self.nbr:
                dx = self.x[:, q] - self.x
                M += torch.einsum("ic,jc->cij", dx, dx)
            self.inv = torch.linalg.inv(M)

    @staticmethod
    def slots(off, lst, nc, fill):
        """One index vector per list slot; a cell whose list is shorter repeats
        itself (fill None) or the list's first entry."""
        off, lst = off.long(), lst.long()
        n = off[1:] - off[:-1]
        own = torch.arange(nc, device=off.device)
        first = own if fill is None else lst[off[:-1]]
        return [torch.where(n > k, lst[(off[:-1] + k).clamp(max=len(lst) - 1)], first)
                for k in range(int(n.max()))]

    def values(self, s):
        D = self.D
        return torch.cat([s[:1 + D], s[1 + D:3 + D], s[4 + D:5 + D]])  # d, v, e, p, a

    def dt(self, s, t):
        D, n, c = self.D, self.nrm, self.c
        best = torch.zeros((), dtype=torch.float64, device=s.device)
        for side in (self.l, self.r):
            v = s[1:1 + D][:, side]
            lam = s[4 + D][side] + (v * n).sum(0).abs()
            best = torch.maximum(best, (lam * self.area / self.vol[side]).max())
        return torch.clamp(c["cfl"] / best, max=self.tf - t)

    def gradients(self, s):
        u, D = self.values(s), self.D
        b = torch.zeros((u.shape[0], D, u.shape[1]), dtype=torch.float64, device=s.device)
        if self.c["order"] == 1:
            return b
        lo, hi = u.clone(), u.clone()
        for q in self.nbr:
            w = u[:, q]
            b += (w - u)[:, None] * (self.x[:, q] - self.x)[None]
            lo, hi = torch.minimum(lo, w), torch.maximum(hi, w)
        g = torch.einsum("cij,kjc->kic", self.inv, b)
        if self.c["limiter"] == "none":
            return g
        phi = torch.ones_like(u)
        for q in self.vtx:
            du = (g * (self.xv[:, q] - self.x)[None]).sum(1)
            lim = torch.where(du > 1e-9, (hi - u) / du, torch.where(du < -1e-9, (lo - u) / du, 1.0))
            phi = torch.minimum(phi, lim)
        return g * phi.clamp(min=0.0)[:, None]

    def side(self, u, g, cell):
        D = self.D
        dx = self.xf - self.x[:, cell]
        du = (g[:, :, cell] * dx[None]).sum(1)
        if self.c["swap"]:  # the reference adds grad e to p and grad p to e
            du = torch.cat([du[:1 + D], du[2 + D:3 + D], du[1 + D:2 + D], du[3 + D:]])
        w = u[:, cell] + du
        return {"d": w[0], "v": w[1:1 + D], "e": w[1 + D], "p": w[2 + D], "a": w[3 + D]}

    def flux(self, w):
        vn = (w["v"] * self.nrm).sum(0)
        m = w["d"] * vn
        et = w["e"] + 0.5 * (w["v"] ** 2).sum(0)
        return torch.cat([m[None], m * w["v"] + w["p"] * self.nrm, (m * (et + w["p"] / w["d"]))[None]])

    @staticmethod
    def conserved(w):
        et = w["e"] + 0.5 * (w["v"] ** 2).sum(0)
        return torch.cat([w["d"][None], w["d"] * w["v"], (w["d"] * et)[None]])

    def fluxes(self, s, g):
        c, D = self.c, self.D
        u = self.values(s)
        l, r = self.side(u, g, self.l), self.side(u, g, self.r)
        vl, vr = (l["v"] * self.nrm).sum(0), (r["v"] * self.nrm).sum(0)
        fl, fr, ul, ur = self.flux(l), self.flux(r), self.conserved(l), self.conserved(r)
        if c["flux"] == "rusanov":
            lam = torch.maximum(l["a"] + vl.abs(), r["a"] + vr.abs())
            f = 0.5 * (fl + fr) - 0.5 * lam * (ur - ul)
        else:
            sl = torch.minimum(vl - l["a"], vr - r["a"])
            sr = torch.maximum(vl + l["a"], vr + r["a"])
            if c["flux"] == "hlle":
                f = (sr * fl - sl * fr + sl * sr * (ur - ul)) / (sr - sl)
            else:
                ml, mr = l["d"] * (sl - vl), r["d"] * (sr - vr)
                sm = (r["p"] - l["p"] + ml * vl - mr * vr) / (ml - mr)
                left = sm >= 0

                def pick(x, y):
                    return torch.where(left, x, y)

                k = {q: pick(l[q], r[q]) for q in "dvepa"}
                sk, mk, vk = pick(sl, sr), pick(ml, mr), pick(vl, vr)
                fac, dv = mk / (sk - sm), sm - vk
                uk = pick(ul, ur)
                star = torch.cat([fac[None], fac * (k["v"] + dv * self.nrm),
                                  (fac * (uk[D + 1] / k["d"] + dv * (sm + k["p"] / mk)))[None]])
                f = pick(fl, fr) + sk * (star - uk)
            f = torch.where(sl >= 0, fl, torch.where(sr <= 0, fr, f))
        if c["boundary"] == "outflow":
            edge = fl
        else:
            edge = torch.zeros_like(fl)
            edge[1:1 + D] = l["p"] * self.nrm
        return torch.where(self.inner, f, edge) * self.area

    def update(self, s, f, dt):
        D = self.D
        du = torch.zeros((D + 2, s.shape[1]), dtype=torch.float64, device=s.device)
        du.index_add_(1, self.l, -f)
        du.index_add_(1, self.r, torch.where(self.inner, f, 0.0))
        du *= dt / self.vol
        d, v, e = s[0], s[1:1 + D], s[1 + D]
        d2 = d + du[0]
        v2 = (d * v + du[1:1 + D]) / d2
        e2 = (d * (e + 0.5 * (v * v).sum(0)) + du[D + 1]) / d2 - 0.5 * (v2 * v2).sum(0)
        p = (self.gamma - 1.0) * d2 * e2
        a = (self.gamma * (self.gamma - 1.0) * e2).sqrt()
        return torch.cat([d2[None], v2, e2[None], p[None], (e2 / self.cv)[None], a[None]])

    def run(self, s, steps, stop):
        t, n = 0.0, 0
        while n < steps and not (stop and n % 10 == 0 and float(t) >= self.tf * (1 - 1e-12)):
            dt = self.dt(s, t)
            for _ in range(2):
                s = self.update(s, self.fluxes(s, self.gradients(s)), 0.5 * dt)
            t, n = t + dt, n + 1
        return s, n


def exact(c, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    p = params(c)
    if c["kind"] == "batch":
        got = []
        for k, n in enumerate(batch_sides(c)):
            m = box(c, (n, n), seed * 64 + k)
            s = torch.as_tensor(initial(c, batch_problem(k), m, p, seed * 64 + k), device=device)
            got.append(Plain(m, c, p, device).run(s, c["steps"], False)[0])
        return got
    mesh = box(c, sizes(c), seed)
    s = torch.as_tensor(initial(c, c["problem"], mesh, p, seed), device=device)
    plain = Plain(mesh, c, p, device)
    if c["kind"] == "tasks":
        dt = plain.dt(s, 0.0)
        g = plain.gradients(s)
        f = plain.fluxes(s, g)
        return {"state": plain.update(s, f, 0.5 * dt), "grads": g.reshape(-1, g.shape[-1]), "flux": f,
                "dt": dt.reshape(1)}
    s, n = plain.run(s, c["steps"], c["stop"] > 0)
    return {"state": s} if c["kind"] == "host" else {"state": s, "steps": None}
