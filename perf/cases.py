"""The work this framework does for its users, as timed cases.

A case names one call sequence through the public entry points:

* ``solve`` -- a steady solve of one mesh: the state goes in from host memory
  (a restart, or a predicted start), ``steps`` outer LU-SGS iterations run, and
  the state and the last residual norms come back to the host;
* ``batch`` -- several independent airfoil solves advanced together;
* ``cavity`` -- inner iterations of the incompressible (SIMPLE) solver;
* ``predict`` / ``train`` -- the warm-start network's inference and training.

Meshes come from the seeded generators, states from the seed of ``prepare``.
``exact`` restates the first-order inviscid solves, the network's inference
and its training in 64 bits with numpy and torch alone."""
import functools

import numpy as np
import torch

from oneflow_b200 import Batch, Solver, meshgen, params as P
from oneflow_b200.mlp import MLP
from oneflow_b200.solver import NS_SOLVER, TURB_SOLVER, Incompressible
from oneflow_b200.walldist import plate_wall_distance


def listed():
    return [
        # one small solve of the warm-start families: 4,096 triangles, every launch counts
        dict(name="bump_4k_fp64", kind="solve", mesh="bump", ni=64, nj=32, precision=0, order=1, ilim=-1, steps=50),
        # the inviscid bump at its benchmark size in the reference's own cell order (hundreds of sweep levels)
        dict(name="bump_65k_fp64_natural", kind="solve", mesh="bump", ni=256, nj=128, precision=0, order=0, ilim=-1,
             steps=10),
        # second order on an odd mesh size, FP32 faces, the reference's zone-wide limiter eps
        dict(name="bump_114k_mixed_venkat", kind="solve", mesh="bump", ni=333, nj=171, precision=1, order=1, ilim=2,
             steps=50),
        # a laminar plate of the size of the reference's regression cases, in its order and precision
        dict(name="plate2d_3k_fp64_laminar", kind="solve", mesh="plate2d", ni=72, nj=48, precision=0, order=0,
             ischeme=12, steps=20),
        # the drop-in's own setting on a 3-D RANS plate: FP64 faces, Green-Gauss, the reference's limiter
        dict(name="plate3d_312k_fp64_sa", kind="solve", mesh="plate3d", nx=100, ny=40, nz=13, precision=0, order=1,
             reference_options=True, steps=5),
        # the RANS-SA plate at its sample size and at its full benchmark size (6.0 M tetrahedra)
        dict(name="plate3d_600k_mixed_sa", kind="solve", mesh="plate3d", nx=200, ny=100, nz=5, precision=1, order=1,
             reference_options=False, steps=20),
        dict(name="plate3d_6m_mixed_sa", kind="solve", mesh="plate3d", nx=200, ny=100, nz=50, precision=1, order=1,
             reference_options=False, steps=20),
        # the transonic wing's hybrid mesh at its parity size: SLAU2, Green-Gauss, Barth
        dict(name="wing_769k_mixed_sa", kind="solve", mesh="wing", n_around=128, n_tet=20, nz_wing=30, nz_tip=10,
             precision=1, order=1, steps=10),
        # eight of the batched airfoils, uneven sizes, one graph launch per iteration
        dict(name="airfoils_8_mixed_sa", kind="batch", count=8, max_cells=120000, order=1, steps=20),
        # one SIMPLE inner iteration of the lid-driven cavity: four GMRES solves
        dict(name="cavity_128_fp64", kind="cavity", n=128, jitter=0.1, triangles=False, inner=1),
        # the warm start's network: a prediction for the cells of an airfoil batch, and a stretch of training
        dict(name="predict_295k", kind="predict", n_in=22, width=256, depth=6, n_out=4, rows=32 * 9216),
        dict(name="train_8192", kind="train", n_in=22, width=256, depth=6, n_out=4, rows=98304, batch=8192, steps=25),
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    kind = rng.choice(["bump", "bump", "plate2d", "plate3d", "wing", "batch", "cavity", "predict", "train"])
    if kind == "bump":
        ni = round(_log(rng, 48, 360))
        order = rng.randrange(2)
        return dict(kind="solve", mesh="bump", ni=ni, nj=max(20, round(ni * rng.uniform(0.4, 0.6))),
                    precision=rng.randrange(2), order=order, ilim=rng.choice([-1, 2]),
                    steps=rng.choice([8, 25]) if order == 0 else rng.choice([10, 30, 50]))
    if kind == "plate2d":
        ni = round(_log(rng, 36, 160))
        return dict(kind="solve", mesh="plate2d", ni=ni, nj=round(ni * rng.uniform(0.5, 0.8)),
                    precision=rng.randrange(2), order=rng.randrange(2), ischeme=rng.choice([1, 12]),
                    steps=rng.choice([10, 20]))
    if kind == "plate3d":
        precision = rng.randrange(2)
        nx, ny = round(_log(rng, 40, 200)), rng.randrange(30, 101)
        nz = round(_log(rng, 5, 25 if precision else 8))
        return dict(kind="solve", mesh="plate3d", nx=nx, ny=ny, nz=nz, precision=precision, order=1,
                    reference_options=rng.random() < 0.5, steps=rng.choice([5, 10]))
    if kind == "wing":
        return dict(kind="solve", mesh="wing", n_around=2 * rng.randrange(24, 65), n_tet=rng.randrange(8, 21),
                    nz_wing=rng.randrange(10, 31), nz_tip=rng.randrange(4, 11), precision=1, order=1,
                    steps=rng.choice([5, 10]))
    if kind == "batch":
        return dict(kind="batch", count=rng.randrange(2, 13), max_cells=round(_log(rng, 25000, 150000)),
                    order=rng.randrange(2), steps=rng.choice([5, 10, 20]))
    if kind == "cavity":
        return dict(kind="cavity", n=round(_log(rng, 32, 256)), jitter=0.1, triangles=rng.random() < 0.3, inner=1)
    net = dict(n_in=rng.choice([8, 22]), width=rng.choice([64, 128, 256]), depth=rng.randrange(3, 7), n_out=4)
    if kind == "predict":
        return dict(kind="predict", **net, rows=round(_log(rng, 4096, 786432)))
    return dict(kind="train", **net, rows=rng.randrange(20000, 200000), batch=64 * round(_log(rng, 8, 256)),
                steps=rng.choice([10, 25]))


# ---------------------------------------------------------------------------
# meshes and parameters
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _mesh(kind, *args):
    if kind == "bump":
        return meshgen.bump_channel(*args)
    if kind == "plate2d":
        return meshgen.plate_2d(*args)
    if kind == "plate3d":
        mesh = meshgen.flat_plate_tets(*args)
        mesh.wall_dist = plate_wall_distance(mesh)
        return mesh
    if kind == "cavity":
        return meshgen.lid_cavity_2d(args[0], jitter=args[1], triangles=args[2])
    n_around, n_tet, nz_wing, nz_tip = args
    return meshgen.swept_wing_hybrid(n_around=n_around, n_tet=n_tet, nz_wing=nz_wing, nz_tip=nz_tip)


@functools.lru_cache(maxsize=2)
def _airfoils(count, max_cells):
    return meshgen.airfoil_cases(count, max_cells=max_cells)


def _solve_mesh(case):
    k = case["mesh"]
    if k in ("bump", "plate2d"):
        return _mesh(k, case["ni"], case["nj"])
    if k == "plate3d":
        return _mesh(k, case["nx"], case["ny"], case["nz"])
    return _mesh(k, case["n_around"], case["n_tet"], case["nz_wing"], case["nz_tip"])


def _solve_params(case):
    kw = dict(precision=case["precision"], sweep_order=case["order"])
    k = case["mesh"]
    if k == "bump":
        if case["ilim"] == 2:
            kw.update(ilim=2, vencat_coef=0.05)
        return P.euler_bump(**kw)
    if k == "plate2d":
        return P.defaults(vismodel=1, ischeme=case["ischeme"], mach_ref=0.2, reynolds=1.0e4, cflst=1.0, cfled=5.0,
                          ncfl=100, **kw)
    if k == "plate3d":
        if case["reference_options"]:
            kw.update(igrad=0, venkat_kh3=0, vencat_coef=0.0001)
        return P.rans_plate(**kw)
    return P.transonic_wing(**kw)


def _inflow(prm):
    a = np.deg2rad(prm.aoa_degree)
    return np.array([1.0, np.cos(a), np.sin(a), 0.0, 1.0 / (prm.gama_ref * prm.mach_ref ** 2)])


def _start(prm, n_t, seed):
    """A start field near the free stream: every cell of it off by up to 0.1 %,
    as an interpolated or predicted start is.  Interior and ghost entries; the
    ghost entries are set again from the boundary conditions on upload."""
    rng = np.random.default_rng(seed)
    q = _inflow(prm)[:, None] * (1.0 + 1e-3 * rng.uniform(-1.0, 1.0, (5, n_t)))
    nut = prm.ref_sa * (1.0 + 1e-3 * rng.uniform(-1.0, 1.0, n_t)) if prm.vismodel >= 3 else None
    return q, nut


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


class _Solve:
    """A solver, its start field in pinned host memory and pinned buffers for what comes back."""

    def __init__(self, mesh, prm, seed):
        self.solver = Solver(mesh, prm)
        self.solver.init_flowfield()
        q, nut = _start(prm, self.solver.nT, seed)
        self.q0, self.q = _pinned(q), _pinned(np.zeros_like(q))
        self.nut0 = None if nut is None else _pinned(nut)
        self.nut = None if nut is None else _pinned(np.zeros_like(nut))

    def upload(self):
        s = self.solver
        s.set_outer_step(0)
        s.upload_state(self.q0)
        if self.nut0 is not None:
            s.upload_state(self.nut0, TURB_SOLVER)

    def download(self):
        s = self.solver
        out = {"q": s.state(out=self.q), "rms": s.residual_norms(NS_SOLVER)}
        if self.nut0 is not None:
            out["nut"] = s.state(TURB_SOLVER, out=self.nut)
            out["rms_sa"] = s.residual_norms(TURB_SOLVER)
        return out


def _samples(case, seed, dtype=np.float32):
    """Scaled features and targets of the network's rows: smooth functions of the inputs plus a little noise."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1.0, 1.0, (case["rows"], case["n_in"])).astype(np.float32)
    a = rng.normal(size=(case["n_in"], case["n_out"])) / np.sqrt(case["n_in"])
    y = np.tanh(2.0 * (x @ a.astype(np.float32))) + 0.01 * rng.standard_normal((case["rows"], case["n_out"]))
    return x.astype(dtype), y.astype(np.float32).astype(dtype)


def _layers(case):
    dims = [case["n_in"]] + [case["width"]] * case["depth"] + [case["n_out"]]
    return list(zip(dims[:-1], dims[1:]))


def _weights(case, seed):
    """Flat FP32 parameters, per layer W [fan_in][fan_out] then b [fan_out], of a network with a few steps behind it."""
    rng = np.random.default_rng(seed + 7)
    flat = []
    for k, n in _layers(case):
        flat += [rng.uniform(-1.0, 1.0, k * n) / np.sqrt(k), rng.uniform(-0.05, 0.05, n)]
    return np.concatenate(flat).astype(np.float32)


LEARNING_RATE, ADAM = 1e-3, (0.9, 0.999, 1e-8)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        return "solve", case, _Solve(_solve_mesh(case), _solve_params(case), seed)
    if kind == "batch":
        parts = [_Solve(mesh, P.rans_airfoil(**dict(fs, sweep_order=case["order"])), seed + i)
                 for i, (mesh, fs) in enumerate(_airfoils(case["count"], case["max_cells"]))]
        return "batch", case, parts, Batch([p.solver for p in parts])
    if kind == "cavity":
        mesh = _mesh("cavity", case["n"], case["jitter"], case["triangles"])
        prm = P.defaults(vismodel=1, reynolds=1000.0, mach_ref=0.1)
        rng = np.random.default_rng(seed)
        s = Incompressible(mesh, prm, meshgen.lid_velocity(mesh, rng.uniform(0.9, 1.1)))
        q = s.q()   # the free stream with its wall ghosts; a little of it perturbed inside
        q[1:4, :mesh.n_cells] *= 1.0 + 1e-3 * rng.uniform(-1.0, 1.0, (3, mesh.n_cells))
        return "cavity", case, s, q
    m = MLP(case["n_in"], case["width"], case["depth"], case["n_out"], seed=seed)
    w = _weights(case, seed)
    m.set_params(w)
    x, y = (torch.from_numpy(v).cuda() for v in _samples(case, seed))
    return kind, case, m, w, x, y, seed


def run(state):
    kind, case = state[0], state[1]
    if kind == "solve":
        s = state[2]
        s.upload()
        s.solver.step(case["steps"])
        return s.download()
    if kind == "batch":
        _, _, parts, batch = state
        for p in parts:
            p.upload()
        batch.step(case["steps"])
        return [p.download() for p in parts]
    if kind == "cavity":
        _, _, s, q = state
        s.upload_state(q)
        for _ in range(case["inner"]):
            s.update_residuals()
        return {"q": s.q(), "pp": s.field("pp"), "fq": s.field("fq"), "remax": s.stats()["remax"]}
    _, _, m, w, x, y, seed = state
    if kind == "predict":
        return m.predict(x)
    m.set_params(w)   # every stretch of training starts from the same network
    losses = m.train(x, y, case["steps"], batch=case["batch"], lr=LEARNING_RATE, seed=seed)
    return {"losses": losses, "params": m.params()}


# ---------------------------------------------------------------------------
# the work of one pass
# ---------------------------------------------------------------------------
def _iteration(n_cells, n_faces, three_d, order2, viscous, sa, precision):
    """Bytes and operations that one outer iteration cannot do without: the
    state read and written, the mesh (face normals, areas, centres and cells;
    cell volumes and centres), and per face the fluxes, increments and source
    terms of the models in use."""
    real = 4 if precision else 8
    cell = 2 * 5 * 8 + 4 * real + (8 * 2 + 8 if sa else 0)
    face = 7 * real + 8
    flops = n_faces * (250 + 2 * 130)
    if order2:
        flops += n_cells * 150 + n_faces * (6 * 15 + 2 * 5 * 20)
    if viscous:
        flops += n_faces * (200 + 2 * 15) + n_cells * 20
    if sa:
        flops += n_faces * 100 + n_cells * 100
    return n_cells * cell + n_faces * face, float(flops)


def work(case):
    kind = case["kind"]
    if kind in ("solve", "batch"):
        if kind == "solve":
            meshes = [(_solve_mesh(case), _solve_params(case))]
        else:
            meshes = [(m, P.rans_airfoil(**fs)) for m, fs in _airfoils(case["count"], case["max_cells"])]
        b = f = 0.0
        for m, p in meshes:
            x, y = _iteration(m.n_cells, m.n_faces, p.dimension == 3, p.ilim != -1, p.vismodel > 0, p.vismodel >= 3,
                              p.precision)
            b, f = b + x * case["steps"], f + y * case["steps"]
        return {"bytes": b, "flops": f}
    if kind == "cavity":
        # the pressure solve's Krylov steps (about 4 n of them, 500 at most) each need the basis so far once;
        # the momentum solves take a handful
        cells = case["n"] ** 2 * (2 if case["triangles"] else 1)
        k = min(500, 4 * case["n"])
        return {"bytes": float(8 * cells * (k * (k + 1) / 2 + 12 * k)) * case["inner"],
                "flops": float(cells * (4 * k * (k + 1) / 2 + 14 * k)) * case["inner"]}
    macs = sum(k * n for k, n in _layers(case))
    if kind == "predict":
        return {"bytes": 4.0 * case["rows"] * (case["n_in"] + case["n_out"]) + 2.0 * macs,
                "flops": 2.0 * case["rows"] * macs}
    rows = case["batch"] * case["steps"]
    return {"bytes": 4.0 * rows * (case["n_in"] + case["n_out"]) + 28.0 * macs * case["steps"],
            "flops": 6.0 * rows * macs}


# ---------------------------------------------------------------------------
# 64-bit restatements (numpy and torch only)
# ---------------------------------------------------------------------------
def exact(case, seed):
    """What ``run`` returns for these inputs in 64 bits, or None: a viscous,
    turbulent or limited solve takes minutes in numpy, and the SIMPLE
    iteration's solutions are defined by its GMRES tolerance alone."""
    kind = case["kind"]
    if kind == "solve" and case["mesh"] == "bump" and case["ilim"] == -1:
        return _exact_euler(case, seed)
    if kind == "predict":
        x, _ = _samples(case, seed, np.float64)
        with torch.no_grad():
            return _forward(torch.from_numpy(x).cuda(), _split(case, torch.from_numpy(_weights(case, seed)).double().cuda()))
    if kind == "train":
        return _exact_train(case, seed)
    return None


def _split(case, flat):
    out, o = [], 0
    for k, n in _layers(case):
        out.append((flat[o:o + k * n].view(k, n), flat[o + k * n:o + k * n + n]))
        o += k * n + n
    return out


def _forward(x, layers):
    for i, (w, b) in enumerate(layers):
        x = x @ w + b
        if i + 1 < len(layers):
            x = torch.nn.functional.gelu(x)
    return x


def _mix64(x):
    x = x ^ (x >> np.uint64(30))
    x = x * np.uint64(0xBF58476D1CE4E5B9)
    x = x ^ (x >> np.uint64(27))
    x = x * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


def _exact_train(case, seed):
    """Adam on the minibatches the seeded hash draws."""
    x, y = (torch.from_numpy(v).cuda() for v in _samples(case, seed, np.float64))
    flat = torch.from_numpy(_weights(case, seed)).double().cuda().requires_grad_()
    m, v = torch.zeros_like(flat), torch.zeros_like(flat)
    b1, b2, eps = ADAM
    losses = []
    for s in range(case["steps"]):
        with np.errstate(over="ignore"):
            h = _mix64(np.uint64(s) * np.uint64(0x9E3779B97F4A7C15) + np.arange(case["batch"], dtype=np.uint64))
            rows = (_mix64(np.uint64(seed) ^ h) % np.uint64(case["rows"])).astype(np.int64)
        i = torch.from_numpy(rows).cuda()
        loss = ((_forward(x[i], _split(case, flat)) - y[i]) ** 2).mean()
        (g,) = torch.autograd.grad(loss, flat)
        m, v = b1 * m + (1 - b1) * g, b2 * v + (1 - b2) * g * g
        with torch.no_grad():
            flat -= LEARNING_RATE * (m / (1 - b1 ** (s + 1))) / ((v / (1 - b2 ** (s + 1))).sqrt() + eps)
        losses.append(float(loss))
    return {"losses": np.array(losses), "params": flat.detach()}


def _greedy_colours(nbr, n):
    col = np.full(n, -1, np.int64)
    for i in range(n):
        used = {col[j] for j in nbr[i]}
        c = 0
        while c in used:
            c += 1
        col[i] = c
    return col


def _sweep_levels(nbr, key, n, lower):
    """Cells grouped so that each group reads only earlier ones of the sweep."""
    lev = np.zeros(n, np.int64)
    for i in np.argsort(key if lower else -key):
        before = [lev[j] for j in nbr[i] if (key[j] < key[i]) == lower]
        lev[i] = 1 + max(before) if before else 0
    order = np.argsort(lev, kind="stable")
    return np.split(order, np.cumsum(np.bincount(lev))[:-1])


def _roe(a, b, n, gam):
    """Roe flux of the face states a, b [5][m] along the unit normals n [2][m], with the entropy fix of the solver."""
    def parts(q):
        vn = n[0] * q[1] + n[1] * q[2]
        k = 0.5 * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2)
        h = gam / (gam - 1) * q[4] / q[0] + k
        e = q[4] / (gam - 1) + q[0] * k
        f = np.array([q[0] * vn, q[0] * vn * q[1] + n[0] * q[4], q[0] * vn * q[2] + n[1] * q[4], q[0] * vn * q[3],
                      q[0] * vn * h])
        return f, h, np.array([q[0], q[0] * q[1], q[0] * q[2], q[0] * q[3], e])
    fa, ha, ua = parts(a)
    fb, hb, ub = parts(b)
    r = np.sqrt(b[0] / a[0])
    mean = lambda s, t: (s + t * r) / (1 + r)  # noqa: E731
    u, v, w, h = mean(a[1], b[1]), mean(a[2], b[2]), mean(a[3], b[3]), mean(ha, hb)
    v2 = u * u + v * v + w * w
    vn = n[0] * u + n[1] * v
    c2 = (gam - 1) * (h - 0.5 * v2)
    c = np.sqrt(np.abs(c2))
    l1, l2, l3 = np.abs(vn), np.abs(vn + c), np.abs(vn - c)
    top = 1e-4 * np.maximum(l2, l3)
    l1, l2, l3 = np.maximum(l1, top), np.maximum(l2, top), np.maximum(l3, top)
    return 0.5 * (fa + fb - _eigen(ub - ua, l1, l2, l3, u, v, w, vn, v2, h, c2, c, n, gam))


def _eigen(d, l1, l2, l3, u, v, w, vn, v2, h, c2, c, n, gam):
    """The flux Jacobian's eigenvalues l1 (vn), l2 (vn + c), l3 (vn - c) applied to the conservative jump d."""
    x1, x2 = (2 * l1 - l2 - l3) / (2 * c2), (l2 - l3) / (2 * c)
    dc = vn * d[0] - n[0] * d[1] - n[1] * d[2]
    dh = (gam - 1) * (d[4] - u * d[1] - v * d[2] - w * d[3] + 0.5 * v2 * d[0])
    t1, t2 = dh * x1 + dc * x2, c2 * dc * x1 + dh * x2
    return np.array([l1 * d[0] - t1, l1 * d[1] - u * t1 + n[0] * t2, l1 * d[2] - v * t1 + n[1] * t2,
                     l1 * d[3] - w * t1, l1 * d[4] - h * t1 + vn * t2])


def _increment(qa, qb, dq, n, area, gam):
    """A neighbour's share of a cell's LU-SGS right-hand side: its split flux increment (Roe-averaged radius)."""
    k = lambda q: 0.5 * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2)  # noqa: E731
    enth = lambda q: gam / (gam - 1) * q[4] / q[0] + k(q)  # noqa: E731
    r = np.sqrt(qb[0] / qa[0])
    mean = lambda s, t: (s + t * r) / (1 + r)  # noqa: E731
    u, v, w, h = mean(qa[1], qb[1]), mean(qa[2], qb[2]), mean(qa[3], qb[3]), mean(enth(qa), enth(qb))
    radius = np.abs(n[0] * u + n[1] * v) + np.sqrt(np.abs((gam - 1) * (h - 0.5 * (u * u + v * v + w * w))))
    c2 = np.abs(gam * qb[4] / qb[0])
    c = np.sqrt(c2)
    vn = n[0] * qb[1] + n[1] * qb[2]
    l1, l2, l3 = 0.5 * (vn - radius), 0.5 * (vn + c - radius), 0.5 * (vn - c - radius)
    return area * _eigen(dq, l1, l2, l3, qb[1], qb[2], qb[3], vn, 2 * k(qb), enth(qb), c2, c, n, gam)


def _ghosts(q, lc, kind, n, inf, gam):
    """Ghost and wall-face states of the boundary faces from their cells' states: slip walls and the far field."""
    s = q[:, lc]
    vn = n[0] * s[1] + n[1] * s[2]
    wall = s.copy()
    wall[1] -= 2 * n[0] * vn
    wall[2] -= 2 * n[1] * vn
    face = 0.5 * (s + wall)
    cr, ci = np.sqrt(gam * inf[4] / inf[0]), np.sqrt(gam * s[4] / s[0])
    vr = n[0] * inf[1] + n[1] * inf[2]
    rp, rm = vn + 2 * ci / (gam - 1), vr - 2 * cr / (gam - 1)
    vb, cb = 0.5 * (rp + rm), 0.25 * (rp - rm) * (gam - 1)
    out = vb >= 0
    ent = np.where(out, s[4] / s[0] ** gam, inf[4] / inf[0] ** gam)
    far = np.empty_like(s)
    far[0] = (cb * cb / (ent * gam)) ** (1 / (gam - 1))
    for e, ne in ((1, n[0]), (2, n[1]), (3, 0.0)):
        far[e] = np.where(out, s[e] - ne * vn, inf[e] - ne * vr) + ne * vb
    far[4] = cb * cb * far[0] / gam
    fast = np.sqrt(s[1] ** 2 + s[2] ** 2 + s[3] ** 2) > ci
    far = np.where(fast, np.where(vn >= 0, s, inf[:, None]), far)
    return np.where(kind == 2, wall, far), face


def _exact_euler(case, seed):
    """The first-order inviscid bump: Roe fluxes, local time step, LU-SGS sweeps in the case's cell order."""
    mesh, prm = _solve_mesh(case), _solve_params(case)
    N, B, gam, inf = mesh.n_cells, mesh.n_bfaces, prm.gama_ref, _inflow(prm)
    nodes = mesh.face_nodes.reshape(-1, 2)
    dx, dy = mesh.x[nodes[:, 1]] - mesh.x[nodes[:, 0]], mesh.y[nodes[:, 1]] - mesh.y[nodes[:, 0]]
    area = np.hypot(dx, dy)
    n = np.array([dy, -dx]) / area
    lc, rc = mesh.lc.astype(np.int64), mesh.rc.astype(np.int64)
    rc[:B] = N + np.arange(B)
    kind = mesh.bc_type
    add = lambda cells, v: np.bincount(cells, v, N)  # noqa: E731
    mx, my = 0.5 * (mesh.x[nodes[:, 0]] + mesh.x[nodes[:, 1]]), 0.5 * (mesh.y[nodes[:, 0]] + mesh.y[nodes[:, 1]])
    flow = 0.5 * (mx * n[0] + my * n[1]) * area   # the divergence theorem's share of a cell's area
    vol = add(lc, flow) - add(rc[B:], flow[B:])
    nbr = [[] for _ in range(N)]
    for f in range(B, len(lc)):
        nbr[lc[f]].append(rc[f])
        nbr[rc[f]].append(lc[f])
    key = np.arange(N)
    if case["order"] == 1:
        key = np.empty(N, np.int64)
        key[np.lexsort((np.arange(N), _greedy_colours(nbr, N)))] = np.arange(N)
    # every cell's faces: {face, neighbour, sign of the normal seen from the cell}, grouped by cell
    own = np.concatenate([lc[B:], rc[B:]])
    face = np.concatenate([np.arange(B, len(lc))] * 2)
    other = np.concatenate([rc[B:], lc[B:]])
    sign = np.concatenate([np.ones(len(lc) - B), -np.ones(len(lc) - B)])
    sweeps = []
    for lower in (True, False):
        use = (key[other] < key[own]) == lower
        o = np.flatnonzero(use)[np.argsort(own[use], kind="stable")]
        start = np.searchsorted(own[o], np.arange(N + 1))
        plan = []
        for cells in _sweep_levels(nbr, key, N, lower):
            cnt = start[cells + 1] - start[cells]
            at = np.repeat(start[cells] - np.concatenate([[0], np.cumsum(cnt)[:-1]]), cnt) + np.arange(cnt.sum())
            plan.append((cells, np.repeat(np.arange(len(cells)), cnt), o[at]))
        sweeps.append(plan)
    q = _start(prm, N + B, seed)[0]
    q[:, N:], wall = _ghosts(q, lc[:B], kind, n[:, :B], inf, gam)
    for _ in range(case["steps"]):
        ql, qr = q[:, lc], q[:, rc]
        m = 0.5 * (ql + qr)
        radius = 0.5 * area * (np.abs(n[0] * m[1] + n[1] * m[2]) + np.sqrt(gam * m[4] / m[0]))
        inv = add(lc, radius) + add(rc[B:], radius[B:])
        rad = inv / prm.cflst + inv   # vol / dt + radius, dt = cfl vol / radius
        a, b = ql.copy(), qr.copy()
        a[:, :B] = b[:, :B] = np.where(kind == 2, wall, m[:, :B])
        fl = area * _roe(a, b, n, gam)
        res = np.array([add(rc[B:], fl[e, B:]) - add(lc, fl[e]) for e in range(5)])
        dq = np.zeros((5, N))
        for k, plan in enumerate(sweeps):
            for cells, at, o in plan:
                rhs = np.zeros((5, len(cells)))
                if len(o):
                    f = face[o]
                    df = _increment(q[:, own[o]], q[:, other[o]], dq[:, other[o]], n[:, f] * sign[o], area[f], gam)
                    rhs = np.array([np.bincount(at, df[e], len(cells)) for e in range(5)])
                dq[:, cells] = (res[:, cells] - rhs) / rad[cells] if k == 0 else dq[:, cells] - rhs / rad[cells]
        p = q[:, :N]
        r = p[0] + dq[0]
        vel = (p[0] * p[1:4] + dq[1:4]) / r
        e = p[4] / (gam - 1) + 0.5 * p[0] * (p[1:4] ** 2).sum(0) + dq[4]
        q[:, :N] = np.concatenate([[r], vel, [(gam - 1) * (e - 0.5 * r * (vel ** 2).sum(0))]])
        q[:, N:], wall = _ghosts(q, lc[:B], kind, n[:, :B], inf, gam)
    return {"q": q, "rms": np.sqrt((res ** 2).mean(1))}
