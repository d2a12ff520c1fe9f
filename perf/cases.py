"""Performance cases of the cloth solver: what its users run, through the public
entry points, from the smallest interactive sheet to the largest drape.

listed() names the cases, draw() makes more of the same ranges, prepare() builds
what a program holds before the call (scene, solver handle, start state), run()
is one pass and returns its results, work() is the least a pass must move and
compute, and exact() is the same result from plain torch in 64 bits where the
result is a mathematical quantity.

A stepping pass uploads its start state and steps from it, so passes repeat. The
reference stepper budget (10 Newton iterations, 60 PCG iterations) truncates the
solve, so its result is the algorithm's and exact() has none for it; the
"exact" Newton mode converges every step, to a solution exact() finds with
dense Newton iterations.
"""
import math

import numpy as np
import torch

import closim_b200 as cb
from closim_b200 import configs
from closim_b200.adjoint import ClothRollout
from closim_b200.avatar import AvatarCollider, LinearMotion, SphereGeometry, Transform, toCollisionObject
from closim_b200.batch import BatchSolver
from closim_b200.broadphase import GpuBroadPhase
from closim_b200.garment import AssembledGarment, AvatarDriver, createFittingScene
from closim_b200.material import OrthotropicStVKMaterial

EXACT_TOL = 3e-4  # PCG tolerance of the exact-Newton mode, as the benchmark sets it


def listed():
    return [
        # the smallest call of an interactive tool: a 41 x 9 strip under moving pins, FP64, Jacobi, step by step
        dict(name="strip_fp64", kind="strip", nx=40, ny=8, steps=2),
        # the reference-equal FP64 step on the standard drape as it lands: Schwarz PCG, floor contact, friction
        dict(name="drape_fp64", kind="drape_fp64", nx=63, ny=63, steps=1, precond="schwarz"),
        # FP64 garment session at an odd size: a moving avatar sphere under a large panel, Jacobi default options
        dict(name="garment_fp64", kind="garment", nx=120, ny=94, steps=1),
        # a small sheet in production mode (mixed precision, converged steps): launch-bound
        dict(name="drape_mixed_small", kind="drape_mixed", nx=16, ny=12, steps=4),
        # the benchmark's drape in production mode, through the landing
        dict(name="drape_mixed", kind="drape_mixed", nx=63, ny=63, steps=3),
        # a mixed sheet near the largest the one-cluster solve takes, ragged sides
        dict(name="drape_mixed_large", kind="drape_mixed", nx=134, ny=108, steps=2),
        # the largest drape: 256 x 256 on a static sphere, mixed precision, reference budget
        dict(name="sphere_mixed", kind="sphere", nx=255, ny=255, steps=1),
        # many uneven sheets in one batched step (dataset generation)
        dict(name="batch", kind="batch", count=96, side_min=16, side_max=80, steps=1),
        # material fit: forward rollout and adjoint of a hung sheet (FP64 exact solves, backward pass)
        dict(name="fit", kind="fit", nx=18, ny=15, steps=2),
        # material model evaluation: energy, gradient and Hessian product of a mesh
        dict(name="material", kind="material", nx=130, ny=97),
        # collision broadphase of a folding sheet, as the FP32 mirror and as the exact set
        dict(name="broadphase_mirror", kind="broadphase", nx=40, ny=33, mode="mirror"),
        dict(name="broadphase_exact", kind="broadphase", nx=159, ny=127, mode="exact"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["strip", "drape_fp64", "garment", "drape_mixed", "drape_mixed", "sphere", "batch", "fit",
                       "material", "broadphase"])
    if kind == "strip":
        return dict(kind=kind, nx=_logint(rng, 10, 120), ny=_logint(rng, 2, 20), steps=rng.randint(1, 3))
    if kind == "drape_fp64":
        return dict(kind=kind, nx=_logint(rng, 9, 90), ny=_logint(rng, 9, 90), steps=1,
                    precond=rng.choice(["jacobi", "schwarz", "mas2"]))
    if kind == "garment":
        return dict(kind=kind, nx=_logint(rng, 24, 125), ny=_logint(rng, 24, 125), steps=1)
    if kind == "drape_mixed":
        return dict(kind=kind, nx=_logint(rng, 10, 135), ny=_logint(rng, 10, 135), steps=rng.randint(1, 3))
    if kind == "sphere":
        return dict(kind=kind, nx=rng.randint(150, 255), ny=rng.randint(150, 255), steps=1)
    if kind == "batch":
        lo = rng.randint(12, 40)
        return dict(kind=kind, count=_logint(rng, 4, 96), side_min=lo, side_max=lo + rng.randint(1, 40), steps=1)
    if kind == "fit":
        return dict(kind=kind, nx=rng.randint(8, 17), ny=rng.randint(8, 16), steps=2)
    if kind == "material":
        return dict(kind=kind, nx=_logint(rng, 8, 255), ny=_logint(rng, 8, 255))
    return dict(kind=kind, nx=_logint(rng, 8, 255), ny=_logint(rng, 8, 255), mode=rng.choice(["mirror", "exact"]))


# ---- workloads -----------------------------------------------------------------------

def _drape(case, seed):
    """The floor drape thrown just above the floor: it lands and slides from the first step."""
    cfg = configs.floor_drape(seed=seed, nx=case["nx"], ny=case["ny"], w=0.0127 * case["nx"], hgt=0.0127 * case["ny"],
                              height=0.002, precond=case.get("precond", "schwarz"))
    cfg["v"] = np.tile([0.3, -0.1, 0.1], cfg["x"].size // 3)
    return cfg


def _fit_config(case, seed):
    cfg = configs.material_fit(seed=seed, nx=case["nx"], ny=case["ny"], w=0.00625 * case["nx"],
                               hgt=0.00625 * case["ny"], steps=case["steps"], grad_tol=1e-10, pcg_max_iters=1500)
    rng = np.random.default_rng(seed + 1000)
    cfg["v"] = rng.normal(0.0, 0.01, cfg["x"].size)
    return cfg


def _garment(case, seed):
    h = 0.01
    pos, uv, idx = configs._grid(case["nx"], case["ny"], 0.008 * case["nx"], 0.008 * case["ny"])
    pos = pos.copy()
    c = (0.004 * case["nx"], 0.004 * case["ny"])
    rng = np.random.default_rng(seed)
    pos[1::3] += rng.uniform(0.0, 2e-4, pos.size // 3).astype(np.float32)
    low, high = Transform((c[0], -0.0606, c[1])), Transform((c[0], -0.0590, c[1]))
    sphere = AvatarCollider("torso", "torso", SphereGeometry(0.06, 24, 12), 0.004,
                            motion=LinearMotion(low, high, 0.0, 4 * h))
    fs = createFittingScene(AssembledGarment(pos, uv, idx), avatar=toCollisionObject(sphere, 0.0),
                            material=cb.ClothMaterial(**configs._material()),
                            contact=cb.ContactParams(1e-3, 50.0, 1e-4, 0.3, 1e-4), arealDensityKgM2=0.2)
    return h, fs, sphere


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, kind=kind)
    if kind == "broadphase":
        nx, ny = case["nx"], case["ny"]
        pos, _, idx = configs._grid(nx, ny, 0.8, 0.8 * ny / nx)
        x0 = pos.astype(np.float64).reshape(-1, 3)
        rng = np.random.default_rng(seed)
        cell = 0.8 / nx
        x0[:, 0] += rng.uniform(-0.1, 0.1, len(x0)) * cell
        x0[:, 2] += rng.uniform(-0.1, 0.1, len(x0)) * cell
        zc = 0.5 * (x0[:, 2].min() + x0[:, 2].max())
        far = x0[:, 2] > zc
        r = x0[far, 2] - zc  # the far half lies folded over the near one, 2 mm above it
        x0[far, 2] = zc - r * math.cos(0.01)
        x0[far, 1] = x0[far, 1] + 0.002 + r * math.sin(0.01)
        x1 = x0.copy()
        x1[far, 1] -= 0.001
        m = idx.size // 3
        st["bp"] = GpuBroadPhase(indices=idx, triCount=m, pad=0.25 * cell, pairCapacity=64 * m + 1024,
                                 mode=case["mode"], n=len(x0))
        st["x0"] = torch.from_numpy(x0.ravel().copy()).cuda()
        st["x1"] = torch.from_numpy(x1.ravel().copy()).cuda()
        return st
    if kind == "batch":
        # the sheets (sides, materials, pins) are the case's; their motion is the seed's
        sheets = configs.batch_sheets(count=case["count"], side_min=case["side_min"], side_max=case["side_max"])
        rng = np.random.default_rng(seed)
        for s in sheets:
            s["v"] = rng.normal(0.0, 0.02, s["x"].size)
        st["batch"] = BatchSolver(sheets)
        return st
    if kind == "material":
        pos, uv, idx = configs._grid(case["nx"], case["ny"], 0.01 * case["nx"], 0.01 * case["ny"])
        st["mesh"] = cb.preprocess(pos, uv, idx, 0.2)
        st["mat"] = OrthotropicStVKMaterial.fromLegacy(cb.ClothMaterial(**configs._material(stretchWeft=3e3)))
        rng = np.random.default_rng(seed)
        st["x"] = pos.astype(np.float64) * 1.01 + rng.normal(0.0, 5e-4, pos.size)
        st["p"] = rng.normal(0.0, 1.0, pos.size)
        st["mat"].energy(st["x"], st["mesh"])  # places the mesh on the GPU
        return st
    if kind == "garment":
        h, fs, sphere = _garment(case, seed)
        s = cb.CudaSolver("fp64")
        s.initialize(fs.scene)
        st.update(solver=s, scene=fs.scene, h=h, driver=AvatarDriver([sphere], s), x=fs.scene.positions.copy(),
                  v=np.zeros_like(fs.scene.positions))
        st["v"][1::3] = -0.05
        return st
    if kind == "strip":
        rng = np.random.default_rng(seed)
        cfg = configs.strip_pull(seed=seed, nx=case["nx"], ny=case["ny"], w=0.025 * case["nx"],
                                 hgt=0.025 * case["ny"])
        cfg["v"] = rng.normal(0.0, 0.01, cfg["x"].size)
    elif kind == "fit":
        cfg = _fit_config(case, seed)
    elif kind == "sphere":
        cfg = configs.sphere_drape(seed=seed, nx=case["nx"], ny=case["ny"], w=case["nx"] / 255.0,
                                   hgt=case["ny"] / 255.0, drop=0.2006)
        cfg["v"] = cfg["v"].copy()
        cfg["v"][1::3] = -0.05
    else:
        cfg = _drape(case, seed)
    sc = configs.make_scene(cfg)
    mixed = kind in ("drape_mixed", "sphere")
    opts = dict(cfg["options"])
    if kind == "drape_mixed":
        opts.update(newtonIters=40, pcgMaxIters=3000, gradTol=1e-10)
    s = cb.CudaSolver("mixed" if mixed else "fp64", **opts)
    s.initialize(sc)
    if kind in ("drape_mixed", "fit"):
        s.setNewtonMode("exact", EXACT_TOL)
    st.update(solver=s, scene=sc, cfg=cfg, h=cfg["h"], x=cfg["x"].copy(), v=cfg["v"].copy())
    if kind == "strip":
        st["pins"] = [configs.pins_at(cfg, k) for k in range(case["steps"])]
    if kind == "fit":
        s.setAdjointOptions(4000, 1e-12)
        st["theta"] = torch.tensor(cfg["theta0"], dtype=torch.float64, requires_grad=True)
        st["v0"] = torch.from_numpy(cfg["v"].copy()).requires_grad_(True)
        st["target"] = torch.from_numpy(_target(cfg))
    return st


def _target(cfg):
    x = cfg["x"].copy()
    x[1::3] -= 0.01
    return x


def run(st):
    kind = st["kind"]
    if kind == "broadphase":
        r = st["bp"].build(st["x0"], st["x1"])
        m = st["bp"].lastMirror
        return dict(pairs=r["pairs"], morton=m["morton"].astype(np.int64), payload=m["payload"].astype(np.int64),
                    left=m["nodeLeft"], right=m["nodeRight"], lo=m["nodeMin"], hi=m["nodeMax"])
    if kind == "batch":
        b = st["batch"]
        b.step(0.01, st["case"]["steps"])
        return b.allPositions(), b.allVelocities()
    if kind == "material":
        mat, mesh = st["mat"], st["mesh"]
        ev = mat.gradient(st["x"], mesh)
        return mat.energy(st["x"], mesh), ev.energy, ev.grad, ev.maxStrain, mat.hessianVector(st["x"], st["p"], mesh)
    if kind == "fit":
        st["theta"].grad = st["v0"].grad = None
        xN = ClothRollout.apply(st["theta"], st["v0"], st["solver"], st["x"], st["h"], st["case"]["steps"], 2)
        loss = ((xN - st["target"]) ** 2).sum() / (xN.numel() // 3)
        loss.backward()
        return xN.detach(), st["theta"].grad, st["v0"].grad
    s, sc = st["solver"], st["scene"]
    sc.positions[:] = st["x"]
    sc.velocities[:] = st["v"]
    s.push_state()
    if kind == "strip":
        for pins in st["pins"]:
            sc.pinned = pins
            s.step(st["h"])
    elif kind == "garment":
        for k in range(st["case"]["steps"]):
            st["driver"].advance_to((k + 1) * st["h"])
            s.step(st["h"])
    else:
        s.advance(st["h"], st["case"]["steps"])
        s.pull()
    return sc.positions, sc.velocities


def work(case):
    """Mesh constants and the start state read once, the results written once;
    floating-point work of one Newton iteration (gradient, one Hessian product
    per 16 PCG iterations' worth of useful search) per step, or of one
    evaluation."""
    kind = case["kind"]
    if kind == "batch":
        side = 0.5 * (case["side_min"] + case["side_max"])
        n, m, copies = side * side, 2 * (side - 1) ** 2, case["count"]
    else:
        n, m, copies = (case["nx"] + 1) * (case["ny"] + 1), 2 * case["nx"] * case["ny"], 1
    mesh = 32 * m + 4 * n + 1.5 * m * 40
    if kind == "broadphase":
        return {"bytes": 48 * n + 12 * m + 100 * m, "flops": 100 * m}
    if kind == "material":
        return {"bytes": 3 * mesh + 24 * n * 5 + 24 * n * 2, "flops": 3 * 200 * m + 2 * 400 * m}
    steps = case["steps"]
    bytes_ = steps * mesh + 96 * n
    flops = steps * (600 * m + 16 * 200 * m)
    if kind == "fit":
        bytes_, flops = 2 * bytes_ + 24 * n * steps, 2 * flops
    return {"bytes": copies * bytes_, "flops": copies * flops}


# ---- the same results in plain torch, 64 bits --------------------------------------------

class _Sheet:
    """Implicit-Euler step of a sheet from its mesh arrays (float32 constants, as
    the mesh holds them): dense Newton on inertia, orthotropic StVK membrane,
    dihedral bending, floor barrier and the frozen-multiplier floor friction."""

    def __init__(self, mesh, mat, dev):
        f64 = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float64)).to(dev)
        i64 = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.int64)).to(dev)
        self.n, self.dev, self.mat = mesh.count, dev, mat
        self.tri = i64(mesh.indices).reshape(-1, 3)
        self.inv = f64(mesh.invDm).reshape(-1, 2, 2)  # [[a, b], [c, d]]
        self.s = f64(mesh.areas)
        self.mass = f64(mesh.masses)
        self.hin = i64(mesh.hinges).reshape(-1, 4)
        meta = f64(mesh.hingeMeta).reshape(-1, 3)
        self.rest, self.w = meta[:, 0], meta[:, 1] ** 2 / meta[:, 2].clamp_min(1e-12)

    @staticmethod
    def membrane(q, inv, s, th):
        F0 = inv[0, 0] * (q[1] - q[0]) + inv[1, 0] * (q[2] - q[0])
        F1 = inv[0, 1] * (q[1] - q[0]) + inv[1, 1] * (q[2] - q[0])
        e0, e1, e2 = 0.5 * (F0 @ F0 - 1), 0.5 * (F1 @ F1 - 1), 0.5 * (F0 @ F1)
        return s * (0.5 * th[0] * e0 * e0 + 0.5 * th[1] * e1 * e1 + 2 * th[2] * e2 * e2)

    @staticmethod
    def bend(q, rest, w, k):
        e, a, b = q[1] - q[0], q[2] - q[0], q[3] - q[0]
        n1, n2 = torch.linalg.cross(e, a), torch.linalg.cross(e, b)
        m2 = -n2
        phi = torch.atan2(torch.linalg.cross(n1, m2) @ (e / e.norm()), n1 @ m2)
        # the angle between the triangles is pi - |phi|; a flat rest state is smooth in phi
        return torch.where(rest > math.pi - 1e-3, 0.5 * k * w * phi * phi,
                           0.5 * k * w * (math.pi - phi.abs() - rest) ** 2)

    def theta(self):
        m = self.mat
        return torch.tensor([m.stretchWarp * m.thickness, m.stretchWeft * m.thickness, m.shear * m.thickness,
                             0.5 * (m.bendWarp + m.bendWeft)], dtype=torch.float64, device=self.dev)

    def _map(self, fm, fb, x, th):
        vm = torch.func.vmap
        return (vm(fm, in_dims=(0, 0, 0, None))(x[self.tri], self.inv, self.s, th[:3]),
                vm(fb, in_dims=(0, 0, 0, None))(x[self.hin], self.rest, self.w, th[3]))

    def energy(self, x, th):
        a, b = self._map(self.membrane, self.bend, x, th)
        return a.sum() + b.sum()

    def grad(self, x, th):
        gm, gb = self._map(torch.func.grad(self.membrane), torch.func.grad(self.bend), x, th)
        g = torch.zeros_like(x)
        g.index_add_(0, self.tri.reshape(-1), gm.reshape(-1, 3))
        return g.index_add_(0, self.hin.reshape(-1), gb.reshape(-1, 3))

    def hessian(self, x, th):
        hm, hb = self._map(torch.func.hessian(self.membrane), torch.func.hessian(self.bend), x, th)
        H = torch.zeros(9 * self.n * self.n, dtype=torch.float64, device=self.dev)
        axis = torch.arange(3, device=self.dev)
        for ids, h in ((self.tri, hm), (self.hin, hb)):
            k = ids.shape[1]
            dof = (ids[:, :, None] * 3 + axis).reshape(-1, 3 * k)
            H.index_add_(0, (dof[:, :, None] * (3 * self.n) + dof[:, None, :]).reshape(-1), h.reshape(-1))
        return H.reshape(3 * self.n, 3 * self.n)

    def step(self, x0, v0, h, g, pins, floor, th):
        """One converged step; returns x1, v1, the Hessian at x1 and the free dofs."""
        free = torch.ones(self.n, 3, dtype=torch.bool, device=self.dev)
        free[pins] = False
        free = free.reshape(-1)
        M = (self.mass / h ** 2)[:, None]
        target = x0 + h * v0 + h * h * g
        x = x0 + h * v0
        x[pins] = x0[pins]
        lagged = None
        if floor:
            level, dhat, kappa, mu, eps = floor
            low = x[:, 1] - level <= 0.2 * dhat  # start above the floor
            x[low, 1] = torch.minimum(x0[low, 1], torch.full_like(x0[low, 1], level + 0.2 * dhat))
        for it in range(80):
            G = M * (x - target) + self.grad(x, th)
            H = self.hessian(x, th)
            H.diagonal().add_(M.expand(-1, 3).reshape(-1))
            if floor:
                d = x[:, 1] - level
                on = d < dhat
                u = d - dhat
                L = torch.log(d.clamp_min(1e-12) / dhat)
                db = torch.where(on, -2 * u * L - u * u / d, 0.0)
                ddb = torch.where(on, -2 * L - 4 * u / d + u * u / d ** 2, 0.0)
                G[:, 1] += kappa * db
                slip = (x - x0) * torch.tensor([1.0, 0.0, 1.0], dtype=torch.float64, device=self.dev)
                mag = torch.sqrt((slip ** 2).sum(1) + eps * eps)
                f = torch.where(on, mu * (-kappa * db).clamp_min(0) / mag, 0.0)
                G += f[:, None] * slip
                D = torch.zeros(self.n, 3, dtype=torch.float64, device=self.dev)
                D[:, 1] = kappa * ddb.clamp_min(0)
                D[:, 0] = D[:, 2] = f
                H.diagonal().add_(D.reshape(-1))
            r = torch.where(free, G.reshape(-1), 0.0)
            if float(r.norm()) < 1e-12 * math.sqrt(self.n) or it == 79:
                break
            Hf = torch.where(free[:, None] & free[None, :], H, 0.0)
            Hf.diagonal().add_((~free).double())
            shift = 0.0
            while True:
                C, bad = torch.linalg.cholesky_ex(Hf)
                if int(bad) == 0:
                    break
                more = float(Hf.diagonal().abs().mean()) * 1e-3 if shift == 0 else shift
                Hf.diagonal().add_(more)
                shift += more
            dx = -torch.cholesky_solve(r[:, None], C)[:, 0].reshape(-1, 3)
            a = min(1.0, 0.01 / max(float(dx.abs().max()), 1e-30))
            if floor:
                while bool((x[:, 1] + a * dx[:, 1] - level <= 0.3 * (x[:, 1] - level)).any()):
                    a *= 0.5
            x = x + a * dx
        damp = 1 - min(max(self.mat.damping, 0.0), 0.1)
        v = (x - x0) / h * damp
        if floor:
            stop = (x[:, 1] - level < dhat) & (v[:, 1] < 0)
            v[stop, 1] = 0.0
        return x, v, H, free


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("drape_mixed", "fit", "material"):
        return None
    if kind == "drape_mixed" and (case["nx"] + 1) * (case["ny"] + 1) > 4600:
        return None  # the dense Newton matrices would take too long
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "material":
        st = prepare(case, seed)
        sh = _Sheet(st["mesh"], cb.ClothMaterial(**configs._material(stretchWeft=3e3)), dev)
        x = torch.from_numpy(st["x"]).to(dev).reshape(-1, 3)
        p = torch.from_numpy(st["p"]).to(dev).reshape(-1, 3)
        th = sh.theta()
        e = sh.energy(x, th).item()
        flat = th.clone()
        flat[3] = 0.0  # the Hessian product is the membrane's
        hp = torch.func.jvp(lambda q: sh.grad(q, flat), (x,), (p,))[1]
        q = x[sh.tri]
        F0 = sh.inv[:, 0, 0, None] * (q[:, 1] - q[:, 0]) + sh.inv[:, 1, 0, None] * (q[:, 2] - q[:, 0])
        F1 = sh.inv[:, 0, 1, None] * (q[:, 1] - q[:, 0]) + sh.inv[:, 1, 1, None] * (q[:, 2] - q[:, 0])
        strain = torch.stack([0.5 * ((F0 * F0).sum(1) - 1), 0.5 * ((F1 * F1).sum(1) - 1), 0.5 * (F0 * F1).sum(1)])
        return e, e, sh.grad(x, th).reshape(-1).cpu(), strain.abs().max().item(), hp.reshape(-1).cpu()
    cfg = _drape(case, seed) if kind == "drape_mixed" else _fit_config(case, seed)
    mesh = cb.preprocess(cfg["pos"], cfg["uv"], cfg["idx"], cfg["density"])
    sh = _Sheet(mesh, cb.ClothMaterial(**cfg["material"]), dev)
    t = lambda a: torch.from_numpy(np.asarray(a, np.float64).copy()).to(dev).reshape(-1, 3)
    x, v, h, g = t(cfg["x"]), t(cfg["v"]), cfg["h"], t(cfg["gravity"])
    c = cfg["contact"]
    floor = (c["floorY"], c["dHatM"], c["kappaJ"], c["frictionMu"], c["frictionEpsM"]) if kind == "drape_mixed" else None
    th = sh.theta()
    pins = cfg["fixed_pins"]
    trace = []
    for _ in range(case["steps"]):
        x0 = x
        x, v, H, free = sh.step(x, v, h, g, pins, floor, th)
        trace.append((x, H, free))
    if kind == "drape_mixed":
        return x.reshape(-1).cpu(), v.reshape(-1).cpu()
    # implicit differentiation of each converged step, backwards
    M = (sh.mass / h ** 2)[:, None].expand(-1, 3).reshape(-1)
    lx = (2 * (x - t(_target(cfg))) / sh.n).reshape(-1)
    lv = torch.zeros_like(lx)
    damp = 1 - min(max(sh.mat.damping, 0.0), 0.1)
    dth = torch.zeros(4, dtype=torch.float64, device=dev)
    for x1, H, free in reversed(trace):
        rhs = torch.where(free, lx + damp * lv / h, 0.0)
        Hf = torch.where(free[:, None] & free[None, :], H, 0.0)
        Hf.diagonal().add_((~free).double())
        mu = torch.where(free, torch.linalg.solve(Hf, rhs), 0.0)
        J = torch.func.jacfwd(lambda q: (sh.grad(x1, q).reshape(-1) * mu).sum())(th)
        dth -= J
        lx, lv = (torch.where(free, M * mu - damp * lv / h, 0.0), torch.where(free, M * mu * h, 0.0))
    thick = sh.mat.thickness
    dth = dth * torch.tensor([thick, thick, thick, 1.0], dtype=torch.float64, device=dev)
    return x.reshape(-1).cpu(), dth.cpu(), lv.cpu()
