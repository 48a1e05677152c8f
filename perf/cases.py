"""The timed cases of the MPM library: what its users run, through its public entry points.

A case is one simulation as a program drives it: the particles of a state are handed over as
device arrays (`set_particles_device`), advanced (`advance` for fixed-dt substeps,
`simulate_frame` for one adaptive frame, `Advance_One_Time_Step` for the backward-Euler solve,
`autograd.rollout` and its backward for gradients) and read back as device arrays
(`get_particles_device`).  The geometries are those of `physbam_b200.scenes` (the 2D block, the
colliding spheres, the dam break, the batch of boxes, snow and sand balls, the differentiable
cube), seeded on the GPU: `ppc` particles uniform in every cell of the body, whole cells only, so
that the particle count depends on the case alone.  States start in mid-simulation: F, V and B
carry smooth random fields, so stresses, collisions and yielding are at work from the first substep.

`exact` restates the substep in FP64 torch (weights, P2G, stress, grid update against the walls,
G2P, plasticity), from the formulas alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from physbam_b200 import autograd as A
from physbam_b200 import driver as D
from physbam_b200 import scenes as S

FP32, FP64 = "fp32", "fp64"
INSET = 0.05          # the walls of every scene that has them
RADIUS = 0.12         # of the spheres, at x = 0.38 and 0.62: in contact
GRAVITY = -9.8

# kind -> (constitutive model, density, (E low, E high), nu)
MATERIALS = {
    "block2d": (S.COROTATED, 1000.0, (1e4, 1e4), 0.3),
    "box": (S.COROTATED, 1000.0, (2e4, 8e4), 0.3),
    "frame": (S.NEO_HOOKEAN, 1000.0, (5e3, 2e4), 0.3),
    "spheres": (S.NEO_HOOKEAN, 1000.0, (5e4, 5e4), 0.35),
    "implicit": (S.NEO_HOOKEAN, 1000.0, (5e4, 5e4), 0.35),
    "dam": (S.COROTATED, 1000.0, (1.4e5, 2.8e5), 0.4),
    "snow": (S.COROTATED, 400.0, (1.4e5, 1.4e5), 0.2),
    "sand": (S.HENCKY, 2200.0, (3.537e5, 3.537e5), 0.3),
    "cube": (S.COROTATED, 1000.0, (5e3, 5e4), 0.3),
    "batch": (None, 1000.0, (1e3, 1e5), 0.3),
}
# kind -> the body as boxes in fractions of the domain (spheres: see _cells)
BOXES = {
    "block2d": ((0.375, 0.475), (0.625, 0.725)),
    "box": ((0.2, 0.12, 0.3), (0.6, 0.5, 0.7)),
    "frame": ((0.25, 0.1, 0.2), (0.7, 0.45, 0.75)),
    "dam": ((0.05, 0.05, 0.05), (0.45, 0.8, 0.95)),
    "cube": ((0.35, 0.35, 0.35), (0.65, 0.65, 0.65)),
}


def listed():
    return [
        # the 2D elastic block on the 64^2 grid, 100 substeps: the smallest scene, all launch latency (the plain
        # path is the only one in 2D)
        {"name": "block2d-64-fp64", "kind": "block2d", "precision": FP64, "grid": "64x64", "ppc": 4, "steps": 100},
        # a small 3D body with walls: a preview or a unit of a parameter study
        {"name": "box-32-fp32", "kind": "box", "precision": FP32, "grid": "32x32x32", "ppc": 8, "steps": 64},
        # the two colliding spheres, the headline workload of the repository's benchmark
        {"name": "spheres-128-fp32", "kind": "spheres", "precision": FP32, "grid": "128x128x128", "ppc": 8, "steps": 64},
        # one adaptive frame (Compute_Dt every substep) of a body in a ragged, non-cubic domain with odd counts
        {"name": "frame-97x83x101-fp32", "kind": "frame", "precision": FP32, "grid": "97x83x101", "ppc": 7, "steps": 1},
        # the dam break at the resolution people iterate at
        {"name": "dam-128-fp32", "kind": "dam", "precision": FP32, "grid": "128x128x128", "ppc": 8, "steps": 12},
        # the dam break at the benchmark's resolution: the largest scene, 36 million particles
        {"name": "dam-256-fp32", "kind": "dam", "precision": FP32, "grid": "256x256x256", "ppc": 8, "steps": 4},
        # 256 independent boxes in one handle, grids 32^3 to 96^3, both elastic models
        {"name": "batch-256-fp32", "kind": "batch", "precision": FP32, "grid": "32..96", "ppc": 6, "steps": 8,
         "scenes": 256},
        # snow (corotated, clamp plasticity fused into G2P)
        {"name": "snow-128-fp32", "kind": "snow", "precision": FP32, "grid": "128x128x128", "ppc": 8, "steps": 32},
        # sand (Hencky strain, Drucker-Prager)
        {"name": "sand-128-fp32", "kind": "sand", "precision": FP32, "grid": "128x128x128", "ppc": 8, "steps": 32},
        # the spheres on the plain path in FP64, the library's reference-precision mode
        {"name": "spheres-128-fp64", "kind": "spheres", "precision": FP64, "grid": "128x128x128", "ppc": 8, "steps": 8},
        # one backward-Euler substep (Newton, CG, line search) of the spheres in contact
        {"name": "implicit-128-fp64", "kind": "implicit", "precision": FP64, "grid": "128x128x128", "ppc": 8, "steps": 1},
        # the differentiable cube: a 64-substep rollout and its gradient
        {"name": "cube-64-grad-fp32", "kind": "cube", "precision": FP32, "grid": "64x64x64", "ppc": 8, "steps": 64},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["block2d", "box", "spheres", "spheres", "frame", "dam", "batch", "snow", "sand", "spheres64",
                       "implicit", "cube"])
    c = {"kind": kind, "precision": FP32, "ppc": rng.randint(4, 9)}
    if kind == "block2d":
        g = log_int(32, 256)
        c.update(precision=FP64, grid="%dx%d" % (g, g), steps=rng.randint(20, 120))
    elif kind == "batch":
        c.update(grid="32..96", ppc=rng.randint(4, 8), scenes=log_int(8, 256), steps=rng.randint(3, 8))
    elif kind == "frame":
        c.update(grid="%dx%dx%d" % tuple(rng.randint(40, 110) for _ in range(3)), steps=1)
    else:
        if kind == "spheres64":
            c.update(kind="spheres", precision=FP64)
            g, steps = log_int(24, 128), rng.randint(4, 10)
        elif kind == "implicit":
            c["precision"] = FP64
            g, steps = log_int(32, 128), 1
        elif kind == "cube":
            c["precision"] = rng.choice([FP32, FP32, FP64])
            g, steps = log_int(24, 72), rng.randint(16, 64)
        elif kind == "dam":
            g, steps = log_int(32, 192), rng.randint(4, 8)
        else:
            g, steps = log_int(24, 160), rng.randint(12, 64)
        c.update(grid="%dx%dx%d" % (g, g, g), steps=steps)
    return c


# ---------------------------------------------------------------------------------------------
# sizes
# ---------------------------------------------------------------------------------------------
def _counts(case):
    return [int(g) for g in case["grid"].split("x")]


def _batch_layout(case):
    """Per scene of a batch: grid side, body (in cells), model, E; the same for every seed."""
    rng = np.random.default_rng(20 + case["scenes"])
    out = []
    for _ in range(case["scenes"]):
        g = int(rng.choice([32, 48, 64, 96]))
        size = rng.uniform(0.1, 0.4, 3)
        lo = rng.uniform(0.1, 0.9 - size)
        c0 = np.ceil(lo * g).astype(int)
        c1 = np.maximum(np.floor((lo + size) * g).astype(int), c0 + 1)
        out.append((g, c0, c1, int(rng.integers(0, 2)), float(np.exp(rng.uniform(math.log(1e3), math.log(1e5))))))
    return out


def _cells(case, device):
    """The body's cells (m, d) in lexicographic order, and each cell's part (spheres: 0 or 1)."""
    counts = _counts(case)
    if case["kind"] in BOXES:
        lo, hi = BOXES[case["kind"]]
        axes = [torch.arange(math.ceil(a * n - 1e-9), math.floor(b * n + 1e-9), device=device)
                for a, b, n in zip(lo, hi, counts)]
        return torch.cartesian_prod(*axes), None
    g = counts[0]
    cells, part = [], []
    for k, cx in enumerate((0.5 - RADIUS, 0.5 + RADIUS)):
        axes = [torch.arange(max(int((c - RADIUS) * g), 0), int((c + RADIUS) * g) + 1, device=device) for c in (cx, 0.5, 0.5)]
        q = torch.cartesian_prod(*axes)
        mid = (q.double() + 0.5) / g - torch.tensor([cx, 0.5, 0.5], dtype=torch.float64, device=device)
        q = q[(mid * mid).sum(1) < RADIUS * RADIUS]
        cells.append(q)
        part.append(torch.full((q.shape[0],), k, device=device))
    return torch.cat(cells), torch.cat(part)


def _particles(case):
    if case["kind"] == "batch":
        return sum(int(np.prod(c1 - c0)) for _, c0, c1, _, _ in _batch_layout(case)) * case["ppc"]
    return _cells(case, "cpu")[0].shape[0] * case["ppc"]


def _dt(case):
    h = 1.0 / max(_counts(case)) if case["kind"] != "batch" else 1.0 / 96
    return {"block2d": 6.4e-3 * h, "box": 3.2e-3 * h, "spheres": 6.4e-3 * h, "implicit": 0.256 * h, "dam": 5e-3 * h,
            "snow": 6.4e-3 * h, "sand": 6.4e-3 * h, "cube": 6.4e-3 * h, "batch": 9.6e-3 * h, "frame": 0.0}[case["kind"]]


def _control(case):
    return S.DtControl(frame_dt=1.0 / 120, cfl=0.1, min_dt=1e-6, max_dt=5e-4)


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _smooth(gen, X, shape, waves=2.5):
    """Smooth random fields of the positions: one sine wave per entry, values in [-1, 1]."""
    d, m = X.shape[1], math.prod(shape)
    k = (torch.rand((d, m), generator=gen, device="cuda", dtype=torch.float64) - 0.5) * (4 * math.pi * waves)
    phase = torch.rand((m,), generator=gen, device="cuda", dtype=torch.float64) * (2 * math.pi)
    return torch.sin(X.double() @ k + phase).to(X.dtype).reshape(-1, *shape)


def _fill(gen, cells, part, ppc, dx, kind, density, E, nu, dtype):
    """Positions jittered in the cells, and a state in mid-simulation."""
    d = cells.shape[1]
    q = cells.repeat_interleave(ppc, 0)
    n = q.shape[0]
    X = ((q.to(dtype) + torch.rand((n, d), generator=gen, device="cuda", dtype=dtype)) * dx).to(dtype)
    del q
    bulk = torch.zeros(d, dtype=dtype, device="cuda")
    bulk[1] = -1.0
    spin = 2.0 * (torch.rand((d, d), generator=gen, device="cuda", dtype=dtype) - 0.5)
    spin = spin - spin.T
    mid = X.mean(0)
    V = bulk + (X - mid) @ spin.T + 0.2 * _smooth(gen, X, (d,))
    if part is not None:                      # the spheres close at 2 m/s each
        V[:, 0] += torch.where(part.repeat_interleave(ppc) == 0, 2.0, -2.0).to(dtype)
    strain = {"snow": 0.015, "sand": 0.006, "block2d": 0.03, "dam": 0.02}.get(kind, 0.04)
    F = torch.eye(d, dtype=dtype, device="cuda") + strain * _smooth(gen, X, (d, d))
    if kind == "sand":
        F = F * 0.995
    B = (spin + 0.5 * _smooth(gen, X, (d, d))) * (0.25 * dx * dx)
    vol = torch.full((n,), dx ** d / ppc, dtype=dtype, device="cuda")
    lo, hi = E
    Ep = lo * torch.exp(math.log(hi / lo) * torch.rand((n,), generator=gen, device="cuda", dtype=dtype))
    return {"X": X, "V": V, "F": F, "B": B, "mass": density * vol, "volume": vol, "mu": Ep / (2 * (1 + nu)),
            "lam": Ep * nu / ((1 + nu) * (1 - 2 * nu))}


def _inputs(case, seed):
    gen = torch.Generator("cuda")
    gen.manual_seed(int(seed))
    dtype = torch.float64 if case["precision"] == FP64 else torch.float32
    kind = case["kind"]
    _, density, E, nu = MATERIALS[kind]
    if kind != "batch":
        cells, part = _cells(case, "cuda")
        return _fill(gen, cells, part, case["ppc"], 1.0 / max(_counts(case)), kind, density, E, nu, dtype)
    parts = []
    for g, c0, c1, _, e in _batch_layout(case):
        cells = torch.cartesian_prod(*[torch.arange(a, b, device="cuda") for a, b in zip(c0.tolist(), c1.tolist())])
        parts.append(_fill(gen, cells, None, case["ppc"], 1.0 / g, kind, density, (e, e), nu, dtype))
    return {k: torch.cat([p[k] for p in parts]) for k in parts[0]}


def _colmajor(M):
    return M.transpose(1, 2).reshape(M.shape[0], -1).contiguous()


def _rowmajor(Mc):
    d = int(round(math.sqrt(Mc.shape[1])))
    return Mc.reshape(-1, d, d).transpose(1, 2).contiguous()


def _walls(case):
    """(axis, True: low side, type) per wall, in object order."""
    kind = case["kind"]
    if kind == "block2d":
        return [(1, True, S.STICK)]
    if kind in ("cube", "batch"):
        return []
    if kind in ("box", "dam", "frame"):
        return [(1, True, S.STICK)] + [(a, low, S.SLIP) for a in range(3) for low in (False, True) if (a, low) != (1, True)]
    return [(a, low, S.SLIP) for a in range(3) for low in (False, True)]


def _scene(case, n, counts, model):
    d = len(counts)
    dx = 1.0 / max(counts)
    dmax = [c * dx for c in counts]
    objects = []
    for axis, low, type_ in _walls(case):
        objects += S.walls(d, counts, [0.0] * d, dmax, 1 << (2 * axis + (1 if low else 0)), type_, 0.0, INSET)
    e = np.broadcast_to(np.zeros(1), (n,))
    gravity = [0.0] * d
    gravity[1] = GRAVITY
    s = S.Scene(case["kind"], d, counts, [0.0] * d, dmax, model, gravity, _dt(case), case["steps"], objects,
                np.broadcast_to(np.zeros(d), (n, d)), np.broadcast_to(np.zeros(d), (n, d)),
                np.broadcast_to(np.zeros((d, d)), (n, d, d)), np.broadcast_to(np.zeros((d, d)), (n, d, d)), e, e, e, e)
    if case["kind"] == "snow":
        s.plasticity = S.Plasticity(max_hardening=10.0)
    if case["kind"] == "sand":
        s.plasticity = S.DruckerPrager.mast_case(2)
    if case["kind"] == "implicit":
        s.implicit = S.Implicit()
    if case["kind"] == "frame":
        s.dt_control = _control(case)
    return s


# ---------------------------------------------------------------------------------------------
# the user's program
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    p = _inputs(case, seed)
    kind, n = case["kind"], p["X"].shape[0]
    fp64 = case["precision"] == FP64
    precision = D.FP64 if fp64 else D.FP32
    path = D.PATH_PLAIN if fp64 or kind == "cube" else D.PATH_FAST
    if kind == "batch":
        drv = D.MPM_BATCH([_scene(case, int(np.prod(c1 - c0)) * case["ppc"], [g] * 3, model)
                           for g, c0, c1, model, _ in _batch_layout(case)])
    else:
        drv = D.MPM_DRIVER(_scene(case, n, _counts(case), MATERIALS[kind][0]), precision=precision, path=path)
    state = {"case": case, "drv": drv, "dtype": p["X"].dtype, "dt": _dt(case)}
    if kind == "cube":
        gen = torch.Generator("cuda")
        gen.manual_seed(int(seed) + 1)
        state["inputs"] = [p[k].requires_grad_(True) for k in ("X", "V", "F", "B", "mu", "lam")]
        state["rest"] = (p["mass"], p["volume"])
        # a loss on the final positions and velocities (a target per particle)
        state["target"] = p["X"].detach() + 0.1 * _smooth(gen, p["X"].detach(), (3,))
        return state
    state["inputs"] = (p["X"], p["V"], _colmajor(p["F"]), _colmajor(p["B"]), p["mass"], p["volume"], p["mu"], p["lam"])
    if kind in ("snow", "sand"):   # the plastic state comes back in device arrays too
        keys = ("Fp", "mu", "lambda_") if kind == "snow" else ("Fp", "plastic_def", "rho_F", "vc")
        v = D.PlasticView()
        v.n, v.dtype, v.on_device = n, D.FP32, 1
        state["plastic"] = {k: torch.empty((n, 9) if k == "Fp" else n, dtype=torch.float32, device="cuda") for k in keys}
        for k, t in state["plastic"].items():
            setattr(v, k, t.data_ptr())
        state["view"] = v
    return state


def run(state):
    case, drv = state["case"], state["drv"]
    kind = case["kind"]
    drv.time = 0.0
    if kind == "cube":
        X, V, F, B, mu, lam = state["inputs"]
        mass, volume = state["rest"]
        X1, V1, F1, B1, _ = A.rollout(drv, X, V, F, B, mu, lam, mass, volume, case["steps"])
        loss = ((X1 - state["target"]) ** 2).sum() + 1e-3 * (V1 ** 2).sum()
        g = torch.autograd.grad(loss, state["inputs"])
        return {"X": X1.detach(), "V": V1.detach(), "F": F1.detach(), "B": B1.detach(), "gX": g[0], "gV": g[1],
                "gF": g[2], "gB": g[3], "gmu": g[4], "glam": g[5]}
    drv.set_particles_device(*state["inputs"])
    if kind == "frame":
        drv.simulate_frame()
    elif kind == "implicit":
        for _ in range(case["steps"]):
            drv.Advance_One_Time_Step(state["dt"])
    else:
        drv.advance(case["steps"], state["dt"])
    X, V, Fc, Bc, valid = drv.get_particles_device(state["dtype"])
    out = {"X": X, "V": V, "F": Fc, "B": Bc, "valid": valid}
    if "view" in state:
        drv._check(drv.L.mpm_get_plastic_state(drv.h, state["view"]), "mpm_get_plastic_state")
        out.update(state["plastic"])
    return out


def work(case):
    """Per substep the particle state (X, V, F, B and four constants) read once and written
    once, plus the hand-over and the read-back; operations of the weights, the stencil sums
    of P2G and G2P and the stress, per particle."""
    n, d = _particles(case), 2 if case["kind"] == "block2d" else 3
    e = 8 if case["precision"] == FP64 else 4
    state = 2 * d + 2 * d * d
    # an adaptive frame of 1/120 s takes about 25 substeps; a backward-Euler substep reads and
    # writes the state once; a rollout's backward reads each recorded state and moves its adjoint
    steps = {"frame": 25, "cube": 2 * case["steps"]}.get(case["kind"], case["steps"])
    plastic = {"snow": 2 * 11, "sand": 2 * 13}.get(case["kind"], 0)
    stencil = 3 ** d
    return {"bytes": float(n) * e * (steps * (2 * state + 4 + plastic) + 2 * state + 4),
            "flops": float(n) * steps * (stencil * (8 * (d + 1) + 8 * (2 * d + 2 * d * d) // 3) + 40 * d * d)}


def tolerance(case):
    """About four times what the path showed against FP64 (the worst output: B, a difference of
    nearly equal sums; for sand the volume correction) and against a second run of its own."""
    kind = case["kind"]
    if kind == "cube":
        return {"rel": 2e-3, "max": 0.05} if case["precision"] == FP32 else {"rel": 1e-10}
    if kind == "implicit":
        # the Newton solve ends anywhere inside its own tolerance
        return {"rel": 1e-4, "max": 0.05}
    if case["precision"] == FP64:
        return {"rel": 1e-11}
    if kind == "sand":
        return {"rel": 2e-3, "max": 0.05}
    return {"rel": 1e-3, "max": 0.05}


# ---------------------------------------------------------------------------------------------
# the substep restated in FP64
# ---------------------------------------------------------------------------------------------
def _cofactor(M):
    """det M times the inverse transpose of M."""
    if M.shape[-1] == 2:
        return torch.stack([torch.stack([M[:, 1, 1], -M[:, 1, 0]], -1), torch.stack([-M[:, 0, 1], M[:, 0, 0]], -1)], -2)
    a, b, c = M.unbind(-1)
    return torch.stack([torch.linalg.cross(b, c), torch.linalg.cross(c, a), torch.linalg.cross(a, b)], -1)


def _det(M, cof):
    return (M[:, :, 0] * cof[:, :, 0]).sum(1)


def _rotation(F):
    """The polar factor R of F = R S (Newton's iteration; Higham, Functions of Matrices, 8.3)."""
    R = F
    for _ in range(7):
        c = _cofactor(R)
        R = 0.5 * (R + c / _det(R, c)[:, None, None])
    return R


def _eigh3(M):
    """Eigenvalues (n, 3) and eigenvectors of symmetric 3x3 matrices by cyclic Jacobi rotations."""
    A_, W = M.clone(), torch.eye(3, dtype=M.dtype, device=M.device).expand_as(M).clone()
    for _ in range(7):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            apq = A_[:, p, q]
            theta = 0.5 * torch.atan2(2 * apq, A_[:, q, q] - A_[:, p, p])
            c, s = torch.cos(theta), torch.sin(theta)
            J = torch.zeros_like(A_)
            J[:, 0, 0] = J[:, 1, 1] = J[:, 2, 2] = 1
            J[:, p, p] = J[:, q, q] = c
            J[:, p, q], J[:, q, p] = s, -s
            A_ = J.transpose(1, 2) @ A_ @ J
            W = W @ J
    return torch.diagonal(A_, dim1=1, dim2=2), W


def _stress(model, F, mu, lam):
    """P(F) F^T."""
    d = F.shape[-1]
    eye = torch.eye(d, dtype=F.dtype, device=F.device)
    FT = F.transpose(1, 2)
    if model == S.HENCKY:
        s, U = _eigh3(F @ FT)
        ln = torch.log(s)
        return (U * (mu[:, None] * ln)[:, None, :]) @ U.transpose(1, 2) + (0.5 * lam * ln.sum(1))[:, None, None] * eye
    J = _det(F, _cofactor(F))
    if model == S.NEO_HOOKEAN:
        return mu[:, None, None] * (F @ FT - eye) + (lam * torch.log(J))[:, None, None] * eye
    return 2 * mu[:, None, None] * ((F - _rotation(F)) @ FT) + (lam * J * (J - 1))[:, None, None] * eye


class _Scene64:
    """One scene's grid, model and walls, and its substep."""

    chunk = 1 << 22

    def __init__(self, counts, model, walls):
        self.counts, self.model, self.walls = counts, model, walls
        self.d, self.dx = len(counts), 1.0 / max(counts)
        self.size = [c + 2 * S.GHOST for c in counts]
        self.gravity = torch.zeros(self.d, dtype=torch.float64, device="cuda")
        self.gravity[1] = GRAVITY

    def stencil(self, X):
        inv = 1.0 / self.dx
        base = torch.floor((X.detach() - self.dx) * inv)
        x = (X - (base + 0.5) * self.dx) * inv
        w = torch.stack([0.5 * (1.5 - x) ** 2, 0.75 - (x - 1) ** 2, 0.5 * (x - 0.5) ** 2])
        dw = torch.stack([(x - 1.5) * inv, -2 * (x - 1) * inv, (x - 0.5) * inv])
        first = base.long() + S.GHOST
        for k in range(3 ** self.d):
            o = [(k // 3 ** (self.d - 1 - a)) % 3 for a in range(self.d)]
            wa = [w[o[a], :, a] for a in range(self.d)]
            flat = torch.zeros_like(first[:, 0])
            for a in range(self.d):
                flat = flat * self.size[a] + (first[:, a] + o[a])
            grad = []
            for a in range(self.d):
                g = dw[o[a], :, a]
                for b in range(self.d):
                    if b != a:
                        g = g * wa[b]
                grad.append(g)
            off = torch.tensor(o, dtype=X.dtype, device=X.device)
            yield flat, math.prod(wa[1:], start=wa[0]), torch.stack(grad, 1), (base + off + 0.5) * self.dx - X

    def grid_positions(self, nodes):
        idx = []
        for a in reversed(range(self.d)):
            idx.append(nodes % self.size[a] - S.GHOST)
            nodes = nodes // self.size[a]
        return (torch.stack(idx[::-1], 1).double() + 0.5) * self.dx

    def substep(self, p, dt):
        """X, V, F, B after one substep of length dt."""
        n, d = p["X"].shape
        grid = torch.zeros((math.prod(self.size), 1 + 2 * d), dtype=torch.float64, device="cuda")
        pieces = [slice(i, min(i + self.chunk, n)) for i in range(0, n, self.chunk)]
        for s in pieces:
            X, V, F, B = p["X"][s], p["V"][s], p["F"][s], p["B"][s]
            m, vol = p["mass"][s], p["volume"][s]
            S_ = vol[:, None, None] * _stress(self.model, F, p["mu"][s], p["lam"][s])
            for flat, w, g, r in self.stencil(X):
                wm = (w * m)[:, None]
                mom = wm * (V + (4.0 / self.dx ** 2) * (B @ r[:, :, None])[:, :, 0])
                f = wm * self.gravity - (S_ @ g[:, :, None])[:, :, 0]
                grid.index_add_(0, flat, torch.cat([wm, mom, f], 1))
        nodes = torch.nonzero(grid[:, 0].detach())[:, 0]
        a = grid[nodes]
        v = (a[:, 1:1 + d] + dt * a[:, 1 + d:]) / a[:, :1]
        Z = self.grid_positions(nodes)
        for axis, low, type_ in self.walls:
            face = INSET if low else self.counts[axis] * self.dx - INSET
            inside = (Z[:, axis] <= face) if low else (Z[:, axis] >= face)
            keep = torch.ones_like(v)
            keep[:, :] = torch.where(inside, 0.0, 1.0)[:, None] if type_ == S.STICK else 1.0
            if type_ == S.SLIP:
                keep[:, axis] = torch.where(inside, 0.0, 1.0)
            v = v * keep
        vel = torch.zeros((grid.shape[0], d), dtype=torch.float64, device="cuda").index_copy(0, nodes, v)
        del grid, a, v, Z
        out = {k: [] for k in ("X", "V", "F", "B")}
        for s in pieces:
            X, F = p["X"][s], p["F"][s]
            V1, G, B1 = torch.zeros_like(X), torch.zeros_like(F), torch.zeros_like(F)
            for flat, w, g, r in self.stencil(X):
                u = vel[flat]
                wu = w[:, None] * u
                V1 = V1 + wu
                G = G + u[:, :, None] * g[:, None, :]
                B1 = B1 + wu[:, :, None] * r[:, None, :]
            out["X"].append(X + dt * V1)
            out["V"].append(V1)
            out["F"].append(F + dt * (G @ F))
            out["B"].append(B1)
        return {**p, **{k: v[0] if len(v) == 1 else torch.cat(v) for k, v in out.items()}}


def _clamp(p, pl):
    """Snow: singular values of F back into [1 - theta_c, 1 + theta_s], hardening with the plastic volume."""
    lam2, W = _eigh3(p["F"].transpose(1, 2) @ p["F"])
    s = torch.sqrt(lam2)
    t = s.clamp(1 - pl.theta_c, 1 + pl.theta_s)
    moved = (t != s).any(1)
    Fp = p["Fp"]
    e = pl.hardening_factor * (1 - s.prod(1) / t.prod(1) * _det(Fp, _cofactor(Fp)))
    c = torch.exp(e.clamp(max=pl.max_hardening)).clamp(min=1e-8)
    WT = W.transpose(1, 2)
    F1, P1 = p["F"] @ ((W * (t / s)[:, None, :]) @ WT), ((W * (s / t)[:, None, :]) @ WT) @ Fp
    pick = moved[:, None, None]
    return {**p, "F": torch.where(pick, F1, p["F"]), "Fp": torch.where(pick, P1, Fp),
            "mu": torch.where(moved, p["mu0"] * c, p["mu"]), "lam": torch.where(moved, p["lam0"] * c, p["lam"])}


def _hardening(q, pl):
    phi = math.pi / 180 * (pl.a0 + (pl.a1 * q - pl.a4) * torch.exp(-pl.a3 * q))
    return math.sqrt(2.0 / 3) * 2 * torch.sin(phi) / (3 - torch.sin(phi))


def _drucker_prager(p, pl):
    """Sand without cohesion: the Hencky strain onto the friction cone, with the volume correction."""
    lam2, W = _eigh3(p["F"].transpose(1, 2) @ p["F"])
    s = torch.sqrt(lam2)
    ln, mu, lam = torch.log(s), p["mu"], p["lam"]
    g, b = 1 / (3 * lam + 2 * mu), 1 / (2 * mu)
    st = ln + p["vc"][:, None] / 3
    k = st.sum(1)
    sh = st - k[:, None] / 3
    norm = sh.norm(dim=1)
    r = p["rho_F"] * k / g
    dg = norm + b * r
    yields = dg > 0
    tip = yields & ((norm == 0) | (k > 0))
    cone = torch.exp((k / 3)[:, None] - (r * b / norm.clamp(min=1e-300))[:, None] * sh)
    t = torch.where(tip[:, None], torch.ones_like(s), torch.where(yields[:, None], cone, s))
    q = p["plastic_def"] + torch.where(tip, ln.norm(dim=1), torch.where(yields, dg, torch.zeros_like(dg)))
    vc = torch.where(tip, p["vc"] + ln.sum(1), torch.where(yields, torch.zeros_like(dg), p["vc"]))
    WT = W.transpose(1, 2)
    pick = yields[:, None, None]
    F1, P1 = p["F"] @ ((W * (t / s)[:, None, :]) @ WT), ((W * (s / t)[:, None, :]) @ WT) @ p["Fp"]
    return {**p, "F": torch.where(pick, F1, p["F"]), "Fp": torch.where(pick, P1, p["Fp"]), "plastic_def": q,
            "rho_F": torch.where(yields, _hardening(q, pl), p["rho_F"]), "vc": vc}


def _frame_dts(scene, p, control):
    """Simulate_To_Frame: the affine CFL bound every substep, fitted to the frame's end."""
    time, end, done = 0.0, control.frame_dt, False
    while not done:
        speed = p["V"].norm(dim=1) + p["B"].flatten(1).norm(dim=1) * (6 * math.sqrt(3.0) / scene.dx)
        v = float(speed.max())
        dt = control.cfl * scene.dx / v if v > control.cfl * scene.dx / control.max_dt else control.max_dt
        dt = min(max(dt, control.min_dt), control.max_dt)
        nxt = time + dt
        if nxt + 1e-4 * dt > end:
            nxt, done = end, True
        elif nxt + dt > end:
            nxt = (time + end) / 2
        p = scene.substep(p, nxt - time)
        time = nxt
    return p


def _returned(p):
    out = {k: p[k] if k in ("X", "V") else _colmajor(p[k]) for k in ("X", "V", "F", "B")}
    out["valid"] = torch.ones(p["X"].shape[0], dtype=torch.uint8, device="cuda")
    return out


def exact(case, seed):
    kind = case["kind"]
    n = _particles(case)
    # the solve stops anywhere inside its own tolerance: no one value; and the largest take too long
    if kind == "implicit" or n * case["steps"] > 1.2e8:
        return None
    p = {k: v.double() for k, v in _inputs(case, seed).items()}
    dt = _dt(case)
    if kind == "batch":
        outs, at = [], 0
        with torch.no_grad():
            for g, c0, c1, model, _ in _batch_layout(case):
                m = int(np.prod(c1 - c0)) * case["ppc"]
                q = {k: v[at:at + m] for k, v in p.items()}
                sc = _Scene64([g] * 3, model, [])
                for _ in range(case["steps"]):
                    q = sc.substep(q, dt)
                outs.append(_returned(q))
                at += m
        return {k: torch.cat([o[k] for o in outs]) for k in outs[0]}
    sc = _Scene64(_counts(case), MATERIALS[kind][0], _walls(case))
    if kind == "cube":
        gen = torch.Generator("cuda")
        gen.manual_seed(int(seed) + 1)
        base = _inputs(case, seed)["X"]
        target = (base + 0.1 * _smooth(gen, base, (3,))).double()
        names = ("X", "V", "F", "B", "mu", "lam")
        leaves = [p[k].requires_grad_(True) for k in names]

        def step(X, V, F, B, mu, lam):
            q = sc.substep({**p, "X": X, "V": V, "F": F, "B": B, "mu": mu, "lam": lam}, dt)
            return q["X"], q["V"], q["F"], q["B"]

        x = tuple(leaves[:4])
        for _ in range(case["steps"]):
            x = checkpoint(step, *x, leaves[4], leaves[5], use_reentrant=False)
        loss = ((x[0] - target) ** 2).sum() + 1e-3 * (x[1] ** 2).sum()
        g = torch.autograd.grad(loss, leaves)
        return {"X": x[0].detach(), "V": x[1].detach(), "F": x[2].detach(), "B": x[3].detach(), "gX": g[0], "gV": g[1],
                "gF": g[2], "gB": g[3], "gmu": g[4], "glam": g[5]}
    with torch.no_grad():
        if kind == "frame":
            return _returned(_frame_dts(sc, p, _control(case)))
        pl = _scene(case, n, _counts(case), MATERIALS[kind][0]).plasticity
        if pl is not None:
            p["Fp"] = torch.eye(3, dtype=torch.float64, device="cuda").expand(n, 3, 3).clone()
            p["mu0"], p["lam0"] = p["mu"], p["lam"]
        if kind == "sand":
            p["plastic_def"] = torch.zeros_like(p["mu"])
            p["rho_F"] = _hardening(p["plastic_def"], pl)
            p["vc"] = torch.zeros_like(p["mu"])
        for _ in range(case["steps"]):
            p = sc.substep(p, dt)
            if kind == "snow":
                p = _clamp(p, pl)
            elif kind == "sand":
                p = _drucker_prager(p, pl)
    out = _returned(p)
    if kind == "snow":
        out.update({"Fp": _colmajor(p["Fp"]), "mu": p["mu"], "lambda_": p["lam"]})
    elif kind == "sand":
        out.update({"Fp": _colmajor(p["Fp"]), "plastic_def": p["plastic_def"], "rho_F": p["rho_F"], "vc": p["vc"]})
    return out
