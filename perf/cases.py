"""What a user of the solver has it do, as cases that can be timed and checked.

Every case is a dict of plain values; its "kind" picks the public entry point:

  solve     Plan.set_sources / set_targets (or set_targets_to_sources) / solve: new points on a kept plan
  facade    FastMultipoleSolver's own call sequence on host arrays (tree, multipoles, locals, calcB)
  batch     many independent coils in one plan (set_coils), one solve
  grad      the autograd wrapper: B = biot_savart(...), then the gradients of 1/2 sum |B|^2 for xyz and J
  replay    new strengths on a fixed tree: update_sources + graph_launch of the captured graph
  direct    calcBioSavartLaplace, the direct sum
  treecode  MultipoleSolver.calcB at query points, on multipoles already computed
  seam      the translation seam: translateAllGPU and translateAllGPUMatrixCuBLAS on one set of expansions

The sources are solid tori (tensor-product quadratures, Gauss-Legendre in the radius, as
bachelors_b200.geometry.torus makes them, generated on the GPU), turned about their axis and shifted by the seed, with a current
that varies by a few per cent from point to point; targets are uniform in a box around the torus, a regular
grid, or the source points themselves.
"""
import math

import numpy as np
import torch

from bachelors_b200 import FastMultipoleSolver, MultipoleSolver, Plan, calcBioSavartLaplace, kernels
from bachelors_b200.autograd import biot_savart

PI = 3.14159265359         # the solver's literals
MU0 = 1.2566370614e-6
DEV = "cuda:0"


def listed():
    return [
        # the smallest call: one coarse coil and a few hundred observation points (the order and leaf size are
        # the plan's defaults); launches and host waits count here
        {"name": "solve_2k", "kind": "solve", "n_phi": 27, "n_theta": 9, "n_rho": 8, "m": 1001, "targets": "box",
         "azimuthal": False, "order": 10, "leaf": 64, "precision": "fp32", "m2l": "simt", "want": 1},
        # the reference program's run: its mesh's 38,400 quadratures, azimuthal current, default leaf
        # capacities 1000 / 100, host arrays, one phase after the other
        {"name": "facade_38k", "kind": "facade", "n_phi": 60, "n_theta": 32, "n_rho": 20, "m": 4001,
         "azimuthal": True, "order": 10, "precision": "fp32", "m2l": "simt"},
        # double precision on a regular grid of observation points
        {"name": "grid_fp64", "kind": "solve", "n_phi": 128, "n_theta": 32, "n_rho": 16, "m": 32768, "targets": "grid",
         "azimuthal": True, "order": 10, "leaf": 32, "precision": "fp64", "m2l": "simt", "want": 1},
        # a million points and targets on the CUDA cores, the plan's default M2L
        {"name": "torus_1m_simt", "kind": "solve", "n_phi": 256, "n_theta": 64, "n_rho": 64, "m": 1048576,
         "targets": "box", "azimuthal": False, "order": 12, "leaf": 64, "precision": "fp32", "m2l": "simt", "want": 1},
        # the same size with odd counts, the tensor-core M2L, field and potential together
        {"name": "torus_1m_bf16x3", "kind": "solve", "n_phi": 251, "n_theta": 65, "n_rho": 63, "m": 1000003,
         "targets": "box", "azimuthal": False, "order": 12, "leaf": 64, "precision": "fp32", "m2l": "bf16x3",
         "want": 3},
        # the largest: 2^24 points, field at the points themselves, order 16
        {"name": "self_16m_p16", "kind": "solve", "n_phi": 512, "n_theta": 128, "n_rho": 256, "m": 0, "targets": "self",
         "azimuthal": False, "order": 16, "leaf": 64, "precision": "fp32", "m2l": "bf16x3", "want": 1},
        # 256 coils of uneven size in one plan
        {"name": "batch_256", "kind": "batch", "coils": 256, "lo": 4096, "hi": 262144, "m": 16384, "order": 8,
         "leaf": 32, "precision": "fp32", "m2l": "bf16x3"},
        # one step of a coil optimisation: field, then gradients for positions and currents
        {"name": "grad_1m", "kind": "grad", "n_phi": 256, "n_theta": 64, "n_rho": 64, "m": 262144, "order": 12,
         "leaf": 64, "precision": "fp32", "m2l": "bf16x3"},
        # currents change, points stay: the captured graph with new strengths each time
        {"name": "replay_256k", "kind": "replay", "n_phi": 128, "n_theta": 32, "n_rho": 64, "m": 0, "targets": "self",
         "order": 10, "leaf": 64, "precision": "fp32", "m2l": "bf16x3"},
        # the direct sum as a check or for small problems (double precision is its default)
        {"name": "direct_38k", "kind": "direct", "n_phi": 60, "n_theta": 32, "n_rho": 20, "m": 10000,
         "azimuthal": True, "precision": "fp64"},
        # point queries against a kept source tree
        {"name": "treecode_64k", "kind": "treecode", "n_phi": 128, "n_theta": 32, "n_rho": 64, "m": 65536, "order": 10,
         "leaf": 1000, "precision": "fp32", "m2l": "simt"},
        # the translation seam at a level's worth of children
        {"name": "seam_64k", "kind": "seam", "count": 65536, "order": 10, "precision": "fp32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _torus_counts(rng, lo, hi):
    """n_phi, n_theta, n_rho with a product log-uniform in [lo, hi], each dimension odd or even."""
    n = _log(rng, lo, hi)
    n_rho = max(3, min(256, int(round(n ** (1 / 3) * rng.uniform(0.4, 0.9)))))
    n_theta = max(5, min(128, int(round(n ** (1 / 3) * rng.uniform(0.5, 1.0)))))
    n_phi = max(7, min(hi, n) // (n_rho * n_theta))
    return {"n_phi": n_phi, "n_theta": n_theta, "n_rho": n_rho}


def draw(rng):
    """Another case of the same ranges."""
    kind = rng.choice(["solve", "solve", "solve", "solve", "facade", "batch", "grad", "replay", "direct", "treecode",
                       "seam"])
    if kind == "solve":
        how = rng.choice(["simt", "bf16x3", "bf16x3", "bf16x6", "tf32", "fp64"])
        fp64 = how == "fp64"
        top_n, top_m, top_p = {"simt": (1 << 20, 1 << 20, 12), "fp64": (100000, 50000, 12)}.get(how, (1 << 22, 1 << 21, 16))
        targets = rng.choice(["box", "box", "grid", "self"])
        return {"kind": "solve", **_torus_counts(rng, 1500, top_n), "targets": targets,
                "m": 0 if targets == "self" else _log(rng, 500, top_m) if targets == "box"
                else _log(rng, 8, round(top_m ** (1 / 3))) ** 3,
                "azimuthal": rng.random() < 0.3, "order": rng.randint(4, top_p), "leaf": rng.choice([32, 50, 64, 100]),
                "precision": "fp64" if fp64 else "fp32", "m2l": "simt" if fp64 else how,
                "want": rng.choice([1, 1, 2, 3])}
    if kind == "facade":
        return {"kind": "facade", **_torus_counts(rng, 2000, 200000), "m": _log(rng, 100, 20000), "azimuthal": True,
                "order": rng.randint(4, 12), "precision": rng.choice(["fp32", "fp32", "fp64"]), "m2l": "simt"}
    if kind == "batch":
        lo = _log(rng, 512, 4096)
        return {"kind": "batch", "coils": _log(rng, 4, 256), "lo": lo, "hi": lo * rng.randint(2, 32),
                "m": _log(rng, 500, 16384), "order": rng.randint(4, 10), "leaf": rng.choice([32, 64]),
                "precision": "fp32", "m2l": rng.choice(["bf16x3", "bf16x3", "simt"])}
    if kind == "grad":
        return {"kind": "grad", **_torus_counts(rng, 2000, 1 << 20), "m": _log(rng, 500, 1 << 18),
                "order": rng.randint(4, 12), "leaf": rng.choice([32, 64]), "precision": "fp32",
                "m2l": rng.choice(["bf16x3", "simt"])}
    if kind == "replay":
        return {"kind": "replay", **_torus_counts(rng, 5000, 1 << 21), "m": 0, "targets": "self",
                "order": rng.randint(6, 14), "leaf": 64, "precision": "fp32", "m2l": "bf16x3"}
    if kind == "direct":
        return {"kind": "direct", **_torus_counts(rng, 1000, 100000), "m": _log(rng, 100, 30000),
                "azimuthal": rng.random() < 0.5, "precision": rng.choice(["fp64", "fp64", "fp32"])}
    if kind == "treecode":
        return {"kind": "treecode", **_torus_counts(rng, 4000, 1 << 18), "m": _log(rng, 1, 65536),
                "order": rng.randint(4, 12), "leaf": rng.choice([100, 1000]),
                "precision": rng.choice(["fp32", "fp32", "fp64"]), "m2l": "simt"}
    return {"kind": "seam", "count": _log(rng, 64, 131072), "order": rng.randint(4, 12),
            "precision": rng.choice(["fp32", "fp32", "fp64"])}


# ------------------------------------------------------------------------------------------ inputs

def _dtype(case):
    return torch.float64 if case["precision"] == "fp64" else torch.float32


def _generator(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 1000003 + salt)
    return g


def _torus(n_phi, n_theta, n_rho, major, minor, centre, axis, turn, magnitude, dtype, g, spread=0.05):
    """Tensor-product torus quadrature on the GPU: xyz [N, 3], w [N], poloidal J [N, 3] (values made in 64 bits)."""
    f64 = dict(dtype=torch.float64, device=DEV)
    f = 2 * math.pi * (torch.arange(n_phi, **f64) + 0.5) / n_phi + turn
    t = 2 * math.pi * (torch.arange(n_theta, **f64) + 0.5) / n_theta
    xg, wg = np.polynomial.legendre.leggauss(n_rho)
    rho = torch.tensor(0.5 * minor * (xg + 1.0), **f64)
    wr = torch.tensor(0.5 * minor * wg, **f64)
    f, t, rho, wr = f[:, None, None], t[None, :, None], rho[None, None, :], wr[None, None, :]
    ring = major + rho * torch.cos(t)
    one = torch.ones((n_phi, n_theta, n_rho), **f64)
    local = torch.stack([ring * torch.cos(f), ring * torch.sin(f), one * (rho * torch.sin(t))], dim=-1).reshape(-1, 3)
    w = (one * ((2 * math.pi / n_phi) * (2 * math.pi / n_theta) * wr * rho * ring)).reshape(-1)
    tangent = torch.stack([one * (-torch.sin(t) * torch.cos(f)), one * (-torch.sin(t) * torch.sin(f)),
                           one * torch.cos(t)], dim=-1).reshape(-1, 3)
    a = np.asarray(axis, dtype=np.float64) / np.linalg.norm(axis)
    v, c = np.cross([0.0, 0.0, 1.0], a), float(a[2])
    vx = np.array([[0, -v[2], v[1]], [v[2], 0, -v[0]], [-v[1], v[0], 0]])
    R = torch.tensor(np.eye(3) + vx + vx @ vx / (1.0 + c), **f64)
    local = local @ R.T + torch.tensor(centre, **f64)
    size = magnitude * (1 + spread * torch.randn((w.shape[0], 1), generator=g, **f64))
    return local.to(dtype), w.to(dtype), ((tangent @ R.T) * size).to(dtype)


def _coil(case, seed):
    """The case's torus (R = 2, a = 0.5, axis z): xyz, w, J (None with the azimuthal current)."""
    r = np.random.default_rng(seed)
    xyz, w, J = _torus(case["n_phi"], case["n_theta"], case["n_rho"], 2.0, 0.5, r.uniform(-0.01, 0.01, 3), (0, 0, 1),
                       r.uniform(0, 1), 1.0, _dtype(case), _generator(seed))
    if case.get("azimuthal"):
        w = w * (1 + 0.05 * torch.rand(w.shape, generator=_generator(seed, 3), device=DEV, dtype=w.dtype))
        J = None
    return xyz, w, J


def _targets(case, seed):
    m, dt = case["m"], _dtype(case)
    if case.get("targets") == "grid":
        k = int(round(m ** (1 / 3)))
        g = torch.linspace(-3, 3, k, dtype=torch.float64, device=DEV)
        return torch.stack(torch.meshgrid(g, g, g, indexing="ij"), dim=-1).reshape(-1, 3).to(dt)
    return (torch.rand((m, 3), generator=_generator(seed, 1), dtype=torch.float64, device=DEV) * 6 - 3).to(dt)


def _batch(case, seed):
    """Uneven tori with random poses, and uniform targets around each."""
    r, g, dt = np.random.default_rng(seed), _generator(seed), _dtype(case)
    xs, ws, Js, ts, so, to = [], [], [], [], [0], [0]
    for _ in range(case["coils"]):
        R, a = r.uniform(1, 3), r.uniform(0.2, 0.6)
        axis, c = r.normal(size=3), r.uniform(-10, 10, 3)
        count = math.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"])))
        x, w, J = _torus(max(4, int(round(count / 64))), 16, 4, R, a, c, axis, 0.0, r.uniform(0.5, 2), dt, g, 0.0)
        t = torch.tensor(c, device=DEV) + 3 * R * (torch.rand((case["m"], 3), generator=g, dtype=torch.float64, device=DEV) - 0.5)
        xs.append(x); ws.append(w); Js.append(J); ts.append(t.to(dt))
        so.append(so[-1] + len(w)); to.append(to[-1] + len(t))
    return torch.cat(xs), torch.cat(ws), torch.cat(Js), torch.cat(ts), np.array(so, np.int64), np.array(to, np.int64)


def _seam(case, seed):
    """Scaled harmonics and expansions of moderate size, and one dense translation matrix."""
    L, g, dt = (case["order"] + 1) ** 2, _generator(seed), _dtype(case)
    degree = torch.tensor([l for l in range(case["order"] + 1) for _ in range(2 * l + 1)], device=DEV)
    fall = torch.pow(0.7, degree.to(torch.float64))
    a = (torch.randn((case["count"], L), generator=g, dtype=torch.float64, device=DEV) * fall).to(dt)
    b = (torch.randn((case["count"], L, 3), generator=g, dtype=torch.float64, device=DEV) * fall[:, None]).to(dt)
    return a, b, (torch.randn((L, L), generator=g, dtype=torch.float64, device=DEV) / math.sqrt(L)).to(dt)


# ------------------------------------------------------------------------------------------ calls

def _warm_plan(case, xyz, w, J, targets):
    """A plan that has solved a little problem before, as a program keeps it: its operators are built."""
    plan = Plan(order=case["order"], leaf_capacity=case["leaf"], precision=case["precision"], m2l=case["m2l"])
    k = max(1, len(w) // 2048)
    plan.set_sources(xyz[::k], w[::k], None if J is None else J[::k])
    plan.set_targets((xyz if targets is None else targets)[:1024])
    plan.solve(1.0, case.get("want", 1))
    return plan


def prepare(case, seed):
    kind = case["kind"]
    if kind == "seam":
        a, b, T = _seam(case, seed)
        return {"kind": kind, "a": a, "b": b, "T": T}
    if kind == "batch":
        xyz, w, J, tgt, so, to = _batch(case, seed)
        return {"kind": kind, "in": (xyz, w, J, tgt), "so": so, "to": to,
                "plan": _warm_plan(case, xyz[so[0]:so[1]], w[so[0]:so[1]], J[so[0]:so[1]], tgt[:to[1]])}
    xyz, w, J = _coil(case, seed)
    tgt = None if case.get("targets") == "self" else _targets(case, seed)
    if kind == "solve":
        return {"kind": kind, "in": (xyz, w, J, tgt), "want": case["want"],
                "plan": _warm_plan(case, xyz, w, J, tgt)}
    if kind == "facade":
        host = [None if v is None else v.cpu().numpy() for v in (xyz, w, J, tgt)]
        return {"kind": kind, "solver": FastMultipoleSolver(tuple(host[:3]), host[3], order=case["order"],
                                                            precision=case["precision"], m2l=case["m2l"])}
    if kind == "grad":
        plan = _warm_plan(case, xyz, w, J, tgt)
        return {"kind": kind, "in": (xyz.requires_grad_(), w, J.requires_grad_(), tgt), "plan": plan}
    if kind == "replay":
        plan = Plan(order=case["order"], leaf_capacity=case["leaf"], precision=case["precision"], m2l=case["m2l"])
        plan.set_sources(xyz, w, torch.flip(J, [0]))
        plan.set_targets_to_sources()
        plan.solve(1.0, 1)
        plan.graph_capture(1)
        return {"kind": kind, "in": (w, J), "plan": plan}
    if kind == "treecode":
        solver = MultipoleSolver((xyz, w, J), quadratureOctreeLeafCapacity=case["leaf"], order=case["order"],
                                 precision=case["precision"], m2l=case["m2l"])
        solver.calcMultipoleExpansionsAtLeaves()
        return {"kind": kind, "solver": solver, "points": tgt}
    return {"kind": kind, "in": (xyz, w, J, tgt), "precision": case["precision"]}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        plan, (xyz, w, J, tgt) = state["plan"], state["in"]
        plan.set_sources(xyz, w, J)
        if tgt is None:
            plan.set_targets_to_sources()
        else:
            plan.set_targets(tgt)
        return [v for v in plan.solve(1.0, state["want"]) if v is not None]
    if kind == "facade":
        s = state["solver"]
        s.calcMultipoleExpansionsAtLeaves()
        s.calclMultipoleExpansions()
        s.calcLocalMultipoleExpansions()
        return s.calcB(1.0)
    if kind == "batch":
        plan, (xyz, w, J, tgt) = state["plan"], state["in"]
        plan.set_sources(xyz, w, J)
        plan.set_targets(tgt)
        plan.set_coils(state["so"], state["to"])
        return plan.solve(1.0, 1)[0]
    if kind == "grad":
        xyz, w, J, tgt = state["in"]
        B = biot_savart(xyz, w, J, tgt, plan=state["plan"])
        dx, dJ = torch.autograd.grad(0.5 * (B * B).sum(), (xyz, J))
        return [B.detach(), dx, dJ]
    if kind == "replay":
        state["plan"].update_sources(*state["in"])
        return state["plan"].graph_launch(1.0)[0]
    if kind == "treecode":
        return state["solver"].calcB(1.0, state["points"])
    if kind == "direct":
        xyz, w, J, tgt = state["in"]
        return calcBioSavartLaplace(1.0, tgt, (xyz, w, J), precision=state["precision"])
    a, b, T = state["a"], state["b"], state["T"]
    return [kernels.translateAllGPU(a, b), kernels.translateAllGPUMatrixCuBLAS(a, T)]


# ------------------------------------------------------------------------------------------ what a pass needs

def work(case):
    """Inputs read once and results written once; the arithmetic of the method (harmonics at every point, the
    translations of a full octree, the direct neighbours) or of the direct sum, counted as multiply and add."""
    kind, es = case["kind"], 8 if case["precision"] == "fp64" else 4
    if kind == "seam":
        p, c = case["order"], case["count"]
        L = (p + 1) ** 2
        terms = sum(min(lam, l - lam) * 2 + 1 if m == 0 else sum((abs(m - mu) <= l - lam) + (abs(m + mu) <= l - lam)
                    for mu in range(-lam, lam + 1)) for l in range(p + 1) for m in range(l + 1) for lam in range(l + 1))
        return {"bytes": es * (c * L * 8 + L * L), "flops": float(c) * (terms * 24 + 2 * L * L)}
    if kind == "batch":
        n = case["coils"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        m = case["coils"] * case["m"]
    else:
        n = case["n_phi"] * case["n_theta"] * case["n_rho"]
        m = n if case.get("targets") == "self" else case["m"]
    io = es * (3 * m + 3 * m * (2 if case.get("want") == 3 else 1) + n * (4 if case.get("azimuthal") else 7))
    if kind == "direct":
        return {"bytes": io, "flops": 20.0 * n * m}
    p = case["order"]
    L, leaf = (p + 1) ** 2, case.get("leaf", 100)
    kept = 2 * p if case["precision"] == "fp64" else p + 8
    entries = sum((2 * l + 1) * (2 * k + 1) for l in range(p + 1) for k in range(p + 1) if l + k <= kept)
    up, down = 12.0 * L * n, 12.0 * L * m
    if kind == "treecode":
        return {"bytes": es * (6 * m + 4 * n), "flops": m * (14.0 * L * 30 + 20.0 * 8 * leaf)}
    boxes = min(n, m) / (0.4 * leaf) * 8 / 7
    m2l = boxes * 60 * 6.0 * entries
    near = 20.0 * m * min(n, 12 * leaf)
    total = up + down + m2l + near
    if kind == "grad":
        return {"bytes": io + es * 6 * n, "flops": 2 * total}
    return {"bytes": io if kind != "replay" else es * (4 * n + 3 * m), "flops": total}


# ------------------------------------------------------------------------------------------ the same in 64 bits

PAIRS = 1 << 40            # direct sums up to this size take some seconds; larger cases have no exact value


def _azimuthal(x):
    v = torch.stack([-x[:, 1], x[:, 0], torch.zeros_like(x[:, 0])], dim=1)
    return v / v.norm(dim=1, keepdim=True).clamp_min(1e-300)


def _powers(x, q, *powers):
    """r^-k of every pair for the k asked, 0 where the points coincide."""
    d = x[:, 0, None] - q[None, :, 0]
    r2 = d * d
    for k in (1, 2):
        torch.sub(x[:, k, None], q[None, :, k], out=d)
        r2.addcmul_(d, d)
    r2.masked_fill_(r2 == 0, math.inf)
    r = r2.rsqrt_()
    return [r if k == 1 else r ** k for k in powers]


def _field(x, q, s, want=1):
    """B and / or A at x from sources q of strength s = w J, in chunks of targets."""
    B, A = torch.empty_like(x), torch.empty_like(x)
    cols = torch.cat([s, torch.linalg.cross(s, q)], dim=1)
    step = max(1, (1 << 22) // max(1, len(q)))
    if len(q) > 1 << 22:
        raise ValueError("more sources than one chunk holds")
    for i in range(0, len(x), step):
        y = x[i:i + step]
        if want & 1:
            k3, = _powers(y, q, 3)
            f = k3 @ cols
            B[i:i + step] = torch.linalg.cross(f[:, :3], y) - f[:, 3:]
        if want & 2:
            k1, = _powers(y, q, 1)
            A[i:i + step] = k1 @ s
    return [MU0 / (4 * PI) * B] * (want & 1) + [A / (4 * PI)] * (want >> 1)


def _gradients(q, w, J, x, g):
    """dLoss/dq and dLoss/dJ for dLoss/dB = g at x."""
    dq, dJ = torch.empty_like(q), torch.empty_like(q)
    c = MU0 / (4 * PI)
    gx = torch.linalg.cross(g, x)
    # moments of the targets for the second term: 1, x_i and x_i x_j times S = J x g, by columns
    second = torch.cat([g] + [x[:, i:i + 1] * g for i in range(3)] +
                       [x[:, i:i + 1] * x[:, j:j + 1] * g for i in range(3) for j in range(3)], dim=1)
    first = torch.cat([g, gx], dim=1)
    step = max(1, (1 << 22) // max(1, len(x)))
    for i in range(0, len(q), step):
        y, Ji, wi = q[i:i + step], J[i:i + step], w[i:i + step, None]
        k3, k5 = _powers(y, x, 3, 5)
        f = k3 @ first                       # sum g / r^3 and sum (g x t) / r^3
        C = torch.linalg.cross(f[:, :3], y) - f[:, 3:]
        dJ[i:i + step] = c * wi * C
        t = (k5 @ second).reshape(len(y), 13, 3)
        S = torch.linalg.cross(Ji[:, None, :].expand(-1, 13, -1), t, dim=2)   # J x (moment of g)
        m0, m1, m2 = S[:, 0], S[:, 1:4], S[:, 4:].reshape(len(y), 3, 3, 3)
        # sum d_i (d . S), d = y - t
        dS = torch.einsum("ni,nj,nj->ni", y, y, m0) - torch.einsum("ni,njj->ni", y, m1) \
            - torch.einsum("nik,nk->ni", m1, y) + torch.einsum("nijj->ni", m2)
        dq[i:i + step] = c * wi * (torch.linalg.cross(Ji, f[:, :3]) - 3 * dS)
    return dq, dJ


def _translate(p, a, b):
    """The translation of real-form expansions b [N, L, 3] by harmonics a [N, L], term by term."""
    s = math.sqrt(0.5)
    k = lambda l, m: l * l + l + m  # noqa: E731
    out = torch.zeros_like(b)

    def view(h, l, m):
        if m == 0:
            return torch.complex(h[:, k(l, 0)], torch.zeros_like(h[:, k(l, 0)]))
        re, im = h[:, k(l, abs(m))] * s, h[:, k(l, -abs(m))] * s
        return torch.complex(re, im if m > 0 else -im)

    A = {(l, m): view(a, l, m)[:, None] for l in range(p + 1) for m in range(-l, l + 1)}
    Bc = {(l, m): view(b, l, m) for l in range(p + 1) for m in range(-l, l + 1)}
    sign = lambda m, mu: -1.0 if ((abs(m - mu) + abs(mu) - abs(m)) >> 1) & 1 else 1.0  # noqa: E731
    for l in range(p + 1):
        for m in range(l + 1):
            if m == 0:
                for lam in range(l + 1):
                    for mu in range(-min(lam, l - lam), min(lam, l - lam) + 1):
                        out[:, k(l, 0)] += sign(0, mu) * b[:, k(lam, mu)] * a[:, k(l - lam, mu), None]
                continue
            plus, minus = torch.zeros_like(Bc[0, 0]), torch.zeros_like(Bc[0, 0])
            for lam in range(l + 1):
                for mu in range(-lam, lam + 1):
                    if abs(m - mu) <= l - lam:
                        plus += sign(m, mu) * (Bc[lam, mu] * A[l - lam, m - mu])
                    if abs(m + mu) <= l - lam:
                        minus += sign(-m, mu) * (Bc[lam, mu] * A[l - lam, -m - mu])
            out[:, k(l, m)] = s * (plus.real + minus.real)
            out[:, k(l, -m)] = s * (plus.imag - minus.imag)
    return out


def exact(case, seed):
    kind = case["kind"]
    f64 = lambda v: v.to(torch.float64)  # noqa: E731
    if kind == "seam":
        a, b, T = (f64(v) for v in _seam(case, seed))
        return [_translate(case["order"], a, b), a @ T]
    if kind == "batch":
        xyz, w, J, tgt, so, to = _batch(case, seed)
        out = [_field(f64(tgt[to[c]:to[c + 1]]), f64(xyz[so[c]:so[c + 1]]),
                      f64(J[so[c]:so[c + 1]]) * f64(w[so[c]:so[c + 1], None]))[0] for c in range(case["coils"])]
        return torch.cat(out)
    xyz, w, J = _coil(case, seed)
    tgt = xyz if case.get("targets") == "self" else _targets(case, seed)
    if len(xyz) * len(tgt) > PAIRS or len(xyz) > 1 << 22:
        return None
    x, q, w = f64(tgt), f64(xyz), f64(w)
    J = _azimuthal(q) if J is None else f64(J)
    if kind == "grad":
        B, = _field(x, q, w[:, None] * J)
        return [B, *_gradients(q, w, J, x, B)]
    out = _field(x, q, w[:, None] * J, case.get("want", 1))
    return out if kind == "solve" else out[0]
