"""The work that users of the package have it do, as measurable cases.

listed() names the cases, draw(rng) gives another one of the same ranges,
prepare(case, seed) makes what a user's program holds before the call, run(state)
is one pass through the public entry points, work(case) the bytes and operations
a pass cannot do without, and exact(case, seed) the result in 64 bits from plain
torch.  A case's "task" is one of

  product       one mobility block times a vector (blobs of shells above a wall or in free space)
  force_torque  [U; W] from forces and torques on every blob
  forces        the right-hand side of a time step: blob forces reduced to body forces and torques
  solve         one rigid-body mobility problem: configuration, preconditioner, GMRES to 1e-8
  step          one Brownian (Euler-Maruyama) step: Lanczos noise, solve, update
  batch         many independent uneven suspensions: Lanczos draws and the solves in lockstep
"""
import math

import numpy as np
import torch

from rigidmultiblobswall_gb300 import forces, integrator, mobility, nearfield, suspensions
from rigidmultiblobswall_gb300.rigid import RigidSystem

ETA = 1.0
KINDS = ("uf", "ut", "wf", "wt")


def listed():
    return [
        # the smallest calls: the reference's drop-in on numpy arrays, 12 bodies (the smoke test's size)
        {"name": "uf_fp64_host_504", "task": "product", "kind": "uf", "mode": "fp64", "bodies": 12, "blobs": 42,
         "extra": 0, "domain": "wall", "periodic": False, "host": True},
        # plain FP64 M.F of 2,048 free blobs (the benchmark's first workload)
        {"name": "uf_fp64_2048", "task": "product", "kind": "uf", "mode": "fp64", "bodies": 0, "blobs": 0,
         "extra": 2048, "domain": "wall", "periodic": False, "host": False},
        # the headline product: 256 shells of 42 blobs, FP64-accurate double-float
        {"name": "uf_df64_10752", "task": "product", "kind": "uf", "mode": "df64", "bodies": 256, "blobs": 42,
         "extra": 0, "domain": "wall", "periodic": False, "host": False},
        # the largest suspension of the benchmark: 4,096 shells
        {"name": "uf_df64_172032", "task": "product", "kind": "uf", "mode": "df64", "bodies": 4096, "blobs": 42,
         "extra": 0, "domain": "wall", "periodic": False, "host": False},
        # a rotational block at an odd size (shells and free blobs together)
        {"name": "wf_df64_5003", "task": "product", "kind": "wf", "mode": "df64", "bodies": 119, "blobs": 42,
         "extra": 5, "domain": "wall", "periodic": False, "host": False},
        # a pseudo-periodic suspension in FP64 (periodic_length of the reference's input files)
        {"name": "uf_fp64_periodic_1500", "task": "product", "kind": "uf", "mode": "fp64", "bodies": 125,
         "blobs": 12, "extra": 0, "domain": "wall", "periodic": True, "host": False},
        # the grand mobility of the lubrication solver: [U; W] of 8,064 blobs
        {"name": "force_torque_df64_8064", "task": "force_torque", "mode": "df64", "bodies": 192, "blobs": 42,
         "extra": 0},
        # the force callback of every time step: 1,024 shells of 12 blobs, the example's Debye length
        {"name": "forces_12288", "task": "forces", "bodies": 1024, "blobs": 12, "debye": 0.1, "periodic": False},
        # the rigid mobility problem in FP64, 256 shells
        {"name": "solve_fp64_256", "task": "solve", "mode": "fp64", "bodies": 256, "blobs": 42, "near": False},
        # the same in mixed precision with the near-field preconditioner
        {"name": "solve_mixed_256", "task": "solve", "mode": "mixed", "bodies": 256, "blobs": 42, "near": True},
        # one Brownian step of 1,024 shells of 12 blobs
        {"name": "step_mixed_1024x12", "task": "step", "mode": "mixed", "bodies": 1024, "blobs": 12},
        # uneven independent suspensions: 16 Lanczos draws and the solve of each
        {"name": "batch_mixed_16", "task": "batch", "mode": "mixed", "suspensions": 16, "low": 16, "high": 512,
         "draws": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    task = rng.choice(["product"] * 5 + ["force_torque", "forces", "solve", "solve", "step", "batch"])
    if task == "product":
        mode = rng.choice(["fp64", "df64", "df64", "mixed"])
        blobs = rng.choice([12, 42])
        periodic = rng.random() < 0.15
        n = _log_int(rng, 100, 5000 if periodic else {"fp64": 30000, "df64": 120000, "mixed": 120000}[mode])
        return {"task": task, "kind": rng.choice(KINDS + ("uf", "uf")), "mode": mode, "bodies": n // blobs,
                "blobs": blobs, "extra": n % blobs,
                "domain": "wall" if periodic else rng.choice(["wall", "wall", "wall", "free"]),
                "periodic": periodic, "host": rng.random() < 0.25}
    if task == "force_torque":
        blobs = rng.choice([12, 42])
        n = _log_int(rng, 200, 16000)
        return {"task": task, "mode": rng.choice(["fp64", "df64"]), "bodies": n // blobs, "blobs": blobs,
                "extra": n % blobs}
    if task == "forces":
        blobs = rng.choice([12, 42])
        return {"task": task, "bodies": _log_int(rng, 16, 1000), "blobs": blobs,
                "debye": round(math.exp(rng.uniform(math.log(0.05), math.log(0.5))), 3),
                "periodic": rng.random() < 0.3}
    if task == "solve":
        mode = rng.choice(["fp64", "df64", "mixed"])
        blobs = rng.choice([12, 42])
        return {"task": task, "mode": mode, "bodies": _log_int(rng, 8, 256 if mode == "fp64" else 700),
                "blobs": blobs, "near": mode == "mixed" and rng.random() < 0.5}
    if task == "step":
        mode = rng.choice(["mixed", "df64"])
        return {"task": task, "mode": mode, "bodies": _log_int(rng, 16, 1500), "blobs": 12}
    return {"task": task, "mode": "mixed", "suspensions": rng.randint(2, 16), "low": 8,
            "high": rng.randint(20, 400), "draws": rng.randint(1, 16)}


# ---------------------------------------------------------------------------
# inputs
def _shell(blobs):
    """(blob positions in the body frame, blob radius, body radius) of the two structures."""
    if blobs == 12:
        return suspensions.icosahedron(1.0), 0.4, 1.0
    shell = suspensions.icosphere_42(suspensions.R42)
    return shell, suspensions.blob_radius_of(shell), suspensions.R42


def _bodies(rng, n, blobs, dense=False):
    """Centres, quaternions and blob positions of n shells that do not touch, in random order: a square
    lattice with jitter (60R x 60R per 256 bodies, heights 1.2R to 5R; dense: area fraction 0.3, 1.1R to 3R)."""
    shell, a, R = _shell(blobs)
    cell = R * (math.sqrt(math.pi / 0.3) if dense else 3.75)
    side = int(math.ceil(math.sqrt(n)))
    site = rng.permutation(side * side)[:n]
    jitter = 0.5 * (cell - 2 * (R + a))
    x = np.empty((n, 3))
    x[:, 0] = cell * (site % side + 0.5) + rng.uniform(-jitter, jitter, n)
    x[:, 1] = cell * (site // side + 0.5) + rng.uniform(-jitter, jitter, n)
    x[:, 2] = rng.uniform(1.1 * R, 3.0 * R, n) if dense else rng.uniform(1.2 * R, 5.0 * R, n)
    q = suspensions.random_quaternions(rng, n)
    return x, q, suspensions.blob_positions(x, q, shell) if n else np.zeros((0, 3)), a, cell * side


def _blobs(case, rng):
    """(r, a, side of the box): the blobs of the case's bodies, then its free blobs (a = 0.5 and the box of
    the 2,048-blob workload without bodies)."""
    n = case["extra"]
    if not case["bodies"]:
        a, side = 0.5, 32.0 * math.sqrt(n / 2048.0)
        r = np.zeros((0, 3))
    else:
        _, _, r, a, side = _bodies(rng, case["bodies"], case["blobs"], dense=case["bodies"] > 2000)
    free = np.empty((n, 3))
    free[:, :2] = rng.uniform(0.0, max(side, 1.0), (n, 2))
    free[:, 2] = rng.uniform(1.5 * a, 10 * a, n)
    return np.concatenate([r, free]), a, max(side, 1.0)


def _product_inputs(case, seed):
    rng = np.random.default_rng(seed)
    r, a, side = _blobs(case, rng)
    if case.get("domain") == "free":
        r = r + np.array([0.0, 0.0, 2.0])
    L = np.array([side, side, 0.0]) if case.get("periodic") else np.zeros(3)
    return r, rng.standard_normal(r.shape), rng.standard_normal(r.shape), a, L


def _batch_counts(case):
    """The same counts for every seed, so that passes over several states do the same work."""
    rng = np.random.default_rng(case["suspensions"] * 1000 + case["high"])
    return [int(c) for c in rng.integers(case["low"], case["high"] + 1, size=case["suspensions"])]


def _batch_inputs(case, seed):
    rng = np.random.default_rng(seed)
    parts = [_bodies(rng, c, 42) for c in _batch_counts(case)]
    return np.concatenate([p[0] for p in parts]), np.concatenate([p[2] for p in parts]), parts[0][3], rng


FORCE_KW = dict(g=1.0, repulsion_strength_wall=0.3, repulsion_strength=0.3)


def _force_kw(case, a, side):
    return dict(FORCE_KW, debye_length_wall=case["debye"] * a, debye_length=case["debye"] * a,
                periodic_length=np.array([side, side, 0.0]) if case["periodic"] else np.zeros(3))


def _gpu(x):
    return torch.as_tensor(x, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    task = case["task"]
    s = {"case": case}
    if task in ("product", "force_torque"):
        r, f, t, a, L = _product_inputs(case, seed)
        if case.get("host"):
            s.update(r=r, f=f, a=a, L=L)
        else:
            s.update(r=_gpu(r), f=_gpu(f), t=_gpu(t), a=a, L=L)
        return s
    if task == "batch":
        x, r, a, rng = _batch_inputs(case, seed)
        counts = _batch_counts(case)
        sys_ = RigidSystem([42] * sum(counts), ETA, a)
        sys_.set_suspensions(counts)
        s.update(sys=sys_, r=_gpu(r), x=_gpu(x), rhs=_gpu(_rhs(rng, len(x), len(r))),
                 z=_gpu(rng.standard_normal((case["draws"], 3 * len(r)))))
        return s
    rng = np.random.default_rng(seed)
    x, q, r, a, side = _bodies(rng, case["bodies"], case["blobs"])
    s.update(sys=RigidSystem([case["blobs"]] * case["bodies"], ETA, a), r=_gpu(r), x=_gpu(x), a=a)
    if task == "forces":
        s["kw"] = _force_kw(case, a, side)
        s["sys"].set_configuration(s["r"], s["x"])
    elif task == "solve":
        s["rhs"] = _gpu(_rhs(rng, len(x), len(r)))
    else:
        st = integrator.BrownianStepper(s["sys"], x, q, np.tile(_shell(case["blobs"])[0], (len(x), 1)), kT=1.0,
                                        mode=case["mode"])
        s.update(stepper=st, q=_gpu(q), ft=_gpu(_forces(rng, len(x))), z=_gpu(rng.standard_normal(3 * len(r))))
    return s


def _forces(rng, bodies):
    """Gravity on every body and a torque on each, as a driven suspension has them."""
    ft = np.zeros((bodies, 6))
    ft[:, 2] = -1.0
    ft[:, 3:] = 0.1 * rng.standard_normal((bodies, 3))
    return ft


def _rhs(rng, bodies, blobs):
    return np.concatenate([np.zeros(3 * blobs), -_forces(rng, bodies).reshape(-1)])


# ---------------------------------------------------------------------------
# one pass
PRODUCTS = {
    ("wall", "uf"): mobility.single_wall_mobility_trans_times_force_pycuda,
    ("wall", "ut"): mobility.single_wall_mobility_trans_times_torque_pycuda,
    ("wall", "wf"): mobility.single_wall_mobility_rot_times_force_pycuda,
    ("wall", "wt"): mobility.single_wall_mobility_rot_times_torque_pycuda,
    ("free", "uf"): mobility.no_wall_mobility_trans_times_force_pycuda,
    ("free", "ut"): mobility.no_wall_mobility_trans_times_torque_pycuda,
    ("free", "wf"): mobility.no_wall_mobility_rot_times_force_pycuda,
    ("free", "wt"): mobility.no_wall_mobility_rot_times_torque_pycuda,
}


def run(s):
    case = s["case"]
    task = case["task"]
    if task == "product":
        return PRODUCTS[case["domain"], case["kind"]](s["r"], s["f"], ETA, s["a"], periodic_length=s["L"],
                                                      mode=case["mode"])
    if task == "force_torque":
        U, W = mobility.wall_force_torque(s["r"], s["f"], s["t"], ETA, s["a"], mode=case["mode"])
        return [U, W]
    if task == "forces":
        return forces.force_torque_calculator_sort_by_bodies(s["sys"], s["r"], blob_radius=s["a"], **s["kw"])
    if task == "step":
        st = s["stepper"]
        st.x, st.q = s["x"], s["q"]  # every pass steps from the same configuration
        out = st.step(1e-3, s["ft"], z=s["z"])
        return [out["velocities"], out["noise"], st.x, st.q]
    sys_ = s["sys"]
    sys_.set_configuration(s["r"], s["x"])
    if task == "solve":
        sys_.build_pc(mode=case["mode"])
        if case["near"]:
            nearfield.attach_exact(sys_, 6.0 * _shell(case["blobs"])[2])
        return [sys_.solve(s["rhs"], tol=1e-8, mode=case["mode"])[0]]
    sys_.build_pc(stochastic=True, mode=case["mode"])
    noise, _ = sys_.lanczos_batched(s["z"], factor=math.sqrt(2.0 / 1e-3), tol=1e-3, mode=case["mode"])
    sol = sys_.solve_batched(s["rhs"], tol=1e-8, mode=case["mode"])[0]
    return [sol, noise]


# ---------------------------------------------------------------------------
# what a pass cannot do without
#: Operations of an unordered pair, both ways: two reciprocal roots, the block's coefficients, two 3 x 3 products.
PAIR = {"uf": 150.0, "ut": 120.0, "wf": 120.0, "wt": 110.0}
#: Operator applications of a solve to 1e-8 and of a Lanczos draw to 1e-3 on these suspensions.
SOLVE, LANCZOS = 10, 6


def work(case):
    task = case["task"]
    if task == "batch":
        n = [42.0 * c for c in _batch_counts(case)]
        pairs = sum(0.5 * k * k for k in n)
        return {"bytes": 8.0 * 3 * sum(n) * (4 + 2 * case["draws"]),
                "flops": pairs * (PAIR["uf"] * SOLVE + (110.0 + 36.0 * case["draws"]) * LANCZOS)}
    n = float(case["bodies"] * case["blobs"] + case.get("extra", 0))
    pairs = 0.5 * n * n * (9 if case.get("periodic") and task == "product" else 1)
    if task == "product":
        return {"bytes": 72.0 * n, "flops": pairs * (PAIR[case["kind"]] if case["domain"] == "wall" else 60.0)}
    if task == "force_torque":
        return {"bytes": 120.0 * n, "flops": pairs * 400.0}
    if task == "forces":
        return {"bytes": 24.0 * n + 48.0 * case["bodies"], "flops": pairs * 20.0}
    products = SOLVE + (LANCZOS if task == "step" else 0)
    return {"bytes": 8.0 * (3 * n * 3 + 12 * case["bodies"]) + 72.0 * n * case["blobs"],
            "flops": pairs * PAIR["uf"] * products}


# ---------------------------------------------------------------------------
# the same in 64 bits with plain torch
def _rpy(kind, d, r2, v):
    """Rotne-Prager-Yamakawa block times v; d = (x, y, z) differences over a, r2 their squared length."""
    x, y, z = d
    r = r2.sqrt()
    if kind in ("ut", "wf"):
        c = torch.where(r < 2, 0.5 * (1 - 0.375 * r), 1 / (r2 * r))
        return [c * (v[1] * z - v[2] * y), c * (v[2] * x - v[0] * z), c * (y * v[0] - x * v[1])]
    if kind == "uf":
        A = torch.where(r <= 2, 4 / 3 * (1 - 9 * r / 32), 1 / r + 2 / (3 * r2 * r))
        B = torch.where(r <= 2, 1 / (8 * r), 1 / (r2 * r) - 2 / (r2 * r2 * r))
    else:
        A = torch.where(r < 2, 1 - 27 * r / 32 + 5 * r2 * r / 64, -0.5 / (r2 * r))
        B = torch.where(r < 2, 9 / (32 * r) - 3 * r / 64, 1.5 / (r2 * r2 * r))
    g = B * (x * v[0] + y * v[1] + z * v[2])
    return [A * v[0] + g * x, A * v[1] + g * y, A * v[2] + g * z]


def _wall(kind, d, Rz, hi, hj, v):
    """Swan-Brady wall correction of the block times v (lengths over a)."""
    x, y = d[0], d[1]
    R = (x * x + y * y + Rz * Rz).sqrt()
    ex, ey, ez = x / R, y / R, Rz / R
    E = ez * ez
    s = 1 / R
    if kind == "uf":
        hh = hi * hj * s * s
        f1 = -((1 + 2 * hh) * s + 2 / 3 * ((1 - 3 * E) * s ** 3 - (1 - 5 * E) * s ** 5))
        f2 = -((1 - 6 * hh) * s - 2 * (1 - 5 * E) * s ** 3 + 10 / 3 * (1 - 7 * E) * s ** 5)
        f3 = 2 / 3 * (3 * hj * s ** 2 - 18 * hh * ez * s + ez * (10 * (2 - 7 * E) * s ** 5 - 6 * (1 - 5 * E) * s ** 3))
        f4 = 2 / 3 * (3 * hj * s ** 2 - 10 * ez * s ** 5)
        f5 = -4 / 3 * (3 * (hj * hj + E) * s ** 3 + (2 - 15 * E) * s ** 5)
        ev = ex * v[0] + ey * v[1] + ez * v[2]
        g = f2 * ev + f3 * v[2]
        return [f1 * v[0] + g * ex, f1 * v[1] + g * ey, f1 * v[2] + g * ez + f4 * ev + f5 * v[2]]
    if kind == "wt":
        f1, f2, f3 = 0.5 * (1 - 6 * E) * s ** 3, -1.5 * s ** 3, 3 * s ** 3
        ev = ex * v[0] + ey * v[1] + ez * v[2]
        c = ey * v[0] - ex * v[1]
        return [f1 * v[0] + f2 * ev * ex + f3 * c * ey, f1 * v[1] + f2 * ev * ey - f3 * c * ex,
                f1 * v[2] - f2 * ev * ez]
    h = hi if kind == "ut" else hj
    f1 = s ** 2
    f2 = 2 * (6 * h * ez * s ** 3 + (1 - 10 * E) * s ** 4)
    f3 = -2 * (3 * h * s ** 3 - 5 * ez * s ** 4)
    f4 = -2 * (h * s ** 3 - ez * s ** 4)
    p, g = f1 * ez + f4, f1 + f2 + f3 * ez
    if kind == "ut":
        c = ey * v[0] - ex * v[1]
        return [f3 * c * ex + f1 * ey * v[2] + p * v[1], f3 * c * ey - f1 * ex * v[2] - p * v[0], -g * c]
    w = f3 * (ex * v[0] + ey * v[1]) + g * v[2]
    return [w * ey - p * v[1], p * v[0] - w * ex, -f1 * (ey * v[0] - ex * v[1])]


def _self(kind, h, v, wall):
    zero = torch.zeros_like(h)
    i = 1 / h
    if kind == "uf":
        xx = 4 / 3 - ((9 * i - 2 * i ** 3 + i ** 5) / 12 if wall else zero)
        zz = 4 / 3 - ((9 * i - 4 * i ** 3 + i ** 5) / 6 if wall else zero)
        return [xx * v[0], xx * v[1], zz * v[2]]
    if kind == "wt":
        xx = 1 - (5 / 16 * i ** 3 if wall else zero)
        return [xx * v[0], xx * v[1], (1 - (i ** 3 / 8 if wall else zero)) * v[2]]
    c = (i ** 4 / 8 if wall else zero) * (1 if kind == "ut" else -1)
    return [c * v[1], -c * v[0], zero]


def _nearest(d, L):
    return d - torch.trunc(d / L + 0.5 * torch.sign(d)) * L if L > 0 else d


def _exact_product(kind, r, v, a, L, wall):
    r, v = _gpu(r), _gpu(v)
    n = r.shape[0]
    z = r[:, 2]
    b = torch.where(z < a, z / a, torch.ones_like(z)) if wall else torch.ones_like(z)
    h = (z.clamp(min=a) if wall else z) / a
    x, y, w = r[:, 0] / a, r[:, 1] / a, (b[:, None] * v).t()
    L = [float(k) / a for k in L]
    out = torch.empty_like(r)
    rows = max(1, min(n, 40_000_000 // max(1, n)))
    for i0 in range(0, n, rows):
        i = slice(i0, min(n, i0 + rows))
        same = torch.arange(n, device=r.device)[None, :] == torch.arange(n, device=r.device)[i, None]
        hi, hj = h[i, None], h[None, :]
        d = [_nearest(x[i, None] - x[None, :], L[0]), _nearest(y[i, None] - y[None, :], L[1]),
             _nearest(hi - hj, L[2])]
        vj = [w[c][None, :] for c in range(3)]
        total = [torch.zeros(same.shape[0], dtype=torch.float64, device=r.device) for _ in range(3)]
        for bx in (-1, 0, 1) if L[0] > 0 else (0,):
            for by in (-1, 0, 1) if L[1] > 0 else (0,):
                e = [d[0] + bx * L[0], d[1] + by * L[1], d[2]]
                r2 = e[0] ** 2 + e[1] ** 2 + e[2] ** 2
                skip = same if bx == 0 and by == 0 else torch.zeros_like(same)
                u = _rpy(kind, e, torch.where(skip, torch.ones_like(r2), r2), vj)
                if wall:
                    u = [p + q for p, q in zip(u, _wall(kind, e, hi + hj, hi, hj, vj))]
                for c in range(3):
                    total[c] += torch.where(skip, torch.zeros_like(u[c]), u[c]).sum(1)
        mine = _self(kind, h[i], [w[c][i] for c in range(3)], wall)
        for c in range(3):
            out[i, c] = b[i] * (total[c] + mine[c])
    return out.reshape(-1) / (8 * math.pi * ETA * a ** {"uf": 1, "wt": 3}.get(kind, 2))


def _exact_solve(x, r, a, rhs, blobs):
    """The saddle-point system solved densely."""
    n, nb = len(r), len(x)
    M = torch.empty(3 * n, 3 * n, dtype=torch.float64, device="cuda")
    R, X = _gpu(r), _gpu(x)
    z = R[:, 2]
    b = torch.where(z < a, z / a, torch.ones_like(z))
    h = z.clamp(min=a) / a
    d = [(R[:, None, 0] - R[None, :, 0]) / a, (R[:, None, 1] - R[None, :, 1]) / a, h[:, None] - h[None, :]]
    same = torch.eye(n, dtype=torch.bool, device="cuda")
    r2 = torch.where(same, torch.ones_like(d[0]), d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
    one, zero = torch.ones_like(r2), torch.zeros_like(r2)
    for c in range(3):
        v = [one if k == c else zero for k in range(3)]
        u = _rpy("uf", d, r2, v)
        w = _wall("uf", d, h[:, None] + h[None, :], h[:, None], h[None, :], v)
        s = _self("uf", h, [torch.ones_like(h) if k == c else torch.zeros_like(h) for k in range(3)], True)
        for k in range(3):
            blk = torch.where(same, torch.diag(s[k]), u[k] + w[k])
            M[k::3, c::3] = blk * b[:, None] * b[None, :] / (8 * math.pi * ETA * a)
    K = torch.zeros(3 * n, 6 * nb, dtype=torch.float64, device="cuda")
    body = torch.arange(n, device="cuda") // blobs
    e = R - X[body]
    i = torch.arange(n, device="cuda")
    for k in range(3):
        K[3 * i + k, 6 * body + k] = 1.0
        p, q = (k + 1) % 3, (k + 2) % 3  # (w x e)_k = w_p e_q - w_q e_p
        K[3 * i + k, 6 * body + 3 + p] = e[:, q]
        K[3 * i + k, 6 * body + 3 + q] = -e[:, p]
    A = torch.cat([torch.cat([M, -K], 1), torch.cat([-K.t(), torch.zeros(6 * nb, 6 * nb, dtype=torch.float64,
                                                                         device="cuda")], 1)])
    return torch.linalg.solve(A, _gpu(rhs))


def _exact_forces(case, x, r, a, kw):
    r, x = _gpu(r), _gpu(x)
    n, nb = r.shape[0], case["blobs"]
    eb, b, L = kw["repulsion_strength"] / kw["debye_length"], kw["debye_length"], kw["periodic_length"]
    f = torch.zeros_like(r)
    rows = max(1, min(n, 40_000_000 // n))
    for i0 in range(0, n, rows):
        i = slice(i0, min(n, i0 + rows))
        d = [_nearest(r[None, :, k] - r[i, None, k], float(L[k])) for k in range(3)]
        rn = (d[0] ** 2 + d[1] ** 2 + d[2] ** 2).sqrt()
        g = torch.where(rn > 2 * a, torch.exp(-(rn - 2 * a) / b), torch.ones_like(rn))
        m = torch.where(rn > 0, eb * g / rn.clamp(min=1e-300), torch.zeros_like(rn))
        for k in range(3):
            f[i, k] = -(m * d[k]).sum(1)
    ew, bw, z = kw["repulsion_strength_wall"], kw["debye_length_wall"], r[:, 2]
    f[:, 2] += -kw["g"] + ew / bw * torch.where(z > a, torch.exp(-(z - a) / bw), torch.ones_like(z))
    f = f.reshape(-1, nb, 3)
    arm = r.reshape(-1, nb, 3) - x[:, None, :]
    return torch.stack([f.sum(1), torch.linalg.cross(arm, f).sum(1)], 1).reshape(-1, 3)


def exact(case, seed):
    task = case["task"]
    if task in ("product", "force_torque"):
        r, f, t, a, L = _product_inputs(case, seed)
        wall = case.get("domain", "wall") == "wall"
        if task == "product":
            return _exact_product(case["kind"], r, f, a, L, wall)
        return [_exact_product("uf", r, f, a, L, wall) + _exact_product("ut", r, t, a, L, wall),
                _exact_product("wf", r, f, a, L, wall) + _exact_product("wt", r, t, a, L, wall)]
    if task in ("step", "batch"):
        return None  # noise of a Lanczos run to 1e-3: no closed form to compare with
    rng = np.random.default_rng(seed)
    x, _, r, a, side = _bodies(rng, case["bodies"], case["blobs"])
    if task == "forces":
        return _exact_forces(case, x, r, a, _force_kw(case, a, side))
    if 3 * len(r) + 6 * len(x) > 12000:
        return None
    return [_exact_solve(x, r, a, _rhs(rng, len(x), len(r)), case["blobs"])]
