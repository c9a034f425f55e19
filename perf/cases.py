"""The work that users of giraffe_gb300 have it do, as timed cases.

Every case goes through the public entry points (`giraffe_gb300.gpu`,
`giraffe_gb300.serve`, the C ABI below them) on structures of the families in
`giraffe_gb300.configs`, drawn from a seed.  Kinds:

  solve    gf_solve on a list of static pipe chains: one call from the
           caller's descriptors to the final nodal states
  static   a device-resident batch of static Beam_1 structures, solved from
           its initial configuration (a load study re-run on one model)
  served   static chains submitted at once to a gf_server and polled until all
           are reported
  riser    Newmark dynamics of driven Beam_1 risers
  pipe     Newmark dynamics of pressurized Pipe_1 risers pinned at the bottom,
           with Rayleigh damping
  plate    Shell_1 plates under follower pressure, Static or Dynamic, plain
           FP64 or the mixed-precision option
  sparse   gf_sparse_solve: the linear solve of a caller's own Newton loop, on
           a host CSR of a 2-D mesh's pattern
  band     gf_band_solve: the same on BandMatrix's GB storage
  mount    gf_beam_mount: tangents and internal forces of many elements on the
           reference's stored Gauss-point state
"""
import ctypes
import math

import numpy as np
import torch

from giraffe_gb300 import configs, gpu, serve
from giraffe_gb300.model import gf_model_desc

_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = gpu.Context(0)
    return _ctx


# ---------------------------------------------------------------------------
def listed():
    return [
        # one small cantilever, 20 load steps: the smallest whole solve, where
        # the latency of a Newton pass is everything
        {"name": "rollup_20", "kind": "static", "form": "rollup", "chains": 1, "n_min": 20, "n_max": 20, "steps": 20},
        # one ordinary pipe chain on its own (an odd element count)
        {"name": "chain_1x401", "kind": "static", "form": "chain", "chains": 1, "n_min": 401, "n_max": 401, "steps": 10},
        # the batched-static benchmark: 512 chains of 50-2000 elements in one call
        {"name": "solve_512_chains", "kind": "solve", "chains": 512, "n_min": 50, "n_max": 2000, "steps": 10},
        # a burst of requests to the served path
        {"name": "served_48_chains", "kind": "served", "chains": 48, "n_min": 83, "n_max": 2000, "steps": 10},
        # batched riser dynamics, ten time steps
        {"name": "risers_64", "kind": "riser", "chains": 64, "n_min": 100, "n_max": 1000, "steps": 10, "damped": False},
        # pressurized, damped Pipe_1 risers, partially constrained at the bottom
        {"name": "pipe_risers_16", "kind": "pipe", "chains": 16, "n_min": 16, "n_max": 100, "steps": 20, "damped": True},
        # the 64 x 64 x 2 benchmark plate, its first load step
        {"name": "plate_64", "kind": "plate", "plates": 1, "n_min": 64, "n_max": 64, "steps": 1, "dynamic": False,
         "mixed": False},
        # four small vibrating plates of different sizes with Rayleigh damping
        {"name": "plates_dynamic_4", "kind": "plate", "plates": 4, "n_min": 5, "n_max": 16, "steps": 4, "dynamic": True,
         "mixed": False},
        # a medium plate with the FP32 factor and FP64 refinement
        {"name": "plate_24_mixed", "kind": "plate", "plates": 1, "n_min": 24, "n_max": 24, "steps": 1, "dynamic": False,
         "mixed": True},
        # the linear solves alone, host matrix in, host solution out
        {"name": "sparse_solve_64x64", "kind": "sparse", "grid_x": 64, "grid_y": 64, "dofs": 5},
        {"name": "band_solve_12000", "kind": "band", "n": 12000, "kl": 17, "ku": 17},
        # the element entry alone
        {"name": "beam_mount_20000", "kind": "mount", "n": 20000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "static", "static", "served", "riser", "pipe", "plate", "plate", "sparse", "band", "mount"])
    if kind == "solve":
        return {"kind": kind, "chains": _log(rng, 2, 400), "n_min": _log(rng, 20, 100), "n_max": _log(rng, 200, 2000),
                "steps": rng.randint(3, 10)}
    if kind == "static":
        if rng.random() < 0.4:
            n = _log(rng, 12, 120)
            return {"kind": kind, "form": "rollup", "chains": 1, "n_min": n, "n_max": n, "steps": rng.randint(16, 24)}
        lo = _log(rng, 10, 1000)
        return {"kind": kind, "form": "chain", "chains": _log(rng, 1, 64), "n_min": lo,
                "n_max": min(2000, lo + _log(rng, 1, 1000)), "steps": rng.randint(2, 10)}
    if kind == "served":
        return {"kind": kind, "chains": rng.randint(4, 60), "n_min": _log(rng, 40, 150), "n_max": _log(rng, 300, 2000),
                "steps": rng.randint(3, 10)}
    if kind == "riser":
        return {"kind": kind, "chains": _log(rng, 1, 96), "n_min": _log(rng, 20, 150), "n_max": _log(rng, 200, 1000),
                "steps": rng.randint(3, 12), "damped": rng.random() < 0.3}
    if kind == "pipe":
        return {"kind": kind, "chains": _log(rng, 1, 32), "n_min": _log(rng, 8, 20), "n_max": _log(rng, 24, 120),
                "steps": rng.randint(5, 25), "damped": rng.random() < 0.7}
    if kind == "plate":
        mixed = rng.random() < 0.2
        one = rng.random() < 0.6
        n = _log(rng, 4, 24 if mixed else 60)
        return {"kind": kind, "plates": 1 if one else rng.randint(2, 6), "n_min": n if one else min(n, 6),
                "n_max": n if one else min(n, 20) + 6, "steps": 1 if n > 24 else rng.randint(1, 3),
                "dynamic": rng.random() < 0.4, "mixed": mixed}
    if kind == "sparse":
        return {"kind": kind, "grid_x": _log(rng, 8, 110), "grid_y": _log(rng, 8, 110), "dofs": rng.randint(3, 6)}
    if kind == "band":
        kl = _log(rng, 3, 160)
        return {"kind": kind, "n": _log(rng, 300, 16000), "kl": kl, "ku": max(1, kl + rng.randint(-2, 2))}
    return {"kind": "mount", "n": _log(rng, 30, 60000)}


# ---------------------------------------------------------------------------
# structures of a case
def _structures(case, seed):
    # the meshes are the case's, the sections and loads the seed's
    kind, steps, lo, hi = case["kind"], case["steps"], case["n_min"], max(case["n_min"], case["n_max"])
    sizes, rng = np.random.default_rng([lo, hi]), np.random.default_rng([seed, 17])
    if kind == "plate":
        out = []
        for n in sizes.integers(lo, hi + 1, case["plates"]):
            p = float(rng.uniform(5e4, 1e5))
            # the residual's round-off floor grows with the mesh: a tolerance above it
            tol = 1e-8 if n <= 24 else 1e-7 if n <= 40 else 1e-6
            if case["dynamic"]:
                out.append(configs.plate_dynamics(int(n), pressure=p, steps=steps, rayleigh_alpha=float(rng.uniform(4.0, 10.0)),
                                                  rayleigh_beta=2e-5, tol=tol))
            else:
                s = configs.square_plate(int(n), pressure=p, steps=20, tol=tol)
                s.solution.end_time = steps / 20.0
                out.append(s)
        return out
    m = case["chains"]
    if kind == "static" and case["form"] == "rollup":
        s = configs.cantilever_rollup(case["n_min"], steps=steps)
        s.loads[0].table.values[1, 5] *= float(rng.uniform(0.8, 1.0))  # rolls most of the circle
        return [s]
    if kind in ("riser", "pipe"):
        ns = sizes.integers(lo, hi + 1, m)
        De, wall = rng.uniform(0.3, 0.5, m), rng.uniform(0.02, 0.04, m)
        amp, per = rng.uniform(0.5, 2.0, m), rng.uniform(5.0, 15.0, m)
        ray = {"rayleigh_alpha": 0.2, "rayleigh_beta": 0.003} if case["damped"] else {}
        if kind == "riser":
            return [configs.riser_chain(int(n), float(d), float(w), float(a), float(p), steps=steps, **ray)
                    for n, d, w, a, p in zip(ns, De, wall, amp, per)]
        return [configs.pipe_riser(int(n), float(d), float(w), 0.25 * float(a), 0.4 * float(p), pressure=float(rng.uniform(1e7, 2e7)),
                                   steps=steps, **ray) for n, d, w, a, p in zip(ns, De, wall, amp, per)]
    ns = np.rint(np.exp(sizes.uniform(math.log(lo), math.log(hi), m))).astype(int)
    De, wall = rng.uniform(0.3, 0.5, m), rng.uniform(0.02, 0.04, m)
    F = rng.normal(0.0, 1e5, (m, 3))
    return [configs.pipe_chain(int(n), float(d), float(w), F[i], steps=steps, element_length=10.0 / int(n))
            for i, (n, d, w) in enumerate(zip(ns, De, wall))]


def _split(flat, structures):
    at, out = 0, []
    for s in structures:
        out.append(flat[at:at + s.n_nodes])
        at += s.n_nodes
    return out


# linear systems: diagonally dominant, as K + a0 M of an implicit step is
def _sparse(case, seed):
    rng = np.random.default_rng([seed, 29])
    gx, gy, d = case["grid_x"], case["grid_y"], case["dofs"]
    node = np.arange(gx * gy)
    ix, iy = node % gx, node // gx
    cols, ok = [], []
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            jx, jy = ix + dx, iy + dy
            ok.append((jx >= 0) & (jx < gx) & (jy >= 0) & (jy < gy))
            cols.append(jy * gx + jx)
    cols, ok = np.stack(cols, 1), np.stack(ok, 1)  # 9 neighbours of each node, ascending
    n = gx * gy * d
    col = (cols[:, :, None] * d + np.arange(d)).reshape(gx * gy, 9 * d)
    keep = np.repeat(ok, d, axis=1)
    col = np.repeat(col, d, axis=0)
    keep = np.repeat(keep, d, axis=0)
    val = rng.uniform(-1.0, 1.0, col.shape)
    val[~keep] = 0.0
    diag = col == np.arange(n)[:, None]
    val[diag] = 0.0
    val[diag] = 1.5 * np.abs(val).sum(axis=1)
    row_ptr = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.int32)
    return row_ptr, col[keep].astype(np.int32), val[keep], rng.normal(size=n)


def _band(case, seed):
    rng = np.random.default_rng([seed, 31])
    n, kl, ku = case["n"], case["kl"], case["ku"]
    ab = np.zeros((n, 2 * kl + ku + 1))  # column j contiguous, entry (i, j) at kl + ku + i - j
    j = np.arange(n)[:, None]
    i = j + np.arange(-ku, kl + 1)[None, :]
    v = rng.uniform(-1.0, 1.0, i.shape)
    v[(i < 0) | (i >= n)] = 0.0
    v[:, ku] = 0.0
    rows = np.zeros(n)
    for t in range(kl + ku + 1):
        inside = (i[:, t] >= 0) & (i[:, t] < n)
        rows[i[inside, t]] += np.abs(v[inside, t])
    v[:, ku] = 1.5 * np.maximum(rows, 1.0)
    ab[:, kl:] = v
    return ab, kl, ku, rng.normal(size=n)


def _elements(case, seed):
    """Beam elements along random directions, each bent and stretched a little."""
    rng = np.random.default_rng([seed, 37])
    n = case["n"]
    e3 = rng.normal(size=(n, 3))
    e3 /= np.linalg.norm(e3, axis=1, keepdims=True)
    e1 = np.cross(e3, rng.normal(size=(n, 3)))
    e1 /= np.linalg.norm(e1, axis=1, keepdims=True)
    L = rng.uniform(0.05, 1.0, (n, 1))
    x0 = rng.uniform(-5.0, 5.0, (n, 3))
    xyz = np.concatenate([x0, x0 + 0.5 * L * e3, x0 + L * e3], axis=1)
    De = rng.uniform(0.3, 0.5, n)
    Di = De - 2.0 * rng.uniform(0.02, 0.04, n)
    A, I = math.pi / 4 * (De ** 2 - Di ** 2), math.pi / 64 * (De ** 4 - Di ** 4)
    mat = np.tile([210e9, 0.3, 7850.0], (n, 1))
    sec = np.stack([A, I, I, 0 * A, 2 * I, 2 * I], axis=1)
    cs = np.concatenate([e1, e3], axis=1)
    ang = rng.normal(0.0, 0.3, (n, 2, 3))
    Q = _rotation(torch.from_numpy(ang)).numpy()
    lag = np.zeros((n, 2, 21))
    lag[..., :9] = Q.swapaxes(-1, -2).reshape(n, 2, 9)  # column-major
    lag[..., 9:12] = ang
    lag[..., 12:15] = rng.normal(0.0, 1e-2, (n, 2, 3))
    lag[..., 15:18] = rng.normal(0.0, 1e-1, (n, 2, 3))
    lag[..., 18:21] = Q[..., 2] + rng.normal(0.0, 1e-3, (n, 2, 3))
    disp = rng.normal(0.0, 1e-3, (n, 18))
    return xyz, mat, sec, cs, lag, disp


# ---------------------------------------------------------------------------
def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    if kind == "sparse":
        return {"kind": kind, "ctx": ctx, "args": _sparse(case, seed)}
    if kind == "band":
        return {"kind": kind, "ctx": ctx, "args": _band(case, seed)}
    if kind == "mount":
        return {"kind": kind, "ctx": ctx, "args": _elements(case, seed)}
    structures = _structures(case, seed)
    st = {"kind": kind, "ctx": ctx, "structures": structures}
    if kind == "served":
        st["server"] = serve.Server(ctx, hbm_budget=4 << 30, max_waves=4, max_wave_structs=64)
        return st
    st["flat"] = np.empty((sum(s.n_nodes for s in structures), 15))
    st["out"] = _split(st["flat"], structures)
    st["ptrs"] = (ctypes.POINTER(ctypes.c_double) * len(structures))(
        *[o.ctypes.data_as(ctypes.POINTER(ctypes.c_double)) for o in st["out"]])
    st["stats"] = (gpu.gf_stats * len(structures))()
    if kind == "solve":
        st["handles"] = [s.desc() for s in structures]
        st["descs"] = (gf_model_desc * len(structures))(*[h.desc for h in st["handles"]])
        st["opts"] = ctx.opts()
    else:
        precision = gpu.GF_PREC_MIXED if case.get("mixed") else gpu.GF_PREC_FP64
        st["batch"] = gpu.BatchSolver(ctx, structures, ctx.opts(precision=precision))
    return st


def run(state):
    ctx, kind = state["ctx"], state["kind"]
    if kind == "sparse":
        x, info = ctx.sparse_solve(*state["args"])
        return {"x": x, "info": info}
    if kind == "band":
        x, info = ctx.band_solve(*state["args"])
        return {"x": x, "info": info}
    if kind == "mount":
        K, f = ctx.beam_mount(*state["args"])
        return {"K": K, "f": f}
    if kind == "served":
        server = state["server"]
        for tag, s in enumerate(state["structures"]):
            server.submit(s, tag)
        done = sorted(server.drain(), key=lambda r: r.tag)
        return {"nodes": [r.final for r in done],
                "steps": np.array([[r.status, r.stats[0], r.stats[2], r.stats[3]] for r in done])}
    if kind == "solve":
        ctx.check(ctx.L.gf_solve(ctx.h, len(state["out"]), state["descs"], ctypes.byref(state["opts"]), state["ptrs"],
                                 state["stats"]), "gf_solve")
    else:
        batch = state["batch"]
        batch.reset()
        batch.run()
        ctx.check(ctx.L.gf_batch_results(batch.h, state["ptrs"], state["stats"]), "gf_batch_results")
    steps = np.array([[x.converged_steps, x.bisections, x.aborted] for x in state["stats"]])
    return {"nodes": state["flat"], "steps": steps}


# ---------------------------------------------------------------------------
def work(case):
    """Bytes: the model and its state read once, the result written once.
    Flops: per Newton pass and element the tangent, force and elimination at
    the fewest operations known for them (Beam_1: 4,000 for the tangent and
    force, 1,600 for a symmetric condensation and block elimination; Shell_1:
    60,000 for the element and 20 (m d)^3 per m x m mesh for a nested
    dissection with d DOFs per grid line and square), about five passes per
    load step and three per time step."""
    kind = case["kind"]
    if kind == "sparse":
        n, m = case["grid_x"] * case["grid_y"] * case["dofs"], math.sqrt(case["grid_x"] * case["grid_y"])
        nnz = 9 * n * case["dofs"]
        return {"bytes": 12.0 * nnz + 20.0 * n, "flops": 20.0 * (m * case["dofs"]) ** 3}
    if kind == "band":
        n, kl, ku = case["n"], case["kl"], case["ku"]
        return {"bytes": 8.0 * n * (kl + ku + 3), "flops": 2.0 * n * kl * ku + 2.0 * n * (kl + ku)}
    if kind == "mount":
        return {"bytes": case["n"] * 8.0 * (9 + 3 + 6 + 6 + 42 + 18 + 324 + 18), "flops": case["n"] * 4000.0}
    if kind == "plate":
        m = 0.5 * (case["n_min"] + case["n_max"])
        el, nodes = case["plates"] * 2 * m * m, case["plates"] * (2 * m + 1) ** 2
        passes = case["steps"] * (3 if case["dynamic"] else 5)
        return {"bytes": 8.0 * (el * 290 + nodes * 36), "flops": passes * (el * 60e3 + case["plates"] * 20.0 * (10.0 * m) ** 3)}
    lo, hi = case["n_min"], max(case["n_max"], case["n_min"])
    uniform = kind in ("riser", "pipe")
    mean = 0.5 * (lo + hi) if uniform else ((hi - lo) / math.log(hi / lo) if hi > lo else lo)
    el = case["chains"] * mean
    passes = case["steps"] * (3 if uniform else 8 if case.get("form") == "rollup" else 5)
    return {"bytes": 8.0 * el * (62 + 2 * 36), "flops": passes * el * 5600.0}


# ---------------------------------------------------------------------------
# 64-bit values without the package: the beam's strain energy in torch, its
# force and tangent as gradient and Hessian, Newton to the last bits
def _skew(v):
    z = torch.zeros_like(v[..., 0])
    return torch.stack([z, -v[..., 2], v[..., 1], v[..., 2], z, -v[..., 0], -v[..., 1], v[..., 0], z], -1).reshape(
        *v.shape[:-1], 3, 3)


def _rotation(a):
    """Rotation tensor of Rodrigues parameters a (length 2 tan(angle / 2))."""
    A = _skew(a)
    g = 4.0 / (4.0 + (a * a).sum(-1))
    return torch.eye(3, dtype=a.dtype, device=a.device) + g[..., None, None] * (A + 0.5 * A @ A)


def _gauss():
    xi = 0.577350269189626
    N = [[0.5 * x * (x - 1.0), 1.0 - x * x, 0.5 * x * (1.0 + x)] for x in (-xi, xi)]
    dN = [[x - 0.5, -2.0 * x, 0.5 + x] for x in (-xi, xi)]
    return N, dN


def _strains(d, jac, T, Q, dz, kap, e3r):
    """Increments and strains at the two Gauss points of one element (18 nodal increments d)."""
    N, dN = (torch.tensor(v, dtype=d.dtype, device=d.device) for v in _gauss())
    d = d.reshape(3, 2, 3)
    u1 = (dN / jac) @ d[:, 0] @ T.T
    a, a1 = N @ d[:, 1] @ T.T, (dN / jac) @ d[:, 1] @ T.T
    g = (4.0 / (4.0 + (a * a).sum(-1)))[:, None]
    z = u1 + dz
    eta = torch.einsum("gij,gi->gj", _rotation(a) @ Q, z) - e3r
    k = torch.einsum("gij,gi->gj", Q, g * (a1 - 0.5 * torch.linalg.cross(a, a1))) + kap
    return a, z, eta, k


def _energy(d, jac, T, Q, dz, kap, e3r, D):
    _, _, eta, k = _strains(d, jac, T, Q, dz, kap, e3r)
    return 0.5 * jac * ((D[:3] * eta * eta).sum() + (D[3:] * k * k).sum())


def _chunked(f, args, size=4096):
    return torch.cat([f(*[a[i:i + size] for a in args]) for i in range(0, len(args[0]), size)])


def _tensors(*arrays):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return [torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev) for a in arrays]


def _frame(x0, x2, cs, E, nu, A, I1, I2, It):
    e1, e3 = cs[:, :3], cs[:, 3:]
    T = np.stack([e1, np.cross(e3, e1), e3], axis=1)
    T = T / np.linalg.norm(T, axis=2, keepdims=True)
    axis = x2 - x0
    length = np.linalg.norm(axis, axis=1)
    G = E / (2 * (1 + nu))
    return length / 2, T, np.einsum("nij,nj->ni", T, axis / length[:, None]), np.stack(
        [G * A, G * A, E * A, E * I1, E * I2, G * It], axis=1)


def _exact_mount(case, seed):
    xyz, mat, sec, cs, lag, disp = _elements(case, seed)
    jac, T, e3r, D = _frame(xyz[:, :3], xyz[:, 6:], cs, mat[:, 0], mat[:, 1], sec[:, 0], sec[:, 1], sec[:, 2], sec[:, 4])
    Q = lag[..., :9].reshape(-1, 2, 3, 3).swapaxes(-1, -2)
    args = _tensors(disp, jac, T, Q, lag[..., 18:21], lag[..., 12:15], e3r, D)
    f = _chunked(torch.func.vmap(torch.func.grad(_energy)), args)
    K = _chunked(torch.func.vmap(torch.func.hessian(_energy)), args)
    return {"K": K.cpu().numpy(), "f": f.cpu().numpy()}


def _exact_static(case, seed):
    """The load steps of one clamped static chain, each by Newton's method with a dense solve."""
    s = _structures(case, seed)[0]
    nodes = np.array(s.nodes)
    ne, nn = (len(nodes) - 1) // 2, len(nodes)
    E, nu, _ = s.materials[0]
    A, I1, I2, _, It, _ = s.sections[0]
    cs = np.tile(np.array(s.cs[0], dtype=float).reshape(-1), (ne, 1))
    jac, T, e3r, D = _frame(nodes[0:-1:2], nodes[2::2], cs, E, nu, *(np.full(ne, v) for v in (A, I1, I2, It)))
    jac, T, e3r, D, x = _tensors(jac, T, e3r, D, nodes)
    dev = x.device
    Q = torch.eye(3, dtype=torch.float64, device=dev).repeat(ne, 2, 1, 1)
    dz = torch.zeros(ne, 2, 3, dtype=torch.float64, device=dev)
    dz[..., 2] = 1.0
    kap = torch.zeros_like(dz)
    rot = torch.zeros_like(x)
    load = torch.as_tensor(s.loads[0].table.values[1], dtype=torch.float64, device=dev)
    dof = (torch.arange(3, device=dev) + 2 * torch.arange(ne, device=dev)[:, None])[:, :, None] * 6 + torch.arange(6, device=dev)
    dof = dof.reshape(ne, 18)
    rows, cols = dof[:, :, None].expand(ne, 18, 18).reshape(-1), dof[:, None, :].expand(ne, 18, 18).reshape(-1)
    tip = 6 * (nn - 1)
    for step in range(case["steps"]):
        F = load * (step + 1) / case["steps"]
        d, last = torch.zeros(6 * nn, dtype=torch.float64, device=dev), math.inf
        for _ in range(40):
            args = (d[dof], jac, T, Q, dz, kap, e3r, D)
            f = torch.func.vmap(torch.func.grad(_energy))(*args)
            K = torch.func.vmap(torch.func.hessian(_energy))(*args)
            R = torch.zeros_like(d).index_add_(0, dof.reshape(-1), -f.reshape(-1))
            M = torch.zeros(6 * nn, 6 * nn, dtype=torch.float64, device=dev).index_put_((rows, cols), K.reshape(-1), True)
            a = d[tip + 3:]
            g = 4.0 / (4.0 + a @ a)
            m = g * (F[3:] - 0.5 * torch.linalg.cross(a, F[3:]))
            R[tip:tip + 3] += F[:3]
            R[tip + 3:] += m
            M[tip + 3:, tip + 3:] -= -0.5 * g * torch.outer(m, a) + 0.5 * g * _skew(F[3:])
            x1 = torch.linalg.solve(M[6:, 6:], R[6:])
            d[6:] += x1
            size = x1.abs().max().item()
            if size < 1e-9 and size > 0.25 * last or size < 1e-16:
                break
            last = size
        a, z, eta, k = torch.func.vmap(_strains)(d[dof], jac, T, Q, dz, kap, e3r)
        Q, dz, kap = _rotation(a) @ Q, z, k
        d = d.reshape(nn, 6)
        x = x + d[:, :3]
        rot = (4.0 / (4.0 - (d[:, 3:] * rot).sum(-1)))[:, None] * (d[:, 3:] + rot + 0.5 * torch.linalg.cross(d[:, 3:], rot))
    out = torch.cat([x, rot, _rotation(rot).reshape(nn, 9)], 1)
    return {"nodes": out.cpu().numpy(), "steps": None}


def _jacobi(rows, cols, vals, b):
    """x with A x = b for a diagonally dominant A, by Jacobi sweeps to the last bits."""
    rows, cols = (torch.as_tensor(v, dtype=torch.int64) for v in (rows, cols))
    vals, b = torch.as_tensor(vals), torch.as_tensor(b)
    A = torch.sparse_coo_tensor(torch.stack([rows, cols]), vals, (len(b), len(b))).coalesce().to_sparse_csr()
    dg = torch.zeros_like(b).index_add_(0, rows[rows == cols], vals[rows == cols])
    x = b / dg
    for _ in range(130):
        x = x + (b - A @ x) / dg
    return x.numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "mount":
        return _exact_mount(case, seed)
    if kind == "static" and case["chains"] == 1 and case["n_min"] == case["n_max"] and case["n_min"] <= 420:
        return _exact_static(case, seed)
    if kind == "sparse":
        rp, ci, v, b = _sparse(case, seed)
        return {"x": _jacobi(np.repeat(np.arange(len(b)), np.diff(rp)), ci, v, b), "info": None}
    if kind == "band":
        ab, kl, ku, b = _band(case, seed)
        n = len(b)
        j = np.repeat(np.arange(n), kl + ku + 1)
        i = j + np.tile(np.arange(-ku, kl + 1), n)
        ok = (i >= 0) & (i < n)
        return {"x": _jacobi(i[ok], j[ok], ab[:, kl:].reshape(-1)[ok], b), "info": None}
    return None
