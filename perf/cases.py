"""Measured cases: what a user of this engine has it do, through its public entry points.

The geometries, frequencies and incidences follow the engine's own workloads (2D TE / TM disks,
3D cubes, k0 L / 2 pi from 5 to 25, up to 64 incident fields, ring and sphere detectors, the
driver's image grid, the batched 2D sweep).  Every case is one of seven operations:

  solve         the fields at the scatterers for given incident fields (the class API's solve)
  transmission  the driver's loop body for one frequency: incident fields, solve, detector fields
  image         the total field on the driver's pixel grid for several incidences in one call
  mean_dos      the mean density of states over measurement points
  ldos          the local density of states over batches of points
  resident      another block of incident fields against a factorisation kept on the device
  sweep         a replay of a captured batch of disorder realisations

The mixed-precision cases ask for a relative residual of 1e-11, so that their fields are
determined well beyond the accuracy at which complex128 results are compared.
"""
import math

import numpy as np
import torch

from magreete_gb300 import Transmission2D_scalar, Transmission2D_vector, Transmission3D_scalar, Transmission3D_vector
from magreete_gb300 import batch, engine, fields, selfterm, workloads

SOLVERS = {"2d_vector": Transmission2D_vector, "2d_scalar": Transmission2D_scalar,
           "3d_vector": Transmission3D_vector, "3d_scalar": Transmission3D_scalar}
COMPONENTS = {"2d_vector": 2, "2d_scalar": 1, "3d_vector": 3, "3d_scalar": 1}
TOL = 1e-11


def _case(op, kind, precision, N, R, kL, device="cuda", points=0, batches=1):
    return {"op": op, "kind": kind, "precision": precision, "N": N, "R": R, "kL": kL, "device": device,
            "points": points, "batches": batches}


def listed():
    cases = [
        # the smallest call: a TM sample of a few hundred scatterers and one incident field, all latency
        ("solve_2d_scalar_fp64_small", _case("solve", "2d_scalar", "fp64", 150, 1, 6.0)),
        # the 2D TE transmission configuration in the default precision
        ("solve_2d_vector_fp64", _case("solve", "2d_vector", "fp64", 1000, 64, 20.0)),
        # a mid-sized 3D dyadic system in the default precision, ragged order and field count
        ("solve_3d_vector_fp64", _case("solve", "3d_vector", "fp64", 1999, 37, 10.0)),
        # the driver's frequency loop on host tensors, default precision
        ("transmission_2d_vector_fp64_host", _case("transmission", "2d_vector", "fp64", 500, 32, 12.0, "cpu", 360)),
        # the driver's full-field image (301 x 301 pixels), five angles in one call
        ("image_2d_vector_fp64", _case("image", "2d_vector", "fp64", 1000, 5, 20.0, points=301 * 301)),
        # the mean DOS configuration: one frequency, 1000 measurement points
        ("mean_dos_2d_vector_fp64", _case("mean_dos", "2d_vector", "fp64", 1000, 0, 20.0, points=1000)),
        # LDOS map of a 3D sample in batches, mixed precision
        ("ldos_3d_vector_mixed", _case("ldos", "3d_vector", "mixed", 1250, 0, 8.0, points=300, batches=3)),
        # the 2D TE transmission configuration in the mixed precision
        ("solve_2d_vector_mixed", _case("solve", "2d_vector", "mixed", 1000, 64, 20.0)),
        # the 3D transmission configuration, a whole frequency on device tensors
        ("transmission_3d_vector_mixed", _case("transmission", "3d_vector", "mixed", 4000, 64, 10.0, points=1024)),
        # a large request of the serving mix
        ("solve_3d_vector_mixed_large", _case("solve", "3d_vector", "mixed", 12001, 33, 15.0)),
        # a re-query: new incident fields against the factorisation of a 3D scalar sample
        ("resident_3d_scalar_mixed", _case("resident", "3d_scalar", "mixed", 6000, 64, 20.0)),
        # disorder realisations of uneven size in one captured graph
        ("sweep_2d_vector", _case("sweep", "2d_vector", "mixed", 1200, 16, 15.0, batches=12)),
    ]
    return [dict(c, name=name) for name, c in cases]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: an operation, then sizes spread over its range."""
    op = rng.choice(["solve"] * 4 + ["transmission"] * 2 + ["image", "mean_dos", "ldos", "resident", "sweep"])
    kind = rng.choice(list(COMPONENTS))
    precision = rng.choice(["fp64", "mixed"])
    d = COMPONENTS[kind]
    kL = round(rng.uniform(5.0, 25.0), 2)
    R = rng.randint(1, 64)
    device = rng.choice(["cuda", "cpu"])
    if op == "solve":
        n = _log_int(rng, 100, 6000) if precision == "fp64" else _log_int(rng, 500, 36000)
        return _case(op, kind, precision, min(16000, max(16, n // d)), R, kL)
    if op == "transmission":
        n = _log_int(rng, 100, 5000) if precision == "fp64" else _log_int(rng, 500, 12000)
        return _case(op, kind, precision, max(16, n // d), R, kL, device, rng.choice([360, 1024]))
    if op == "image":
        side = _log_int(rng, 60, 301)
        return _case(op, kind, precision, _log_int(rng, 100, 1000), rng.randint(1, 9), kL, points=side * side)
    if op == "mean_dos":
        n = _log_int(rng, 200, 3000)
        return _case(op, kind, precision, max(32, n // d), 0, kL, points=_log_int(rng, 50, 1000))
    if op == "ldos":
        n = _log_int(rng, 200, 4000)
        return _case(op, kind, precision, max(32, n // d), 0, kL, points=_log_int(rng, 20, 300), batches=rng.randint(1, 4))
    if op == "resident":
        n = _log_int(rng, 200, 3000) if precision == "fp64" else _log_int(rng, 500, 9000)
        return _case(op, kind, precision, max(16, n // d), R, kL)
    return _case("sweep", rng.choice(["2d_vector", "2d_scalar"]), "mixed", _log_int(rng, 300, 1500), rng.randint(1, 32),
                 kL, batches=rng.randint(4, 16))


# ---------------------------------------------------------------- inputs

def _scatterers(kind, N, seed):
    """N random points of the unit disk (2D) or cube (3D), thinned to a smallest separation as a
    sample of particles has: about a particle's diameter in 2D, its radius in 3D."""
    g = torch.Generator().manual_seed(int(seed))
    u = torch.rand(2 * N, 3, dtype=torch.float64, generator=g)
    if kind.startswith("2d"):
        r, phi = torch.sqrt(u[:, 0]), 2 * math.pi * u[:, 1]
        pts = torch.stack([r * torch.cos(phi), r * torch.sin(phi)], 1)
        apart = 0.4 / math.sqrt(N)
    else:
        pts = u - 0.5
        apart = 0.35 / N ** (1 / 3)
    p = pts.to("cuda")
    index = torch.arange(2 * N, device="cuda")
    crowded = torch.zeros(2 * N, dtype=torch.bool, device="cuda")
    for i in range(0, 2 * N, 4096):
        dist2 = sum((p[i:i + 4096, None, c] - p[None, :, c]) ** 2 for c in range(p.shape[1]))
        near = (dist2 < apart * apart) & (index[None, :] < index[i:i + 4096, None])
        crowded[i:i + 4096] = near.any(1)
    # the points with room first; a small sample may have to take some of the others
    return pts[torch.argsort(crowded.to("cpu"), stable=True)[:N]].clone()


def _physics(kind, N, kL):
    """(k0, polarisability, radius) of N scatterers: index 1.6, 5% (2D) or 10% (3D) of the volume."""
    if kind.startswith("2d"):
        V = 0.05 * math.pi / N
        a = math.sqrt(V / math.pi)
    else:
        V = 0.1 / N
        a = (3 * V / (4 * math.pi)) ** (1 / 3)
    return 2 * math.pi * kL, complex(V * (1.6 ** 2 - 1)), a


def _directions(kind, R):
    """2D: R angles; 3D: R directions in the plane z = 0 and their polarisations, two per direction."""
    if kind.startswith("2d"):
        return np.arange(R) / R * 2 * np.pi
    nd = (R + 1) // 2
    th = np.arange(nd) / nd * 2 * np.pi
    u = np.stack([np.cos(th), np.sin(th), np.zeros(nd)], 1)
    vertical = np.tile([0.0, 0.0, 1.0], (nd, 1))
    horizontal = np.stack([np.sin(th), -np.cos(th), np.zeros(nd)], 1)
    return (torch.from_numpy(np.concatenate([u, u])[:R].copy()),
            torch.from_numpy(np.concatenate([vertical, horizontal])[:R].copy()))


def _plane_waves(kind, points, k0, directions):
    """Plane waves at `points`: (M, R) or (M, d, R) complex128 on the points' device."""
    dev = points.device
    if kind.startswith("2d"):
        th = torch.as_tensor(directions, dtype=torch.float64)
        c, s = torch.cos(th).to(dev), torch.sin(th).to(dev)
        phase = points[:, 0:1] * c + points[:, 1:2] * s
        # the reference keeps the TE polarisation in single precision
        pol = torch.stack([torch.sin(-th), torch.cos(-th)]).to(torch.float32).to(torch.float64).to(dev)
    else:
        u, p = directions
        phase = points @ u.to(dev).T
        pol = p.to(dev).T
    E = torch.exp(1j * k0 * phase)
    if kind.endswith("scalar"):
        return E
    return E[:, None, :] * pol[None]


def _detectors(kind, M):
    if kind.startswith("2d"):
        t = torch.arange(M, dtype=torch.float64) / M * 2 * math.pi
        return 2.0 * torch.stack([torch.cos(t), torch.sin(t)], 1)
    i = torch.arange(M, dtype=torch.float64)
    z = 1 - 2 * (i + 0.5) / M
    t = i * math.pi * (math.sqrt(5.0) - 1.0)
    r = torch.sqrt(1 - z * z)
    return 3.0 * torch.stack([r * torch.cos(t), r * torch.sin(t), z], 1)


def _grid(kind, P):
    side = math.isqrt(P)
    return fields.grid_points(2 if kind.startswith("2d") else 3, side, side, 1.0, 2.4)


def _measure_points(kind, P, seed):
    u = torch.rand(P, 3, dtype=torch.float64, generator=torch.Generator().manual_seed(int(seed) + 7919))
    if kind.startswith("2d"):
        r, phi = 0.5 * torch.sqrt(u[:, 0]), 2 * math.pi * u[:, 1]
        return torch.stack([r * torch.cos(phi), r * torch.sin(phi)], 1)
    return 0.5 * (u - 0.5)


def _options(case):
    return {"precision": "fp64"} if case["precision"] == "fp64" else {"precision": "mixed", "tol": TOL}


def _sweep_problems(case, seed):
    out = []
    for i in range(case["batches"]):
        # sizes from a third of the largest up to it, frequencies spread around the case's
        N = case["N"] * (i + 1 + case["batches"] // 2) // (case["batches"] + case["batches"] // 2)
        kL = case["kL"] * (0.8 + 0.4 * i / case["batches"])
        k0, alpha, a = _physics(case["kind"], N, kL)
        out.append(workloads.Problem(case["kind"], _scatterers(case["kind"], N, seed * 1009 + i), k0, alpha, a,
                                     thetas=_directions(case["kind"], case["R"])))
    return out


def prepare(case, seed):
    kind, N, R = case["kind"], case["N"], case["R"]
    if case["op"] == "sweep":
        sweep = batch.BatchedSweep(_sweep_problems(case, seed), branches=8, tol=TOL)
        sweep.warmup()
        return {"op": "sweep", "sweep": sweep.capture()}
    k0, alpha, a = _physics(kind, N, case["kL"])
    pts = _scatterers(kind, N, seed).to(case["device"])
    s = {"op": case["op"], "kind": kind, "k0": k0, "alpha": alpha, "a": a, "pts": pts}
    if case["op"] in ("solve", "resident"):
        s["E0"] = _plane_waves(kind, pts, k0, _directions(kind, R)).contiguous()
    if case["op"] == "resident":
        opt = _options(case)
        s["factors"] = engine.SystemFactorization(kind, pts, k0, alpha * k0 * k0,
                                                  selfterm.diagonal_shift(kind, k0, alpha, a), opt["precision"],
                                                  opt.get("tol", engine.DEFAULT_TOL))
        s["E0"] = s["E0"].reshape(COMPONENTS[kind] * N, R)
        return s
    s["solver"] = SOLVERS[kind](pts, source="plane", **_options(case))
    if case["op"] == "transmission":
        s["directions"] = _directions(kind, R)
        s["det"] = _detectors(kind, case["points"]).to(case["device"])
    elif case["op"] == "image":
        dirs = _directions(kind, R)
        s["grid"] = _grid(kind, case["points"]).to(case["device"])
        s["E0"] = _plane_waves(kind, s["grid"], k0, dirs).contiguous()
        s["Ej"] = _image_fields(case, pts, k0, dirs, seed)
        s["columns"] = list(range(R))
    elif case["op"] in ("mean_dos", "ldos"):
        mp = _measure_points(kind, case["points"] * case["batches"], seed).to(case["device"])
        s["measure"] = mp if case["op"] == "mean_dos" else list(mp.split(case["points"]))
    return s


def _image_fields(case, pts, k0, dirs, seed):
    """Solved fields as the image step gets them: plane waves modulated by the sample's disorder."""
    E = _plane_waves(case["kind"], pts, k0, dirs).reshape(-1, case["R"])
    g = torch.Generator().manual_seed(int(seed) + 31)
    noise = torch.randn(E.shape + (2,), dtype=torch.float64, generator=g).to(E.device)
    return E * (1 + 0.3 * torch.view_as_complex(noise))


def run(s):
    op = s["op"]
    if op == "sweep":
        s["sweep"].replay()
        return s["sweep"].solutions()
    if op == "resident":
        return s["factors"].solve(s["E0"])
    solver, k0, alpha, a = s["solver"], s["k0"], s["alpha"], s["a"]
    if op == "solve":
        return solver.solve(k0, alpha, a, s["E0"])
    if op == "transmission":
        def source(points):
            if s["kind"].startswith("2d"):
                return solver.generate_source(points, k0, s["directions"], 0.2)
            if s["kind"] == "3d_vector":
                return solver.generate_source(points, k0, s["directions"][0], s["directions"][1], 0.2)
            return solver.generate_source(points, k0, s["directions"][0], 0.2)
        Ek = solver.solve(k0, alpha, a, source(s["pts"]))
        return [Ek, solver.propagate(s["det"], Ek, k0, alpha, source(s["det"]))]
    if op == "image":
        return fields.full_fields(solver, s["grid"], s["Ej"], s["columns"], s["E0"], k0, alpha)
    if op == "mean_dos":
        return solver.mean_DOS_measurements(s["measure"], k0, alpha, a)
    return solver.batch_LDOS_measurements(s["measure"], k0, alpha, a)


# ---------------------------------------------------------------- work

def _solve_work(n, R):
    """LU of order n (8/3 n^3 real operations), solves and one read / write of the fields."""
    return {"bytes": 8.0 * 3 * n + 32.0 * n * R, "flops": 8.0 / 3 * n ** 3 + 8.0 * n * n * R}


def work(case):
    kind, N, R, P = case["kind"], case["N"], case["R"], case["points"]
    d = COMPONENTS[kind]
    n = d * N
    if case["op"] == "sweep":
        parts = [_solve_work(p.n, R) for p in _sweep_problems(case, 1)]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    if case["op"] == "solve":
        return _solve_work(n, R)
    if case["op"] == "resident":
        # both triangular factors (complex64 or complex128) are read for a block of fields
        per = 16.0 if case["precision"] == "fp64" else 8.0
        return {"bytes": per * n * n + 32.0 * n * R, "flops": 8.0 * n * n * R}
    if case["op"] == "transmission":
        w = _solve_work(n, R)
        return {"bytes": w["bytes"] + 32.0 * d * P * R, "flops": w["flops"] + 8.0 * d * P * n * R}
    if case["op"] == "image":
        return {"bytes": 16.0 * n * R + 32.0 * d * P * R, "flops": 8.0 * d * P * n * R}
    cols = d * P * case["batches"]
    return {"bytes": 24.0 * (N + P * case["batches"]) + 8.0 * P * case["batches"],
            "flops": 8.0 / 3 * n ** 3 + 8.0 * n * n * cols}


# ---------------------------------------------------------------- the same in 64 bits, in plain torch

def _hankel_small(x):
    """H0, H1 for 0 < x < 25: J_k by Miller's backward recurrence, Y0 from Neumann's series
    Y0 = (2/pi) (ln(x/2) + gamma) J0 - (4/pi) sum (-1)^k J_2k / k, and Y1 = -Y0' term by term."""
    top = 90
    jp, j = torch.zeros_like(x), torch.full_like(x, 1e-300)
    norm, y0, y1 = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(x)
    j1 = torch.zeros_like(x)
    for m in range(top, 0, -1):
        # j = J_m, jp = J_{m+1}; next is J_{m-1}
        jm = (2.0 * m / x) * j - jp
        if m % 2 == 0:
            k = m // 2
            sign = -1.0 if k % 2 else 1.0
            norm = norm + 2.0 * j
            y0 = y0 + sign * j / k
            y1 = y1 + sign * 0.5 * (jm - jp) / k
        jp, j = j, jm
        if m == 1:
            j1 = jp
        big = j.abs() > 1e200
        if bool(big.any()):
            f = torch.where(big, torch.full_like(x, 1e-200), torch.ones_like(x))
            jp, j, norm, y0, y1 = jp * f, j * f, norm * f, y0 * f, y1 * f
            j1 = j1 * f
    norm = norm + j
    j0, j1, y0, y1 = j / norm, j1 / norm, y0 / norm, y1 / norm
    lg = torch.log(0.5 * x) + np.euler_gamma
    c = 2.0 / math.pi
    return (torch.complex(j0, c * lg * j0 - 2.0 * c * y0),
            torch.complex(j1, -c * (j0 / x - lg * j1) + 2.0 * c * y1))


def _hankel_large(x):
    """H0, H1 for x >= 25: Hankel's asymptotic expansion."""
    out = []
    for nu in (0, 1):
        mu = 4.0 * nu * nu
        term = torch.ones_like(x)
        P, Q = torch.ones_like(x), torch.zeros_like(x)
        for k in range(1, 24):
            term = term * ((mu - (2 * k - 1) ** 2) / (8.0 * k)) / x
            if k % 2:
                Q = Q + (term if (k // 2) % 2 == 0 else -term)
            else:
                P = P + (term if (k // 2) % 2 == 0 else -term)
        chi = x - (0.5 * nu + 0.25) * math.pi
        out.append(torch.sqrt(2.0 / (math.pi * x)) * torch.complex(P, Q) * torch.exp(1j * chi))
    return out


def _hankel(x):
    """H0, H1 of positive x (zeros elsewhere)."""
    h0 = torch.zeros(x.shape, dtype=torch.complex128, device=x.device)
    h1 = torch.zeros_like(h0)
    for mask, f in (((x > 0) & (x < 25), _hankel_small), (x >= 25, _hankel_large)):
        v = x[mask]
        if v.numel():
            h0[mask], h1[mask] = f(v)
    return h0, h1


def _greens(kind, targets, sources, k0):
    """Dense Green's matrix (d T, d S) complex128, zero blocks at zero separation."""
    d = COMPONENTS[kind]
    r = targets[:, None, :] - sources[None, :, :]
    R = torch.sqrt((r * r).sum(-1))
    same = R == 0
    R = torch.where(same, torch.ones_like(R), R)
    kR = k0 * R
    if kind.startswith("2d"):
        h0, h1 = _hankel(kR)
        if d == 1:
            g = 0.25j * h0
        else:
            P = r[..., :, None] * r[..., None, :] / (R * R)[..., None, None]
            eye = torch.eye(2, dtype=torch.float64, device=r.device)
            g = 0.25j * ((eye - P) * h0[..., None, None] - (eye - 2 * P) * (h1 / kR)[..., None, None])
    else:
        e = torch.exp(1j * kR) / (4 * math.pi * R)
        if d == 1:
            g = e
        else:
            P = r[..., :, None] * r[..., None, :] / (R * R)[..., None, None]
            eye = torch.eye(3, dtype=torch.float64, device=r.device)
            f = 1 / (1j * kR) + 1 / (kR * kR)
            g = (eye - P - (eye - 3 * P) * f[..., None, None]) * e[..., None, None]
    T, S = targets.shape[0], sources.shape[0]
    if d == 1:
        return torch.where(same, torch.zeros_like(g), g)
    g = torch.where(same[..., None, None], torch.zeros_like(g), g)
    return g.permute(0, 2, 1, 3).reshape(d * T, d * S)


def _greens_rows(kind, targets, sources, k0, step=0):
    step = step or max(1, (1 << 21) // sources.shape[0])
    for t0 in range(0, targets.shape[0], step):
        yield t0, _greens(kind, targets[t0:t0 + step], sources, k0)


def _self_over_volume(kind, k0, a):
    if kind.startswith("2d"):
        log = 2.0 * np.euler_gamma - 1.0 + 2.0 * math.log(k0 * a / 2.0) - 1j * math.pi
        s = -a * a / 4.0 * log if kind == "2d_scalar" else -1 / (2.0 * k0 * k0) - a * a / 8.0 * log
        return s / (math.pi * a * a)
    V = 4.0 * math.pi * a ** 3 / 3.0
    if kind == "3d_scalar":
        return (a * a / 2.0 + 1j * k0 * V / (4.0 * math.pi)) / V
    return (-1.0 / (3.0 * k0 * k0) + a * a / 3.0 + 1j * k0 * V / (6.0 * math.pi)) / V


def _system(kind, pts, k0, alpha, a):
    d, n = COMPONENTS[kind], COMPONENTS[kind] * pts.shape[0]
    M = torch.empty((n, n), dtype=torch.complex128, device=pts.device)
    for t0, g in _greens_rows(kind, pts, pts, k0):
        M[d * t0:d * t0 + g.shape[0]] = -alpha * k0 * k0 * g
    # the reference subtracts the self-term in single precision
    shift = complex(np.complex64(alpha * k0 * k0 * _self_over_volume(kind, k0, a)))
    M.fill_diagonal_(1.0 - shift)
    return M


def _solved(M, B):
    """M^-1 B with one refinement step."""
    LU, piv = torch.linalg.lu_factor(M)
    X = torch.linalg.lu_solve(LU, piv, B)
    return X + torch.linalg.lu_solve(LU, piv, B - M @ X)


def exact(case, seed):
    kind, N, R = case["kind"], case["N"], case["R"]
    d = COMPONENTS[kind]
    n = d * N
    if case["op"] != "image" and n > 12500:
        return None      # a 64-bit factorisation of this order takes too long
    if case["op"] == "sweep":
        out = []
        for p in _sweep_problems(case, seed):
            pts = p.points.to("cuda")
            B = _plane_waves(kind, pts, p.k0, p.thetas).reshape(-1, R)
            out.append(_solved(_system(kind, pts, p.k0, p.alpha, p.radius), B))
        return out
    k0, alpha, a = _physics(kind, N, case["kL"])
    pts = _scatterers(kind, N, seed).to("cuda")
    if case["op"] == "image":
        dirs, grid = _directions(kind, R), _grid(kind, case["points"]).to("cuda")
        Ej = _image_fields(case, pts, k0, dirs, seed)
        E = _plane_waves(kind, grid, k0, dirs)
        flat = E.reshape(-1, R).clone()
        for t0, g in _greens_rows(kind, grid, pts, k0):
            flat[d * t0:d * t0 + g.shape[0]] += alpha * k0 * k0 * (g @ Ej)
        return flat.reshape(E.shape)
    M = _system(kind, pts, k0, alpha, a)
    if case["op"] in ("mean_dos", "ldos"):
        mp = _measure_points(kind, case["points"] * case["batches"], seed).to("cuda")
        G = torch.cat([g for _, g in _greens_rows(kind, mp, pts, k0)])
        dots = (G.T * _solved(M, G.T.contiguous())).sum(0)
        pref = {"2d_vector": 4.0 * k0 * k0, "2d_scalar": 4.0 * k0 * k0, "3d_vector": 2.0 * math.pi * k0,
                "3d_scalar": 4.0 * math.pi * k0}[kind] * alpha
        if case["op"] == "mean_dos":
            return torch.imag(dots.sum() / case["points"] * pref)
        v = torch.imag(dots * pref)
        return v.reshape(-1, d, 1).sum(1) if d > 1 else v
    dirs = _directions(kind, R)
    E0 = _plane_waves(kind, pts, k0, dirs).reshape(n, R)
    X = _solved(M, E0)
    if case["op"] == "transmission":
        det = _detectors(kind, case["points"]).to("cuda")
        E = _plane_waves(kind, det, k0, dirs)
        flat = E.reshape(-1, R) + alpha * k0 * k0 * (_greens(kind, det, pts, k0) @ X)
        return [X.to(case["device"]), flat.reshape(E.shape).to(case["device"])]
    return X
