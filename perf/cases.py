"""Performance cases: what a program built on openvort_b200 spends its time on.

Every case goes through the public entry points, over seeded synthetic
tangles.  The kinds are

  update     update_tangle on a host tangle (the reference's two calls):
             tangents, normals and velocities of every node
  run        a device-resident state: upload, a few RK4 steps, positions back
  batch      an ensemble of independent ring pairs stepped together
  adjoint    a trajectory and the gradient of a loss on its final positions
  points     Biot-Savart velocity at probe points of a device-resident state
  reconnect  one vortex-vortex reconnection pass over a host tangle

`listed` holds one point of each path's range, `draw` draws others.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import openvort_b200 as ov
from openvort_b200 import geometry as G
from openvort_b200.adjoint import Adjoint, centroid_length_loss, trajectory
from openvort_b200.tangle import IMAGE_TABLES, Flow, Params

KAPPA = 9.97e-4
DT = 1e-6                       # time step of the tangle runs
DT_FINE = 2.5e-7                # of the ensembles, whose finest rings carry fast Kelvin waves
R_FRAC = (0.02, 0.05)           # ring radii of a tangle, in box lengths


def listed():
    return [
        # the smallest call: tangents and velocities of one ring, from and to host memory
        {"name": "ring_update", "kind": "update", "shape": "ring", "points": 256, "boundary": "open",
         "method": "direct", "precision": "fp64"},
        # the 256-point ring stepped with RK4 (launches and latency count)
        {"name": "ring_run", "kind": "run", "shape": "ring", "points": 256, "boundary": "open", "method": "direct",
         "precision": "fp64", "steps": 50},
        # the 22.4k-point periodic tangle by direct summation over its 26 images, FP64
        {"name": "direct_fp64_22k", "kind": "update", "shape": "tangle", "points": 22400, "boundary": "periodic-26",
         "method": "direct", "precision": "fp64"},
        # and one RK4 step of it in the mixed form
        {"name": "direct_mixed_22k", "kind": "run", "shape": "tangle", "points": 22400, "boundary": "periodic-26",
         "method": "direct", "precision": "mixed", "steps": 1},
        # the same tangle stepped with the Barnes-Hut sum at theta = 0.4
        {"name": "bh_mixed_22k", "kind": "run", "shape": "tangle", "points": 22400, "boundary": "periodic-26",
         "method": "bh", "theta": 0.4, "precision": "mixed", "steps": 4},
        # velocities of a 200k-point tangle, Barnes-Hut, FP64
        {"name": "bh_fp64_200k", "kind": "update", "shape": "tangle", "points": 200000, "boundary": "periodic-26",
         "method": "bh", "theta": 0.5, "precision": "fp64"},
        # one RK4 step of the 1M-point tangle, Barnes-Hut, mixed form: the headline workload
        {"name": "bh_mixed_1m", "kind": "run", "shape": "tangle", "points": 1000000, "boundary": "periodic-26",
         "method": "bh", "theta": 0.5, "precision": "mixed", "steps": 1},
        # ensembles of ring pairs: a parameter study of a few hundred systems in FP64, and a
        # large one in the mixed form at the kernel shape its autotuner settles on
        {"name": "batch_fp64_256", "kind": "batch", "systems": 256, "precision": "fp64", "steps": 2},
        {"name": "batch_mixed_2048", "kind": "batch", "systems": 2048, "precision": "mixed", "steps": 2,
         "targets": 64, "sources": 256},
        # gradient of a loss through a ring's trajectory (forward and backward)
        {"name": "adjoint_2048", "kind": "adjoint", "points": 2048, "steps": 4, "every": 2},
        # the velocity field of a Barnes-Hut tangle at probe points (spectra, structure functions)
        {"name": "points_bh_4096", "kind": "points", "points": 50000, "boundary": "periodic-26", "probes": 4096,
         "method": "bh", "theta": 0.4, "precision": "fp64"},
        # the reconnection pass that precedes every step of a simulation
        {"name": "reconnect_100k", "kind": "reconnect", "points": 100000, "boundary": "periodic-26",
         "precision": "mixed"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["update_direct", "run_ring", "run_direct", "run_bh", "update_bh", "batch", "adjoint", "points",
                       "reconnect"])
    boundary = rng.choice(["open", "periodic-6", "periodic-26", "periodic-26"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "update_direct":
        return {"kind": "update", "shape": "tangle", "points": _log_int(rng, 200, 24000), "boundary": boundary,
                "method": "direct", "precision": "fp64"}
    if kind == "run_ring":
        return {"kind": "run", "shape": "ring", "points": _log_int(rng, 64, 2048), "boundary": "open",
                "method": "direct", "precision": "fp64", "steps": rng.randint(10, 50)}
    if kind == "run_direct":
        n = _log_int(rng, 300, 24000)
        return {"kind": "run", "shape": "tangle", "points": n, "boundary": boundary, "method": "direct",
                "precision": "mixed", "steps": 1 if n > 8000 else rng.randint(1, 8)}
    if kind == "run_bh":
        theta = rng.choice([0.3, 0.4, 0.5])
        n = _log_int(rng, 3000, 250000 if precision == "mixed" else 100000)
        return {"kind": "run", "shape": "tangle", "points": n, "boundary": boundary, "method": "bh", "theta": theta,
                "precision": precision, "steps": 1 if n > 40000 else rng.randint(1, 3)}
    if kind == "update_bh":
        return {"kind": "update", "shape": "tangle", "points": _log_int(rng, 5000, 300000), "boundary": boundary,
                "method": "bh", "theta": rng.choice([0.4, 0.5]), "precision": "fp64"}
    if kind == "batch":
        if precision == "fp64":
            return {"kind": "batch", "systems": _log_int(rng, 8, 400), "precision": "fp64", "steps": rng.randint(1, 3)}
        return {"kind": "batch", "systems": _log_int(rng, 8, 2048), "precision": "mixed", "steps": rng.randint(1, 2),
                "targets": 64, "sources": 256}
    if kind == "adjoint":
        return {"kind": "adjoint", "points": _log_int(rng, 128, 4096), "steps": rng.randint(2, 5),
                "every": rng.randint(1, 4)}
    if kind == "points":
        return {"kind": "points", "points": _log_int(rng, 2000, 100000), "boundary": boundary,
                "probes": _log_int(rng, 512, 8192), "method": rng.choice(["bh", "bh", "direct"]),
                "theta": rng.choice([0.4, 0.5]), "precision": "fp64"}
    return {"kind": "reconnect", "points": _log_int(rng, 5000, 150000), "boundary": rng.choice(["open", "periodic-26"]),
            "precision": precision}


# ---------------------------------------------------------------- inputs

def _tangle_scale(points):
    """Box side and point spacing of a tangle of about `points` points: up to
    30k the box of the repository's 22.4k-point tangle (D/200 at D = 0.1 cm),
    above it the line density of its 1M-point one (spacing 5e-4 cm, D = 0.4
    cm at 1M points)."""
    if points <= 30000:
        return 0.1, 0.1 / 200
    return 0.4 * (points / 1e6) ** (1 / 3), 5e-4


def _tangle(case, seed):
    """Rings with seeded centres and directions; their sizes depend on the
    case alone, so every seed gives exactly `points` nodes."""
    points = case["points"]
    D, dl = _tangle_scale(points)
    lo, hi = (max(5, int(2 * math.pi * f * D / dl)) for f in R_FRAC)
    sizes, left, rng = [], points, np.random.default_rng(points)
    while left > 0:
        n = int(rng.integers(lo, hi + 1))
        if left - n < lo:
            n = left
        sizes.append(n)
        left -= n
    rng = np.random.default_rng(seed)
    rings = []
    for n in sizes:
        d = rng.normal(size=3)
        rings.append(G.ring_points(rng.uniform(0.0, D, size=3), d / np.sqrt(d @ d), n * dl / (2 * math.pi), n))
    if case["boundary"] == "open":   # whole rings in a box that holds them all
        return G.rings_to_tangle(rings, (-0.1 * D,) * 3, (1.1 * D,) * 3, "open"), dl
    return G.rings_to_tangle(rings, (0.0,) * 3, (D,) * 3, case["boundary"], wrap=True), dl


def _ensemble(case, seed):
    """Coaxial ring pairs, leapfrogging or head-on, 64 to 2048 points each;
    sizes from the case alone."""
    sizes = np.random.default_rng(case["systems"]).integers(64, 2049, size=case["systems"])
    rng = np.random.default_rng(seed)
    systems = [G.ring_pair_system(rng, "leapfrog" if rng.uniform() < 0.5 else "headon", int(n)) for n in sizes]
    t = G.rings_to_tangle([r for pair in systems for r in pair], (-0.09,) * 3, (0.09,) * 3, "open")
    return t, np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)


def _ring(case, seed):
    n, radius = case["points"], 1e-2
    pos = G.kelvin_ring(seed, n=n, radius=radius, modes=(2, 8), sigma=1e-4)
    return G.rings_to_tangle([pos], (-0.05,) * 3, (0.05,) * 3, "open"), 2 * math.pi * radius / n


def _params(case, dl):
    kind = case["kind"]
    if kind == "batch":
        return Params(core_a=1e-8, alpha=0.098, alpha_p=0.016, use_mf=1, dl_max=1e-2, hyperfriction=0, use_bh=0)
    if kind == "adjoint" or case.get("shape") == "ring":
        # dl_max below dl keeps hyperfriction off the ring's own curvature
        return Params(core_a=1e-8, alpha=0.098, alpha_p=0.016, use_mf=1, dl_max=dl / 2, hyperfriction=1, use_bh=0,
                      vn=Flow("simple", {"external_v": (0.2, 0.0, 0.0)}))
    return Params(core_a=1e-8, alpha=0.098, alpha_p=0.016, use_mf=1, dl_max=2 * dl, hyperfriction=1,
                  use_bh=1 if case.get("method") == "bh" else 0, bh_theta=case.get("theta", 0.4), bh_grain=1e-8,
                  vn=Flow("simple", {"external_v": (0.5, 0.0, 0.0)}))


def _inputs(case, seed):
    """Tangle, parameters, time step and (ensembles) slot offsets."""
    if case["kind"] == "batch":
        t, offsets = _ensemble(case, seed)
        return t, _params(case, 0.0), DT_FINE, offsets
    if case["kind"] == "adjoint" or case.get("shape") == "ring":
        t, dl = _ring(case, seed)
        # grid-scale Kelvin waves: omega ~ dl^-2, so the step shrinks with it
        return t, _params(case, dl), 2e-6 * min(1.0, (dl / 2.45e-4) ** 2), None
    t, dl = _tangle(case, seed)
    return t, _params(case, dl), DT, None


def _probes(case, seed):
    D, _ = _tangle_scale(case["points"])
    return np.random.default_rng(seed + 77).uniform(0.0, D, size=(case["probes"], 3))


def prepare(case, seed):
    kind = case["kind"]
    t, p, dt, offsets = _inputs(case, seed)
    precision = ov.OV_PREC_MIXED if case.get("precision") == "mixed" else ov.OV_PREC_FP64
    lib = ov.configure(p, precision)
    s = {"kind": kind, "t": t, "dt": dt, "case": dict(case), "lib": lib}
    if kind == "run":
        s["state"] = ov.DeviceState(t)
        s["pos0"] = t.pos.copy()
    elif kind == "points":
        s["state"] = ov.DeviceState(t)
        s["pts"] = _probes(case, seed)
    elif kind == "batch":
        s["batch"] = ov.DeviceBatch(t, offsets)
        if "targets" in case:
            s["batch"].set_tuning(case["targets"], case["sources"])
    elif kind == "adjoint":
        s["adj"] = Adjoint(t)
        s["x0"] = torch.tensor(t.pos, dtype=torch.float64)
        s["vn"] = torch.tensor([0.2, 0.0, 0.0], dtype=torch.float64)
    elif kind == "reconnect":
        ov.update_tangle(t, 0.0)      # the pass needs current tangents
        t.set_images_from_library(lib)
        s["links0"], s["vels0"] = t.links.copy(), t.vels.copy()
        s["rec_dist"], s["rec_angle"] = _tangle_scale(case["points"])[1], 0.087
    return s


def run(s):
    kind, t, case = s["kind"], s["t"], s["case"]
    if kind == "update":
        ov.update_tangle(t, 0.0)
        return {"vels": t.vels, "vs": t.vs, "tangents": t.tangents, "normals": t.normals, "dxi": t.dxi}
    if kind == "run":
        t.pos[:] = s["pos0"]
        st = s["state"]
        st.upload()
        st.run(0.0, s["dt"], case["steps"])
        st.download(ov.OV_FIELD_POS)
        return {"pos": t.pos}
    if kind == "batch":
        b = s["batch"]
        b.run(0.0, s["dt"], case["steps"])
        b.download(ov.OV_FIELD_POS)
        return {"pos": t.pos}
    if kind == "adjoint":
        x0 = s["x0"].clone().requires_grad_(True)
        vn = s["vn"].clone().requires_grad_(True)
        xf = trajectory(s["adj"], x0, vn, 0.0, s["dt"], case["steps"], case["every"])
        centroid_length_loss(xf, t.links[:, 0], t.active, LOSS_TARGET).backward()
        return {"x": xf.detach(), "x0_grad": x0.grad, "vn_grad": vn.grad}
    if kind == "points":
        return {"v": s["state"].eval_points(s["pts"], method=1 if case["method"] == "bh" else 0)}
    # reconnect: the pass works in place on the host tangle's links and flags
    t.links[:] = s["links0"]
    t.vels[:] = s["vels0"]
    t.recalc[:] = 0
    n = s["lib"].ov_reconnect_vortices(t.ptr(), 0.0, s["rec_dist"], s["rec_angle"])
    ov.check(s["lib"])
    return {"reconnections": n, "links": t.links, "flags": t.recalc, "vels": t.vels}


LOSS_TARGET = (0.004, -0.002, 0.003)


# ---------------------------------------------------------------- work

FLOPS_PAIR = 43      # one segment at one target (multiply, add, root and divide count one each)
FLOPS_CELL = 60      # one cell's expansion with its opening test


def _images(case):
    return 1 + len(IMAGE_TABLES[case.get("boundary", "open")])


def _bh_flops(n, targets, theta, images):
    """Cells and leaf segments grow with log N and about theta^-2.15: 744
    cells per target and image and 619 segments per target at 1M points,
    theta = 0.5."""
    levels = math.log2(max(2, n)) / 20 * (0.5 / theta) ** 2.15
    return targets * (min(744 * levels, n) * FLOPS_CELL * images + min(619 * levels, n) * FLOPS_PAIR)


def work(case):
    kind = case["kind"]
    images = _images(case)
    if kind == "batch":
        # points uniform in 64..2048 per system
        n = 1056.0 * case["systems"]
        pairs = case["systems"] * (64 * 64 + 64 * 2048 + 2048 * 2048) / 3
        return {"bytes": n * (40 + 24), "flops": 4 * case["steps"] * pairs * FLOPS_PAIR}
    n = float(case["points"])
    if kind == "adjoint":
        # forward, its recomputation and the reverse: 4 sums and 4 products per
        # step, a product costing about three evaluations
        return {"bytes": n * (24 * 3 + 16), "flops": 4 * case["steps"] * n * n * FLOPS_PAIR * 4}
    if kind == "points":
        flops = (_bh_flops(n, case["probes"], case["theta"], images) if case["method"] == "bh"
                 else case["probes"] * n * images * FLOPS_PAIR)
        return {"bytes": n * 40 + 48 * case["probes"], "flops": flops}
    if kind == "reconnect":
        # about 0.5% of the nodes are tested, each against every segment and image
        return {"bytes": n * (40 + 72 + 24), "flops": 0.0054 * n * n * images * FLOPS_PAIR}
    evals = 1 if kind == "update" else 4 * case["steps"]
    flops = evals * (_bh_flops(n, n, case["theta"], images) if case["method"] == "bh" else n * n * images * FLOPS_PAIR)
    return {"bytes": n * (40 + (104 if kind == "update" else 24)), "flops": flops}


# ---------------------------------------------------------------- exact values
#
# The same equations in 64-bit torch: tangents and normals by the 4-point
# Lagrange stencils, local induction, the sum over straight segments and
# their periodic images, mutual friction, RK4 (whose fourth stage advances
# dt/2).  Closed loops of free nodes only, as every case here has.

def _wrap(d, L):
    if L is None:
        return d
    return d - L * (d > L / 2).to(d.dtype) + L * (d < -L / 2).to(d.dtype)


def _norm(v):
    return (v * v).sum(-1).sqrt()


def _stencils(x, f, r, L):
    """dxi, tangents, normals; f and r are the forward and reverse nodes."""
    nodes = (f[f], f, r, r[r])
    dxi = _norm(_wrap(x[f] - x, L))
    arc = (dxi + dxi[f], dxi, -dxi[r], -(dxi[r] + dxi[r[r]]))
    tan, nrm = torch.zeros_like(x), torch.zeros_like(x)
    for j in range(4):
        o0, o1, o2 = arc[(j + 1) % 4], arc[(j + 2) % 4], arc[(j + 3) % 4]
        den = arc[j] * (arc[j] - o0) * (arc[j] - o1) * (arc[j] - o2)
        d = _wrap(x[nodes[j]] - x, L)
        tan = tan + d * (-(o0 * o1 * o2) / den)[:, None]
        nrm = nrm + d * (2 * (o0 * o1 + o0 * o2 + o1 * o2) / den)[:, None]
    return dxi, tan, nrm


def _segments_at(pts, r1, r2, skip):
    """Sum over the segments r1 -> r2 at pts; skip: (targets, segments) left out."""
    a = [r1[None, :, c] - pts[:, c, None] for c in range(3)]
    b = [r2[None, :, c] - pts[:, c, None] for c in range(3)]
    a2, b2 = sum(u * u for u in a), sum(u * u for u in b)
    off = (a2 < 1e-16) | (b2 < 1e-16)
    if skip is not None:
        off = off | skip
    la, lb = torch.where(off, 1.0, a2).sqrt(), torch.where(off, 1.0, b2).sqrt()
    ab, dot = la * lb, sum(u * v for u, v in zip(a, b))
    off = off | ((dot / ab - 1).abs() < 1e-8)
    w = torch.where(off, 0.0, (la + lb) / torch.where(off, 1.0, ab * (ab + dot)))
    return torch.stack([((a[1] * b[2] - a[2] * b[1]) * w).sum(1), ((a[2] * b[0] - a[0] * b[2]) * w).sum(1),
                        ((a[0] * b[1] - a[1] * b[0]) * w).sum(1)], 1) * (KAPPA / 4 / math.pi)


def _nonlocal(pts, x, f, L, boundary, own):
    """Tangle and image sums at pts; own: pts are the nodes, whose two
    segments the tangle's own sum leaves out."""
    r2 = x + _wrap(x[f] - x, L)
    n, out = x.shape[0], []
    ids = torch.arange(n, device=x.device)
    for i in range(0, pts.shape[0], max(1, (1 << 25) // n)):
        p = pts[i:i + max(1, (1 << 25) // n)]
        skip = None
        if own:
            k = ids[i:i + p.shape[0], None]
            skip = (ids[None, :] == k) | (f[None, :] == k)
        v = _segments_at(p, x, r2, skip)
        for shift, _ in IMAGE_TABLES[boundary]:
            v = v + _segments_at(p - torch.tensor(shift, dtype=x.dtype, device=x.device) * L, x, r2, None)
        out.append(v)
    return torch.cat(out)


def _velocity(x, f, r, L, boundary, p, vn):
    dxi, tan, nrm = _stencils(x, f, r, L)
    lia_f = p.kappa * torch.log(2 * (dxi * dxi[r]).sqrt() / math.sqrt(math.sqrt(math.e)) / p.core_a) / 4 / math.pi
    lia = torch.linalg.cross(tan, nrm) * lia_f[:, None]
    vs = lia + _nonlocal(x, x, f, L, boundary, True)
    v = vs
    if p.hyperfriction:
        v = v - torch.where((_norm(nrm) > p.max_curv_scale / p.dl_max)[:, None],
                            p.hyperalpha * torch.linalg.cross(tan, lia), torch.zeros_like(x))
    if p.use_mf:
        dv = vn[None, :] - vs
        v = v + p.alpha * torch.linalg.cross(tan, dv) - p.alpha_p * torch.linalg.cross(tan, torch.linalg.cross(tan, dv))
    return v, vs, tan, nrm, dxi


def _rk4(x, vel, dt):
    k1 = vel(x)
    k2 = vel(x + k1 * (dt / 2))
    k3 = vel(x + k2 * (dt / 2))
    k4 = vel(x + k3 * (dt / 2))
    return x + k1 * (dt / 6) + k2 * (dt / 3) + k3 * (dt / 3) + k4 * (dt / 6)


def exact(case, seed):
    kind = case["kind"]
    if kind == "reconnect" or (kind == "batch" and case["systems"] * case["steps"] > 600):
        return None        # whole decisions; thousands of systems one by one take too long
    if kind == "run" and case["method"] == "bh":
        return None        # the Barnes-Hut sum is an approximation without a closed form
    if kind == "points" and case["method"] == "bh":
        return None
    evals = {"update": 1, "run": 4 * case.get("steps", 1)}.get(kind, 1)
    t, p, dt, offsets = _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.tensor(t.pos, dtype=torch.float64, device=dev)
    f = torch.tensor(t.links[:, 0], dtype=torch.long, device=dev)
    r = torch.tensor(t.links[:, 1], dtype=torch.long, device=dev)
    vn = torch.tensor(p.vn.params.get("external_v", (0.0, 0.0, 0.0)), dtype=torch.float64, device=dev)
    boundary = t.boundary
    L = t.box_hi[0] - t.box_lo[0] if boundary.startswith("periodic") else None
    direct_pairs = float(x.shape[0]) ** 2 * _images(case) * evals
    if kind in ("update", "run") and case["method"] == "direct" and direct_pairs > 8e10:
        return None
    if kind == "update":
        if case["method"] == "bh":
            dxi, tan, nrm = _stencils(x, f, r, L)
            return {"vels": None, "vs": None, "tangents": tan, "normals": nrm, "dxi": dxi}
        v, vs, tan, nrm, dxi = _velocity(x, f, r, L, boundary, p, vn)
        return {"vels": v, "vs": vs, "tangents": tan, "normals": nrm, "dxi": dxi}
    if kind == "run":
        for _ in range(case["steps"]):
            x = _rk4(x, lambda y: _velocity(y, f, r, L, boundary, p, vn)[0], dt)
        return {"pos": x}
    if kind == "batch":
        out = x.clone()
        for a, b in zip(offsets[:-1], offsets[1:]):
            y, fy, ry = x[a:b], f[a:b] - int(a), r[a:b] - int(a)
            for _ in range(case["steps"]):
                y = _rk4(y, lambda z: _velocity(z, fy, ry, None, "open", p, vn)[0], dt)
            out[a:b] = y
        return {"pos": out}
    if kind == "points":
        if float(case["probes"]) * x.shape[0] * _images(case) > 8e10:
            return None
        pts = torch.tensor(_probes(case, seed), dtype=torch.float64, device=dev)
        return {"v": _nonlocal(pts, x, f, L, boundary, False)}
    # adjoint: the same trajectory under autograd, every evaluation recomputed in the backward
    from torch.utils.checkpoint import checkpoint
    x0, vn = x.clone().requires_grad_(True), vn.clone().requires_grad_(True)

    def vel(y):
        return checkpoint(lambda z, w: _velocity(z, f, r, L, boundary, p, w)[0], y, vn, use_reentrant=False)

    y = x0
    for _ in range(case["steps"]):
        y = _rk4(y, vel, dt)
    target = torch.tensor(LOSS_TARGET, dtype=torch.float64, device=dev)
    loss = ((y.mean(0) - target) ** 2).sum() + _norm(y[f] - y).sum()
    gx, gv = torch.autograd.grad(loss, (x0, vn))
    return {"x": y.detach(), "x0_grad": gx, "vn_grad": gv}
