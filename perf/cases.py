"""The work that programs have this engine do, as timed cases.

Every case is one call that a simulation, a post-processing script or a training loop makes through the package's
public classes:

  product    the RPY grand mobility of segments (and blobs), RpyMobilitySolver
  fcm        the fast force-coupling mobility in a periodic box, FcmSolver
  flow       flow velocities at field points, FlowFieldEvaluator
  mlp        the learned preconditioner's network, forward or with gradients, FilamentMLP
  step       one implicit time step of one wall array, WallCiliaSimulation
  batch      one implicit time step of many uneven arrays, WallCiliaBatch
  swim       one time step of a free ciliated sphere, CiliatedSwimmer
  elastic    one Broyden step of elastic cilia, ElasticCiliaSimulation

Sizes are the repository's own configurations and the ranges between its smallest tests and its largest benchmark.
Inputs depend on the seed alone.  Time steps continue their simulation from pass to pass, as a run does.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cufcm_fil_b200 import RpyMobilitySolver, _lib, swim, workloads
from cufcm_fil_b200.elastic import ElasticCiliaSimulation
from cufcm_fil_b200.fcm import FcmSolver
from cufcm_fil_b200.flow import FlowFieldEvaluator
from cufcm_fil_b200.mlp import FilamentMLP
from cufcm_fil_b200.sim import WallCiliaBatch, WallCiliaSimulation, arclength_table

NSEG, SEG_SEP = 20, 2.6
N_IN, HIDDEN, N_OUT = 182, 256, 62  # the network of 20-segment cilia


def listed():
    return [
        # The smallest matrix-vector product (16 vertical cilia, FP32 on the device): a call of a few launches.
        {"name": "wall product 320", "kind": "product", "wall": True, "dof": 3, "n_fil": 16, "n_seg": 20, "n_blob": 0,
         "host": False},
        # The 32 x 32 lattice of prescribed cilia, forces only: the product inside every large implicit solve.
        {"name": "wall product 20480", "kind": "product", "wall": True, "dof": 3, "n_fil": 1024, "n_seg": 20,
         "n_blob": 0, "host": False},
        # A swimmer with forces and torques through the host arrays, as the reference's driver calls it.
        {"name": "swimmer product host", "kind": "product", "wall": False, "dof": 6, "n_fil": 159, "n_seg": 20,
         "n_blob": 2562, "host": True},
        # The precision-study box: 1000 cilia on a sphere of 10 000 blobs, 512^3 grid, arrays on the device.
        {"name": "fcm 512", "kind": "fcm", "n_fil": 1000, "n_blob": 10000, "grid": 512, "radius": 100.0,
         "host": False},
        # A small swimmer on a coarser grid through the host layouts of the mobility interface.
        {"name": "fcm 128 host", "kind": "fcm", "n_fil": 100, "n_blob": 1000, "grid": 128, "radius": 30.0,
         "host": True},
        # One flow-field frame: a 160 x 100 plane of points above the 16 x 16 array, from saved forces.
        {"name": "flow plane", "kind": "flow", "n_flow": 16000, "n_seg": 5120, "n_blob": 0},
        # The network of the learned preconditioner, once per GMRES iteration of the 32 x 32 lattice.
        {"name": "mlp forward 1024", "kind": "mlp", "grad": False, "batch": 1024},
        # A training batch of that network: loss and gradients.
        {"name": "mlp gradients 2048", "kind": "mlp", "grad": True, "batch": 2048},
        # One time step of the 16 x 16 array with the line-patch preconditioner, state and forces saved.
        {"name": "step 256", "kind": "step", "n_fil": 256, "n_line": 16, "spacing": 80.0},
        # A sweep: 64 arrays of 16 to 256 cilia stepped together with the block-diagonal preconditioner.
        {"name": "batch 64", "kind": "batch", "n_arrays": 64, "most": 256, "spacing": 80.0},
        # One time step of a free sphere of 256 cilia and 2562 blobs.
        {"name": "swimmer step", "kind": "swim", "n_fil": 256, "n_blob": 2562},
        # One time step of 16 x 16 elastic cilia (forces and torques, Broyden's method).
        {"name": "elastic step", "kind": "elastic", "n_fil": 256, "n_seg": 20, "spacing": 80.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product", "product", "fcm", "flow", "mlp", "step", "batch", "swim", "elastic"])
    if kind == "product":
        wall = rng.random() < 0.5
        return {"kind": kind, "wall": wall, "dof": rng.choice([3, 6]), "n_fil": _log_int(rng, 1, 500),
                "n_seg": rng.randint(5, 25), "n_blob": 0 if wall or rng.random() < 0.3 else _log_int(rng, 100, 6000),
                "host": rng.random() < 0.4}
    if kind == "fcm":
        grid = rng.choice([128, 144, 160, 192, 200, 256, 270, 320, 384])
        radius = round(rng.uniform(0.4, 1.0) * min(100.0, 0.8 * grid - 46.0), 1)
        return {"kind": kind, "n_fil": int(rng.uniform(0.03, 0.1) * radius ** 2), "n_blob": int(radius ** 2),
                "grid": grid, "radius": radius, "host": rng.random() < 0.4}
    if kind == "flow":
        blobs = rng.random() < 0.5
        return {"kind": kind, "n_flow": _log_int(rng, 100, 40000), "n_seg": NSEG * _log_int(rng, 4, 400),
                "n_blob": _log_int(rng, 100, 4000) if blobs else 0}
    if kind == "mlp":
        return {"kind": kind, "grad": rng.random() < 0.5, "batch": _log_int(rng, 16, 8192)}
    if kind == "step":
        line = rng.randint(2, 20)
        return {"kind": kind, "n_fil": line * rng.randint(2, 16), "n_line": line, "spacing": rng.uniform(70.0, 100.0)}
    if kind == "batch":
        return {"kind": kind, "n_arrays": _log_int(rng, 4, 60), "most": rng.randint(32, 240),
                "spacing": rng.uniform(70.0, 100.0)}
    if kind == "swim":
        return {"kind": kind, "n_fil": _log_int(rng, 12, 256), "n_blob": _log_int(rng, 300, 2562)}
    return {"kind": kind, "n_fil": _log_int(rng, 4, 256), "n_seg": rng.randint(13, 20),
            "spacing": rng.uniform(60.0, 100.0)}


# ------------------------------------------------------------------------------------------------ inputs

def _lattice(n_fil, spacing, height):
    return workloads.lattice_bases(n_fil, max(1, math.ceil(math.sqrt(n_fil))), spacing, height)


def _leaning_cilia(n_fil, n_seg, gen):
    """Straight cilia on a wall lattice of spacing 20, each leaning up to 0.15 rad."""
    bases = _lattice(n_fil, 20.0, 2.0)
    lean, turn = gen.uniform(0.0, 0.15, n_fil), gen.uniform(0.0, 2.0 * math.pi, n_fil)
    d = np.stack([np.sin(lean) * np.cos(turn), np.sin(lean) * np.sin(turn), np.cos(lean)], 1)
    return (bases[:, None, :] + 2.2 * np.arange(n_seg)[None, :, None] * d[:, None, :]).reshape(-1, 3)


def _rotation(gen):
    q, r = np.linalg.qr(gen.standard_normal((3, 3)))
    return q * np.sign(np.diag(r))


def _ciliated_sphere(n_fil, n_seg, n_blob, radius, centre, gen):
    """Radial cilia and surface blobs of a sphere in a random orientation: (segments, blobs)."""
    segs, blobs = workloads.sphere_with_cilia(n_fil, n_seg, max(n_blob, 1), radius, centre=(0.0, 0.0, 0.0))
    rot = _rotation(gen)
    c = np.asarray(centre)
    return segs @ rot.T + c, (blobs @ rot.T + c)[:n_blob]


def _particles(case, seed):
    gen = np.random.default_rng(seed)
    f32 = np.float32
    if case["kind"] == "product":
        ns, nb = case["n_fil"] * case["n_seg"], case["n_blob"]
        if case["wall"]:
            x, xb = _leaning_cilia(case["n_fil"], case["n_seg"], gen), np.zeros((0, 3))
        else:
            radius = max(20.0, 0.7 * math.sqrt(max(nb, 40 * case["n_fil"])))
            x, xb = _ciliated_sphere(case["n_fil"], case["n_seg"], nb, radius, (0.0, 0.0, 0.0), gen)
    else:
        nb, ns = case["n_blob"], case["n_fil"] * NSEG
        box = 2.0 * case["grid"]
        x, xb = _ciliated_sphere(case["n_fil"], NSEG, nb, case["radius"], gen.uniform(0.0, box, 3), gen)
    f = gen.standard_normal((ns, 6))
    if case.get("dof") == 3:
        f[:, 3:] = 0.0
    fb = gen.standard_normal((nb, 3))
    return x.astype(f32), f.astype(f32), xb.astype(f32), fb.astype(f32)


def _flow_data(case, seed):
    gen = np.random.default_rng(seed)
    n_seg, n_blob, nf = case["n_seg"], case["n_blob"], case["n_flow"]
    if n_blob:
        x, xb = _ciliated_sphere(n_seg // NSEG, NSEG, n_blob, 60.0, (0.0, 0.0, 0.0), gen)
        xf = gen.uniform(-150.0, 150.0, (nf, 3))
        xf *= np.maximum(1.0, 125.0 / np.linalg.norm(xf, axis=1))[:, None]
    else:
        x, xb = _leaning_cilia(n_seg // NSEG, NSEG, gen), np.zeros((0, 3))
        half = 20.0 * math.sqrt(n_seg / NSEG)
        nx = max(1, int(math.sqrt(1.6 * nf)))
        k = np.arange(nf)
        xf = np.stack([half * (2.0 * (k % nx) / nx - 1.0), np.full(nf, 3.7),
                       50.0 + half * (k // nx) / math.ceil(nf / nx)], 1)
    f32 = np.float32
    return (xf.astype(f32), x.astype(f32), gen.standard_normal((n_seg, 6)).astype(f32), xb.astype(f32),
            gen.standard_normal((n_blob, 3)).astype(f32))


def _mlp_data(case, seed):
    """(parameters W1, b1, W2, b2, W3, b3 flat, features, targets): unit residual rows and shapes in cilium lengths."""
    gen = np.random.default_rng(seed)
    parts = []
    for a, b in ((N_IN, HIDDEN), (HIDDEN, HIDDEN), (HIDDEN, N_OUT)):
        lim = math.sqrt(6.0 / a)
        parts += [gen.uniform(-lim, lim, a * b), gen.normal(0.0, 0.05, b)]
    n = case["batch"]
    n_res = N_IN - 3 * NSEG
    x = np.concatenate([gen.standard_normal((n, n_res)) / math.sqrt(n_res), gen.uniform(-0.5, 1.0, (n, 3 * NSEG))], 1)
    t = gen.standard_normal((n, N_OUT))
    return tuple(a.astype(np.float32) for a in (np.concatenate(parts), x, t))


def _forcing():
    from pathlib import Path
    data = np.load(Path(_lib.LIB_PATH).parent / "data" / "fulford_blake_nseg20_sep2.6.npz")
    return {"phase_refs": data["phase"], "angle_refs": data["angle"],
            "s_table": arclength_table(nseg=NSEG, seg_sep=SEG_SEP, steps=300)}


def prepare(case, seed):
    kind = case["kind"]
    gen = np.random.default_rng(seed)
    if kind in ("product", "fcm"):
        x, f, xb, fb = _particles(case, seed)
        if kind == "product":
            solver = RpyMobilitySolver(len(x), len(xb), wall=case["wall"], seg_dof=case["dof"])
        else:
            g = case["grid"]
            solver = FcmSolver(len(x) + len(xb), rh=1.0, alpha=1.0, beta=10.0, eta=6.0, nx=g, ny=g, nz=g,
                               boxsize=2.0 * g)
            if not case["host"]:
                f = np.ascontiguousarray(f[:, :3])
                x, f = np.concatenate([x, xb]), np.concatenate([f, fb])
        if case["host"]:
            return {"case": case, "solver": solver, "in": (x, f, xb, fb)}
        dev = [torch.as_tensor(a.reshape(-1), device="cuda") for a in (x, f, xb, fb)]
        return {"case": case, "solver": solver, "in": dev,
                "out": (torch.zeros_like(dev[1]), torch.zeros_like(dev[2]))}
    if kind == "flow":
        data = _flow_data(case, seed)
        return {"case": case, "solver": FlowFieldEvaluator(case["n_flow"], case["n_seg"], case["n_blob"]), "in": data}
    if kind == "mlp":
        p, x, t = _mlp_data(case, seed)
        net = FilamentMLP(N_IN, HIDDEN, N_OUT, max_batch=case["batch"])
        net.set_params(p)
        x, t = torch.as_tensor(x, device="cuda"), torch.as_tensor(t, device="cuda")
        return {"case": case, "solver": net, "in": (x, t), "out": torch.zeros_like(t)}
    if kind == "elastic":
        n = case["n_fil"]
        return {"case": case, "nt": 0, "solver": ElasticCiliaSimulation(
            bases=_lattice(n, case["spacing"], 1.3), nseg=case["n_seg"], ic_type=2,
            perturbations=gen.normal(0.0, 1.6, (n, 2, 3)))}
    if kind == "step":
        n = case["n_fil"]
        sim = WallCiliaSimulation(
            bases=workloads.lattice_bases(n, n // case["n_line"], case["spacing"], 0.5 * SEG_SEP), nseg=NSEG,
            seg_sep=SEG_SEP, precond=_lib.CF_PRECOND_LINE, phase0=gen.uniform(0.0, 2.0 * math.pi, n),
            angle0=gen.normal(0.0, 0.05, n), **_forcing())
        pinned = [torch.zeros(n, dtype=torch.float64).pin_memory() for _ in range(4)]
        x = torch.zeros(3 * n * NSEG).pin_memory()
        f = torch.zeros(6 * n * NSEG).pin_memory()
        return {"case": case, "nt": 0, "solver": sim, "state": pinned, "segs": (x, f)}
    if kind == "batch":
        sizes = np.random.default_rng(case["n_arrays"]).integers(16, case["most"] + 1, case["n_arrays"])
        arrays = [{"bases": _lattice(n, case["spacing"], 0.5 * SEG_SEP), "phase0": gen.normal(0.0, 0.05, n)}
                  for n in sizes]
        return {"case": case, "nt": 0, "solver": WallCiliaBatch(arrays, nseg=NSEG, seg_sep=SEG_SEP, **_forcing())}
    n, nb = case["n_fil"], case["n_blob"]
    geo = swim.sphere_geometry(swim.fibonacci_normals(n), swim.fibonacci_normals(nb, 0.3), ar=6.0)
    return {"case": case, "nt": 0, "solver": swim.CiliatedSwimmer(
        geometry=geo, nseg=NSEG, seg_sep=SEG_SEP, phase0=gen.uniform(0.0, 2.0 * math.pi, n),
        angle0=gen.normal(0.0, 0.05, n), **_forcing())}


# ------------------------------------------------------------------------------------------------ one pass

def _single(d):
    """Results of a time step as they are handed on for files and plots: single precision, that of the pair sums."""
    if isinstance(d, dict):
        return {k: _single(v) for k, v in d.items()}
    if isinstance(d, (list, tuple)):
        return [_single(v) for v in d]
    return np.asarray(d, np.float32)


def run(state):
    case, s = state["case"], state["solver"]
    kind = case["kind"]
    if kind == "product":
        x, f, xb, fb = state["in"]
        if case["host"]:
            return s.apply(x, f, xb, fb)
        v, vb = state["out"]
        s.apply_device(x, f, v, xb, fb, vb)
        return v, vb
    if kind == "fcm":
        if case["host"]:
            return s.evaluate_full_mobility(*state["in"])
        s.apply_device(state["in"][0], state["in"][1], state["out"][0])
        return state["out"][0]
    if kind == "flow":
        xf, x, f, xb, fb = state["in"]
        if len(xb):
            return s.velocities(xf, x, f, x_blobs=xb, f_blobs=fb, n_blob_per_body=len(xb))
        return s.velocities(xf, x, f)
    if kind == "mlp":
        if case["grad"]:
            return s.gradients(*state["in"])
        s.forward(state["in"][0], state["out"], stream=torch.cuda.current_stream())
        return state["out"]
    nt = state["nt"]
    state["nt"] = nt + 1
    if kind == "step":
        s.step_io(nt, state_out=state["state"], x_segs=state["segs"][0], f_segs=state["segs"][1])
        return list(state["segs"]) + [v.float() for v in state["state"]]
    s.step(nt)
    if kind == "batch":
        return _single([np.concatenate(s.segments()), {k: np.concatenate([a[k] for a in s.state()])
                                                       for k in ("phase", "angle", "phase_dot", "angle_dot")}])
    if kind == "swim":
        return _single([s.state(), s.particles()])
    return _single(s.segments())


# ------------------------------------------------------------------------------------------------ work

def work(case):
    """Inputs read once, outputs written once; operations by the fixed counts below (one pair: one ordered
    3 x 3 block 150 near a wall, 40 without one, twice that with torques; one flow term 60)."""
    kind = case["kind"]

    def product(n, wall=True, dof=3):
        return n * n * (150.0 if wall else 40.0) * (1 if dof == 3 else 2)

    if kind == "product":
        n, b = case["n_fil"] * case["n_seg"], case["n_blob"]
        return {"bytes": 4.0 * (15 * n + 9 * b), "flops": product(n + b, case["wall"], case["dof"])}
    if kind == "fcm":
        n, m = case["n_fil"] * NSEG + case["n_blob"], float(case["grid"]) ** 3
        # spreading and gathering 10^3 points each, six real transforms, the projector
        return {"bytes": 36.0 * n, "flops": n * 1000 * 14.0 + 6 * 2.5 * m * math.log2(m) + 12 * m}
    if kind == "flow":
        n = case["n_seg"] + case["n_blob"]
        return {"bytes": 24.0 * case["n_flow"] + 36.0 * n, "flops": 60.0 * case["n_flow"] * n}
    if kind == "mlp":
        p = N_IN * HIDDEN + HIDDEN * HIDDEN + HIDDEN * N_OUT
        n = case["batch"]
        if case["grad"]:
            return {"bytes": 4.0 * (2 * p + n * (N_IN + N_OUT)), "flops": 6.0 * n * p - 2.0 * n * N_IN * HIDDEN}
        return {"bytes": 4.0 * (p + n * (N_IN + N_OUT)), "flops": 2.0 * n * p}
    if kind == "step":  # the patch inverses and one product per iteration, four of them
        n, line = case["n_fil"], case["n_line"]
        lines = n / line
        return {"bytes": 4.0 * n * (9 * NSEG + 16), "flops": 2.0 * lines * (62.0 * line) ** 3 + 4 * product(n * NSEG)}
    if kind == "batch":  # one product per iteration, eight of them, of arrays of mean size
        n = 0.5 * (16 + case["most"])
        return {"bytes": case["n_arrays"] * 8.0 * n * (3 * NSEG + 8),
                "flops": case["n_arrays"] * 8 * product(n * NSEG)}
    if kind == "swim":
        n = case["n_fil"] * NSEG + case["n_blob"]
        return {"bytes": 8.0 * 6 * n, "flops": 8 * product(n, False)}
    n = case["n_fil"] * case["n_seg"]
    return {"bytes": 8.0 * 13 * n, "flops": 3 * product(n, True, 6) + case["n_fil"] * 2.0 * (6 * case["n_seg"]) ** 3}


# ------------------------------------------------------------------------------------------------ in 64 bits

_PI = math.pi


def _wall_block(xi, xj, f):
    """Velocities and spins of targets [m, 1, 3] from unit spheres [1, n, 3] above the wall z = 0, without the
    diagonal; f [1, n, 6]."""
    F, T = f[..., :3], f[..., 3:]
    d = xi - xj
    r = d.norm(dim=-1, keepdim=True)
    self_pair = r == 0
    r = torch.where(self_pair, torch.ones_like(r), r)
    u = d / r
    uf, ut = (u * F).sum(-1, keepdim=True), (u * T).sum(-1, keepdim=True)
    v = ((1 + 2 / (3 * r * r)) * F + (1 - 2 / (r * r)) * uf * u) / (8 * _PI * r)
    v = v + torch.linalg.cross(T.expand_as(u), u) / (8 * _PI * r * r)
    w = torch.linalg.cross(F.expand_as(u), u) / (8 * _PI * r * r) + (3 * ut * u - T) / (16 * _PI * r ** 3)

    R = torch.cat([d[..., :2], xi[..., 2:] + xj[..., 2:]], -1)
    s = 1 / R.norm(dim=-1, keepdim=True)
    e = R * s
    ez, h = e[..., 2:], xj[..., 2:] / R[..., 2:]
    ez2, g = ez * ez, 1 - h
    Fz, ef = F[..., 2:], (e * F).sum(-1, keepdim=True)
    z = torch.zeros_like(e)
    z[..., 2] = 1
    k0 = -(0.75 * s * (1 + 2 * h * g * ez2) + 0.5 * (s ** 3 * (1 - 3 * ez2) - s ** 5 * (1 - 5 * ez2)))
    k1 = -(0.75 * s * (1 - 6 * h * g * ez2) - 1.5 * s ** 3 * (1 - 5 * ez2) + 2.5 * s ** 5 * (1 - 7 * ez2))
    k2 = ez * (1.5 * h * s * (1 - 6 * g * ez2) - 3 * s ** 3 * (1 - 5 * ez2) + 5 * s ** 5 * (2 - 7 * ez2))
    k3 = 1.5 * h * s - 5 * s ** 5
    k4 = -((3 * h * h * s + 3 * s ** 3) * ez2 + (2 - 15 * ez2) * s ** 5)
    img = k0 * F + (k1 * ef + k2 * Fz) * e + (k3 * ef * ez + k4 * Fz) * z

    def spin(e, F, h):  # spin of the target from a force on the image's source
        c = 0.75 * s * s
        b = F[..., 2:] * (9 * h * ez2 * s * s + (1.5 - 15 * ez2) * s ** 4) - ez * (e * F).sum(-1, keepdim=True) * (
            4.5 * h * s * s - 7.5 * s ** 4)
        q = -1.5 * ez * (h * s * s - s ** 4)
        return -c * torch.linalg.cross(F.expand_as(e), e) - b * torch.linalg.cross(z, e) - q * torch.linalg.cross(
            F.expand_as(e), z)

    rot = spin(e, F, h)
    Tx, Ty = T[..., 0:1], T[..., 1:2]
    et = (e * T).sum(-1, keepdim=True)
    curl = e[..., 0:1] * Ty - e[..., 1:2] * Tx
    flat = torch.cat([-e[..., 1:2], e[..., 0:1], torch.zeros_like(ez)], -1)
    rot = rot + s ** 3 * ((0.375 - 2.25 * ez2) * T - 1.125 * et * e + 2.25 * ez * et * z + 2.25 * curl * flat)
    # velocity from a torque: the transpose of the spin block seen from the source
    back = torch.cat([-e[..., :2], ez], -1)
    p = 0.75 * s * s
    ez_t = torch.linalg.cross(z, back)
    along = (ez_t * T).sum(-1, keepdim=True)
    b1 = (9 * g * ez2 * s * s + (1.5 - 15 * ez2) * s ** 4) * along
    b2 = -ez * (4.5 * g * s * s - 7.5 * s ** 4) * along
    b3 = -1.5 * ez * (g * s * s - s ** 4)
    vel = -p * torch.linalg.cross(back, T.expand_as(back)) - b1 * z - b2 * back - b3 * torch.linalg.cross(
        z, T.expand_as(z))
    v = v + (img + vel) / (6 * _PI)
    w = w + rot / (6 * _PI)
    return torch.where(self_pair, torch.zeros_like(v), v), torch.where(self_pair, torch.zeros_like(w), w)


def _wall_self(x, f):
    h = 1 / x[:, 2:]
    c6, c8 = 1 / (6 * _PI), 1 / (8 * _PI)
    F, T = f[:, :3], f[:, 3:]
    flat = torch.tensor([1.0, 1.0, 0.0], dtype=x.dtype, device=x.device)
    up = 1 - flat
    par = c6 * (1 - (9 * h - 2 * h ** 3 + h ** 5) / 16)
    perp = c6 * (1 - (9 * h - 4 * h ** 3 + h ** 5) / 8)
    tr = 3 / 32 * c6 * h ** 4
    z = up.expand_as(F)
    v = (par * flat + perp * up) * F - tr * torch.linalg.cross(z, T)
    w = tr * torch.linalg.cross(z, F)
    w = w + ((c8 - 15 / 64 * c6 * h ** 3) * flat + (c8 - 3 / 32 * c6 * h ** 3) * up) * T
    return v, w


def _free_block(xi, xj, f):
    """The same for unit spheres without a wall; touching and coincident spheres included."""
    F, T = f[..., :3], f[..., 3:]
    d = xi - xj
    r = d.norm(dim=-1, keepdim=True)
    one = torch.where(r == 0, torch.ones_like(r), r)
    u = d / one
    far = r > 2
    uf, ut = (u * F).sum(-1, keepdim=True), (u * T).sum(-1, keepdim=True)
    a = torch.where(far, (1 + 2 / (3 * one * one)) / (8 * _PI * one), (1 - 9 / 32 * r) / (6 * _PI))
    b = torch.where(far, (1 - 2 / (one * one)) / (8 * _PI * one), 3 / 32 * r / (6 * _PI))
    c = torch.where(far, 1 / (8 * _PI * one * one), r * (1 - 3 / 8 * r) / (16 * _PI))
    p = torch.where(far, -1 / (16 * _PI * one ** 3), (1 - 27 / 32 * r + 5 / 64 * r ** 3) / (8 * _PI))
    q = torch.where(far, 3 / (16 * _PI * one ** 3), (9 / 32 * r - 3 / 64 * r ** 3) / (8 * _PI))
    v = a * F + b * uf * u + c * torch.linalg.cross(T.expand_as(u), u)
    w = c * torch.linalg.cross(F.expand_as(u), u) + p * T + q * ut * u
    return v, w


def _exact_product(case, seed):
    x, f, xb, fb = (torch.as_tensor(a, device="cuda").double() for a in _particles(case, seed))
    n, dof = len(x), case["dof"]
    X = torch.cat([x, xb])
    Fa = torch.cat([f, torch.cat([fb, torch.zeros_like(fb)], 1)])
    v, w = torch.zeros_like(X), torch.zeros_like(X)
    block = _wall_block if case["wall"] else _free_block
    rows = max(1, (1 << 22) // len(X))
    for i in range(0, len(X), rows):
        a, b = block(X[i:i + rows, None], X[None], Fa[None])
        v[i:i + rows], w[i:i + rows] = a.sum(1), b.sum(1)
    if case["wall"]:
        a, b = _wall_self(X, Fa)
        v, w = v + a, w + b
    spins = w[:n] if dof == 6 else torch.zeros_like(w[:n])
    return torch.cat([v[:n], spins], 1).reshape(-1), v[n:].reshape(-1)


def _exact_fcm(case, seed):
    """The force-coupling method as defined (truncated kernels on the grid, corrections within the cut-off)."""
    x, f, xb, fb = (torch.as_tensor(a, device="cuda").double() for a in _particles(case, seed))
    X, F = torch.cat([x, xb]), torch.cat([f[:, :3], fb])
    g, ngd, dx = case["grid"], 10, 2.0
    box = g * dx
    X = X - torch.floor(X / box) * box
    sig, Sig = 1 / math.sqrt(_PI), dx
    pd = sig ** 2 - Sig ** 2
    off = torch.arange(ngd, device="cuda") - ngd // 2
    V = torch.zeros_like(X)

    def support(lo, hi):
        at = torch.round(X[lo:hi] / dx)[:, :, None] + off  # [m, 3, ngd]
        y = at * dx - X[lo:hi, :, None]
        e = torch.exp(-y * y / (2 * Sig * Sig)) / math.sqrt(2 * _PI * Sig * Sig)
        r2 = (y * y)[:, 0, None, None, :] + (y * y)[:, 1, None, :, None] + (y * y)[:, 2, :, None, None]
        wgt = e[:, 0, None, None, :] * e[:, 1, None, :, None] * e[:, 2, :, None, None] * (
            1 - 1.5 * pd / Sig ** 2 + 0.5 * pd / Sig ** 4 * r2)
        at = torch.remainder(at, g).long()
        ind = at[:, 0, None, None, :] + g * at[:, 1, None, :, None] + g * g * at[:, 2, :, None, None]
        return wgt.reshape(hi - lo, -1), ind.reshape(hi - lo, -1)

    spec = []
    step = 4096
    for c in range(3):
        grid = torch.zeros(g ** 3, dtype=torch.float64, device="cuda")
        for lo in range(0, len(X), step):
            hi = min(len(X), lo + step)
            wgt, ind = support(lo, hi)
            grid.index_add_(0, ind.reshape(-1), (wgt * F[lo:hi, c, None]).reshape(-1))
        spec.append(torch.fft.rfftn(grid.view(g, g, g)))
    k = 2 * _PI / box * torch.fft.fftfreq(g, 1.0 / g, device="cuda", dtype=torch.float64)
    kr = 2 * _PI / box * torch.arange(g // 2 + 1, device="cuda", dtype=torch.float64)
    k[g // 2] = abs(k[g // 2])  # the Nyquist planes count as positive frequencies
    q = (kr[None, None, :], k[None, :, None], k[:, None, None])
    qq = q[0] ** 2 + q[1] ** 2 + q[2] ** 2
    qq[0, 0, 0] = 1
    dot = (q[0] * spec[0] + q[1] * spec[1] + q[2] * spec[2]) / qq
    for c in range(3):
        spec[c] = (spec[c] - q[c] * dot) / qq
        spec[c][0, 0, 0] = 0
    del dot, qq
    for c in range(3):
        u = torch.fft.irfftn(spec[c], s=(g, g, g)).reshape(-1)
        for lo in range(0, len(X), step):
            hi = min(len(X), lo + step)
            wgt, ind = support(lo, hi)
            V[lo:hi, c] = (u[ind] * wgt).sum(1) * dx ** 3

    def pair(r, s2):
        erf, gauss = torch.erf(r / math.sqrt(2 * s2)), torch.exp(-r * r / (2 * s2)) / (2 * _PI * s2) ** 1.5
        a = (1 + s2 / r ** 2) * erf / (8 * _PI * r) - 0.5 * s2 * s2 / r ** 2 * gauss
        b = (1 - 3 * s2 / r ** 2) * erf / (8 * _PI * r ** 3) + 1.5 * s2 * s2 / r ** 4 * gauss
        return a, b, erf, gauss

    cut = 6.0 * dx
    for lo in range(0, len(X), 2048):
        d = X[lo:lo + 2048, None] - X[None]
        d -= box * torch.trunc(d / (0.5 * box))
        r = d.norm(dim=-1)
        i, j = torch.nonzero((r < cut) & (r > 0), as_tuple=True)
        d, r = d[i, j], r[i, j][:, None]
        av, bv, _, _ = pair(r, 2 * sig * sig)
        s2 = 2 * Sig * Sig
        a, b, erf, gauss = pair(r, s2)
        qi = erf / (4 * _PI * r ** 3) - (1 + s2 / r ** 2) * gauss
        qx = -3 * erf / (4 * _PI * r ** 5) + (1 + 3 * s2 / r ** 2) / r ** 2 * gauss
        ti, tx = (2 - r ** 2 / s2) / s2 * gauss, gauss / (s2 * s2)
        t1, t2 = av - a - qi * pd - ti * pd * pd / 4, bv - b - qx * pd - tx * pd * pd / 4
        V.index_add_(0, lo + i, t1 * F[j] + t2 * d * (d * F[j]).sum(-1, keepdim=True))
    root = math.sqrt(_PI)
    own = 1 / (6 * _PI) - 1 / (6 * _PI * Sig * root) + pd / (12 * (root * Sig) ** 3) - pd * pd / (
        32 * _PI ** 1.5 * Sig ** 5)
    V = V + own * F
    if not case["host"]:
        return V.reshape(-1)
    n = len(x)
    return torch.cat([V[:n], torch.zeros_like(V[:n])], 1).reshape(-1), V[n:].reshape(-1)


def _exact_flow(case, seed):
    xf, x, f, xb, fb = (torch.as_tensor(a, device="cuda").double() for a in _flow_data(case, seed))
    out = torch.zeros_like(xf)

    def stokeslet(d, F):
        r = d.norm(dim=-1, keepdim=True)
        return F / r + d * (d * F).sum(-1, keepdim=True) / r ** 3

    for lo in range(0, len(xf), max(1, (1 << 22) // len(x))):
        hi = min(len(xf), lo + max(1, (1 << 22) // len(x)))
        p = xf[lo:hi, None]
        d, F, T = p - x[None], f[None, :, :3], f[None, :, 3:]
        r = d.norm(dim=-1, keepdim=True)
        v = stokeslet(d, F) + torch.linalg.cross(T.expand_as(d), d) / r ** 3
        if not len(xb):  # a no-slip wall at z = 0
            D = torch.cat([d[..., :2], p[..., 2:] + x[None, :, 2:]], -1)
            R = D.norm(dim=-1, keepdim=True)
            v = v - stokeslet(D, F)
            h, X3 = x[None, :, 2:], D[..., 2:]
            z = p[..., 2:]
            mirror = torch.cat([F[..., :2], -F[..., 2:]], -1)
            a = (D * mirror).sum(-1, keepdim=True)
            e3 = torch.zeros_like(D)
            e3[..., 2] = 1
            # the source doublet and the Stokes doublet of the image, at the field height z
            v = v + 2 * h / R ** 5 * (z * (3 * a * D - R ** 2 * mirror) + R ** 2 * (
                (D * F).sum(-1, keepdim=True) - X3 * F[..., 2:]) * e3
                + R ** 2 * F[..., 2:] * torch.cat([d[..., :2], torch.zeros_like(X3)], -1))
        out[lo:hi] = v.sum(1)
        if len(xb):
            out[lo:hi] += stokeslet(p - xb[None], fb[None]).sum(1)
    return out / (8 * _PI)


def _exact_mlp(case, seed):
    p, x, t = (torch.as_tensor(a, device="cuda").double() for a in _mlp_data(case, seed))
    parts, o = [], 0
    for a, b in ((N_IN, HIDDEN), (HIDDEN, HIDDEN), (HIDDEN, N_OUT)):
        parts += [p[o:o + a * b].view(a, b).clone().requires_grad_(),
                  p[o + a * b:o + a * b + b].clone().requires_grad_()]
        o += a * b + b
    y = torch.relu(x @ parts[0] + parts[1])
    y = torch.relu(y @ parts[2] + parts[3])
    y = y @ parts[4] + parts[5]
    if not case["grad"]:
        return y.detach()
    loss = (y - t).square().mean()
    loss.backward()
    return float(loss.detach()), torch.cat([a.grad.reshape(-1) for a in parts])


def exact(case, seed):
    """What run() gives, from the definitions in 64 bits.  A time step's solver stops at its tolerance: the iterate
    it returns has no value of its own in more bits."""
    made = {"product": _exact_product, "fcm": _exact_fcm, "flow": _exact_flow, "mlp": _exact_mlp}.get(case["kind"])
    return made(case, seed) if made else None
