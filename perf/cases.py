"""Workloads that the speed of this framework is measured on: frames of the two simulators at the sizes of the
application's menu and of the benchmark, the renderer, batched rollouts and the two differentiable uses.

    listed(), draw(rng)      the cases, as dicts of plain values
    prepare(case, seed)      what a program holds before the call: simulators, renderers, device buffers, host inputs
    run(state)               one pass through the public entry points; its outputs
    work(case)               bytes and operations that one pass cannot do without
    exact(case, seed)        the same outputs from plain torch in 64 bits, where that is quick enough
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

from __graft_entry__ import load_package  # noqa: E402  (the package's directory name is not an identifier)

FOV = 45 * math.pi / 180
MPM_RADIUS, MPM_DIAMETER = 0.6, 1.2


def listed():
    return [
        # The smallest interactive scene: a frame is a few microseconds of arithmetic, so launches decide.
        {"name": "mpm_3k_frame", "kind": "mpm", "n": 3001, "x": 24, "y": 20, "z": 28, "wall": False, "w": 0, "h": 0},
        # The application's default scene and its whole frame: box size, two substeps, fluid image at its canvas.
        {"name": "mpm_70k_app_frame", "kind": "mpm", "n": 70000, "x": 40, "y": 30, "z": 60, "wall": False, "w": 896, "h": 504},
        # The application's largest scene while the user drags the box slider: the wall moves on every frame.
        {"name": "mpm_200k_wall_frame", "kind": "mpm", "n": 200000, "x": 50, "y": 50, "z": 80, "wall": True, "w": 0, "h": 0},
        # The benchmark's scene: a million particles on a 128^3 grid, one frame.
        {"name": "mpm_1m_frame", "kind": "mpm", "n": 1000000, "x": 128, "y": 128, "z": 128, "wall": False, "w": 0, "h": 0},
        # Data generation: 64 scenes of uneven sizes restarted from host records and rolled out 100 substeps.
        {"name": "batch_64_rollout", "kind": "batch", "scenes": 64, "lo": 4000, "hi": 64000, "substeps": 100},
        # Differentiable simulation with the default tape: forward, centroid loss, backward.
        {"name": "adjoint_32k_fp64", "kind": "adjoint", "n": 32768, "side": 48, "substeps": 40, "every": 10, "tape": "fp64"},
        # One iteration of the batched inverse problem on the solver's own trajectory, every substep taped.
        {"name": "inverse_64_step", "kind": "inverse", "scenes": 64, "lo": 16000, "hi": 32000, "substeps": 40, "every": 1},
        # The renderer alone: the sphere view of the default scene, and the fluid view of the benchmark's scene.
        {"name": "render_70k_spheres", "kind": "render", "n": 70000, "x": 40, "y": 30, "z": 60, "w": 896, "h": 504, "spheres": True, "dist": 70.0},
        {"name": "render_1m_fluid", "kind": "render", "n": 1000000, "x": 128, "y": 128, "z": 128, "w": 1344, "h": 756, "spheres": False, "dist": 160.0},
        # The second simulator: its smallest and largest menu entries, and the benchmark's large scene.
        {"name": "sph_10k_frame", "kind": "sph", "n": 10000, "hx": 0.7, "hy": 2.0, "hz": 0.7},
        {"name": "sph_40k_frame", "kind": "sph", "n": 40000, "hx": 1.4, "hy": 2.0, "hz": 1.4},
        {"name": "sph_400k_frame", "kind": "sph", "n": 400000, "hx": 1.9, "hy": 2.0, "hz": 1.9},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box_for(rng, n):
    """A box that a dam-break block of n particles fills to a third or so, sides odd and even alike."""
    side = (n / 4.0 * 6.0) ** (1.0 / 3.0)
    return [max(16, min(128, int(side * rng.uniform(0.85, 1.3)) + 6)) for _ in range(3)]


def draw(rng):
    kind = rng.choice(["mpm", "mpm", "mpm", "batch", "adjoint", "inverse", "render", "render", "sph", "sph", "sph"])
    if kind == "mpm":
        n = _log_int(rng, 1500, 700000)
        x, y, z = _box_for(rng, n)
        image = n <= 200000 and rng.random() < 0.4
        return {"kind": kind, "n": n, "x": x, "y": y, "z": z, "wall": rng.random() < 0.3,
                "w": rng.randint(300, 1344) if image else 0, "h": rng.randint(200, 756) if image else 0}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(3, 60), "lo": 4000, "hi": rng.randint(8000, 64000), "substeps": rng.randint(10, 100)}
    if kind == "adjoint":
        return {"kind": kind, "n": _log_int(rng, 2000, 32000), "side": rng.randint(40, 56), "substeps": rng.randint(5, 40),
                "every": rng.randint(1, 20), "tape": rng.choice(["fp64", "fp64", "fixed"])}
    if kind == "inverse":
        every = rng.choice([1, 10])
        return {"kind": kind, "scenes": rng.randint(3, 48), "lo": 8000, "hi": rng.randint(12000, 32000),
                "substeps": 10 * rng.randint(1, 4), "every": every}
    if kind == "render":
        n = _log_int(rng, 5000, 800000)
        x, y, z = _box_for(rng, n)
        return {"kind": kind, "n": n, "x": x, "y": y, "z": z, "w": rng.randint(300, 1344), "h": rng.randint(200, 756),
                "spheres": rng.random() < 0.4, "dist": round(1.25 * max(x, y, z) * rng.uniform(0.9, 1.3), 2)}
    n = _log_int(rng, 2000, 380000)
    # the menu's boxes grow with the particle count so that a column stays about as high
    h = min(1.9, max(0.5, 0.7 * math.sqrt(n / 10000.0) * rng.uniform(0.8, 1.1)))
    return {"kind": kind, "n": n, "hx": round(h, 3), "hy": 2.0, "hz": round(min(1.9, h * rng.uniform(0.9, 1.2)), 3)}


# ---------------------------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------------------------

def _dambreak(n, box, seed):
    """(n', 20) records of a block at one end of the box, filled layer by layer from the floor: lattice spacing
    0.65 and one random shift of up to 2 for all three axes of a particle, as the application's reset() makes it."""
    y = np.arange(0.0, box[1] * 0.8, 0.65)
    x = np.arange(3.0, box[0] - 4, 0.65)
    z = np.arange(3.0, box[2] / 2, 0.65)
    p = np.stack(np.meshgrid(y, x, z, indexing="ij"), axis=-1).reshape(-1, 3)[:n, [1, 0, 2]]
    rec = np.zeros((len(p), 20), np.float32)
    rec[:, 0:3] = p + 2.0 * np.random.default_rng(seed).random((len(p), 1))
    return rec


def _lattice(n, origin, seed):
    """(n, 20) records: the first n points of a cubic lattice of spacing 0.5, jittered by 0.05."""
    a = round(n ** (1.0 / 3.0))
    while a ** 3 < n:
        a += 1
    i = np.arange(n)
    p = np.stack([i // (a * a), (i // a) % a, i % a], axis=1) * 0.5 + origin
    rec = np.zeros((n, 20), np.float32)
    rec[:, 0:3] = p + 0.05 * (2.0 * np.random.default_rng(seed).random((n, 3)) - 1.0)
    return rec


def _mpm_records(case, seed):
    box = [float(case["x"]), float(case["y"]), float(case["z"])]
    # The application's scenes are shifted lattices; the benchmark's is the jittered one, from one corner.
    if case["n"] > 200000:
        rec = _lattice(case["n"], 4.0, seed)
        return rec[(rec[:, 0:3] < np.array(box) - 4.0).all(axis=1)], box
    return _dambreak(case["n"], box, seed), box


def _pool(case, seed):
    """(n, 8) posvel records of a pool with waves at rest density (4 particles per cell) and its velocities."""
    rng = np.random.default_rng(seed)
    n, sx, sz = case["n"], case["x"] - 6.0, case["z"] - 6.0
    p = rng.random((n, 3)) * np.array([sx, 1.0, sz]) + 3.0
    depth = n / 4.0 / (sx * sz)
    wave = 1.0 + 0.35 * np.sin(2 * math.pi * (p[:, 0] / sx + rng.random())) * np.cos(2 * math.pi * (p[:, 2] / sz + rng.random()))
    pv = np.zeros((n, 8), np.float32)
    pv[:, 0], pv[:, 2] = p[:, 0], p[:, 2]
    pv[:, 1] = np.minimum(3.0 + (p[:, 1] - 3.0) * depth * wave, case["y"] - 3.0)
    pv[:, 4:7] = rng.normal(0.0, 0.5, (n, 3))
    return pv


def _sph_records(case, seed):
    """(n, 16) records: half of the box filled from the floor, spacing half a kernel radius, as reset() makes it."""
    h, step = (case["hx"], case["hy"], case["hz"]), 0.035
    x = np.arange(-0.95 * h[0], 0.95 * h[0], step)
    z = np.arange(-0.95 * h[2], 0.0, step)
    layers = -(-case["n"] // (len(x) * len(z)))
    y = -0.95 * h[1] + step * np.arange(layers)
    p = np.stack(np.meshgrid(y, x, z, indexing="ij"), axis=-1).reshape(-1, 3)[:case["n"], [1, 0, 2]]
    rec = np.zeros((len(p), 16), np.float32)
    rec[:, 0:3] = p + 0.001 * np.random.default_rng(seed).random((len(p), 1))
    return rec


def _camera(pkg, case):
    """The application's orbit camera, looking at the lower half of the box."""
    box = (case["x"], case["y"], case["z"])
    dist = case.get("dist") or 1.17 * max(box)
    return pkg.camera_uniforms(case["w"], case["h"], dist, [box[0] / 2.0, box[1] / 4.0, box[2] / 2.0], FOV, MPM_DIAMETER)


class _DeviceImage:
    """The renderer's colour buffer for torch (the array interface of a device pointer); the renderer, which owns
    the memory, lives as long as a tensor of it."""

    def __init__(self, renderer):
        self.renderer = renderer
        self.__cuda_array_interface__ = {"data": (renderer.colorDevicePtr(), False), "typestr": "<f4", "version": 2,
                                         "shape": (renderer.height, renderer.width, 4)}


def _renderer(pkg, case):
    r = pkg.FluidRenderer(case["w"], case["h"], MPM_RADIUS, FOV)
    return r, torch.as_tensor(_DeviceImage(r), device="cuda"), _camera(pkg, case)


def _walls(box):
    """The box widths of a slider dragged to 70 % and back, one per frame, at the application's closing speed."""
    steps = [1.0 - 0.007 * k for k in range(44)]
    return [[box[0], box[1], box[2] * r] for r in steps + steps[::-1]]


# ---------------------------------------------------------------------------------------------------------------
# State and passes
# ---------------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    pkg = load_package()
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "mpm":
        rec, box = _mpm_records(case, seed)
        s["posvel"] = torch.zeros((len(rec), 8), dtype=torch.float32, device="cuda")
        s["sim"] = pkg.MLSMPMSimulator(None, s["posvel"], MPM_DIAMETER, maxParticles=len(rec),
                                       maxGrid=tuple(int(b) for b in box))
        s["sim"].upload(rec, box)
        s["boxes"] = _walls(box) if case["wall"] else ([box] if case["w"] else None)
        s["frame"] = 0
        s["renderer"] = None
        if case["w"]:
            s["renderer"], s["image"], s["camera"] = _renderer(pkg, case)
    elif kind == "sph":
        rec = _sph_records(case, seed)
        half = [case["hx"], case["hy"], case["hz"]]
        s["posvel"] = torch.zeros((len(rec), 8), dtype=torch.float32, device="cuda")
        s["sim"] = pkg.SPHSimulator(None, s["posvel"], 0.08, maxParticles=len(rec))
        s["sim"].upload(rec, half)
        s["half"] = half
    elif kind == "render":
        s["posvel"] = torch.from_numpy(_pool(case, seed)).cuda()
        s["renderer"], s["image"], s["camera"] = _renderer(pkg, case)
        s["spheres"] = case["spheres"]
    elif kind == "batch":
        # the case has its scenes (sizes, boxes, constants); the seed shifts every particle
        descs, s["rec"] = pkg.batch_scenes(case["scenes"], seed=case["scenes"], n_range=(case["lo"], case["hi"]))
        s["rec"][:, 0:3] += 0.04 * np.random.default_rng(seed).random((len(s["rec"]), 3)).astype(np.float32) - 0.02
        s["batch"] = pkg.MLSMPMBatch(descs, s["rec"])
        s["substeps"] = case["substeps"]
    elif kind == "adjoint":
        s["rec"] = _adjoint_records(case, seed)
        box = [float(case["side"])] * 3
        s["adj"] = pkg.MLSMPMAdjoint([pkg.scene_desc(len(s["rec"]), box)], case["substeps"], case["every"], tape=case["tape"])
        s["substeps"], s["centroid_loss"] = case["substeps"], pkg.centroid_loss
    else:
        hidden, s["rec"], _ = pkg.inverse.inverse_scenes(case["scenes"], seed=seed, n_range=(case["lo"], case["hi"]))
        adj = pkg.MLSMPMAdjoint(hidden, case["substeps"], case["every"], tape="fixed")
        steps = list(range(10, case["substeps"] + 1, 10))
        adj.setObservations(pkg.inverse.observe(adj, s["rec"], case["substeps"], steps))
        s["guess"] = [pkg.inverse.with_constants(d, 3.0, 0.1) for d in hidden]
        s["adj"], s["substeps"] = adj, case["substeps"]
    return s


def _adjoint_records(case, seed):
    rec = _lattice(case["n"], 8.0, seed)
    rec[:, 4:7] = np.random.default_rng(seed + 1).normal(0.0, 0.1, (len(rec), 3))
    return rec


def run(s):
    kind = s["kind"]
    if kind == "mpm":
        stream = torch.cuda.current_stream()
        if s["boxes"]:
            s["sim"].changeBoxSize(s["boxes"][s["frame"] % len(s["boxes"])])
            s["frame"] += 1
        s["sim"].execute(stream)
        if s["renderer"] is None:
            return s["posvel"]
        s["renderer"].execute(s["posvel"], s["sim"].numParticles, s["camera"], stream)
        return {"posvel": s["posvel"], "image": s["image"]}
    if kind == "sph":
        s["sim"].changeBoxSize(s["half"])
        s["sim"].execute(torch.cuda.current_stream())
        return s["posvel"]
    if kind == "render":
        s["renderer"].execute(s["posvel"], len(s["posvel"]), s["camera"], torch.cuda.current_stream(), sphereRenderFl=s["spheres"])
        return s["image"]
    if kind == "batch":
        s["batch"].upload(s["rec"])
        s["batch"].step(s["substeps"])
        return s["batch"].downloadParticles()
    if kind == "adjoint":
        s["adj"].forward(s["rec"], s["substeps"])
        state = s["adj"].state(s["substeps"])
        loss, seed = s["centroid_loss"](state, [30.0, 10.0, 30.0])
        grad, grad_params = s["adj"].backward({s["substeps"]: seed})
        return {"state": state, "loss": loss, "grad": grad, "grad_params": grad_params}
    for i, d in enumerate(s["guess"]):
        s["adj"].setScene(i, d)
    s["adj"].forward(s["rec"], s["substeps"])
    loss = s["adj"].observationLoss()
    _, grad_params = s["adj"].backwardObserved(grad_init=False)
    return {"loss": loss, "grad_params": grad_params}


# ---------------------------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------

def work(case):
    """Bytes: inputs read once and outputs written once: a particle's state (64 B) and its posvel record (32 B) for a
    frame, 80-byte records for host states, gradients and tapes' ends, 12 bytes for an observed position, 20 bytes a
    pixel for an image.  Operations: per particle and substep of MPM 27 cells x (p2g_1 20, p2g_2 35, g2p 30), of its
    adjoint three times that, of SPH about 30 neighbours x 60; per pixel of a fluid image the filters' taps x 30."""
    kind = case["kind"]
    per_substep = 27 * 85.0
    pixels = float(case.get("w", 0) * case.get("h", 0))
    fluid = {"bytes": 20.0 * pixels, "flops": pixels * 8 * 17 * 30}
    if kind == "mpm":
        n = len(_mpm_records(case, 0)[0])
        return {"bytes": n * (2 * 64 + 32.0) + fluid["bytes"], "flops": 2 * n * per_substep + fluid["flops"]}
    if kind == "sph":
        return {"bytes": case["n"] * (2 * 32 + 32.0), "flops": 2 * case["n"] * 30 * 60.0}
    if kind == "render":
        return {"bytes": 32.0 * case["n"] + fluid["bytes"], "flops": pixels * 100 if case["spheres"] else fluid["flops"]}
    t = case["substeps"]
    if kind == "adjoint":
        return {"bytes": case["n"] * 4 * 80.0, "flops": 4 * t * case["n"] * per_substep}
    n = case["scenes"] * (case["lo"] + case["hi"]) / 2.0
    if kind == "batch":
        return {"bytes": n * 2 * 80.0, "flops": t * n * per_substep}
    return {"bytes": n * (80.0 + 12 * (t // 10)), "flops": 4 * t * n * per_substep}


# ---------------------------------------------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _mpm_substep(x, v, C, init, real, k, mu):
    """One substep of the continuous model (no fixed point): positions, velocities and C as (n, 3, 3) matrices."""
    rest, dt, gravity = 4.0, float(np.float32(0.2)), float(np.float32(-0.3))
    Y, Z = int(init[1]), int(init[2])
    cells = int(math.ceil(init[0])) * int(math.ceil(init[1])) * int(math.ceil(init[2]))
    base = torch.floor(x)
    d = x - (base + 0.5)
    w = torch.stack([0.5 * (0.5 - d) ** 2, 0.75 - d ** 2, 0.5 * (0.5 + d) ** 2])  # [offset][particle][axis]
    nodes = []
    b = base.to(torch.int64)
    for gx in range(3):
        for gy in range(3):
            for gz in range(3):
                o = torch.tensor([gx - 1, gy - 1, gz - 1], device=x.device)
                at = b + o
                idx = (at[:, 0] * Y + at[:, 1]) * Z + at[:, 2]
                ok = (idx >= 0) & (idx < cells)
                wt = torch.where(ok, w[gx, :, 0] * w[gy, :, 1] * w[gz, :, 2], torch.zeros_like(x[:, 0]))
                nodes.append((idx.clamp(0, cells - 1), wt, base + o + 0.5 - x))
    mass = torch.zeros(cells, dtype=x.dtype, device=x.device)
    mom = torch.zeros(cells, 3, dtype=x.dtype, device=x.device)
    for idx, wt, dist in nodes:
        mass = mass.index_add(0, idx, wt)
        mom = mom.index_add(0, idx, wt[:, None] * (v + torch.einsum("nij,nj->ni", C, dist)))
    rho = sum(mass[idx] * wt for idx, wt, _ in nodes)
    pressure = torch.clamp(k * ((rho / rest) ** 5 - 1.0), min=0.0)
    stress = mu * (C + C.transpose(1, 2)) - pressure[:, None, None] * torch.eye(3, dtype=x.dtype, device=x.device)
    T = -4.0 * dt / rho[:, None, None] * stress
    for idx, wt, dist in nodes:
        mom = mom.index_add(0, idx, wt[:, None] * torch.einsum("nij,nj->ni", T, dist))
    full = mass > 0
    vel = torch.where(full[:, None], mom / torch.where(full, mass, torch.ones_like(mass))[:, None], mom)
    vel = vel + torch.where(full, gravity * dt, 0.0)[:, None] * torch.tensor([0.0, 1.0, 0.0], dtype=x.dtype, device=x.device)
    i = torch.arange(cells, device=x.device)
    coord = torch.stack([i // Z // Y, (i // Z) % Y, i % Z], dim=1)
    top = torch.tensor([math.ceil(r) - 3 for r in real], device=x.device)
    vel = torch.where(full[:, None] & ((coord < 2) | (coord > top)), torch.zeros_like(vel), vel)
    vp, B = torch.zeros_like(v), torch.zeros_like(C)
    for idx, wt, dist in nodes:
        wv = wt[:, None] * vel[idx]
        vp = vp + wv
        B = B + wv[:, :, None] * dist[:, None, :]
    hi = torch.tensor([float(np.float32(r)) for r in real], dtype=x.dtype, device=x.device)
    x = torch.minimum(torch.clamp(x + vp * dt, min=1.0), hi - 2.0)
    nx = x + vp * dt * 3.0
    vp = vp + torch.where(nx < 3.0, 0.3 * (3.0 - nx), 0.0) + torch.where(nx > hi - 4.0, 0.3 * (hi - 4.0 - nx), 0.0)
    return x, vp, 4.0 * B


def _posvel(x, v):
    zero = torch.zeros_like(x[:, :1])
    return torch.cat([x, zero, v, zero], dim=1)


def _exact_mpm(case, seed):
    rec, box = _mpm_records(case, seed)
    x = torch.from_numpy(rec[:, 0:3]).to(_device(), torch.float64)
    v, C = torch.zeros_like(x), torch.zeros(len(x), 3, 3, dtype=x.dtype, device=x.device)
    for _ in range(2):
        x, v, C = _mpm_substep(x, v, C, box, _walls(box)[0], 3.0, float(np.float32(0.1)))
    posvel = _posvel(x, v)
    return {"posvel": posvel, "image": _exact_image(case, posvel, False)} if case["w"] else posvel


def _exact_adjoint(case, seed):
    from torch.utils.checkpoint import checkpoint
    rec, box = _adjoint_records(case, seed), [float(case["side"])] * 3
    dev = _device()

    def leaf(a):
        return torch.as_tensor(a, dtype=torch.float64, device=dev).requires_grad_(True)

    x0, v0 = leaf(rec[:, 0:3]), leaf(rec[:, 4:7])
    C0, k, mu = leaf(np.zeros((len(rec), 3, 3))), leaf(3.0), leaf(float(np.float32(0.1)))
    x, v, C = x0, v0, C0
    for _ in range(case["substeps"]):
        x, v, C = checkpoint(_mpm_substep, x, v, C, box, box, k, mu, use_reentrant=False)
    loss = ((x.mean(dim=0) - torch.tensor([30.0, 10.0, 30.0], dtype=x.dtype, device=dev)) ** 2).sum()
    gx, gv, gC, gk, gmu = torch.autograd.grad(loss, [x0, v0, C0, k, mu])

    def records(a, b, c):  # 80-byte records: x, v, the columns of C, each padded to four floats
        r = torch.zeros(len(a), 5, 4, dtype=a.dtype, device=dev)
        r[:, 0, 0:3], r[:, 1, 0:3], r[:, 2:5, 0:3] = a, b, c.transpose(1, 2)
        return r.reshape(-1, 20)

    return {"state": records(x.detach(), v.detach(), C.detach()), "loss": loss.detach().reshape(1),
            "grad": records(gx, gv, gC), "grad_params": torch.stack([gk, gmu]).reshape(1, 2)}


def _exact_sph(case, seed):
    rec = _sph_records(case, seed)
    x = torch.from_numpy(rec[:, 0:3]).to(_device(), torch.float64)
    v, kr = torch.zeros_like(x), 0.07
    half = torch.tensor([case["hx"], case["hy"], case["hz"]], dtype=x.dtype, device=x.device)
    for _ in range(2):
        i, j = _pairs(x, kr)
        diff = x[j] - x[i]
        r = diff.norm(dim=1)
        dens = torch.zeros_like(x[:, 0]).index_add(0, i, 315.0 / (64 * math.pi * kr ** 9) * (kr ** 2 - r ** 2) ** 3)
        near = torch.zeros_like(dens).index_add(0, i, 15.0 / (math.pi * kr ** 6) * (kr - r) ** 3)
        apart = r > 0
        i, j, diff, r = i[apart], j[apart], diff[apart], r[apart]
        p = 20.0 * (dens - 15000.0)
        grad, near_grad, lap = (c * (kr - r) ** q for c, q in ((45.0 / (math.pi * kr ** 6), 2), (45.0 / (math.pi * kr ** 5), 2),
                                                                (45.0 / (math.pi * kr ** 6), 1)))
        along = -0.5 * ((p[i] + p[j]) * grad / dens[j] + (near[i] + near[j]) * near_grad / near[j]) / r
        term = along[:, None] * diff + 100.0 * (lap / dens[j])[:, None] * (v[j] - v[i])
        force = torch.zeros_like(x).index_add(0, i, term)
        a = force / dens[:, None]
        a[:, 1] -= 9.8
        a += 8000.0 * (torch.clamp(half - x, max=0.0) - torch.clamp(half + x, max=0.0))
        v = v + 0.006 * a
        x = x + 0.006 * v
    return _posvel(x, v)


def _pairs(x, radius):
    """All ordered pairs (i, j), i == j too, closer than radius: particles sorted by cell, the 27 cells around."""
    c = torch.floor((x + 3.0) / radius).to(torch.int64)
    m = 128
    key = (c[:, 2] * m + c[:, 1]) * m + c[:, 0]
    skey, order = torch.sort(key)
    left, right = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            row = key + (dz * m + dy) * m
            lo, hi = torch.searchsorted(skey, row - 1), torch.searchsorted(skey, row + 1, right=True)
            count = hi - lo
            i = torch.repeat_interleave(torch.arange(len(x), device=x.device), count)
            first = torch.cumsum(count, 0) - count
            j = order[lo[i] + torch.arange(len(i), device=x.device) - first[i]]
            close = ((x[i] - x[j]) ** 2).sum(dim=1) < radius * radius
            left.append(i[close])
            right.append(j[close])
    return torch.cat(left), torch.cat(right)


def _mat(column_major, x, y, z, w):
    m = column_major
    return [m[r] * x + m[4 + r] * y + m[8 + r] * z + m[12 + r] * w for r in range(4)]


def _matrices(case):
    """The application's perspective and orbit camera: projection, its inverse, view and its inverse, by columns."""
    w, h = case["w"], case["h"]
    box = (case["x"], case["y"], case["z"])
    dist, target = case.get("dist") or 1.17 * max(box), np.array([box[0] / 2.0, box[1] / 4.0, box[2] / 2.0])
    f, r = 1.0 / math.tan(FOV / 2.0), 1.0 / (0.1 - 500.0)
    P = np.array([[f * h / w, 0, 0, 0], [0, f, 0, 0], [0, 0, 500.0 * r, 0.1 * 500.0 * r], [0, 0, -1.0, 0]])
    yt, xt = -math.pi / 12, math.pi / 4
    eye = np.array([0.0, 0.0, dist])
    eye = np.array([eye[0], math.cos(yt) * eye[1] - math.sin(yt) * eye[2], math.sin(yt) * eye[1] + math.cos(yt) * eye[2]])
    eye = target + np.array([math.cos(xt) * eye[0] + math.sin(xt) * eye[2], eye[1], -math.sin(xt) * eye[0] + math.cos(xt) * eye[2]])
    back = (eye - target) / np.linalg.norm(eye - target)
    side = np.cross([0.0, 1.0, 0.0], back)
    side /= np.linalg.norm(side)
    V = np.eye(4)
    V[:3, :3] = np.stack([side, np.cross(back, side), back])
    V[:3, 3] = -V[:3, :3] @ eye
    return [m.astype(np.float32).astype(np.float64).T.reshape(-1).tolist() for m in (P, np.linalg.inv(P), V, np.linalg.inv(V))]


def _fragments(case, posvel, P, V):
    """Every fragment of the particles' billboards, a window offset at a time: (particle, pixel, nx, ny, nz, view z)."""
    w, h = case["w"], case["h"]
    x, y, z, _ = _mat(V, posvel[:, 0], posvel[:, 1], posvel[:, 2], 1.0)
    s = MPM_DIAMETER
    cm, cp, cc = (_mat(P, x + o, y + o, z, 1.0) for o in (-0.5 * s, 0.5 * s, 0.0))
    zq = cc[2] / cc[3]
    keep = (cc[3] > 0) & (zq >= 0) & (zq <= 1)
    fx = [(c[0] / c[3] + 1.0) * 0.5 * w for c in (cm, cp)]
    fy = [(1.0 - c[1] / c[3]) * 0.5 * h for c in (cm, cp)]
    x0, y0 = torch.ceil(torch.minimum(*fx) - 0.5), torch.ceil(torch.minimum(*fy) - 0.5)
    x1, y1 = torch.ceil(torch.maximum(*fx) - 0.5) - 1, torch.ceil(torch.maximum(*fy) - 0.5) - 1
    wide, high = (int(torch.where(keep, t, torch.zeros_like(t)).max().item()) + 1 for t in (x1 - x0, y1 - y0))
    for oy in range(high):
        for ox in range(wide):
            px, py = x0 + ox, y0 + oy
            nx = 2.0 * (px + 0.5 - fx[0]) / (fx[1] - fx[0]) - 1.0
            ny = 2.0 * (py + 0.5 - fy[0]) / (fy[1] - fy[0]) - 1.0
            rr = nx * nx + ny * ny
            i = torch.nonzero(keep & (px <= x1) & (py <= y1) & (px >= 0) & (px < w) & (py >= 0) & (py < h) & (rr <= 1.0))[:, 0]
            nz = torch.sqrt(1.0 - rr[i])
            yield i, (py[i] * w + px[i]).to(torch.int64), nx[i], ny[i], nz, z[i] + nz * s / 2.0


def _exact_image(case, posvel, spheres):
    P, Pinv, V, Vinv = _matrices(case)
    w, h = case["w"], case["h"]
    near = torch.full((w * h,), -math.inf, dtype=posvel.dtype, device=posvel.device)
    thick = torch.zeros_like(near)
    for _, p, _, _, nz, vz in _fragments(case, posvel, P, V):
        near = near.scatter_reduce(0, p, vz, "amax")
        thick = thick.index_add(0, p, 0.05 * nz)
    hit = torch.isfinite(near)
    if spheres:
        image = torch.full((w * h, 3), 0.8, dtype=posvel.dtype, device=posvel.device)
        stops = torch.tensor([[0, 0.4, 0.8], [35 / 256, 161 / 256, 165 / 256], [95 / 256, 254 / 256, 150 / 256],
                              [243 / 256, 250 / 256, 49 / 256], [1.0 - 1 / 256, 165 / 256, 0.0]], dtype=posvel.dtype, device=posvel.device)
        for i, p, nx, ny, nz, vz in _fragments(case, posvel, P, V):
            won = vz == near[p]
            value = posvel[i[won], 4:7].norm(dim=1) / 1.5
            band = torch.clamp(torch.floor(value * 4.0), 0, 3)
            t = (value * 4.0 - band)[:, None]
            band = band.to(torch.int64)
            light = torch.clamp((nx + ny + nz)[won] / math.sqrt(3.0), min=0.0)
            image[p[won]] = (stops[band] * (1.0 - t) + stops[band + 1] * t) * light[:, None]
        return torch.cat([image, torch.ones_like(image[:, :1])], dim=1).reshape(h, w, 4)
    depth = torch.where(hit, near, torch.zeros_like(near)).abs().reshape(h, w)
    ys, xs = torch.meshgrid(torch.arange(h, device=depth.device), torch.arange(w, device=depth.device), indexing="ij")
    ppc = 12.0 * 2.0 * MPM_RADIUS * 0.05 * (h / 2.0) / math.tan(FOV / 2.0)
    for k in range(8):
        dx, dy = (1, 0) if k % 2 == 0 else (0, 1)
        size = torch.where(depth > 0, torch.ceil(ppc / torch.where(depth > 0, depth, torch.ones_like(depth))), torch.zeros_like(depth)).clamp(max=100)
        top, weight = torch.zeros_like(depth), torch.zeros_like(depth)
        for o in range(-int(size.max().item()), int(size.max().item()) + 1):
            tap = depth[(ys + o * dy).clamp(0, h - 1), (xs + o * dx).clamp(0, w - 1)]
            g = torch.exp(-2.0 * o * o / (2.0 * (size / 3.0).clamp(min=1e-9) ** 2)) * torch.exp(-(tap - depth) ** 2 / (2.0 * (MPM_RADIUS * 10.0 / 3.0) ** 2))
            g = torch.where(abs(o) <= size, g, torch.zeros_like(g))
            top, weight = top + tap * g, weight + g
        depth = torch.where(depth > 0, top / weight, depth)
    thick = thick.reshape(h, w)
    for dx, dy in ((1, 0), (0, 1)):
        top, total = torch.zeros_like(thick), 0.0
        for o in range(-30, 31):
            g = math.exp(-o * o / 200.0)
            top, total = top + g * thick[(ys + o * dy).clamp(0, h - 1), (xs + o * dx).clamp(0, w - 1)], total + g
        thick = torch.where(thick != 0, top / total, thick)
    return _shade(P, Pinv, V, Vinv, w, h, depth, thick, xs, ys)


def _shade(P, Pinv, V, Vinv, w, h, depth, thick, xs, ys):
    tx, ty = (xs + 0.5).to(depth.dtype) / w, (ys + 0.5).to(depth.dtype) / h

    def view(ox, oy):
        d = depth[(ys + oy).clamp(0, h - 1), (xs + ox).clamp(0, w - 1)]
        e = _mat(Pinv, (tx + ox / w) * 2.0 - 1.0, 1.0 - 2.0 * (ty + oy / h), -P[10] + P[14] / d, 1.0)
        return torch.stack(e[:3], dim=-1) / e[3][..., None]

    def unit(a):
        return a / a.norm(dim=-1, keepdim=True)

    at = view(0, 0)
    ddx, ddy, ddx2, ddy2 = view(1, 0) - at, view(0, 1) - at, at - view(-1, 0), at - view(0, -1)
    ddx = torch.where((ddx[..., 2:].abs() > ddx2[..., 2:].abs()), ddx2, ddx)
    ddy = torch.where((ddy[..., 2:].abs() > ddy2[..., 2:].abs()), ddy2, ddy)
    normal, ray = -unit(torch.cross(ddx, ddy, dim=-1)), unit(at)
    light = unit(torch.tensor(_mat(V, 0.0, 0.0, -1.0, 0.0)[:3], dtype=depth.dtype, device=depth.device))
    facing = (unit(light - ray) * normal).sum(dim=-1)
    specular = torch.where(torch.isnan(facing), torch.zeros_like(facing), facing.clamp(min=0.0)) ** 250
    diffuse = torch.tensor([0.085, 0.6375, 0.9], dtype=depth.dtype, device=depth.device)
    refracted = 0.8 * torch.exp(-1.5 * thick[..., None] * (1.0 - diffuse))
    along = (normal * ray).sum(dim=-1, keepdim=True)
    fresnel = (0.02 + 0.98 * (1.0 + along) ** 5).clamp(0.0, 1.0)
    mirror = ray - normal * 2.0 * along
    to = torch.stack(_mat(Vinv, mirror[..., 0], mirror[..., 1], mirror[..., 2], 0.0)[:3], dim=-1)
    image = specular[..., None] + refracted * (1.0 - fresnel) + _sky(to) * fresnel
    image = torch.where((depth > 0)[..., None], image, torch.full_like(image, 0.8))
    return torch.cat([image, torch.ones_like(image[..., :1])], dim=-1)


def _sky(d):
    """The renderer's built-in sky (brighter above the horizon), sampled as its 32 x 32 cube faces are: bilinear
    within a face, clamped at its edges."""
    size = 32
    x, y, z = d[..., 0], d[..., 1], d[..., 2]
    ax, ay, az = x.abs(), y.abs(), z.abs()
    on_x, on_y = (ax >= ay) & (ax >= az), ay >= az
    face = torch.where(on_x, torch.where(x >= 0, 0, 1), torch.where(on_y, torch.where(y >= 0, 2, 3), torch.where(z >= 0, 4, 5)))
    ma = torch.where(on_x, ax, torch.where(on_y, ay, az))
    sc = torch.where(on_x, torch.where(x >= 0, -z, z), torch.where(on_y, x, torch.where(z >= 0, x, -x)))
    tc = torch.where(on_x, -y, torch.where(on_y, torch.where(y >= 0, z, -z), -y))
    f = torch.stack([(sc / ma + 1.0) * 0.5 * size - 0.5, (tc / ma + 1.0) * 0.5 * size - 0.5])
    base = torch.floor(torch.nan_to_num(f))
    frac = f - base
    color = 0.0
    for ox, oy in ((0, 0), (1, 0), (0, 1), (1, 1)):
        s, t = (2.0 * ((base[k] + o).clamp(0, size - 1) + 0.5) / size - 1.0 for k, o in ((0, ox), (1, oy)))
        one = torch.ones_like(s)
        up = torch.where(face == 2, one, torch.where(face == 3, -one, -t))
        up = up / torch.sqrt(s * s + t * t + 1.0)
        high, low = up.clamp(min=0.0), up.clamp(max=0.0)
        texel = torch.stack([0.55 + 0.25 * high + 0.2 * low, 0.65 + 0.25 * high + 0.2 * low, 0.8 + 0.2 * high + 0.1 * low], dim=-1)
        weight = (frac[0] if ox else 1.0 - frac[0]) * (frac[1] if oy else 1.0 - frac[1])
        color = color + texel * weight[..., None]
    return color


def exact(case, seed):
    kind = case["kind"]
    if kind == "mpm":
        return _exact_mpm(case, seed)
    if kind == "sph":
        return _exact_sph(case, seed)
    if kind == "render":
        return _exact_image(case, torch.from_numpy(_pool(case, seed)).to(_device(), torch.float64), case["spheres"])
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    return None  # batch, inverse: dozens of scenes over dozens of substeps, minutes in 64 bits
