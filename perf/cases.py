"""Performance cases of the projector: what they are, how a program runs them, what they must cost.

Three kinds of work, each through the package's public entry points:

* ``scan``: ``dpt_b200.torch.Projector`` on a device volume, forward alone (inference) or
  forward and backward of an image cotangent to the volume, to the per-view pose tangent, or
  to both;
* ``render``: the same forward through ``dpt_b200.project`` into a caller's image buffer;
* ``likelihood``: ``dpt_b200.torch.transmit`` (counts from a per-pixel open beam) and the
  Poisson ``objective`` of an optical-depth image, forward and backward.

A case is a dict of plain values.  ``listed()`` names the representative ones, ``draw(rng)``
gives more of the same ranges, ``prepare``/``run`` are what a user's program does, ``work`` is
the arithmetic and traffic no implementation can avoid and ``exact`` the result in plain FP64
Torch.
"""

from __future__ import annotations

import math

import torch

import dpt_b200
from dpt_b200.geometry import BatchedGeometry, CurvedDetectorGeometry, DetectorGeometry, ParallelGeometry
from dpt_b200.objectives import ObjectiveSpec, prepare_objective
from dpt_b200.phantoms import centred_grid
from dpt_b200.torch import Projector
from dpt_b200.torch.operators import objective, transmit
from dpt_b200.transmission import TransmissionSpec, prepare_transmission

DEVICE = "cuda:0"
STORAGE = {"float32": torch.float32, "float64": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}


def _scan(name, shape, spacing, views, detector, pitch, samples, *, sid=1000.0, sdd=1500.0, arc=360.0, panel="cone",
          arithmetic="float32", volume=False, pose=False, turn=0.0, kind="scan"):
    case = {"kind": kind, "nz": shape[0], "ny": shape[1], "nx": shape[2], "sx": spacing[0], "sy": spacing[1],
            "sz": spacing[2], "views": views, "rows": detector[0], "cols": detector[1], "pitch": pitch,
            "samples": samples, "sid": sid, "sdd": sdd, "arc": arc, "panel": panel, "arithmetic": arithmetic,
            "volume": volume, "pose": pose, "turn": turn}
    return {"name": name, **case} if name else case


def listed():
    cube = ((256, 256, 256), (0.8, 0.8, 0.8))
    return [
        # a preview of a small volume: the smallest call, latency and launches
        _scan("preview_64", (64, 64, 64), (1.0,) * 3, 8, (64, 64), 1.5, 128, sid=500.0, sdd=1000.0),
        # one iteration of a reconstruction on that volume
        _scan("train_64", (64, 64, 64), (1.0,) * 3, 8, (64, 64), 1.5, 128, sid=500.0, sdd=1000.0, volume=True),
        # digitally reconstructed radiographs of an odd-sized volume into a caller's buffer
        _scan("drr_odd", (117, 131, 149), (1.4, 1.4, 1.9), 5, (243, 201), 2.1, 333, kind="render"),
        # two-view registration of an anisotropic, rotated head volume: pose gradient alone
        _scan("register_head", (76, 507, 512), (0.45, 0.45, 2.5), 2, (256, 256), 1.6, 768, arc=180.0, pose=True,
              turn=15.0),
        # sparse-view reconstruction: forward and volume gradient
        _scan("sparse_256", *cube, 24, (512, 512), 0.8, 1024, volume=True),
        # the full scan: forward, volume and pose gradients of 360 views (the headline workload)
        _scan("full_scan", *cube, 360, (512, 512), 0.8, 1024, volume=True, pose=True),
        # the same step on a BF16 volume, a batch of views
        _scan("bf16_step", *cube, 16, (512, 512), 0.8, 1024, volume=True, pose=True, arithmetic="bfloat16"),
        # forward of an FP16 volume larger than L2, under two samples per cell
        _scan("fp16_512", (512, 512, 512), (0.5,) * 3, 12, (512, 512), 0.8, 1024, arithmetic="float16"),
        # strict FP64: a step of a few views
        _scan("fp64_step", *cube, 6, (512, 512), 0.8, 1024, volume=True, pose=True, arithmetic="float64"),
        # strict FP64 forward of a CT chest grid, three views
        _scan("fp64_chest", (139, 512, 512), (0.7617, 0.7617, 2.5), 3, (512, 512), 1.6, 1024, arc=180.0,
              arithmetic="float64"),
        # parallel panels, odd sizes, a sample count that is no power of two
        _scan("parallel_odd", (203, 187, 211), (0.9, 1.1, 0.7), 31, (301, 233), 1.1, 611, panel="parallel",
              arc=180.0, volume=True),
        # Poisson likelihood of a scan's image and its gradient
        {"name": "likelihood", "kind": "likelihood", "pixels": 90 * 512 * 512},
    ]


def _log(rng, low, high):
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def draw(rng):
    if rng.random() < 0.1:
        return {"kind": "likelihood", "pixels": int(_log(rng, 1 << 12, 94e6))}
    n = [max(24, round(_log(rng, 40, 330) * rng.choice((0.5, 0.8, 1.0)))) for _ in range(3)]
    spacing = [round(rng.uniform(0.85, 1.15) * 205.0 / max(n), 4) for _ in range(3)]
    detector = [round(_log(rng, 40, 700)) for _ in range(2)]
    arithmetic = rng.choice(("float32",) * 5 + ("bfloat16", "bfloat16", "float16", "float64", "float64"))
    volume, pose = rng.choice(((False, False), (True, False), (True, True), (False, True)))
    panel = rng.choice(("cone",) * 6 + ("parallel", "curved"))
    views, samples = round(_log(rng, 1, 360)), round(_log(rng, 96, 1100))
    # no more work than the full scan, whose three directions cost about three forwards
    passes = (1 + volume + pose) * (3 if arithmetic == "float64" else 1)
    most = 360 * 512 * 512 * 1024 * 3 // (passes * samples * detector[0] * detector[1])
    extent = max(k * s for k, s in zip(reversed(n), spacing))
    pitch = round(rng.uniform(1.0, 1.4) * extent * (1.0 if panel == "parallel" else 1.5) / max(detector), 4)
    return _scan(None, n, spacing, max(1, min(views, most)), detector, pitch, samples, panel=panel,
                 arc=rng.choice((180.0, 360.0)), arithmetic=arithmetic, volume=volume, pose=pose,
                 turn=rng.choice((0.0, 0.0, 15.0)),
                 kind="render" if not (volume or pose) and rng.random() < 0.3 else "scan")


# ------------------------------------------------------------------ geometry of a case

def _panels(case):
    """Per view: the vectors of its panel (world mm), evenly spaced around z."""
    panels = []
    rows, cols, pitch, sid, sdd = case["rows"], case["cols"], case["pitch"], case["sid"], case["sdd"]
    for k in range(case["views"]):
        a = math.radians(case["arc"]) * k / case["views"] + 0.05
        n, u, v = (math.cos(a), math.sin(a), 0.0), (-math.sin(a), math.cos(a), 0.0), (0.0, 0.0, 1.0)
        source = tuple(sid * c for c in n)
        centre = tuple(-(sdd - sid) * c for c in n)
        left, top = -0.5 * (cols - 1) * pitch, -0.5 * (rows - 1) * pitch
        if case["panel"] == "curved":
            # a cylinder of radius sdd about the source; pixel (0, 0) at arc angle `first`
            first = left / sdd
            radial = tuple(-math.cos(first) * n[i] + math.sin(first) * u[i] for i in range(3))
            u = tuple(math.sin(first) * n[i] + math.cos(first) * u[i] for i in range(3))
            origin = tuple(source[i] + sdd * radial[i] + top * v[i] for i in range(3))
        else:
            origin = tuple(centre[i] + left * u[i] + top * v[i] for i in range(3))
        panels.append({"source": source, "origin": origin, "u": u, "v": v, "direction": tuple(-c for c in n)})
    return panels


def _geometry(case):
    shape, spacing = (case["rows"], case["cols"]), (case["pitch"], case["pitch"])
    views = []
    for p in _panels(case):
        if case["panel"] == "parallel":
            views.append(ParallelGeometry(p["origin"], p["direction"], case["sdd"], p["u"], p["v"], spacing, shape))
        elif case["panel"] == "curved":
            views.append(CurvedDetectorGeometry(p["source"], p["origin"], p["u"], p["v"], spacing, shape))
        else:
            views.append(DetectorGeometry(p["source"], p["origin"], p["u"], p["v"], spacing, shape))
    return BatchedGeometry(tuple(views))


def _turned(case):
    c, s = math.cos(math.radians(case["turn"])), math.sin(math.radians(case["turn"]))
    return (c, -s, 0.0, s, c, 0.0, 0.0, 0.0, 1.0)


def _grid(case):
    return centred_grid((case["nz"], case["ny"], case["nx"]), (case["sx"], case["sy"], case["sz"]), _turned(case))


def _segments(case, view, rows, cols):
    """Sources and end points (world mm, FP64) of the pixels (rows x cols index tensors) of one view."""
    p = _panels(case)[view]
    r, c = rows.double()[:, None], cols.double()[None, :]

    def vec(key):
        return torch.tensor(p[key], dtype=torch.float64, device=rows.device)

    pitch = case["pitch"]
    if case["panel"] == "curved":
        angle = c * pitch / case["sdd"]
        radial = (vec("origin") - vec("source")) - torch.dot(vec("origin") - vec("source"), vec("v")) * vec("v")
        end = (vec("origin") + (torch.cos(angle) - 1.0)[..., None] * radial
               + (torch.sin(angle) * case["sdd"])[..., None] * vec("u") + (r * pitch)[..., None] * vec("v"))
    else:
        end = vec("origin") + (c * pitch)[..., None] * vec("u") + (r * pitch)[..., None] * vec("v")
    if case["panel"] == "parallel":
        source = end - case["sdd"] * vec("direction")
    else:
        source = vec("source").expand_as(end)
    return source.reshape(-1, 3), end.reshape(-1, 3)


def _grid_map(case, device):
    """(matrix, origin): grid index = matrix (object point - origin), FP64."""
    h = torch.tensor([case["sx"], case["sy"], case["sz"]], dtype=torch.float64, device=device)
    n = torch.tensor([case["nx"], case["ny"], case["nz"]], dtype=torch.float64, device=device)
    turn = torch.tensor(_turned(case), dtype=torch.float64, device=device).reshape(3, 3)
    return turn.T / h[:, None], -(turn @ ((n - 1) / 2 * h))


# ------------------------------------------------------------------ inputs

def _field(case, generator):
    """Attenuation of a noisy ellipse with random ellipsoids in it (1/mm, non-negative)."""
    axes = [torch.linspace(-1.0, 1.0, case[k], device=DEVICE) for k in ("nz", "ny", "nx")]
    z, y, x = axes[0][:, None, None], axes[1][None, :, None], axes[2][None, None, :]
    shape = (case["nz"], case["ny"], case["nx"])
    inside = (((y / 0.8) ** 2 + (x / 0.92) ** 2) < 1.0).expand(shape)
    field = torch.randn(shape, device=DEVICE, generator=generator).mul_(0.0008).add_(0.0206).mul_(inside)
    picks = torch.rand((6, 7), generator=generator, device=DEVICE).tolist()
    for p in picks:
        r2 = sum(((axis - (q - 0.5)) / (0.08 + 0.35 * w)) ** 2 for axis, q, w in zip((z, y, x), p[:3], p[3:6]))
        field += torch.where(r2 < 1.0, 0.04 * p[6] - 0.018, 0.0)
    return field.clamp_(min=0.0)


def _inputs(case, seed):
    """(field, tangent or None, cotangent or None) of a scan, from the seed alone."""
    generator = torch.Generator(device=DEVICE).manual_seed(1000003 * (seed % 65521) + 17)
    field = _field(case, generator).to(STORAGE[case["arithmetic"]]).contiguous()
    tangent = cotangent = None
    if case["pose"]:
        # a few millimetres and a degree or two from the planned pose
        scale = torch.tensor([3.0, 3.0, 3.0, 0.02, 0.02, 0.02], dtype=torch.float64, device=DEVICE)
        tangent = scale * torch.randn((case["views"], 6), dtype=torch.float64, device=DEVICE, generator=generator)
    if case["volume"] or case["pose"]:
        # the residual image of a fit: of both signs, a structured and a noisy part
        dtype = torch.float64 if case["arithmetic"] == "float64" else torch.float32
        shape = (case["views"], case["rows"], case["cols"])
        cotangent = torch.randn(shape, dtype=dtype, device=DEVICE, generator=generator)
        wave = torch.sin(torch.arange(case["cols"], device=DEVICE, dtype=dtype) * (9.0 / case["cols"]))
        cotangent = cotangent.mul_(0.3).add_(wave).mul_(1e-3)
    return field, tangent, cotangent


def _likelihood_inputs(case, seed):
    generator = torch.Generator(device=DEVICE).manual_seed(1000003 * (seed % 65521) + 29)
    n = case["pixels"]
    depth = torch.rand(n, device=DEVICE, generator=generator).mul_(6.0)
    beam = torch.rand(n, device=DEVICE, generator=generator).mul_(1000.0).add_(500.0)
    observation = torch.poisson(beam * torch.exp(-depth), generator=generator)
    return depth, beam, observation


def prepare(case, seed):
    if case["kind"] == "likelihood":
        depth, beam, observation = _likelihood_inputs(case, seed)
        return {"kind": "likelihood", "depth": depth.requires_grad_(), "beam": beam, "observation": observation,
                "transmission": prepare_transmission(TransmissionSpec(beam="per-pixel"), max_pixels=case["pixels"],
                                                     device=DEVICE),
                "objective": prepare_objective(ObjectiveSpec(kind="poisson", domain="counts"),
                                               max_pixels=case["pixels"], device=DEVICE)}
    field, tangent, cotangent = _inputs(case, seed)
    projector = Projector(grid=_grid(case), geometry=_geometry(case), samples_per_ray=case["samples"],
                          precision="fp64" if case["arithmetic"] == "float64" else "fp32")
    state = {"kind": case["kind"], "projector": projector, "field": field.requires_grad_(case["volume"]),
             "tangent": None if tangent is None else tangent.requires_grad_(), "cotangent": cotangent}
    if case["kind"] == "render":
        dtype = torch.float64 if case["arithmetic"] == "float64" else torch.float32
        state["out"] = torch.empty((case["views"], case["rows"], case["cols"]), dtype=dtype, device=DEVICE)
    return state


def run(state):
    if state["kind"] == "likelihood":
        depth = state["depth"]
        counts = transmit(depth, state["beam"], output="counts", workspace=state["transmission"])
        loss = objective(counts, state["observation"], workspace=state["objective"])
        (grad,) = torch.autograd.grad(loss, depth)
        return {"counts": counts.detach(), "loss": loss.detach(), "grad": grad}
    projector, field, tangent = state["projector"], state["field"], state["tangent"]
    if state["kind"] == "render":
        with torch.no_grad():
            return {"image": dpt_b200.project(field, prepared=projector, pose=tangent, out=state["out"])}
    image = projector(field, tangent)
    result = {"image": image.detach()}
    inputs = {}
    if field.requires_grad:
        inputs["volume"] = field
    if tangent is not None:
        inputs["pose"] = tangent
    if inputs:
        grads = torch.autograd.grad(image, list(inputs.values()), state["cotangent"])
        result.update(zip(inputs, grads))
    return result


# ------------------------------------------------------------------ what a pass cannot do without

def _clip(case, matrix, origin, source, end):
    """Grid-index origin and direction of the rays and their clipped parameter interval."""
    o, d = (source - origin) @ matrix.T, (end - source) @ matrix.T
    high = torch.tensor([case["nx"], case["ny"], case["nz"]], dtype=torch.float64, device=o.device) - 0.5
    moving = d != 0
    safe = torch.where(moving, d, torch.ones_like(d))
    a, b = (-0.5 - o) / safe, (high - o) / safe
    inf = torch.full_like(a, math.inf)
    outside = ~moving & ((o < -0.5) | (o > high))
    lower = torch.where(moving, torch.minimum(a, b), -inf).amax(1).clamp(min=0.0)
    upper = torch.where(moving, torch.maximum(a, b), inf).amin(1).clamp(max=1.0)
    upper = torch.where(outside.any(1), torch.full_like(upper, -1.0), upper)
    return o, d, lower, upper


def work(case):
    """Inputs read once, outputs written once; per sample inside the volume the arithmetic of a
    position (6), the trilinear value and its sum (15), for the volume gradient the eight
    weights and their accumulation (28) and for the pose gradient the slope and its moments (45)."""
    if case["kind"] == "likelihood":
        return {"bytes": case["pixels"] * 4.0 * 5, "flops": case["pixels"] * 30.0}
    matrix, origin = _grid_map(case, "cpu")
    rows = torch.linspace(0, case["rows"] - 1, min(24, case["rows"])).round()
    cols = torch.linspace(0, case["cols"] - 1, min(24, case["cols"])).round()
    hits = []
    for view in range(0, case["views"], max(1, case["views"] // 8)):
        _, _, lower, upper = _clip(case, matrix, origin, *_segments(case, view, rows, cols))
        hits.append(float((upper > lower).double().mean()))
    rays = case["views"] * case["rows"] * case["cols"]
    samples = rays * case["samples"] * sum(hits) / len(hits)
    voxels = case["nx"] * case["ny"] * case["nz"]
    stored = 2 if case["arithmetic"] in ("float16", "bfloat16") else 4
    element = 8 if case["arithmetic"] == "float64" else 4
    active = case["volume"] or case["pose"]
    size = voxels * stored * (2 if case["volume"] else 1) + rays * element * (2 if active else 1)
    flops = 21 + (28 if case["volume"] else 0) + (45 if case["pose"] else 0)
    return {"bytes": float(size), "flops": samples * flops}


# ------------------------------------------------------------------ the result in FP64

def _rigid(tangent):
    """Rotation and translation of exp of the (6,) twist."""
    rho, w = tangent[:3], tangent[3:]
    zero = torch.zeros_like(w[0])
    twist = torch.stack((zero, -w[2], w[1], rho[0], w[2], zero, -w[0], rho[1], -w[1], w[0], zero, rho[2],
                         zero, zero, zero, zero)).reshape(4, 4)
    motion = torch.linalg.matrix_exp(twist)
    return motion[:3, :3], motion[:3, 3]


def _ray_sums(case, field, o, d, lower, upper, seed, gradient, pose):
    """Sum of the trilinear samples of each ray (and their slope sums with ``pose``); adds
    ``seed`` times every sample's corner weights to ``gradient`` when it is given."""
    n = (case["nx"], case["ny"], case["nz"])
    alpha = (torch.arange(case["samples"], dtype=torch.float64, device=o.device) + 0.5) / case["samples"]
    t = lower[:, None] + alpha * (upper - lower)[:, None]
    base, fraction, interior = 0, [], []
    strides = (1, n[0], n[0] * n[1])
    for k in range(3):
        p = o[:, k, None] + t * d[:, k, None]
        interior.append((p >= 0) & (p < n[k] - 1))
        p = p.clamp(0.0, n[k] - 1.0)
        cell = p.floor().clamp(max=max(n[k] - 2, 0))
        fraction.append(p - cell)
        base = base + cell.long() * strides[k]
    weights = [(1.0 - f, f) for f in fraction]
    total, slopes = 0.0, [0.0, 0.0, 0.0]
    for corner in range(8):
        bits = (corner & 1, corner >> 1 & 1, corner >> 2 & 1)
        index = base + sum(b * s for b, s, m in zip(bits, strides, n) if m > 1)
        w = [weights[k][bits[k]] for k in range(3)]
        product = w[0] * w[1] * w[2]
        value = field[index]
        total = total + product * value
        if gradient is not None:
            gradient.index_add_(0, index.reshape(-1), (product * seed[:, None]).reshape(-1))
        if pose:
            for k in range(3):
                sign = 1.0 if bits[k] else -1.0
                slopes[k] = slopes[k] + sign * w[(k + 1) % 3] * w[(k + 2) % 3] * value
    moments = None
    if pose:
        g = torch.stack([torch.where(m, s, torch.zeros_like(t)) for m, s in zip(interior, slopes)], -1)
        along = (g * d[:, None, :]).sum(-1)
        moments = (g.sum(1), (g * t[..., None]).sum(1), ((1.0 - alpha) * along).sum(1), (alpha * along).sum(1))
    return total.sum(1), moments


def exact(case, seed):
    if case["kind"] == "likelihood":
        depth, beam, observation = (v.double() for v in _likelihood_inputs(case, seed))
        counts = beam * torch.exp(-depth)
        deviance = counts - observation + torch.xlogy(observation, observation / counts)
        return {"counts": counts, "loss": deviance.sum(), "grad": observation - counts}
    rays = case["rows"] * case["cols"]
    cost = case["views"] * rays * case["samples"] * (1 + 2 * case["volume"] + 2 * case["pose"])
    if cost > 26e9:
        return None
    field, tangent, cotangent = _inputs(case, seed)
    field = field.double().reshape(-1)
    image = torch.zeros((case["views"], rays), dtype=torch.float64, device=DEVICE)
    volume = torch.zeros_like(field) if case["volume"] else None
    pose = torch.zeros_like(tangent) if case["pose"] else None
    matrix, origin = _grid_map(case, DEVICE)
    rows, cols = torch.arange(case["rows"], device=DEVICE), torch.arange(case["cols"], device=DEVICE)
    step = max(1, 4_000_000 // case["samples"])
    for view in range(case["views"]):
        source, end = _segments(case, view, rows, cols)
        for first in range(0, rays, step):
            part = slice(first, min(first + step, rays))
            s, e = source[part], end[part]
            length = (e - s).norm(dim=1)
            twist = None
            if tangent is not None:
                twist = tangent[view].clone().requires_grad_(case["pose"])
                rotation, translation = _rigid(twist)
                s, e = (s - translation) @ rotation, (e - translation) @ rotation
            o, d, lower, upper = _clip(case, matrix, origin, s, e)
            hit = (upper > lower).nonzero().reshape(-1)
            if hit.numel() == 0:
                continue
            o, d, lower, upper, length = o[hit], d[hit], lower[hit], upper[hit], length[hit]
            with torch.no_grad():
                scale = length * (upper - lower) / case["samples"]
                cot = cotangent[view].reshape(-1)[part][hit].double() if cotangent is not None else None
                total, moments = _ray_sums(case, field, o, d, lower, upper, None if cot is None else cot * scale,
                                           volume, case["pose"])
                image[view, part.start + hit] = total * scale
            if case["pose"]:
                # the ray sum to first order in the ray's own quantities, whose dependence on
                # the pose autograd follows
                g, tg, low, high = moments
                ray = (total + (g * (o - o.detach())).sum(1) + (tg * (d - d.detach())).sum(1)
                       + low * (lower - lower.detach()) + high * (upper - upper.detach()))
                value = (cot * length * (upper - lower) / case["samples"] * ray).sum()
                pose[view] += torch.autograd.grad(value, twist)[0]
    result = {"image": image.reshape(case["views"], case["rows"], case["cols"])}
    if volume is not None:
        result["volume"] = volume.reshape(case["nz"], case["ny"], case["nx"])
    if pose is not None:
        result["pose"] = pose
    return result
