"""Performance cases: what a user of this package has it do, through its public
entry points, from the smallest problem of the 2D sweep to the 512^3 cone beam.

``listed()`` names the cases, ``draw(rng)`` makes one more of the same ranges,
``prepare`` makes what a program holds before the call (geometry with its plan,
volumes, sinograms), ``run`` is the call, ``work`` what it cannot do without and
``exact`` the same results in 64 bits from plain torch and numpy.

Inputs are seeded ellipse / ellipsoid phantoms and their analytic line
integrals with photon noise (I0 = 1e4), as in the benchmark's workloads.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

FORWARD_STEP_FLOPS = {2: 9, 3: 18}   # position, linear filter, sum
BACKWARD_STEP_FLOPS = {2: 10, 3: 14}  # perspective, linear filter, sum
BATCH_SIZES = (128, 192, 256, 384, 512, 768, 1024)


# ------------------------------------------------------------ the cases


def listed():
    return [
        # The smallest problem of the 2D sweep (64 x 64, 360 views): launches and
        # latency, as in an interactive tool or an inner loop over small images.
        fan("forward_64", "forward", 64, 360, 91, dso=256.0, dsd=384.0),
        fan("backward_64", "backward", 64, 360, 91, dso=256.0, dsd=384.0),
        # A clinical-size slice backprojected on its own.
        fan("backward_512", "backward", 512, 512, 725),
        # The headline problem: 2048 x 2048, 2048 views, 2897 cells.
        fan("forward_2048", "forward", 2048, 2048, 2897),
        fan("backward_2048", "backward", 2048, 2048, 2897),
        # Half-precision storage, both directions, on the published benchmark's
        # geometry (360 views, detector int(sqrt(2) n), DSO 20 n, DSD 22 n).
        fan("half_1024", "half", 1024, 360, 1448, spacing=1.0, dso=20480.0, dsd=22528.0),
        # A served filtered backprojection.
        fan("fbp_1024", "fbp", 1024, 1024, 1449),
        # A training step on a calibrated (jittered, per-view vector) trajectory:
        # FP32 forward through autograd and its exact (matched) gradient.
        fan("matched_vec_513", "matched", 513, 437, 726, vec=True),
        # Many problems of mixed sizes per launch, differentiated.
        {"name": "batch_12", "op": "batch", "count": 12, "mix": 3},
        # Circular cone beam: forward at 256^3, backprojection at 512^3, and a
        # training step / CGLS-style product pair (matched) at 128^3.
        cone("cone_forward_256", "forward", 256, 256, 256, 360, 384, 384),
        cone("cone_backward_512", "backward", 512, 512, 512, 720, 768, 768),
        cone("cone_matched_128", "matched", 128, 128, 128, 180, 192, 192),
    ]


def fan(name, op, n, views, det, width=0, spacing=1.5, dso=0.0, dsd=0.0, vec=False):
    """A fan-beam case; by default the sweep's DSO = 2 n and DSD = 3 n."""
    c = {"op": op, "height": n, "width": width or n, "views": views, "det": det,
         "spacing": spacing, "dso": dso or 2.0 * n, "dsd": dsd or (dso + n if dso else 3.0 * n),
         "vec": vec}
    return dict(c, name=name) if name else c


def cone(name, op, depth, height, width, views, rows, cols, tilt=0.0):
    """A circular cone-beam case (DSO = 2 n, DSD = 3 n, cells of 1.5)."""
    n = max(depth, height, width)
    c = {"op": "cone_" + op, "depth": depth, "height": height, "width": width, "views": views,
         "rows": rows, "cols": cols, "spacing": 1.5, "dso": 2.0 * n, "dsd": 3.0 * n, "tilt": tilt}
    return dict(c, name=name) if name else c


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    op = rng.choice(["forward", "forward", "backward", "backward", "fbp", "half", "matched",
                     "batch", "cone_forward", "cone_backward", "cone_matched"])
    if op == "batch":
        return {"op": op, "count": rng.randint(4, 16), "mix": rng.randint(10, 10 ** 6)}
    if op.startswith("cone_"):
        n = log_int(rng, 24, 160 if op == "cone_matched" else 288)
        shape = [max(16, int(n * rng.uniform(0.7, 1.0))) if rng.random() < 0.4 else n
                 for _ in range(3)]
        side = math.ceil(1.5 * n)
        rows = side if rng.random() < 0.6 else int(side * rng.uniform(0.7, 1.1))
        tilt = rng.uniform(0.005, 0.03) if rng.random() < 0.25 else 0.0
        return cone("", op[5:], *shape, log_int(rng, 40, 360), rows, side, tilt)
    n = log_int(rng, 128 if op in ("fbp", "half") else 64, 1024 if op == "matched" else 2048)
    width = int(n * rng.uniform(0.75, 1.0)) if rng.random() < 0.3 else n
    if op == "half":
        return fan("", op, n, rng.choice([180, 360, 361, 500]), int(math.sqrt(2) * n), width,
                   1.0, 20.0 * n, 22.0 * n)
    views = n if rng.random() < 0.4 else log_int(rng, 60, max(120, n))
    det = math.ceil(math.sqrt(2) * n) if rng.random() < 0.6 else int(n * rng.uniform(1.2, 1.6))
    return fan("", op, n, views, det, width, vec=rng.random() < (0.5 if op == "matched" else 0.2))


def batch_problems(case):
    """(n, views) of each problem of a batch."""
    rng = random.Random(case["mix"])
    return [(rng.choice(BATCH_SIZES), rng.randint(180, 720)) for _ in range(case["count"])]


def batch_fans(case):
    return [fan("", "matched", n, views, math.ceil(math.sqrt(2) * n), vec=True)
            for n, views in batch_problems(case)]


# ------------------------------------------------------------ geometry in 64 bits


def fan_angles(case):
    return np.linspace(0, 2 * np.pi, case["views"], endpoint=False).astype(np.float32)


def fan_vectors(case, seed):
    """Per view [source x, y, detector centre x, y, cell step x, y]."""
    a = fan_angles(case).astype(np.float64)
    cs, sn, dod = np.cos(a), np.sin(a), case["dsd"] - case["dso"]
    v = np.stack([case["dso"] * sn, case["dso"] * cs, -dod * sn, -dod * cs,
                  case["spacing"] * cs, -case["spacing"] * sn], axis=1)
    if case["vec"]:
        rng = np.random.default_rng(seed)
        v[:, :4] += rng.normal(0.0, 0.5, (len(v), 4))
        v = v.astype(np.float32).astype(np.float64)  # what the plan takes
    return v


def fan_geometry(case, seed, prec=32):
    import curadon_gb300 as cg

    shape = (case["height"], case["width"])
    if case["vec"]:
        return cg.FanVecGeometry(shape, case["det"], fan_vectors(case, seed))
    return cg.FanGeometry(DSD=np.full(case["views"], case["dsd"], np.float32),
                          DSO=np.full(case["views"], case["dso"], np.float32),
                          angles=fan_angles(case), vol_shape=shape, det_shape=case["det"],
                          det_spacing=case["spacing"], vol_prec=prec, sino_prec=prec)


def cone_rotation(case):
    """The detector's own rotation as (pitch, roll, yaw)."""
    t = case["tilt"]
    return (t, -0.5 * t, 0.7 * t)


def cone_geometry(case):
    import curadon_gb300 as cg

    return cg.ConeGeometry(DSD=case["dsd"], DSO=case["dso"], angles=fan_angles(case),
                           vol_shape=(case["depth"], case["height"], case["width"]),
                           det_shape=(case["rows"], case["cols"]),
                           det_spacing=(case["spacing"], case["spacing"]),
                           det_rotation=cone_rotation(case) if case["tilt"] else None)


def rpy_matrix(rotation):
    pitch, roll, yaw = rotation
    cr, sr, cp, sp = math.cos(roll), math.sin(roll), math.cos(pitch), math.sin(pitch)
    cy, sy = math.cos(yaw), math.sin(yaw)
    return np.array([[cr * cp, cr * sp * sy - sr * cy, cr * sp * cy + sr * sy],
                     [sr * cp, sr * sp * sy + cr * cy, sr * sp * cy - cr * sy],
                     [-sp, cp * sy, cp * cy]])


def orbit_matrix(phi):
    c, s = math.cos(phi), math.sin(phi)
    return np.array([[c, 0.0, s], [0.0, 1.0, 0.0], [-s, 0.0, c]])


def cone_rays(case):
    """Per view, in voxel indices: source, centre of cell (0, 0), u and v steps."""
    shape = np.array([case["width"], case["height"], case["depth"]], np.float64)
    ds, dod = case["spacing"], case["dsd"] - case["dso"]
    R = rpy_matrix(cone_rotation(case))
    o = R @ np.array([-ds * case["cols"] / 2 + ds / 2, -ds * case["rows"] / 2 + ds / 2, 0.0])
    o[2] += dod
    out = []
    for phi in fan_angles(case).astype(np.float64):
        M = orbit_matrix(phi)
        shift = shape / 2 - 0.5
        out.append((M @ np.array([0.0, 0.0, -case["dso"]]) + shift, M @ o + shift,
                    M @ (R @ np.array([ds, 0.0, 0.0])), M @ (R @ np.array([0.0, ds, 0.0]))))
    return [np.stack([v[k] for v in out]) for k in range(4)]


# ------------------------------------------------------------ inputs


def fan_ellipses(case, seed):
    """(centre, semi-axes, rotation, value) of 10 ellipses on the image."""
    rng = np.random.default_rng(seed)
    s = min(case["height"], case["width"]) / 64.0
    return [(rng.uniform(-24, 24, 2) * s, rng.uniform(3, 20, 2) * s, rng.uniform(0, math.pi),
             rng.uniform(0, 1)) for _ in range(10)]


def fan_image(case, seed, device):
    h, w = case["height"], case["width"]
    y = torch.arange(h, device=device, dtype=torch.float32)[:, None] - h / 2 + 0.5
    x = torch.arange(w, device=device, dtype=torch.float32)[None, :] - w / 2 + 0.5
    img = torch.zeros((h, w), device=device)
    for c, a, rot, val in fan_ellipses(case, seed):
        co, si = math.cos(rot), math.sin(rot)
        p = ((x - c[0]) * co + (y - c[1]) * si) / a[0]
        q = ((y - c[1]) * co - (x - c[0]) * si) / a[1]
        img += val * (p * p + q * q <= 1.0)
    return img.clamp_(0, 2)


def fan_sinogram(case, seed, device):
    """Line integrals of the ellipses along the rays, with photon noise."""
    v = torch.as_tensor(fan_vectors(case, seed), device=device)
    t = torch.arange(case["det"], device=device, dtype=torch.float64) - (case["det"] - 1) / 2
    src = v[:, None, 0:2]
    d = v[:, None, 2:4] + t[None, :, None] * v[:, None, 4:6] - src
    d = d / d.norm(dim=-1, keepdim=True)
    out = torch.zeros((case["views"], case["det"]), device=device, dtype=torch.float64)
    for c, a, rot, val in fan_ellipses(case, seed):
        co, si = math.cos(rot), math.sin(rot)
        m = torch.tensor([[co / a[0], si / a[0]], [-si / a[1], co / a[1]]], device=device,
                         dtype=torch.float64)
        p = (src - torch.tensor(c, device=device, dtype=torch.float64)) @ m.T
        out += val * chord((d @ m.T).square().sum(-1), (p * (d @ m.T)).sum(-1),
                           p.square().sum(-1))
    return with_noise(out.float(), seed)


def chord(qa, qb, qc):
    """Length of a unit-speed ray inside a unit ball: qa t^2 + 2 qb t + qc = 1."""
    return 2.0 * (qb * qb - qa * (qc - 1.0)).clamp_min(0.0).sqrt() / qa


def with_noise(s, seed):
    """Log-transformed counts at I0 = 1e4 photons, line integrals up to 2.5."""
    gen = torch.Generator(device=s.device).manual_seed(seed)
    mu = 2.5 / s.max().clamp_min(1e-6)
    noise = torch.randn(s.shape, device=s.device, generator=gen)
    return (s + noise * (torch.exp(0.5 * mu * s) / 100.0 / mu)).contiguous()


def cone_ellipsoids(case, seed):
    """(centre, matrix into the unit ball, value) of 20 ellipsoids, voxel indices."""
    rng = np.random.default_rng(seed)
    ext = np.array([case["width"], case["height"], case["depth"]], np.float64)
    out = []
    for _ in range(20):
        c = rng.uniform(-0.7, 0.7, 3) * ext / 2 + ext / 2 - 0.5
        a = rng.uniform(0.05, 0.4, 3) * ext
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        out.append((c, q / a[:, None], rng.uniform(0, 1)))
    return out


def quadric(p, du, dv, rows, cols, device):
    """The vectors p + u du + v dv on the (views, rows, cols) grid, per component."""
    u = torch.arange(cols, device=device, dtype=torch.float32)[None, None, :]
    v = torch.arange(rows, device=device, dtype=torch.float32)[None, :, None]
    return [p[:, k, None, None] + u * du[:, k, None, None] + v * dv[:, k, None, None]
            for k in range(3)]


def cone_volume(case, seed, device):
    shape = (case["depth"], case["height"], case["width"])
    out = torch.zeros(shape, device=device)
    z, y, x = (torch.arange(s, device=device, dtype=torch.float32) for s in shape)
    for c, m, val in cone_ellipsoids(case, seed):
        q = 0.0
        for k in range(3):
            q = q + ((m[k, 2] * (z - c[2]))[:, None, None] + (m[k, 1] * (y - c[1]))[None, :, None]
                     + (m[k, 0] * (x - c[0]))[None, None, :]).square_()
        out += val * (q <= 1.0)
    return out.clamp_(0, 2)


def cone_projections(case, seed, device):
    src, org, du, dv = cone_rays(case)
    rows, cols = case["rows"], case["cols"]
    out = torch.zeros((case["views"], rows, cols), device=device)
    step = max(1, (1 << 25) // (rows * cols))
    f32 = lambda a: torch.as_tensor(a, device=device, dtype=torch.float32)  # noqa: E731
    for v0 in range(0, case["views"], step):
        part = slice(v0, v0 + step)
        ray = quadric(f32(org[part] - src[part]), f32(du[part]), f32(dv[part]), rows, cols, device)
        length = (ray[0] * ray[0] + ray[1] * ray[1] + ray[2] * ray[2]).sqrt_()
        for c, m, val in cone_ellipsoids(case, seed):
            mt = m.T
            d = quadric(f32((org[part] - src[part]) @ mt), f32(du[part] @ mt), f32(dv[part] @ mt),
                        rows, cols, device)
            p = f32((src[part] - c) @ mt)[:, :, None, None]
            qa = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
            qb = d[0] * p[:, 0] + d[1] * p[:, 1] + d[2] * p[:, 2]
            qc = (p * p).sum(1)
            out[part] += val * length * chord(qa, qb, qc)
    return with_noise(out, seed)


def prepare(case, seed):
    import curadon_gb300 as cg

    dev = torch.device("cuda", 0)
    op = case["op"]
    if op == "batch":
        from curadon_gb300.batch import BatchProjector

        fans = batch_fans(case)
        proj = BatchProjector([fan_geometry(f, seed + k) for k, f in enumerate(fans)], dev)
        x = torch.cat([fan_image(f, seed + k, dev).reshape(-1) for k, f in enumerate(fans)])
        y = torch.cat([fan_sinogram(f, seed + k, dev).reshape(-1) for k, f in enumerate(fans)])
        return {"op": op, "projector": proj, "x": x.requires_grad_(True), "y": y}
    if op.startswith("cone_"):
        geom = cone_geometry(case)
        state = {"op": op, "geom": geom, "cg": cg}
        if op != "cone_backward":
            state["x"] = cone_volume(case, seed, dev)
        if op != "cone_forward":
            state["y"] = cone_projections(case, seed, dev)
        if op == "cone_forward":
            state["out"] = torch.zeros(geom.sinogram_shape(), device=dev)
        if op == "cone_matched":
            state["x"] = (0.8 * state["x"]).requires_grad_(True)
            geom.exact_plan
        else:
            geom.plan
        return state
    geom = fan_geometry(case, seed, 16 if op == "half" else 32)
    state = {"op": op, "geom": geom, "cg": cg}
    if op in ("forward", "half", "matched"):
        state["x"] = fan_image(case, seed, dev)
    if op != "forward":
        state["y"] = fan_sinogram(case, seed, dev)
    if op == "half":
        # attenuation per pixel, so that sums over views stay in half's range
        state["x"] = (state["x"] * (2.0 / case["height"])).half()
        state["y"] = (state["y"] * (2.0 / case["height"])).half()
    if op == "matched":
        state["x"] = (0.8 * state["x"]).requires_grad_(True)
        geom.exact_plan
    else:
        geom.plan
    if op in ("forward", "half"):
        state["out"] = torch.zeros(geom.sinogram_shape(), device=dev,
                                   dtype=torch.float16 if op == "half" else torch.float32)
    return state


# ------------------------------------------------------------ the calls


def run(state):
    op = state["op"]
    if op == "batch":
        y = state["projector"](state["x"])
        (grad,) = torch.autograd.grad(y, state["x"], y.detach() - state["y"])
        return {"sinograms": y.detach(), "grad": grad}
    cg, geom = state["cg"], state["geom"]
    if op in ("forward", "cone_forward"):
        return cg.forward(state["x"], state["out"], geom)
    if op in ("backward", "cone_backward"):
        shape = tuple(int(n) for n in geom.vol_shape)
        return cg.backward(state["y"], torch.zeros(shape, device=state["y"].device), geom)
    if op == "half":
        cg.forward(state["x"], state["out"], geom)
        return {"sinogram": state["out"],
                "volume": cg.backward(state["y"], torch.zeros_like(state["x"]), geom)}
    if op == "fbp":
        from curadon_gb300.fbp import fbp

        return fbp(state["y"], geom)
    # matched, cone_matched: y = A x and the gradient of 1/2 |A x - data|^2
    y = cg.TorchForward.apply(state["x"], geom, True)
    (grad,) = torch.autograd.grad(y, state["x"], y.detach() - state["y"])
    return {"sinogram": y.detach(), "grad": grad}


# ------------------------------------------------------------ what a pass cannot do without


def fan_steps(case):
    """Samples of all rays (estimated on 16 views: chord along the main axis)."""
    v = fan_vectors(dict(case, vec=False), 0)
    v = v[np.linspace(0, len(v) - 1, min(16, len(v))).astype(int)]
    t = np.arange(case["det"]) - (case["det"] - 1) / 2
    src = v[:, None, 0:2] + np.array([case["width"], case["height"]]) / 2
    d = v[:, None, 2:4] + t[None, :, None] * v[:, None, 4:6] - v[:, None, 0:2]
    return case["views"] * chord_steps(src, d, (case["width"], case["height"]), 0).mean(0).sum()


def cone_steps(case):
    src, org, du, dv = cone_rays(case)
    pick = np.linspace(0, len(src) - 1, min(4, len(src))).astype(int)
    u, v = np.arange(case["cols"])[None, None, :, None], np.arange(case["rows"])[None, :, None, None]
    s = src[pick][:, None, None, :]
    d = org[pick][:, None, None, :] - s + u * du[pick][:, None, None, :] + v * dv[pick][:, None, None, :]
    steps = chord_steps(s, d, (case["width"], case["height"], case["depth"]), 1)
    return case["views"] * steps.mean(0).sum()


def chord_steps(src, d, shape, grow):
    """Steps inside the box [-1, n + grow]: along the main axis (2D) or unit length (3D)."""
    lo = np.full(d.shape[:-1], 0.0)
    hi = np.full(d.shape[:-1], np.inf)
    for k, n in enumerate(shape):
        with np.errstate(divide="ignore", invalid="ignore"):
            t1, t2 = (-1 - src[..., k]) / d[..., k], (n + grow - src[..., k]) / d[..., k]
        lo, hi = np.fmax(lo, np.fmin(t1, t2)), np.fmin(hi, np.fmax(t1, t2))
    speed = np.abs(d).max(-1) if len(shape) == 2 else np.sqrt((d * d).sum(-1))
    return np.clip(hi - lo, 0, None) * speed


def work(case):
    op = case["op"]
    if op == "batch":
        parts = [work(f) for f in batch_fans(case)]
        # the drop-in gradient is the backprojection: as many steps as pixels x views
        return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}
    dims = 3 if op.startswith("cone_") else 2
    if dims == 3:
        voxels = case["depth"] * case["height"] * case["width"]
        rays = case["views"] * case["rows"] * case["cols"]
    else:
        voxels = case["height"] * case["width"]
        rays = case["views"] * case["det"]
    kind = op[5:] if dims == 3 else op
    size = 2 if kind == "half" else 4
    bwd = BACKWARD_STEP_FLOPS[dims] * voxels * case["views"]
    if kind == "backward":
        return {"bytes": size * (rays + voxels), "flops": bwd}
    if kind == "fbp":
        fft = 2 * 2.5 * 2 * case["det"] * math.log2(2 * case["det"]) * case["views"]
        return {"bytes": size * (rays + voxels), "flops": bwd + fft}
    fwd = FORWARD_STEP_FLOPS[dims] * (cone_steps(case) if dims == 3 else fan_steps(case))
    if kind == "forward":
        return {"bytes": size * (rays + voxels), "flops": fwd}
    if kind == "half":
        return {"bytes": 2 * size * (rays + voxels), "flops": fwd + bwd}
    # matched: x and data in, y and gradient out; the transpose takes the same steps
    return {"bytes": size * (2 * rays + 2 * voxels), "flops": 2 * fwd}


# ------------------------------------------------------------ the same in 64 bits


class FanRays:
    """All rays of a fan case: first sample, step, count and step length."""

    def __init__(self, case, vectors, device):
        v = torch.as_tensor(vectors, device=device, dtype=torch.float64)
        t = torch.arange(case["det"], device=device, dtype=torch.float64) - (case["det"] - 1) / 2
        size = (case["width"], case["height"])
        src = [v[:, None, k] + size[k] / 2 for k in range(2)]
        d = [v[:, None, 2 + k] - v[:, None, k] + t[None, :] * v[:, None, 4 + k] for k in range(2)]
        lo = torch.full_like(d[0], torch.finfo(torch.float32).tiny)
        hi = torch.full_like(d[0], torch.finfo(torch.float32).max)
        for k in range(2):
            t1, t2 = (-1 - src[k]) / d[k], (size[k] - src[k]) / d[k]
            lo = torch.minimum(torch.maximum(t1, lo), torch.maximum(t2, lo))
            hi = torch.maximum(torch.minimum(t1, hi), torch.minimum(t2, hi))
        # a ray that misses, or only touches a corner (lo == hi), takes no steps;
        # its positions are finite all the same, since they become indices
        hit = lo <= hi - 1e-6
        zero = torch.zeros_like(lo)
        lo, length = torch.where(hit, lo, zero), torch.where(hit, hi - lo, zero)
        m = torch.maximum((d[0] * length).abs(), (d[1] * length).abs())
        self.steps = m.round().reshape(-1)
        m = torch.where(hit, m, torch.ones_like(m))
        self.v = [(d[k] * length / m).reshape(-1) for k in range(2)]
        self.p = [(src[k] + d[k] * lo).reshape(-1) - 0.5 for k in range(2)]
        self.norm = torch.hypot(*self.v)
        self.pitch = size[0] + 4
        self.size = size

    def cells(self):
        """Per step: the four (index, weight) of every ray into the padded image."""
        for j in range(int(self.steps.max()) if self.steps.numel() else 0):
            idx, w = [], []
            for k in range(2):
                p = self.p[k] + j * self.v[k]
                f = p.floor()
                w.append(p - f)
                idx.append(f.clamp_(-2, self.size[k]).long() + 2)
            base = idx[1] * self.pitch + idx[0]
            on = (self.steps > j).double()
            hi = w[1] * on
            lo = on - hi
            yield ((base, lo * (1 - w[0])), (base + 1, lo * w[0]),
                   (base + self.pitch, hi * (1 - w[0])), (base + self.pitch + 1, hi * w[0]))

    def forward(self, image):
        flat = torch.nn.functional.pad(image.double(), (2, 2, 2, 2)).reshape(-1)
        acc = torch.zeros_like(self.norm)
        for cells in self.cells():
            for at, w in cells:
                acc += w * flat[at]
        return torch.where(self.steps > 0, acc * self.norm, torch.zeros_like(acc))

    def adjoint(self, y):
        acc = torch.zeros((self.size[1] + 4) * self.pitch, device=y.device, dtype=torch.float64)
        c = torch.where(self.steps > 0, y.reshape(-1) * self.norm, torch.zeros_like(self.norm))
        for cells in self.cells():
            for at, w in cells:
                acc.index_add_(0, at, w * c)
        return acc.view(self.size[1] + 4, self.pitch)[2:-2, 2:-2].contiguous()


def fan_forward64(case, vectors, image):
    step = max(1, (1 << 24) // case["det"])
    parts = [FanRays(case, vectors[v0:v0 + step], image.device).forward(image)
             for v0 in range(0, case["views"], step)]
    return torch.cat(parts).view(case["views"], case["det"])


def fan_adjoint64(case, vectors, y):
    step = max(1, (1 << 24) // case["det"])
    return sum(FanRays(case, vectors[v0:v0 + step], y.device).adjoint(y[v0:v0 + step])
               for v0 in range(0, case["views"], step))


def fan_backward64(case, vectors, sino):
    h, w, det = case["height"], case["width"], case["det"]
    dev = sino.device
    X = torch.arange(w, device=dev, dtype=torch.float64)[None, :] - w / 2 + 0.5
    Y = torch.arange(h, device=dev, dtype=torch.float64)[:, None] - h / 2 + 0.5
    rows = torch.nn.functional.pad(sino.double(), (2, 2))
    acc = torch.zeros((h, w), device=dev, dtype=torch.float64)
    for row, (sx, sy, cx, cy, ux, uy) in zip(rows, np.asarray(vectors).tolist()):
        dx, dy = X - sx, Y - sy
        den = dx * uy - dy * ux                          # (P - S) x U
        mag = ((cx - sx) * uy - (cy - sy) * ux) / den
        t = (dy * (sx - cx) - dx * (sy - cy)) / -den     # cells from the centre
        u = t + (det / 2 - 0.5)
        f = u.floor()
        i = f.clamp(-2, det).long() + 2
        a, b = row[i], row[(i + 1).clamp_max_(det + 3)]
        acc += (a + (u - f) * (b - a)) * mag
    return acc / case["spacing"]


def ramp64(sino):
    n = sino.shape[-1]
    w = torch.as_tensor(np.fft.fftshift(np.abs(np.linspace(-1, 1, n))), device=sino.device)
    return torch.fft.ifft(torch.fft.fft(sino.double()) * w).real


class ConeRays:
    """The rays of some views: entry, step, count."""

    def __init__(self, case, rays, device):
        src, org, du, dv = (torch.as_tensor(a, device=device) for a in rays)
        u = torch.arange(case["cols"], device=device, dtype=torch.float64)[None, None, :]
        v = torch.arange(case["rows"], device=device, dtype=torch.float64)[None, :, None]
        self.size = (case["width"], case["height"], case["depth"])
        g = lambda a, k: a[:, k, None, None]  # noqa: E731
        d = [g(org, k) - g(src, k) + u * g(du, k) + v * g(dv, k) for k in range(3)]
        lo = torch.full_like(d[0], torch.finfo(torch.float32).tiny)
        hi = torch.full_like(d[0], torch.finfo(torch.float32).max)
        for k, n in enumerate(self.size):
            t1, t2 = (-1 - g(src, k)) / d[k], (n + 1 - g(src, k)) / d[k]
            lo = torch.minimum(torch.maximum(t1, lo), torch.maximum(t2, lo))
            hi = torch.maximum(torch.minimum(t1, hi), torch.minimum(t2, hi))
        samples = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]).sqrt_().ceil_()
        steps = torch.where(lo <= hi, ((hi - lo) * samples).ceil(), torch.zeros_like(lo))
        hit = (steps > 0).reshape(-1)
        self.hit = hit.nonzero()[:, 0]
        self.count = hit.numel()
        take = lambda a: a.reshape(-1)[self.hit]  # noqa: E731
        self.steps = take(steps)
        h = take(hi - lo) / self.steps
        full = [g(src, k) + d[k] * lo for k in range(3)]
        self.p = [take(p) for p in full]
        self.v = [take(x) * h for x in d]
        self.pitch = (self.size[0] + 5, self.size[1] + 5)

    def cells(self):
        for j in range(int(self.steps.max()) + 1 if self.steps.numel() else 0):
            w, idx = [], []
            for k in range(3):
                p = self.p[k] + j * self.v[k]
                f = p.floor()
                w.append(p - f)
                idx.append(f.clamp_(-2, self.size[k] + 1).long() + 2)
            base = (idx[2] * self.pitch[1] + idx[1]) * self.pitch[0] + idx[0]
            on = (self.steps >= j).double()
            for c in (0, 1):
                wz = on * (w[2] if c else 1 - w[2])
                for b in (0, 1):
                    wy = wz * (w[1] if b else 1 - w[1])
                    at = base + (c * self.pitch[1] + b) * self.pitch[0]
                    wx = wy * w[0]
                    yield at, wy - wx
                    yield at + 1, wx

    def forward(self, vol):
        flat = torch.nn.functional.pad(vol.double(), (2, 3, 2, 3, 2, 3)).reshape(-1)
        acc = torch.zeros_like(self.steps)
        for at, w in self.cells():
            acc += w * flat[at]
        out = torch.zeros(self.count, device=vol.device, dtype=torch.float64)
        out[self.hit] = acc
        return out

    def adjoint(self, y, acc):
        c = y.reshape(-1)[self.hit]
        for at, w in self.cells():
            acc.index_add_(0, at, w * c)


def cone_parts(case):
    rays = cone_rays(case)
    step = max(1, (1 << 24) // (case["rows"] * case["cols"]))
    for v0 in range(0, case["views"], step):
        yield v0, [a[v0:v0 + step] for a in rays]


def cone_forward64(case, vol):
    shape = (case["views"], case["rows"], case["cols"])
    return torch.cat([ConeRays(case, part, vol.device).forward(vol)
                      for _, part in cone_parts(case)]).view(shape)


def cone_adjoint64(case, y):
    size = (case["depth"] + 5, case["height"] + 5, case["width"] + 5)
    acc = torch.zeros(size[0] * size[1] * size[2], device=y.device, dtype=torch.float64)
    for v0, part in cone_parts(case):
        ConeRays(case, part, y.device).adjoint(y[v0:v0 + len(part[0])], acc)
    return acc.view(size)[2:-3, 2:-3, 2:-3].contiguous()


def cone_backward64(case, sino):
    dev, shape = sino.device, (case["width"], case["height"], case["depth"])
    R, dod = rpy_matrix(cone_rotation(case)), case["dsd"] - case["dso"]
    src = R @ np.array([0.0, 0.0, -case["dso"] - dod]) + np.array([0.0, 0.0, dod])
    x, y, z = (torch.arange(n, device=dev, dtype=torch.float64) - n / 2 + 0.5 for n in shape)
    acc = torch.zeros(shape[::-1], device=dev, dtype=torch.float64)
    rows, cols = case["rows"], case["cols"]
    pitch = cols + 4
    for view, phi in zip(sino, fan_angles(case).astype(np.float64)):
        flat = torch.nn.functional.pad(view.double(), (2, 2, 2, 2)).reshape(-1)
        M = R @ orbit_matrix(phi)
        off = R @ np.array([0.0, 0.0, -dod]) + np.array([0.0, 0.0, dod]) - src
        d = [(M[k, 2] * z)[:, None, None] + (M[k, 1] * y)[None, :, None]
             + (M[k, 0] * x)[None, None, :] + off[k] for k in range(3)]
        t = (case["dso"] - case["dsd"] - src[2]) / d[2]
        idx, w = [], []
        for k, n in ((0, cols), (1, rows)):
            p = d[k] * t + (src[k] + n // 2 - 0.5)
            f = p.floor()
            w.append(p - f)
            idx.append(f.clamp_(-2, n).long() + 2)
        at = idx[1] * pitch + idx[0]
        top = torch.lerp(flat[at], flat[at + 1], w[0])
        low = torch.lerp(flat[at + pitch], flat[at + pitch + 1], w[0])
        acc += torch.lerp(top, low, w[1])
    return acc


def exact(case, seed):
    dev = torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")
    op = case["op"]
    if op == "batch":
        ys, grads = [], []
        for k, f in enumerate(batch_fans(case)):
            v = fan_vectors(f, seed + k)
            y = fan_forward64(f, v, fan_image(f, seed + k, dev))
            r = y - fan_sinogram(f, seed + k, dev).double()
            ys.append(y.reshape(-1))
            grads.append(fan_backward64(f, v, r).reshape(-1))
        return {"sinograms": torch.cat(ys), "grad": torch.cat(grads)}
    if op.startswith("cone_"):
        if case["depth"] * case["height"] * case["width"] * case["views"] > 2.5e10:
            return None  # minutes in 64 bits
        if op == "cone_forward":
            return cone_forward64(case, cone_volume(case, seed, dev))
        if op == "cone_backward":
            return cone_backward64(case, cone_projections(case, seed, dev))
        y = cone_forward64(case, 0.8 * cone_volume(case, seed, dev))
        return {"sinogram": y,
                "grad": cone_adjoint64(case, y - cone_projections(case, seed, dev).double())}
    v = fan_vectors(case, seed)
    if op == "forward":
        return fan_forward64(case, v, fan_image(case, seed, dev))
    sino = fan_sinogram(case, seed, dev)
    if op == "backward":
        return fan_backward64(case, v, sino)
    if op == "half":
        scale = 2.0 / case["height"]
        return {"sinogram": fan_forward64(case, v, (fan_image(case, seed, dev) * scale).half()),
                "volume": fan_backward64(case, v, (sino * scale).half())}
    if op == "fbp":
        return fan_backward64(case, v, ramp64(sino) * (math.pi / (2 * case["views"])))
    y = fan_forward64(case, v, 0.8 * fan_image(case, seed, dev))
    return {"sinogram": y, "grad": fan_adjoint64(case, v, y - sino.double())}
