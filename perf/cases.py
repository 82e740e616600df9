"""Performance cases of the projector framework: the work its users have it do, through the public ops.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` makes what a
program holds before the call (inputs on the GPU and the scan's geometry), ``run`` is one pass, ``work`` the
bytes and operations a pass cannot do without, and ``exact`` the same results in 64-bit torch arithmetic.

Inputs are synthetic: ellipse / ellipsoid phantoms and their analytic line integrals, drawn from the seed.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pyro-nn-layers_b200"))

import pyronn_layers as pl  # noqa: E402
from pyronn_layers import fbp, geometry  # noqa: E402

DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
DEV = "cuda"


# ------------------------------------------------------------------ the cases


def _case2d(name, op, beam, batch, y, x, views, width, dtype="fp32"):
    # pixel pitches as the fan batch and the parallel slice of the benchmark have them
    return {"name": name, "op": op, "beam": beam, "batch": batch, "y": y, "x": x, "views": views, "width": width,
            "dtype": dtype}


def _case3d(name, op, batch, z, y, x, views, height, width, pitch, voxel, sid, sdd, dtype="fp32", hw=False):
    return {"name": name, "op": op, "beam": "cone", "batch": batch, "z": z, "y": y, "x": x, "views": views,
            "height": height, "width": width, "pitch": pitch, "voxel": voxel, "sid": sid, "sdd": sdd, "dtype": dtype,
            "hw": hw}


def listed():
    return [
        # one parallel-beam slice in a training loop (forward and gradient): the smallest call, latency counts
        _case2d("par2d_256_train", "train", "par", 1, 256, 256, 180, 367),
        # a batch of fan-beam slices as a data pipeline projects it, 16-bit storage
        _case2d("fan2d_512_b64_fwd_fp16", "fwd", "fan", 64, 512, 512, 360, 1024, "fp16"),
        # the same batch backprojected
        _case2d("fan2d_512_b64_back_fp16", "back", "fan", 64, 512, 512, 360, 1024, "fp16"),
        # a small mini-batch of odd-sized slices trained in FP32
        _case2d("fan2d_odd_b3_train", "train", "fan", 3, 387, 451, 301, 777),
        # filtered backprojection of a stack of parallel-beam slices (odd detector rows)
        _case2d("par2d_fbp_b16", "fbp", "par", 16, 256, 256, 360, 367),
        # the unrolled-reconstruction mini-batch: four volumes, forward and paired gradient, FP32
        _case3d("cone128_b4_train", "train", 4, 128, 128, 128, 180, 256, 256, 1.5, 1.0, 600.0, 1000.0),
        # the same scan with the exact transpose as gradient, one volume
        _case3d("cone128_matched_train", "matched", 1, 128, 128, 128, 180, 256, 256, 1.5, 1.0, 600.0, 1000.0),
        # an odd-sized volume and detector in BF16, forward and gradient
        _case3d("cone_odd_train_bf16", "train", 1, 181, 203, 219, 271, 287, 347, 0.8, 0.5, 750.0, 1200.0, "bf16"),
        # the texture-interpolation option, forward and gradient
        _case3d("cone160_hw_train", "train", 1, 160, 160, 160, 240, 320, 320, 1.0, 0.5, 750.0, 1200.0, hw=True),
        # the large scan: forward projection, 16-bit storage
        _case3d("cone512_fwd_fp16", "fwd", 1, 512, 512, 512, 360, 768, 1024, 1.0, 0.5, 750.0, 1200.0, "fp16"),
        # the large scan: backprojection
        _case3d("cone512_back_fp16", "back", 1, 512, 512, 512, 360, 768, 1024, 1.0, 0.5, 750.0, 1200.0, "fp16"),
        # FDK reconstruction of a mid-size scan (ramp filter into FP32, then backprojection)
        _case3d("cone256_fdk_fp16", "fdk", 1, 256, 256, 256, 360, 512, 512, 1.0, 0.5, 750.0, 1200.0, "fp16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    dtype = rng.choice(["fp32", "fp32", "fp16", "bf16"])
    if rng.random() < 0.5:
        op = rng.choice(["train", "train", "fwd", "back", "fbp"])
        y = _log_int(rng, 128, 640)
        x = max(96, min(640, int(y * rng.uniform(0.8, 1.25))))
        batch = _log_int(rng, 1, 48)
        c = _case2d("", op, rng.choice(["par", "fan"]), batch, y, x, _log_int(rng, 90, 480),
                    int(max(x, y) * rng.uniform(1.3, 2.0)), dtype)
    else:
        op = rng.choice(["train", "train", "matched", "fwd", "back", "fdk"])
        n = _log_int(rng, 56, 128 if op == "matched" else 288)
        z, y, x = (max(40, int(n * rng.uniform(0.8, 1.2))) for _ in range(3))
        batch = rng.choice([1, 1, 2, 3]) if n <= 160 else 1
        height, width = int(n * rng.uniform(1.4, 2.0)), int(n * rng.uniform(1.5, 2.1))
        voxel, sid, sdd = rng.choice([(0.5, 750.0, 1200.0), (1.0, 600.0, 1000.0)])
        # a detector 1.2 to 2.4 times as wide as the volume's shadow
        pitch = round(rng.uniform(1.2, 2.4) * voxel * sdd / sid * max(x, y) / width, 2)
        c = _case3d("", op, batch, z, y, x, _log_int(rng, 60, 360), height, width, pitch, voxel, sid, sdd, dtype,
                    op in ("train", "fwd", "back") and rng.random() < 0.2)
    del c["name"]
    return c


# ------------------------------------------------------------------- geometry


def _geometry(c):
    if c["beam"] == "par":
        return geometry.ParallelBeam2D((c["y"], c["x"]), (1.0, 1.0), c["width"], 1.0, c["views"])
    if c["beam"] == "fan":
        return geometry.FanBeam2D((c["y"], c["x"]), (0.5, 0.5), c["width"], 0.5, c["views"], 750.0, 1200.0)
    return geometry.ConeBeam3D((c["z"], c["y"], c["x"]), (c["voxel"],) * 3, (c["height"], c["width"]),
                               (c["pitch"],) * 2, c["views"], c["sid"], c["sdd"], step_size=0.5)


# --------------------------------------------------------------------- inputs


def _ellipsoids(rng, n, half):
    """n ellipsoids inside the box of half extents `half` (mm, x y [z]): centre, semi-axes, angle, density."""
    out = []
    for k in range(n):
        big = k == 0
        axes = [h * (rng.uniform(0.7, 0.9) if big else rng.uniform(0.06, 0.35)) for h in half]
        centre = [0.0 if big else rng.uniform(-0.5, 0.5) * h for h in half]
        out.append((centre, axes, rng.uniform(0.0, math.pi), 0.02 if big else rng.uniform(-0.008, 0.02)))
    return out


def _phantoms(c, geo, seed):
    half = [0.5 * float(n) * float(s) for n, s in zip(geo.volume_shape[::-1], geo.volume_spacing[::-1])]
    rng = random.Random(seed)
    return [_ellipsoids(rng, 10, half) for _ in range(c["batch"])]


def _volume(c, geo, seed):
    """[batch, (z), y, x] FP32 phantom volumes."""
    axes = [torch.arange(n, device=DEV, dtype=torch.float32) * float(s) + float(o)
            for n, s, o in zip(geo.volume_shape, geo.volume_spacing, geo.volume_origin)]
    y, x = axes[-2][:, None], axes[-1][None, :]
    out = torch.zeros((c["batch"],) + geo.volume_shape, device=DEV)
    for b, bodies in enumerate(_phantoms(c, geo, seed)):
        for ctr, ax, phi, rho in bodies:
            cs, sn = math.cos(phi), math.sin(phi)
            p = ((x - ctr[0]) * cs + (y - ctr[1]) * sn) / ax[0]
            q = ((y - ctr[1]) * cs - (x - ctr[0]) * sn) / ax[1]
            r = p * p + q * q
            if len(axes) == 3:
                w = (axes[0] - ctr[2]) / ax[2]
                for k in range(0, len(w), 64):
                    out[b, k:k + 64] += rho * ((w[k:k + 64] ** 2)[:, None, None] + r <= 1.0)
            else:
                out[b] += rho * (r <= 1.0)
    return out


def _sinogram(c, geo, seed):
    """[batch, views, (height), width] FP32 line integrals of the phantoms."""
    width = geo.detector_shape[-1]
    out = torch.zeros((c["batch"],) + tuple(geo.detector_shape), device=DEV)
    full = math.pi if c["beam"] == "par" else 2.0 * math.pi
    theta = torch.arange(c["views"], device=DEV, dtype=torch.float32) * (full / c["views"])
    three = c["beam"] == "cone"
    if three:
        u = (torch.arange(width, device=DEV) - (width - 1) / 2.0) * geo.detector_spacing[1]
        height = geo.detector_shape[1]
        v = ((torch.arange(height, device=DEV) - (height - 1) / 2.0) * geo.detector_spacing[0])[None, :, None]
        u = u[None, None, :]
    else:
        u = (torch.arange(width, device=DEV) * float(geo.detector_spacing[0]) + float(geo.detector_origin[0]))[None, :]
    chunk = max(1, (1 << 25) // (geo.detector_shape[-1] * (geo.detector_shape[1] if three else 1)))
    for k in range(0, c["views"], chunk):
        t = theta[k:k + chunk].reshape((-1, 1, 1) if three else (-1, 1))
        ct, st = torch.cos(t), torch.sin(t)
        if c["beam"] == "par":
            sx, sy, dx, dy = -st * u, ct * u, ct + 0 * u, st + 0 * u
        else:
            sid, sdd = (geo.sid, geo.sdd) if three else (float(geo.sid[0]), float(geo.sdd[0]))
            sx, sy, dx, dy = -sid * ct, -sid * st, ct * sdd - st * u, st * sdd + ct * u
        norm = torch.sqrt(dx * dx + dy * dy + v * v) if three else torch.sqrt(dx * dx + dy * dy)
        for b, bodies in enumerate(_phantoms(c, geo, seed)):
            for ctr, ax, phi, rho in bodies:
                cs, sn = math.cos(phi), math.sin(phi)
                ox, oy = sx - ctr[0], sy - ctr[1]
                o0, o1 = (ox * cs + oy * sn) / ax[0], (oy * cs - ox * sn) / ax[1]
                d0, d1 = (dx * cs + dy * sn) / ax[0], (dy * cs - dx * sn) / ax[1]
                dd, od, oo = d0 * d0 + d1 * d1, o0 * d0 + o1 * d1, o0 * o0 + o1 * o1
                if three:
                    dd, od, oo = dd + (v / ax[2]) ** 2, od - ctr[2] * v / ax[2] ** 2, oo + (ctr[2] / ax[2]) ** 2
                disc = (od * od - dd * (oo - 1.0)).clamp_min_(0.0)
                out[b, k:k + chunk] += (2.0 * rho) * torch.sqrt(disc) / dd * norm
    return out


def prepare(case, seed):
    c = dict(case)
    geo = _geometry(c)
    dt = DTYPES[c["dtype"]]
    s = {"case": c, "geo": geo, "args": geo.args()}
    if c["op"] in ("fwd", "train", "matched"):
        s["x"] = _volume(c, geo, seed).to(dt).requires_grad_(c["op"] != "fwd")
    if c["op"] in ("back", "fbp", "fdk"):
        s["p"] = _sinogram(c, geo, seed).to(dt)
    if c["op"] in ("train", "matched"):
        # the loss's gradient with respect to the projections: a noisy residual
        gen = torch.Generator(device=DEV).manual_seed(int(seed))
        r = _sinogram(c, geo, seed + 1000)
        s["r"] = (0.1 * r + 0.05 * torch.randn(r.shape, device=DEV, generator=gen)).to(dt)
    return s


# ------------------------------------------------------------------- one pass


def _project(c, geo, args, x):
    if c["beam"] == "cone":
        more = {"matched_adjoint": True} if c["op"] == "matched" else {"hardware_interp": c["hw"]}
        return pl.cone_projection3d(x, geo.detector_shape, *args, **more)
    f = pl.fan_projection2d if c["beam"] == "fan" else pl.parallel_projection2d
    return f(x, geo.detector_shape, *args)


def _backproject(c, geo, args, p):
    if c["beam"] == "cone":
        return pl.cone_backprojection3d(p, geo.volume_shape, *args, hardware_interp=c["hw"])
    f = pl.fan_backprojection2d if c["beam"] == "fan" else pl.parallel_backprojection2d
    return f(p, geo.volume_shape, *args)


def run(state):
    c, geo, args = state["case"], state["geo"], state["args"]
    if c["op"] == "fwd":
        return _project(c, geo, args, state["x"])
    if c["op"] == "back":
        return _backproject(c, geo, args, state["p"])
    if c["op"] == "fbp":
        return fbp.fbp_reconstruct_2d(state["p"], geo)
    if c["op"] == "fdk":
        return fbp.fdk_reconstruct(state["p"], geo)
    y = _project(c, geo, args, state["x"])
    (gx,) = torch.autograd.grad(y, state["x"], state["r"])
    return y.detach(), gx


def _samples(c, geo):
    """Ray samples of a forward projection (rays through the volume times its extent, over the step)."""
    voxels = float(np.prod(geo.volume_shape))
    if c["beam"] == "cone":
        pitch = c["pitch"] * c["sid"] / (c["sdd"] * c["voxel"])
        return c["batch"] * c["views"] * voxels / (pitch * pitch * 0.5)
    mag = 1.6 if c["beam"] == "fan" else 1.0
    pitch = float(geo.detector_spacing[0]) / (mag * float(geo.volume_spacing[0]))
    return c["batch"] * c["views"] * voxels / (pitch * 0.2)


def work(case):
    c = dict(case)
    geo = _geometry(c)
    e = 2 if c["dtype"] != "fp32" else 4
    vol = float(c["batch"]) * float(np.prod(geo.volume_shape))
    sino = float(c["batch"]) * float(np.prod(geo.detector_shape))
    three = c["beam"] == "cone"
    fwd_flops = _samples(c, geo) * (15 if three else 7)   # the sample's lerps and its addition
    back_flops = vol * c["views"] * (8 if three else 4)   # the update's lerps, weight and addition
    one = (vol + sino) * e
    if c["op"] == "fwd":
        return {"bytes": one, "flops": fwd_flops}
    if c["op"] == "back":
        return {"bytes": one, "flops": back_flops}
    if c["op"] in ("fbp", "fdk"):
        n = 1 << (2 * c["width"] - 1).bit_length()
        return {"bytes": sino * e + vol * 4, "flops": back_flops + sino / c["width"] * 5 * n * math.log2(n)}
    if c["op"] == "matched":
        return {"bytes": one + sino * e + vol * 4, "flops": 2 * fwd_flops}
    return {"bytes": 2 * one, "flops": fwd_flops + back_flops}


# ---------------------------------------------------------- 64-bit restatement


def _t64(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=DEV)


def _box(lo, hi, src, d):
    """Entry and exit parameters of rays (per axis lists) with the box, as the ops' slab test has them."""
    amin = amax = None
    for k in range(len(src)):
        a0, a1 = (lo[k] - src[k]) / d[k], (hi[k] - src[k]) / d[k]
        n, f = torch.minimum(a0, a1), torch.maximum(a0, a1)
        n, f = torch.where(d[k] == 0, torch.zeros_like(n), n), torch.where(d[k] == 0, torch.full_like(f, math.inf), f)
        if amin is None:
            amin, amax = n, f
        else:
            amin = torch.where(d[k] == 0, amin, torch.maximum(amin, n))
            amax = torch.where(d[k] == 0, amax, torch.minimum(amax, f))
    return amin, amax


class _Grid:
    """Multilinear interpolation of [batch, ...] values on a grid, zero outside it; coordinates x first."""

    def __init__(self, vol):
        self.b = vol.shape[0]
        self.n = list(vol.shape[1:])[::-1]
        pad = [2, 2] * len(self.n)
        padded = torch.nn.functional.pad(vol.double(), pad)
        self.m = list(padded.shape[1:])[::-1]
        self.flat = padded.reshape(self.b, -1)

    def corners(self, pos):
        base, frac, stride = 0, [], []
        s = 1
        for k, p in enumerate(pos):
            p = p.clamp(-2.0, self.n[k] + 0.999)
            f = torch.floor(p)
            frac.append(p - f)
            base = base + (f.long() + 2) * s
            stride.append(s)
            s *= self.m[k]
        for c in range(1 << len(pos)):
            w, off = 1.0, 0
            for k in range(len(pos)):
                hi = (c >> k) & 1
                w = w * (frac[k] if hi else 1.0 - frac[k])
                off += hi * stride[k]
            yield base + off, w

    def __call__(self, pos):
        out = 0.0
        for idx, w in self.corners(pos):
            out = out + self.flat[:, idx] * w
        return out


def _march(grid, origin, gain, a, am, step, scale):
    """The ops' trapezoid march: positions origin + alpha gain (index units), alpha kept in 32 bits."""
    n = a.numel()
    total = torch.zeros((grid.b, n), dtype=torch.float64, device=DEV)
    last, a_end = torch.zeros_like(total), a.clone()
    ids = torch.nonzero(a < am).reshape(-1)
    k = 0
    while ids.numel():
        o, g, ca, cam = [t[ids] for t in origin], [t[ids] for t in gain], a_end[ids], am[ids]
        acc, lv = total[:, ids], last[:, ids]
        for _ in range(32):
            live = ca < cam
            v = grid([p + ca.double() * q for p, q in zip(o, g)])
            lv = torch.where(live, v, lv)
            acc = acc + torch.where(live, v * (0.5 if k == 0 else 1.0), torch.zeros_like(v))
            ca = torch.where(live, ca + step, ca)
            k += 1
        total[:, ids], last[:, ids], a_end[ids] = acc, lv, ca
        ids = ids[ca < cam]
    st = float(step)
    end = grid([p + am.double() * q for p, q in zip(origin, gain)])
    seg = am.double() - (a_end - step).double()
    total *= st
    fixed = total - 0.5 * st * last + 0.5 * seg * last + 0.5 * seg * end
    total = torch.where((total > 0) & (a < am), fixed, total)
    return total * scale


def _rays_2d(c, geo):
    """Per ray (view major): index-space origin and gain, entry, exit, step, millimetre scale."""
    s = [float(v) for v in geo.volume_spacing[::-1]]
    o = [float(v) for v in geo.volume_origin[::-1]]
    n = [geo.volume_shape[1], geo.volume_shape[0]]
    rays = _t64(geo.ray_vectors)
    f32 = np.float32
    uu = torch.arange(c["width"], device=DEV, dtype=torch.float64)[None, :]
    uu = uu * float(geo.detector_spacing[0]) + float(geo.detector_origin[0])
    rx, ry = rays[:, :1], rays[:, 1:]
    if c["beam"] == "par":
        uu = uu.float().double()
        sx, sy = f32(s[0]), f32(s[1])
        sid = float(f32(np.sqrt(f32(f32(n[0]) * sx * f32(n[0]) * sx + f32(n[1]) * sy * f32(n[1]) * sy)) * f32(1.2)))
        src = [((rx.float() * -sid).double() - ry * uu).float().double(),
               ((ry.float() * -sid).double() + rx * uu).float().double()]
        d = [rx.expand_as(src[0]), ry.expand_as(src[0])]
    else:
        sid, sdd = float(geo.sid[0]), float(geo.sdd[0])
        lx, ly = rx * sdd - ry * uu, ry * sdd + rx * uu
        inv = 1.0 / torch.sqrt(lx * lx + ly * ly)
        d = [lx * inv, ly * inv]
        src = [(rx * -sid).expand_as(lx), (ry * -sid).expand_as(lx)]
    d, src = [t.reshape(-1) for t in d], [t.reshape(-1) for t in src]
    amin, amax = _box([o[k] - 0.5 for k in (0, 1)], [n[k] * s[k] + o[k] - 0.5 for k in (0, 1)], src, d)
    step = float(f32(0.2) * min(f32(s[0]), f32(s[1])))
    hit = amin < amax
    a, am = amin.float(), torch.where(hit, amax, amin).float()
    scale = torch.sqrt((d[0] * s[0]) ** 2 + (d[1] * s[1]) ** 2)
    return [(src[k] - o[k]) / s[k] for k in (0, 1)], [d[k] / s[k] for k in (0, 1)], a, am, step, scale


def _decomposed(geo):
    p = _t64(geo.projection_matrices)
    s, o = _t64(geo.volume_spacing[::-1].copy()), _t64(geo.volume_origin[::-1].copy())
    inv = torch.linalg.inv(p[:, :, :3])
    src = (-(inv @ p[:, :, 3:])[:, :, 0] - o) / s
    return inv / s[None, :, None], src, s


def _rays_3d(c, geo, views):
    inv, src, s = _decomposed(geo)
    inv, src = inv[views], src[views]
    h, w = c["height"], c["width"]
    v = torch.arange(h, device=DEV, dtype=torch.float64)[None, :, None]
    u = torch.arange(w, device=DEV, dtype=torch.float64)[None, None, :]
    d = [inv[:, k, 2, None, None] + v * inv[:, k, 1, None, None] + u * inv[:, k, 0, None, None] for k in range(3)]
    length = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
    d = [(t / length).reshape(-1) for t in d]
    o = [src[:, k, None, None].expand(-1, h, w).reshape(-1) for k in range(3)]
    lo = -0.5 if c["hw"] else 0.0
    amin, amax = _box([lo] * 3, [n + lo for n in geo.volume_shape[::-1]], o, d)
    step = float(np.float32(0.5))
    hit = amin < amax
    a, am = amin.float() + np.float32(0.5 * step), torch.where(hit, amax, amin).float()
    a = torch.where(hit, a, am)
    scale = torch.sqrt(sum((d[k] * s[k]) ** 2 for k in range(3)))
    return o, d, a, am, step, scale


def _exact_forward(c, geo, x):
    grid = _Grid(x)
    shape = (c["batch"],) + tuple(geo.detector_shape)
    if c["beam"] != "cone":
        return _march(grid, *_rays_2d(c, geo)).reshape(shape)
    out = torch.zeros(shape, dtype=torch.float64, device=DEV)
    chunk = max(1, (1 << 22) // (c["height"] * c["width"]))
    for k in range(0, c["views"], chunk):
        views = slice(k, min(k + chunk, c["views"]))
        part = _march(grid, *_rays_3d(c, geo, views))
        out[:, views] = part.reshape(c["batch"], -1, c["height"], c["width"])
    return out


def _exact_back_2d(c, geo, p):
    ax = [_t64(np.arange(n) * float(s) + float(o)) for n, s, o in
          zip(geo.volume_shape, geo.volume_spacing, geo.volume_origin)]
    cy, cx = ax[0][:, None], ax[1][None, :]
    rays = np.asarray(geo.ray_vectors, dtype=np.float64)
    p = torch.nn.functional.pad(p.double(), (2, 2))
    out = torch.zeros((c["batch"],) + geo.volume_shape, dtype=torch.float64, device=DEV)
    for n in range(c["views"]):
        rx, ry = rays[n]
        s, w = cy * rx - cx * ry, 1.0
        if c["beam"] == "fan":
            sid, sdd = float(geo.sid[0]), float(geo.sdd[0])
            rr = rx * rx + ry * ry
            s = sdd * rr * s / (cx * rx + cy * ry + sid * rr)
            w = 1.0 / ((cx + rx * sid) ** 2 + (cy + ry * sid) ** 2)
        i = (s - float(geo.detector_origin[0])) / float(geo.detector_spacing[0])
        i = i.clamp(-2.0, c["width"] + 0.999)
        f = torch.floor(i)
        t, k = i - f, f.long() + 2
        row = p[:, n]
        out += (row[:, k] * (1.0 - t) + row[:, k + 1] * t) * w
    scale = float(np.float32(3.14159265359)) / c["views"]
    return out * (scale * float(geo.sid[0]) * float(geo.sdd[0]) if c["beam"] == "fan" else scale)


def _exact_back_3d(c, geo, p, mult=1.0):
    z, y, x = (_t64(np.arange(n)) * float(s) + float(o) for n, s, o in
               zip(geo.volume_shape, geo.volume_spacing, geo.volume_origin))
    x, y = x[None, None, :], y[None, :, None]
    m = np.asarray(geo.projection_matrices, dtype=np.float64)
    h, w, total = c["height"], c["width"], c["views"] * c["height"] * c["width"]
    # software taps with 0 <= x <= W, 0 <= y <= H come from the flat buffer; texture taps stop at W - 1, H - 1
    wmax, hmax = (w - 1, h - 1) if c["hw"] else (w, h)
    flat = torch.cat([p.reshape(c["batch"], -1), torch.zeros((c["batch"], 1), device=DEV, dtype=p.dtype)], 1)
    out = torch.zeros((c["batch"],) + geo.volume_shape, dtype=torch.float64, device=DEV)
    slab = max(1, (1 << 26) // (geo.volume_shape[1] * geo.volume_shape[2]))
    for k in range(0, geo.volume_shape[0], slab):
        zk = z[k:k + slab, None, None]
        for n in range(c["views"]):
            un, vn, wn = (m[n, r, 0] * x + m[n, r, 1] * y + (m[n, r, 2] * zk + m[n, r, 3]) for r in range(3))
            rw = 1.0 / wn
            u, v = (un * rw).clamp(-2.0, w + 2.0), (vn * rw).clamp(-2.0, h + 2.0)
            fu, fv = torch.floor(u), torch.floor(v)
            tu, tv = u - fu, v - fv
            val = 0.0
            for j in range(4):
                du, dv = j & 1, j >> 1
                xx, yy = fu.int() + du, fv.int() + dv
                idx = (yy + n * h) * w + xx
                ok = (xx >= 0) & (xx <= wmax) & (yy >= 0) & (yy <= hmax) & (idx < total)
                weight = (tu if du else 1.0 - tu) * (tv if dv else 1.0 - tv)
                tap = flat[:, torch.where(ok, idx, total)]
                val = val + tap.double() * weight
            out[:, k:k + slab] += val * rw * rw
    return out * mult


def _exact_matched(c, geo, r):
    """The transpose of the forward march (its end correction always applied)."""
    grid = _Grid(torch.zeros((c["batch"],) + geo.volume_shape, device=DEV))
    acc = torch.zeros_like(grid.flat)
    chunk = max(1, (1 << 22) // (c["height"] * c["width"]))
    for k in range(0, c["views"], chunk):
        views = slice(k, min(k + chunk, c["views"]))
        o, d, a, am, step, scale = _rays_3d(c, geo, views)
        val = r[:, views].reshape(c["batch"], -1).double() * scale

        def put(ids, al, weight):
            pos = [o[j][ids] + al.double() * d[j][ids] for j in range(3)]
            for idx, w in grid.corners(pos):
                for b in range(c["batch"]):
                    acc[b].index_add_(0, idx, w * weight * val[b, ids])

        ids = torch.nonzero(a < am).reshape(-1)
        al = a[ids]
        first = True
        while ids.numel():
            nxt = al + step
            end = ~(nxt < am[ids])
            seg = am[ids].double() - al.double()
            weight = torch.full_like(seg, 0.5 * step if first else step)
            weight = torch.where(end, weight - 0.5 * step + 0.5 * seg, weight)
            put(ids, al, weight)
            if bool(end.any()):
                put(ids[end], am[ids[end]], 0.5 * seg[end])
            ids, al, first = ids[~end], nxt[~end], False
    m = grid.m
    full = acc.reshape(c["batch"], m[2], m[1], m[0])
    return full[:, 2:-2, 2:-2, 2:-2]


def _exact_filter(c, geo, p):
    w = c["width"]
    if c["beam"] == "cone":
        du, (dv, _) = geo.detector_spacing[1], geo.detector_spacing
        sdd = geo.sdd
        u = (_t64(np.arange(w)) - (w - 1) / 2.0) * du
        v = (_t64(np.arange(c["height"])) - (c["height"] - 1) / 2.0) * dv
        r2 = u[None, :] ** 2 + v[:, None] ** 2
    else:
        du = float(geo.detector_spacing[0])
        sdd = float(geo.sdd[0]) if c["beam"] == "fan" else 0.0
        r2 = (_t64(np.arange(w)) * du + float(geo.detector_origin[0])) ** 2
    m = np.arange(-(w - 1), w)
    h = np.where(m == 0, 0.25 / du ** 2, np.where(m % 2 != 0, -1.0 / (math.pi ** 2 * np.maximum(m * m, 1) * du ** 2), 0.0))
    toeplitz = _t64(du * h)[(torch.arange(w, device=DEV)[:, None] - torch.arange(w, device=DEV)[None, :]) + w - 1]
    out = torch.empty(p.shape, dtype=torch.float64, device=DEV)
    for b in range(c["batch"]):
        for k in range(0, c["views"], 32):
            g = p[b, k:k + 32].double()
            if sdd > 0.0:
                g = g * (sdd / torch.sqrt(sdd * sdd + r2))
            out[b, k:k + 32] = g @ toeplitz
    return out


def exact(case, seed):
    c = dict(case)
    geo = _geometry(c)
    vol = float(np.prod(geo.volume_shape)) * c["batch"] * c["views"]
    # about 20 seconds of 64-bit arithmetic at most
    if c["op"] in ("fwd", "train", "matched") and _samples(c, geo) > 1.2e11 / (2.0 if c["beam"] == "cone" else 1.0):
        return None
    if c["op"] == "fwd" and vol > 1e10 and c["beam"] == "cone":
        return None
    s = prepare(case, seed)
    with torch.no_grad():
        if c["op"] == "fwd":
            return _exact_forward(c, geo, s["x"])
        if c["op"] in ("back", "fbp", "fdk"):
            p = s["p"]
            if c["op"] != "back":
                p = _exact_filter(c, geo, p)
            if c["beam"] != "cone":
                return _exact_back_2d(c, geo, p)
            return _exact_back_3d(c, geo, p, geo.sid * geo.sdd * math.pi / c["views"] if c["op"] == "fdk" else 1.0)
        y = _exact_forward(c, geo, s["x"])
        if c["op"] == "matched":
            return y, _exact_matched(c, geo, s["r"])
        return y, _exact_back_3d(c, geo, s["r"]) if c["beam"] == "cone" else _exact_back_2d(c, geo, s["r"])
