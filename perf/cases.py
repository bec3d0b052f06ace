"""What users of this framework have it do, as measurable cases: the plane
transform (both samplers, single, batched, through the drop-in call), the ray
transform (z-slices and rotated layers), the ray-to-Radon reduction, the
backprojection, and the serving loop.  Sizes are those of the benchmark, the
tests and the drop-in programs' defaults, from a few hundred plane integrals
to 7 million, odd and ragged ones among them.

The transforms compute in FP32 (their stated accuracy is 1e-5 against FP64)
and hand their sums over as doubles; the programs modelled here keep results
as float32, the precision they hold.  ``exact`` gives the reference's own FP64
arithmetic (cell index by truncation, fraction by fmod) wherever that is
affordable, so the accuracy is also checked against 64 bits.
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = Path(__file__).resolve().parents[1] / "wrt-project_b200"


def _package():
    if "wrt_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            "wrt_b200", _PKG / "__init__.py", submodule_search_locations=[str(_PKG)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["wrt_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["wrt_b200"]


_shared = {}


def _context():
    """One library context per program, as the drop-in programs and bench.py have."""
    if "ctx" not in _shared:
        torch.zeros(1, device="cuda")
        wrt = _package()
        _shared["ctx"] = wrt.Context(torch.cuda.current_device())
        _shared["stream"] = torch.cuda.ExternalStream(wrt.lib().wrt_ctx_stream(_shared["ctx"].handle))
    return _shared["ctx"], _shared["stream"]


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: one small volume, a coarse sphere grid (the sizes of smoke and
        # of the small-batch benchmark); launches and host work are all of it
        {"name": "planes_24", "op": "planes", "n": 24, "ntheta": 8, "nphi": 16, "nshift": 32,
         "sampler": "trilinear", "half": 24, "storage": "f32"},
        # many small volumes of uneven sizes in one batched launch
        {"name": "batch_32_small", "op": "batch", "count": 32, "nmin": 16, "nmax": 48,
         "thmin": 8, "thmax": 16, "smin": 32, "smax": 64},
        # the drop-in call on host arrays, radon_grid at 64^3 with the 128 x 128 quadrature
        {"name": "radon_grid_64", "op": "dropin", "n": 64, "ntheta": 32, "nphi": 64, "nshift": 128,
         "sampler": "trilinear", "half": 64},
        # radon_grid's default sampler and lattice (nearest, 4n x 4n) on a resident volume
        {"name": "planes_nearest_128", "op": "planes", "n": 128, "ntheta": 64, "nphi": 128,
         "nshift": 256, "sampler": "nearest", "half": 0, "storage": "f32"},
        # the benchmark's workload
        {"name": "planes_128", "op": "planes", "n": 128, "ntheta": 64, "nphi": 128, "nshift": 256,
         "sampler": "trilinear", "half": 128, "storage": "f32"},
        # nothing even, the reference's full lattice
        {"name": "planes_113_ragged", "op": "planes", "n": 113, "ntheta": 37, "nphi": 75,
         "nshift": 101, "sampler": "trilinear", "half": 0, "storage": "f32"},
        # the largest transform the framework is set up for, volume stored in bfloat16
        {"name": "planes_256_bf16", "op": "planes", "n": 256, "ntheta": 96, "nphi": 192,
         "nshift": 384, "sampler": "trilinear", "half": 256, "storage": "bf16"},
        # layer-by-layer rays, the reference's z-slices
        {"name": "rays_128", "op": "rays", "n": 128, "nslices": 128, "nshift": 128, "nphi": 128,
         "frames": 0},
        # ... and layers about other axes, odd sizes
        {"name": "rays_rotated_101", "op": "rays", "n": 101, "nslices": 101, "nshift": 127,
         "nphi": 90, "frames": 3},
        # ray data of one orientation to Radon data
        {"name": "reduction_128", "op": "reduction", "n": 128, "nshift_ray": 128, "ntheta": 64,
         "nphi": 128, "nshift": 256},
        # backprojection of the benchmark's Radon data
        {"name": "adjoint_128", "op": "adjoint", "n": 128, "ntheta": 64, "nphi": 128,
         "nshift": 256},
        # the serving loop: mixed requests of several callers, submitted together and waited for
        {"name": "serve_mix", "op": "serve", "requests": 12, "nmax": 96},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["planes", "planes", "planes", "dropin", "batch", "rays", "reduction",
                     "adjoint", "adjoint", "serve"])
    n = _log_int(rng, 20, 176)
    nth = _log_int(rng, 6, 64)
    nph = 2 * nth + rng.choice([0, 0, 1, -3])
    ns = _log_int(rng, 24, 256)
    if op in ("planes", "dropin"):
        c = {"op": op, "n": n, "ntheta": nth, "nphi": nph, "nshift": ns,
             "sampler": rng.choice(["trilinear", "trilinear", "nearest"]),
             "half": rng.choice([0, n])}
        if op == "planes":
            c["storage"] = rng.choice(["f32", "bf16"]) if c["sampler"] == "trilinear" else "f32"
        return c
    if op == "batch":
        lo = _log_int(rng, 12, 40)
        return {"op": "batch", "count": rng.randint(3, 40), "nmin": lo,
                "nmax": lo + rng.randint(3, 40), "thmin": 4, "thmax": rng.randint(8, 24),
                "smin": 16, "smax": rng.randint(24, 96)}
    if op == "rays":
        return {"op": "rays", "n": n, "nslices": max(4, n - rng.choice([0, 1, 7])),
                "nshift": _log_int(rng, 16, 160), "nphi": _log_int(rng, 16, 160),
                "frames": rng.choice([0, 0, 1, 2, 4])}
    if op == "reduction":
        return {"op": "reduction", "n": n, "nshift_ray": _log_int(rng, 16, 192), "ntheta": nth,
                "nphi": nph, "nshift": ns}
    if op == "adjoint":
        return {"op": "adjoint", "n": n, "ntheta": nth, "nphi": nph, "nshift": ns}
    return {"op": "serve", "requests": rng.randint(4, 16), "nmax": _log_int(rng, 32, 128)}


# ------------------------------------------------------------------ the inputs
def _phantom(n, seed, k=12):
    """A seeded phantom as the benchmark's: sums of ellipsoids inside radius 0.9."""
    _package()
    from wrt_b200.phantom import ellipsoid_phantom
    return ellipsoid_phantom(n, k, seed, dtype=np.float32)


def _frames(count, seed):
    from wrt_b200.phantom import layer_frames
    return list(layer_frames(count + 1, seed)[1:]) if count else [None]


def _batch_sizes(c, seed):
    """Sizes of the batch's requests: the same for every seed of a case."""
    r = np.random.default_rng(c["count"] * 1000 + c["nmin"])
    out = []
    for _ in range(c["count"]):
        nth = int(r.integers(c["thmin"], c["thmax"] + 1))
        out.append((int(r.integers(c["nmin"], c["nmax"] + 1)), nth, 2 * nth,
                    int(r.integers(c["smin"], c["smax"] + 1))))
    return out


def _serve_sizes(c):
    r = np.random.default_rng(c["requests"] * 1000 + c["nmax"])
    out = []
    for k in range(c["requests"]):
        op = ("forward", "forward", "adjoint", "forward", "rays", "reduction")[k % 6]
        n = int(r.integers(max(16, c["nmax"] // 3), c["nmax"] + 1))
        nth = int(r.integers(max(4, n // 6), max(6, n // 3) + 1))
        out.append((op, n, nth, 2 * nth, int(r.integers(n, 2 * n + 1))))
    return out


def _radon(nshift, nphi, ntheta, seed):
    """Radon data as the backprojection meets it: a smooth bump per direction and noise."""
    r = np.random.default_rng(seed)
    s = np.linspace(-1.0, 1.0, nshift)[:, None, None]
    c = r.uniform(-0.3, 0.3, (1, nphi, ntheta))
    g = np.clip(1.0 - ((s - c) / 0.7) ** 2, 0.0, None)
    return np.ascontiguousarray(g + 0.05 * r.standard_normal((nshift, nphi, ntheta)))


def _rays(n, nshift, nphi, seed):
    """Ray data [z][s][phi] of smooth layers (zero at the ends) with noise."""
    r = np.random.default_rng(seed)
    z = np.linspace(-1.0, 1.0, n)[:, None, None]
    s = np.linspace(-1.0, 1.0, nshift)[None, :, None]
    c = r.uniform(-0.2, 0.2, (1, 1, nphi))
    g = np.clip(1.0 - z ** 2 - (s - c) ** 2, 0.0, None)
    return np.ascontiguousarray(g * (1.0 + 0.1 * r.standard_normal((n, nshift, nphi))))


class _State:
    pass


def _f64_out(*shape):
    return torch.zeros(shape, dtype=torch.float64, device="cuda")


def prepare(c, seed):
    wrt, s = _package(), _State()
    s.c, s.op = c, c["op"]
    s.ctx, s.stream = _context()
    if s.op in ("planes", "dropin"):
        s.sampler = wrt.TRILINEAR if c["sampler"] == "trilinear" else wrt.NEAREST
        v = _phantom(c["n"], seed)
        if s.op == "dropin":
            s.volume = v.astype(np.float64)
            return s
        s.vol = wrt.Volume(s.ctx, c["n"],
                           wrt.STORAGE_BF16 if c["storage"] == "bf16" else wrt.STORAGE_F32)
        s.vol.upload(v)
        s.grid = wrt.Grid(s.ctx, c["nphi"], c["ntheta"], c["nshift"])
        s.out = _f64_out(c["nshift"], c["nphi"], c["ntheta"])
    elif s.op == "batch":
        s.reqs, s.keep = [], []
        for k, (n, nth, nph, ns) in enumerate(_batch_sizes(c, seed)):
            vol = wrt.Volume(s.ctx, n)
            vol.upload(_phantom(n, seed * 64 + k, 6))
            grid = wrt.Grid(s.ctx, nph, nth, ns)
            out = _f64_out(ns, nph, nth)
            s.keep.append(out)
            s.reqs.append((vol, grid, out.data_ptr(), n))
    elif s.op == "rays":
        s.vol = wrt.Volume(s.ctx, c["n"])
        s.vol.upload(_phantom(c["n"], seed))
        s.frames = _frames(c["frames"], seed)
        s.out = [_f64_out(c["nslices"], c["nshift"], c["nphi"]) for _ in s.frames]
    elif s.op == "reduction":
        s.data = torch.from_numpy(_rays(c["n"], c["nshift_ray"], c["nphi"], seed)).cuda()
        s.grid = wrt.Grid(s.ctx, c["nphi"], c["ntheta"], c["nshift"])
        s.out = _f64_out(c["nshift"], c["nphi"], c["ntheta"])
    elif s.op == "adjoint":
        s.data = torch.from_numpy(_radon(c["nshift"], c["nphi"], c["ntheta"], seed)).cuda()
        s.grid = wrt.Grid(s.ctx, c["nphi"], c["ntheta"], c["nshift"])
        s.out = _f64_out(c["n"], c["n"], c["n"])
    else:
        if "server" not in _shared:  # one serving process
            _shared["server"] = wrt.Server(torch.cuda.current_device(), budget_bytes=8 << 30)
        s.server = _shared["server"]
        s.jobs = []
        for k, (op, n, nth, nph, ns) in enumerate(_serve_sizes(c)):
            sd = seed * 64 + k
            if op == "forward":
                s.jobs.append((op, _phantom(n, sd, 6), nph, nth, ns, np.empty((ns, nph, nth))))
            elif op == "adjoint":
                s.jobs.append((op, _radon(ns, nph, nth, sd), n, np.empty((n, n, n))))
            elif op == "rays":
                s.jobs.append((op, _phantom(n, sd, 6), n, ns, nph, np.empty((n, ns, nph))))
            else:
                s.jobs.append((op, _rays(n, n, nph, sd), ns, nth, np.empty((ns, nph, nth))))
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    wrt, c = _package(), s.c
    if s.op == "dropin":
        return s.ctx.radon_grid(s.volume, c["nphi"], c["ntheta"], c["nshift"], sampler=s.sampler,
                                half_extent=c["half"]).astype(np.float32)
    if s.op == "serve":
        ids = []
        for j in s.jobs:
            if j[0] == "forward":
                ids.append(s.server.submit_forward(j[1], j[2], j[3], j[4], j[5],
                                                   half_extent=j[1].shape[0]))
            elif j[0] == "adjoint":
                ids.append(s.server.submit_adjoint(j[1], j[2], j[3]))
            elif j[0] == "rays":
                ids.append(s.server.submit_ray(j[1], j[2], j[3], j[4], j[5]))
            else:
                ids.append(s.server.submit_reduce(j[1], j[2], j[3], j[4]))
        for rid in ids:
            s.server.wait(rid, 60000)
        return [j[-1].astype(np.float32) for j in s.jobs]
    with torch.cuda.stream(s.stream):  # the library's stream: its work and torch's in order
        if s.op == "planes":
            wrt.radon_forward_device(s.ctx, s.vol, s.grid, s.out.data_ptr(), sampler=s.sampler,
                                     half_extent=c["half"])
            return s.out.float()
        if s.op == "batch":
            wrt.radon_forward_batch(s.ctx, s.reqs)
            return [o.float() for o in s.keep]
        if s.op == "rays":
            for f, o in zip(s.frames, s.out):
                wrt.ray_forward_device(s.ctx, s.vol, c["nslices"], c["nshift"], c["nphi"],
                                       o.data_ptr(), frame=f)
            return [o.float() for o in s.out]
        if s.op == "reduction":
            wrt.radon_reduction_device(s.ctx, s.data.data_ptr(), c["n"], c["nshift_ray"], s.grid,
                                       s.out.data_ptr())
            return s.out.float()
        wrt.radon3d_adjoint_device(s.ctx, s.data.data_ptr(), s.grid, c["n"], s.out.data_ptr())
        return s.out.float()


# ------------------------------------------------------------------ its work
def _planes_work(n, ndir, ns, vol_bytes):
    # one value read per node, one written per plane; a plane integral is at least one
    # multiply-add per lattice row of the unit ball's chord (a row's sum can be shared)
    return vol_bytes * n ** 3 + 8.0 * ndir * ns, 2.0 * ndir * ns * n


def _adjoint_work(n, ndir, ns):
    return 8.0 * ndir * ns + 8.0 * n ** 3, 2.0 * ndir * ns + 2.0 * n ** 3


def _rays_work(n, rays):
    return 4.0 * n ** 3 + 8.0 * rays, 2.0 * rays * n


def _reduction_work(n, nsr, nph, nth, ns):
    return 8.0 * n * nsr * nph + 8.0 * ns * nph * nth, 2.0 * ns * nph * nth * n


def work(c):
    if c["op"] in ("planes", "dropin"):
        b, f = _planes_work(c["n"], c["nphi"] * c["ntheta"], c["nshift"],
                            {"f32": 4, "bf16": 2}.get(c.get("storage"), 8))
    elif c["op"] == "batch":
        w = [_planes_work(n, nth * nph, ns, 4) for n, nth, nph, ns in _batch_sizes(c, 0)]
        b, f = sum(x[0] for x in w), sum(x[1] for x in w)
    elif c["op"] == "rays":
        k = max(1, c["frames"])
        b, f = _rays_work(c["n"], k * c["nslices"] * c["nshift"] * c["nphi"])
    elif c["op"] == "reduction":
        b, f = _reduction_work(c["n"], c["nshift_ray"], c["nphi"], c["ntheta"], c["nshift"])
    elif c["op"] == "adjoint":
        b, f = _adjoint_work(c["n"], c["nphi"] * c["ntheta"], c["nshift"])
    else:
        b = f = 0.0
        for op, n, nth, nph, ns in _serve_sizes(c):
            w = (_planes_work(n, nth * nph, ns, 4) if op == "forward" else
                 _adjoint_work(n, nth * nph, ns) if op == "adjoint" else
                 _rays_work(n, n * ns * nph) if op == "rays" else
                 _reduction_work(n, n, nph, nth, ns))
            b, f = b + w[0], f + w[1]
    return {"bytes": b, "flops": f}


# --------------------------------------------------- the same in 64 bits, torch
_CHUNK = 1 << 26  # samples at a time


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _sphere(nphi, ntheta, nshift):
    x, w = np.polynomial.legendre.leggauss(ntheta)
    phi = (2 * math.pi / nphi) * np.arange(nphi)
    return phi, np.arccos(x), w, -1.0 + np.arange(nshift) * (2.0 / (nshift - 1))


def _trilinear(v, n, x, y, z):
    """cube_trilinear_interp in torch: cell by truncation, fraction by fmod."""
    d = _dev([2.0 / (n - 1)])  # on the device: torch divides by it (a number it would invert)
    inside = (x.abs() <= 1.0) & (y.abs() <= 1.0) & (z.abs() <= 1.0)
    idx, fr = [], []
    for a in (x, y, z):
        a1 = (a + 1.0).clamp_(0.0, 2.0)
        i = (a1 / d).to(torch.int64)
        f = torch.fmod(a1, d) / d
        top = i >= n - 1
        fr.append(torch.where(top, torch.ones_like(f), f))
        idx.append(torch.where(top, torch.full_like(i, n - 2), i))
    base = (idx[0] * n + idx[1]) * n + idx[2]
    out = 0.0
    for k in range(8):
        w = 1.0
        for a in range(3):
            w = w * (fr[a] if (k >> a) & 1 else 1.0 - fr[a])
        out = out + w * v[base + ((k & 1) * n + ((k >> 1) & 1)) * n + (k >> 2)]
    return torch.where(inside, out, torch.zeros_like(out))


def _nearest(v, n, x, y, z):
    d = _dev([2.0 / n])
    inside = (x.abs() <= 1.0) & (y.abs() <= 1.0) & (z.abs() <= 1.0)
    b = 0
    for a in (x, y, z):
        b = b * n + ((a + 1.0) / d).to(torch.int64).clamp_(0, n - 1)
    return torch.where(inside, v[b], torch.zeros((), dtype=torch.float64, device=v.device))


def _support(v):
    """A radius that holds every sample that can be non-zero, in either sampler."""
    n = v.shape[0]
    t = -1.0 + np.arange(n) * (2.0 / (n - 1))
    r2 = t[:, None, None] ** 2 + t[None, :, None] ** 2 + t[None, None, :] ** 2
    r = math.sqrt(r2[v != 0].max()) if (v != 0).any() else 0.0
    return r + 3.5 * (4.0 / n + 2.0 / (n - 1))


def _exact_planes(v, nphi, ntheta, nshift, nearest, half):
    n = v.shape[0]
    L = half or 2 * n
    k = min(L, int(_support(v) * n) + 2)
    i = torch.arange(-k, min(k + 1, L), dtype=torch.float64, device="cuda")
    total = float(nphi) * ntheta * nshift * len(i) ** 2
    if total > 1.5e11:
        return None  # beyond about 20 seconds
    # the largest go through torch's own FP64 interpolation (no cell rule of the reference)
    big = total > 2e10 and not nearest
    cube = _dev(v)[None, None] if big else None
    phi, theta, _, shift = _sphere(nphi, ntheta, nshift)
    p, t = np.meshgrid(phi, theta, indexing="ij")
    om = lambda th: np.stack([np.sin(th) * np.cos(p), np.sin(th) * np.sin(p), np.cos(th)], -1)
    nrm, v1 = om(t).reshape(-1, 3), om(t + math.pi / 2).reshape(-1, 3)
    v2 = np.stack([nrm[:, 1] * v1[:, 2] - nrm[:, 2] * v1[:, 1],
                   -(nrm[:, 0] * v1[:, 2] - nrm[:, 2] * v1[:, 0]),
                   nrm[:, 0] * v1[:, 1] - nrm[:, 1] * v1[:, 0]], -1)
    nrm, v1, v2, sh, flat = _dev(nrm), _dev(v1), _dev(v2), _dev(shift), _dev(v).reshape(-1)
    delta = 1.0 / n
    out = torch.empty(nshift, nphi * ntheta, dtype=torch.float64, device="cuda")
    step = max(1, _CHUNK // (len(i) ** 2 * nshift))
    shifts = max(1, min(nshift, _CHUNK // len(i) ** 2))
    for d0 in range(0, nphi * ntheta, step):
        for s0 in range(0, nshift, shifts):
            sl, ss = slice(d0, d0 + step), slice(s0, s0 + shifts)
            q = []
            for a in range(3):
                row = (sh[ss, None, None] * nrm[sl, a][None, :, None] +
                       (delta * v1[sl, a])[None, :, None] * i)
                q.append(row[..., None] + (delta * v2[sl, a])[None, :, None, None] * i)
            if big:
                g = torch.stack(torch.broadcast_tensors(q[2], q[1], q[0]), -1)
                f = torch.nn.functional.grid_sample(
                    cube, g.reshape(1, 1, 1, -1, 3), align_corners=True).reshape(g.shape[:-1])
            else:
                f = (_nearest if nearest else _trilinear)(flat, n, *q)
            out[ss, sl] = f.sum(dim=(2, 3)) * delta ** 2
    return out.reshape(nshift, nphi, ntheta)


def _exact_rays(v, nslices, nshift, nphi, frame):
    n = v.shape[0]
    if float(nslices) * nshift * nphi * 2 * n > 3e10:
        return None
    flat = _dev(v).reshape(-1)
    delta = (2.0 / (n - 1)) / 2.0
    z = _dev(-1.0 + np.arange(nslices) * (2.0 / (nslices - 1)))
    sh = _dev(-1.0 + np.arange(nshift) * (2.0 / (nshift - 1)))
    phi = (2 * math.pi / nphi) * np.arange(nphi)
    m = min(2 * n, int(math.sqrt(3.0) / delta) + 2)
    k = torch.arange(-m, m + 1, dtype=torch.float64, device="cuda")
    cp, sp = _dev(np.cos(phi)), _dev(np.sin(phi))
    dx, dy = _dev(np.cos(phi + math.pi / 2)), _dev(np.sin(phi + math.pi / 2))
    out = torch.empty(nslices, nshift, nphi, dtype=torch.float64, device="cuda")
    step = max(1, _CHUNK // (nshift * nphi * len(k)))
    x0 = (sh[:, None] * cp)[:, :, None] + (delta * dx)[None, :, None] * k
    y0 = (sh[:, None] * sp)[:, :, None] + (delta * dy)[None, :, None] * k
    for z0 in range(0, nslices, step):
        zz = z[z0:z0 + step, None, None, None]
        x, y = x0[None].expand(len(zz), -1, -1, -1), y0[None].expand(len(zz), -1, -1, -1)
        zz = zz.expand_as(x)
        if frame is not None:
            F = [float(f) for f in np.asarray(frame, np.float64).reshape(9)]
            x, y, zz = [F[3 * r] * x + F[3 * r + 1] * y + F[3 * r + 2] * zz for r in range(3)]
        out[z0:z0 + step] = _trilinear(flat, n, x, y, zz).sum(-1) * delta
    return out


def _curvatures(y):
    """Second derivatives of the natural splines of y's last axis, knots -1 .. 1."""
    ns = y.shape[-1]
    h = 2.0 / (ns - 1)
    A = np.diag(np.full(ns - 2, 4.0)) + np.diag(np.ones(ns - 3), 1) + np.diag(np.ones(ns - 3), -1)
    rhs = (y[..., 2:] - 2.0 * y[..., 1:-1] + y[..., :-2]) * (6.0 / h ** 2)
    M = torch.zeros_like(y)
    M[..., 1:-1] = rhs @ torch.linalg.inv(_dev(A))
    return M, h


def _spline(y, M, h, line, s):
    """Values at s of the splines number `line` (y, M flat lines x knots)."""
    ns = y.shape[-1]
    i = ((s + 1.0) / h).to(torch.int64).clamp_(0, ns - 2)
    b = (s - (-1.0 + i * h)) / h
    a, o = 1.0 - b, line * ns + i
    y, M = y.reshape(-1), M.reshape(-1)
    return (a * y[o] + b * y[o + 1] +
            ((a ** 3 - a) * M[o] + (b ** 3 - b) * M[o + 1]) * (h * h / 6.0))


def _exact_reduction(rays, nshift, ntheta):
    n, nsr, nphi = rays.shape
    if float(nshift) * nphi * ntheta * 2 * n > 3e9:
        return None
    y = _dev(rays).permute(0, 2, 1).contiguous()  # [z][phi][s]
    M, h = _curvatures(y)
    _, theta, _, shift = _sphere(nphi, ntheta, nshift)
    dz = 2.0 / (n - 1)
    dtau = dz / 2.0
    m = min(2 * n, int(1.0 / dtau) + 2)
    tau = torch.arange(-m, m + 1, dtype=torch.float64, device="cuda") * dtau
    sh, ph = _dev(shift), torch.arange(nphi, device="cuda")
    out = torch.empty(nshift, nphi, ntheta, dtype=torch.float64, device="cuda")
    step = max(1, (_CHUNK >> 2) // (nphi * len(tau)))
    for t, th in enumerate(theta):
        for s0 in range(0, nshift, step):
            p = sh[s0:s0 + step, None]
            z = p * math.cos(th) + tau * math.sin(th)
            s = p * math.sin(th) - tau * math.cos(th)
            keep = ((tau * tau + p * p).abs() <= 1.0) & (z.abs() <= 1.0) & (s.abs() <= 1.0)
            iz = ((z + 1.0) / _dev([dz])).to(torch.int64).clamp_(0, n - 2)
            f = ((z - (-1.0 + dz * iz)) / dz)[:, None, :]
            sc = s.clamp(-1.0, 1.0)[:, None, :]
            val = []
            for q in range(3):
                line = (iz + q).clamp_max(n - 1)[:, None, :] * nphi + ph[None, :, None]
                val.append(_spline(y, M, h, line, sc))
            # the reference's third layer is 0 past the last one (slicing.c:62-74)
            v2 = torch.where((iz >= n - 2)[:, None, :], torch.zeros_like(val[2]), val[2])
            g = val[0] + f * (val[1] - val[0]) + 0.5 * f * (f - 1.0) * (v2 - 2.0 * val[1] + val[0])
            g = torch.where(keep[:, None, :], g, torch.zeros_like(g))
            out[s0:s0 + step, :, t] = g.sum(-1) * dtau
    return out


def _exact_adjoint(radon, n):
    nshift, nphi, ntheta = radon.shape
    if float(n) ** 3 * nphi * ntheta > 3e10:
        return None
    phi, theta, w, _ = _sphere(nphi, ntheta, nshift)
    y = _dev(radon).reshape(nshift, -1).T.contiguous()
    M, h = _curvatures(y)
    x = _dev(-1.0 + 1.0 / n + np.arange(n) * (2.0 / n))
    out = torch.zeros(n, n, n, dtype=torch.float64, device="cuda")
    zero = torch.zeros((), dtype=torch.int64, device="cuda")
    for ip in range(nphi):
        for it in range(ntheta):
            o = (math.sin(theta[it]) * math.cos(phi[ip]), math.sin(theta[it]) * math.sin(phi[ip]),
                 math.cos(theta[it]))
            s = o[0] * x[None, :, None] + o[1] * x[None, None, :] + o[2] * x[:, None, None]
            d = ip * ntheta + it
            val = _spline(y[d], M[d], h, zero, s.clamp(-1.0, 1.0))
            val = torch.where(s.abs() <= 1.0, val, torch.zeros_like(val))
            out += val * (2.0 * math.pi / nphi * float(w[it]))
    return out


def _bf16(v):
    return torch.from_numpy(np.ascontiguousarray(v)).to(torch.bfloat16).to(torch.float64).numpy()


def exact(c, seed):
    op = c["op"]
    if op in ("planes", "dropin"):
        v = _phantom(c["n"], seed)
        v = _bf16(v) if c.get("storage") == "bf16" else v.astype(np.float64)
        return _exact_planes(v, c["nphi"], c["ntheta"], c["nshift"], c["sampler"] == "nearest",
                             c["half"])
    if op == "batch":
        return [_exact_planes(_phantom(n, seed * 64 + k, 6).astype(np.float64), nph, nth, ns,
                              False, n)
                for k, (n, nth, nph, ns) in enumerate(_batch_sizes(c, seed))]
    if op == "rays":
        _package()
        v = _phantom(c["n"], seed).astype(np.float64)
        return [_exact_rays(v, c["nslices"], c["nshift"], c["nphi"], f)
                for f in _frames(c["frames"], seed)]
    if op == "reduction":
        return _exact_reduction(_rays(c["n"], c["nshift_ray"], c["nphi"], seed), c["nshift"],
                                c["ntheta"])
    if op == "adjoint":
        return _exact_adjoint(_radon(c["nshift"], c["nphi"], c["ntheta"], seed), c["n"])
    out = []
    for k, (kind, n, nth, nph, ns) in enumerate(_serve_sizes(c)):
        sd = seed * 64 + k
        if kind == "forward":
            out.append(_exact_planes(_phantom(n, sd, 6).astype(np.float64), nph, nth, ns, False, n))
        elif kind == "adjoint":
            out.append(_exact_adjoint(_radon(ns, nph, nth, sd), n))
        elif kind == "rays":
            out.append(_exact_rays(_phantom(n, sd, 6).astype(np.float64), n, ns, nph, None))
        else:
            out.append(_exact_reduction(_rays(n, n, nph, sd), ns, nth))
    return out
