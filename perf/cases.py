"""Workloads for measuring the warp path through its public entry points.

The listed cases follow the workloads this repository is benchmarked and
tested on: the plain TPS warp, the affine warp, the large TPS warp, the
serving mix and host-resident volumes, with the solve and the node grid also
taken by themselves.  `draw` gives more cases of the same ranges.

A case is a dict:
    op        tps | affine | rotate | scale | resample | solve | nodes | serve | host
    x, y, z   volume dims in voxels (for `nodes`: of the volume the grid covers)
    channels  volumes per call
    dtype     u8 | u16
    n         landmark pairs
    g         control-grid spacing
    interp    0 trilinear, 1 nearest neighbour
    ox, oy, oz   output dims where the call resizes (0: the input's)
    jobs, mix    jobs of a serving batch and the seed of its sizes and kinds
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

import terawarp_b200 as tw
from terawarp_b200 import synth
from terawarp_b200.api import Server

_ctx = None


def _context():
    """The context a program creates once and keeps."""
    global _ctx
    if _ctx is None:
        _ctx = tw.Context(0)
    return _ctx


def _case(op, x=0, y=0, z=0, channels=1, dtype="u8", n=0, g=0, interp=0, out=(0, 0, 0), jobs=0, mix=0, name=None):
    c = {"op": op, "x": x, "y": y, "z": z, "channels": channels, "dtype": dtype, "n": n, "g": g, "interp": interp,
         "ox": out[0], "oy": out[1], "oz": out[2], "jobs": jobs, "mix": mix}
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest volume of the serving mix, aligned by a few
        # landmarks: latency and launches
        _case("affine", 128, 128, 128, dtype="u8", n=16, name="affine_128_u8"),
        # the plain TPS warp (the reference's CPU-runnable mode)
        _case("tps", 256, 256, 128, dtype="u8", n=64, g=16, name="tps_256_u8"),
        # an ordinary two-channel acquisition whose dims are multiples of nothing
        _case("tps", 517, 389, 203, channels=2, dtype="u16", n=500, g=8, name="tps_ragged_2ch_u16"),
        # the command's default grid spacing, 4, on the largest serving volume
        _case("tps", 1024, 1024, 256, dtype="u8", n=1000, g=4, name="tps_spacing4_u8"),
        # the large TPS warp
        _case("tps", 2048, 2048, 1024, dtype="u16", n=2000, g=16, name="tps_large_u16"),
        # the affine warp
        _case("affine", 1024, 1024, 512, dtype="u16", n=32, name="affine_1024_u16"),
        # a rigid re-orientation onto a larger canvas, ragged dims
        _case("rotate", 723, 611, 187, dtype="u8", out=(800, 700, 240), name="rotate_resize_u8"),
        # a label volume carried along a field that is already there
        _case("resample", 768, 640, 256, dtype="u16", n=400, g=16, interp=1, name="labels_nearest_u16"),
        # the landmark solve at the most landmarks of the serving mix
        _case("solve", 2048, 2048, 1024, n=4096, name="solve_4096"),
        # the node grid of the large TPS warp
        _case("nodes", 2048, 2048, 1024, n=2000, g=16, name="nodes_large"),
        # a burst of the serving mix on device-resident volumes
        _case("serve", jobs=12, mix=2, name="serve_burst"),
        # a volume in pinned host memory, warped through the device in slabs
        _case("host", 1024, 1024, 256, dtype="u16", n=500, g=16, name="host_stream_u16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, most):
    """Dims over the range of the serving mix and beyond, often ragged, below `most` voxels."""
    while True:
        d = [_log_int(rng, 128, 2048), _log_int(rng, 128, 2048), _log_int(rng, 64, 1024)]
        if rng.random() < 0.4:  # stacks cropped to round sizes
            d = [max(64, 32 * round(v / 32)) for v in d]
        if d[0] * d[1] * d[2] <= most:
            return d


def draw(rng):
    op = rng.choice(["tps"] * 7 + ["affine"] * 3 + ["rotate", "scale"] + ["resample"] * 3 + ["solve"] * 2 + ["nodes"] * 2
                    + ["serve", "host"])
    dtype = rng.choice(["u8", "u16"])
    if op == "serve":
        return _case(op, jobs=rng.randint(4, 24), mix=rng.randrange(1 << 20))
    if op in ("solve", "nodes"):
        x, y, z = _dims(rng, 1 << 31)
        n = _log_int(rng, 16, 4096)
        if op == "solve":
            return _case(op, x, y, z, n=n)
        g = rng.choice([4, 8, 16, 32])
        while (x // g + 4) * (y // g + 4) * (z // g + 4) * n > 3_000_000_000 and g < 64:
            g *= 2
        return _case(op, x, y, z, n=n, g=g)
    x, y, z = _dims(rng, (1 << 28) if op == "host" else (1 << 30))
    if op == "affine":
        return _case(op, x, y, z, dtype=dtype, n=_log_int(rng, 16, 512))
    if op in ("rotate", "scale"):
        out = tuple(max(64, int(v * rng.uniform(0.6, 1.3))) for v in (x, y, z)) if rng.random() < 0.5 else (0, 0, 0)
        return _case(op, x, y, z, dtype=dtype, out=out, interp=int(rng.random() < 0.2))
    n = _log_int(rng, 16, 2000)
    g = rng.choice([4, 8, 16, 16, 32])
    while (x // g + 4) * (y // g + 4) * (z // g + 4) * n > 8_000_000_000:
        g *= 2
    if op == "host":
        return _case(op, x, y, z, dtype=dtype, n=n, g=max(g, 8))
    channels = rng.choice([1, 1, 1, 2, 3]) if op == "tps" and x * y * z < (1 << 28) else 1
    return _case(op, x, y, z, channels=channels, dtype=dtype, n=n, g=g, interp=int(rng.random() < 0.2))


# ------------------------------------------------------------------ inputs

def _volume(shape, dtype, seed, labels=False):
    """A (z, y, x) volume on the GPU: smooth bright spots on a dark ground,
    noise 0..10 and thin bright fibres (uint16 values up to 4095), or a
    volume of piecewise constant labels."""
    Z, Y, X = shape
    gen = torch.Generator(device="cuda").manual_seed(seed)
    vmax = 255 if dtype == "u8" else 4095
    out = torch.empty(shape, dtype=torch.uint8 if dtype == "u8" else torch.uint16, device="cuda")
    raw = out if dtype == "u8" else out.view(torch.int16)
    cell = 8
    coarse = torch.rand((Z // cell + 2, Y // cell + 2, X // cell + 2), generator=gen, device="cuda")
    coarse = torch.floor(coarse * (vmax + 1)) if labels else coarse.pow(8) * (1.2 * vmax)
    step = max(cell, (1 << 26) // (X * Y) // cell * cell)
    for z0 in range(0, Z, step):
        z1 = min(Z, z0 + step)
        part = coarse[None, None, z0 // cell:(z1 - 1) // cell + 2]
        if labels:
            v = F.interpolate(part, scale_factor=cell, mode="nearest")[0, 0, :z1 - z0, :Y, :X]
        else:
            v = F.interpolate(part, scale_factor=cell, mode="trilinear")[0, 0, cell // 2:cell // 2 + z1 - z0,
                                                                         cell // 2:cell // 2 + Y,
                                                                         cell // 2:cell // 2 + X]
            v = v + torch.randint(0, 11, v.shape, generator=gen, device="cuda")
        raw[z0:z1] = v.clamp_(0, vmax).to(raw.dtype)
    if not labels:
        nf = max(8, min(4000, (X * Y * Z) >> 20))
        p = torch.rand((nf, 1, 3), generator=gen, device="cuda") * torch.tensor([X, Y, Z], device="cuda")
        d = torch.randn((nf, 1, 3), generator=gen, device="cuda")
        d = d / d.norm(dim=-1, keepdim=True) + 0.35 * torch.randn((nf, 300, 3), generator=gen, device="cuda")
        p = (p + torch.cumsum(d / d.norm(dim=-1, keepdim=True), 1)).round().long().reshape(-1, 3)
        ok = ((p >= 0) & (p < torch.tensor([X, Y, Z], device="cuda"))).all(1)
        lin = (p[ok, 2] * Y + p[ok, 1]) * X + p[ok, 0]
        raw.view(-1)[lin] = int(0.9 * vmax)
    return out


def _landmarks(c, seed):
    """(subject, target) landmark pairs of the smooth displacement model."""
    dims = (c["x"], c["y"], c["z"])
    if c["op"] == "affine":
        return synth.affine_landmarks(synth.random_affine(seed, dims), dims, c["n"], seed + 7,
                                      margin=min(16.0, min(dims) / 8))
    return synth.lattice_landmarks(dims, c["n"], seed + 7, margin=min(8.0, min(dims) / 8))


def _in_shape(c):
    s = (c["z"], c["y"], c["x"])
    return s if c["channels"] == 1 else (c["channels"],) + s


def _out_dims(c):
    return tuple(c["o" + a] or c[a] for a in "xyz")


def _gsz(c):
    return tuple(tw.grid_size(c[a], c["g"]) for a in "xyz")


def _mix(c):
    """Sizes, kinds and grids of a serving batch (from the case alone), in the serving mix's ranges."""
    return synth.serving_jobs(c["jobs"], seed=c["mix"])


def prepare(case, seed):
    c, ctx = case, _context()
    op = c["op"]
    if op == "serve":
        jobs = []
        for i, j in enumerate(_mix(c)):
            src = _volume(j.shape_zyx, j.dtype, seed + 31 * i)
            dst = torch.empty_like(src)
            dims = j.shape_zyx[::-1]
            if j.kind == "tps":
                sub, tar = synth.lattice_landmarks(dims, len(j.centres), seed + 31 * i + 7, margin=min(dims) / 16)
                jobs.append((src, dst, None, tar, sub, j.g))
            else:
                rot, sc = (15.0, (0.9, 1.1)) if j.kind == "affine" else (30.0, (1.0, 1.0))
                jobs.append((src, dst, synth.random_affine(seed + 31 * i, dims, rot, sc), None, None, 0))
        torch.cuda.synchronize()
        return {"op": op, "server": Server(ctx), "jobs": jobs}
    s = {"op": op, "ctx": ctx, "case": c}
    if c["n"]:
        s["sub"], s["tar"] = _landmarks(c, seed)
    if op in ("solve", "nodes"):
        if op == "nodes":
            s["tps"] = tw.tps_solve(ctx, s["tar"], s["sub"])
            gx, gy, gz = _gsz(c)
            s["out"] = torch.empty((gz, gy, gx, 4), dtype=torch.float32, device="cuda")
        return s
    shape = _in_shape(c)
    if c["channels"] == 1:
        src = _volume(shape, c["dtype"], seed, labels=c["interp"] == 1)
    else:
        src = torch.stack([_volume(shape[1:], c["dtype"], seed + 101 * k, labels=c["interp"] == 1).view(
            torch.uint8 if c["dtype"] == "u8" else torch.int16) for k in range(c["channels"])])
        src = src if c["dtype"] == "u8" else src.view(torch.uint16)
    out_shape = shape[:-3] + _out_dims(c)[::-1]
    if op == "host":
        s["src"] = torch.empty(shape, dtype=src.dtype, pin_memory=True)
        s["src"].copy_(src)
        s["out"] = torch.empty(out_shape, dtype=src.dtype, pin_memory=True)
    else:
        s["src"] = src
        s["out"] = torch.empty(out_shape, dtype=src.dtype, device="cuda")
    if op == "resample":
        tps = tw.tps_solve(ctx, s["tar"], s["sub"])
        s["nodes"] = tw.tps_eval_grid(ctx, tps, _gsz(c), c["g"])
        tps.close()
    if op in ("rotate", "scale"):
        rng = np.random.default_rng(seed)
        s["para"] = tuple(rng.uniform(-25, 25, 3)) if op == "rotate" else tuple(rng.uniform(0.7, 1.4, 3))
    torch.cuda.synchronize()
    return s


def _bytes_of(t):
    """The same voxels under a type every torch operation takes."""
    return t.view(torch.int16) if t.dtype == torch.uint16 else t


def run(s):
    op = s["op"]
    if op == "serve":
        srv, ids = s["server"], []
        for src, dst, M, centres, values, g in s["jobs"]:
            ids.append(srv.submit_affine(M, src, dst) if M is not None
                       else srv.submit_tps(centres, values, g, src, dst))
        for i in ids:
            srv.wait(i)
        return [_bytes_of(j[1]) for j in s["jobs"]]
    ctx, c = s["ctx"], s["case"]
    if op in ("tps", "host"):
        g = c["g"]
        return _bytes_of(tw.imgwarp_smallmemory_image(ctx, s["sub"], s["tar"], g, g, g, 1, c["interp"], s["src"],
                                                      out=s["out"]))
    if op == "affine":
        return _bytes_of(tw.q_imagewarp_affine_image(ctx, s["tar"], s["sub"], s["src"], out=s["out"]))
    if op in ("rotate", "scale"):
        kw = {"warp_mode": 1, "deformation_mode": 0} if op == "rotate" else {"warp_mode": 0, "deformation_mode": 2}
        if c["ox"]:
            kw.update(resize_mode=1, newsize=_out_dims(c))
        return _bytes_of(tw.bigimagewarp(ctx, s["src"], out=s["out"], para=s["para"], interp=c["interp"], **kw))
    if op == "resample":
        tw.warp_tps_device(ctx, s["nodes"], c["g"], s["src"], s["out"], interp=c["interp"])
        return _bytes_of(s["out"])
    if op == "solve":
        tps = tw.tps_solve(ctx, s["tar"], s["sub"])
        out = tps.coeffs()
        tps.close()
        return out
    return tw.tps_eval_grid(ctx, s["tps"], _gsz(c), c["g"], out=s["out"])


# -------------------------------------------------------------------- work

def _solve_flops(n):
    return 2.0 * n ** 3 / 3.0


def _tps_work(dims, dtype, channels, n, g, field=True):
    """Source and output once each; with `field`, the solve and the node grid (15 operations per node and
    landmark).  Per voxel: 24 operations of the spline's last contraction, 30 of the sample."""
    vox = float(dims[0]) * dims[1] * dims[2] * channels
    nodes = 1.0
    for v in dims:
        nodes *= tw.grid_size(v, g)
    es = 1 if dtype == "u8" else 2
    flops = 54.0 * vox + (_solve_flops(n) + 15.0 * nodes * n if field else 0.0)
    return {"bytes": 2.0 * es * vox + (24.0 * n if field else 12.0 * nodes), "flops": flops}


def work(case):
    c, op = case, case["op"]
    if op == "serve":
        b = f = 0.0
        for j in _mix(c):
            if j.kind == "tps":
                w = _tps_work(j.shape_zyx[::-1], j.dtype, 1, len(j.centres), j.g)
            else:
                vox = float(np.prod(j.shape_zyx))
                w = {"bytes": (2.0 if j.dtype == "u8" else 4.0) * vox, "flops": 48.0 * vox}
            b, f = b + w["bytes"], f + w["flops"]
        return {"bytes": b, "flops": f}
    if op == "solve":
        return {"bytes": 24.0 * c["n"] + 32.0 * c["n"], "flops": _solve_flops(c["n"])}
    if op == "nodes":
        nodes = float(np.prod(_gsz(c)))
        return {"bytes": 16.0 * nodes + 32.0 * c["n"], "flops": 15.0 * nodes * c["n"]}
    dims = (c["x"], c["y"], c["z"])
    if op in ("tps", "host", "resample"):
        return _tps_work(dims, c["dtype"], c["channels"], c["n"], c["g"], field=op != "resample")
    es = 1 if c["dtype"] == "u8" else 2
    out = float(np.prod(_out_dims(c)))
    # what a call must read of its source: no more than the source, nor than the samples it takes touch
    return {"bytes": es * (out + min(float(np.prod(dims)), 8.0 * out)), "flops": 48.0 * out}


# ------------------------------------------------------------- exact values

def exact(case, seed):
    """Coefficients and node displacements in 64 bits.  The warped volumes are
    whole numbers and have to be equal; they have no value here."""
    c = case
    if c["op"] not in ("solve", "nodes"):
        return None
    sub, tar = _landmarks(c, seed)
    s = torch.from_numpy(tar).cuda().double()
    t = torch.from_numpy(sub).cuda().double()
    n = len(s)
    one = torch.ones((n, 1), dtype=torch.float64, device="cuda")
    X, Y = torch.cat([one, s], 1), torch.cat([one, t], 1)

    def dist(a, b):
        d = torch.zeros((len(a), len(b)), dtype=torch.float64, device="cuda")
        for k in range(3):
            d += (a[:, k:k + 1] - b[:, k][None, :]) ** 2
        return d.sqrt()

    A = torch.zeros((n + 4, n + 4), dtype=torch.float64, device="cuda")
    A[:n, :n] = -dist(s, s)
    A[:n, :n] += 0.2 * torch.eye(n, dtype=torch.float64, device="cuda")
    A[:n, n:], A[n:, :n] = X, X.T
    sol = torch.linalg.solve(A, torch.cat([Y, torch.zeros((4, 4), dtype=torch.float64, device="cuda")]))
    coef, aff = sol[:n], sol[n:]
    if c["op"] == "solve":
        return coef.cpu().numpy(), aff.cpu().numpy()
    gx, gy, gz = _gsz(c)
    axes = [(torch.arange(k, device="cuda", dtype=torch.float64) - 1) * c["g"] for k in (gx, gy, gz)]
    out = torch.zeros((gz, gy, gx, 4), dtype=torch.float64, device="cuda")
    flat = out.view(-1, 4)
    step = max(1, (1 << 27) // n)
    for i in range(0, gx * gy * gz, step):
        k = torch.arange(i, min(i + step, gx * gy * gz), device="cuda")
        p = torch.stack([axes[0][k % gx], axes[1][k // gx % gy], axes[2][k // (gx * gy)]], 1)
        f = -dist(p, s) @ coef + torch.cat([torch.ones_like(p[:, :1]), p], 1) @ aff
        flat[k, :3] = f[:, 1:] - p
    return out
