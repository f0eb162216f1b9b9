"""The calls whose speed this framework is judged by, through its public entry points.

A case names one call of a user's program: compressing or decompressing a 2D or
3D float vector field with its critical points kept, a batch of fields, the
learned bounds, or the archive path with the lossless stage behind it.  Fields
are Gaussian-windowed linear flows with noise, rescaled to [-1, 1]: the
definition of ``cpsz_b200/workloads.py``, made on the GPU.  Simulation output
sits in device memory, so most cases take device fields and write device
blobs; the archive and the offline_log cases go through host memory instead.

Blobs are bytes.  Decompressed values are defined by the format's own
single-precision recurrence (every rounding of it is part of the format, and
another rounding diverges point by point), so no 64-bit value stands beside
them: ``exact`` has none to give.
"""
import math

import numpy as np
import torch

import cpsz_b200
from cpsz_b200 import learned, workloads

EBS = (0.01, 0.05, 0.1)  # relative bounds of the repository's workloads


def listed():
    return [
        # one small field of an ensemble or a time step: launches and host latency decide
        {"name": "compress2d_128x128", "kind": "compress2d", "r1": 128, "r2": 128, "eb": 0.1},
        # a regional model's layer, sides that fit no tile
        {"name": "compress2d_1021x1537", "kind": "compress2d", "r1": 1021, "r2": 1537, "eb": 0.05},
        # the benchmark's field, the largest 2D call
        {"name": "compress2d_8192x8192", "kind": "compress2d", "r1": 8192, "r2": 8192, "eb": 0.1},
        # writing an archive: fields in pinned host memory, the blob's Zstandard frame back in it
        {"name": "archive2d_2048x3001", "kind": "archive2d", "r1": 2048, "r2": 3001, "eb": 0.01},
        # reading fields back onto the device, ragged and the largest
        {"name": "decompress2d_1021x1537", "kind": "decompress2d", "r1": 1021, "r2": 1537, "eb": 0.05},
        {"name": "decompress2d_8192x8192", "kind": "decompress2d", "r1": 8192, "r2": 8192, "eb": 0.1},
        # the offline_log pair as a program moving over from the reference calls it: host arrays, both directions
        {"name": "log2d_1200x1800", "kind": "log2d", "r1": 1200, "r2": 1800, "eb": 0.05},
        # a small ragged volume
        {"name": "compress3d_57x64x101", "kind": "compress3d", "r1": 57, "r2": 64, "r3": 101, "eb": 0.1},
        # the benchmark's volume, the largest 3D call
        {"name": "compress3d_384x384x384", "kind": "compress3d", "r1": 384, "r2": 384, "r3": 384, "eb": 0.05},
        # reading a volume back onto the device
        {"name": "decompress3d_256x256x256", "kind": "decompress3d", "r1": 256, "r2": 256, "r3": 256, "eb": 0.05},
        # an ensemble of many fields of different sizes and bounds in one call
        {"name": "batch2d_128", "kind": "batch2d", "fields": 128, "lo": 128, "hi": 2048, "layout": 3},
        # the learned bounds with the exact check and its fallback loop
        {"name": "learned2d_1100x1536", "kind": "learned2d", "r1": 1100, "r2": 1536, "eb": 0.1},
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["compress2d", "compress2d", "archive2d", "decompress2d", "decompress2d", "log2d", "compress3d",
                       "decompress3d", "batch2d", "learned2d"])
    eb = rng.choice(EBS)
    if kind in ("compress2d", "decompress2d"):
        return {"kind": kind, "r1": _side(rng, 64, 8192), "r2": _side(rng, 64, 8192), "eb": eb}
    if kind == "archive2d":
        return {"kind": kind, "r1": _side(rng, 256, 4096), "r2": _side(rng, 256, 4096), "eb": eb}
    if kind == "log2d":
        return {"kind": kind, "r1": _side(rng, 64, 2048), "r2": _side(rng, 64, 2048), "eb": eb}
    if kind in ("compress3d", "decompress3d"):
        return {"kind": kind, "r1": _side(rng, 24, 320), "r2": _side(rng, 24, 320), "r3": _side(rng, 24, 320), "eb": eb}
    if kind == "batch2d":
        return {"kind": kind, "fields": _side(rng, 8, 128), "lo": 128, "hi": rng.choice([512, 1024, 2048]),
                "layout": rng.randrange(1 << 20)}
    return {"kind": kind, "r1": _side(rng, 256, 2048), "r2": _side(rng, 256, 2048), "eb": 0.1}


# ---- fields -----------------------------------------------------------------------

def _axis(gen, flows, n, sigma):
    """Per flow and grid line: the Gaussian window and its product with the distance from the centre."""
    c = torch.rand(flows, generator=gen, dtype=torch.float64) * n
    d = torch.arange(n, device="cuda", dtype=torch.float64)[None, :] - c.cuda()[:, None]
    g = torch.exp(d * d * (-0.5 / sigma ** 2))
    return g.float(), (g * d).float()


def _finish(fields, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    for f in fields:
        f += workloads.NOISE * torch.randn(f.shape, generator=gen, device="cuda")
    scale = 1.0 / max(float(f.abs().max()) for f in fields)
    return [f.mul_(scale) for f in fields]


def _field_2d(seed, r1, r2, flows, sigma):
    gen = torch.Generator().manual_seed(seed)
    gi, di = _axis(gen, flows, r1, sigma)
    gj, dj = _axis(gen, flows, r2, sigma)
    a = torch.randn(2, 2, flows, 1, generator=gen).cuda()
    return _finish([torch.cat([a[c, 0] * di, a[c, 1] * gi]).T @ torch.cat([gj, dj]) for c in range(2)], seed)


def _field_3d(seed, r1, r2, r3, flows, sigma):
    gen = torch.Generator().manual_seed(seed)
    (gi, di), (gj, dj), (gk, dk) = (_axis(gen, flows, n, sigma) for n in (r1, r2, r3))
    a = torch.randn(3, 3, flows, 1, generator=gen).cuda()
    out = []
    for c in range(3):
        f = ((a[c, 0] * di).T[:, None, :] * gj.T[None] + gi.T[:, None, :] * (a[c, 1] * dj).T[None]) @ gk
        f += (gi.T[:, None, :] * gj.T[None]) @ (a[c, 2] * dk)
        out.append(f)
    return _finish(out, seed)


def _case_2d(case, seed):
    # the benchmark's flows (2000 of sigma 60 on 8192 x 8192) at its density
    r1, r2 = case["r1"], case["r2"]
    return _field_2d(seed, r1, r2, max(1, round(2000 / 8192 ** 2 * r1 * r2)), 60.0)


def _case_3d(case, seed):
    # the benchmark's flows (500 of sigma 20 on 384^3) at its density
    r = case["r1"], case["r2"], case["r3"]
    return _field_3d(seed, *r, max(1, round(500 / 384 ** 3 * math.prod(r))), 20.0)


def _sides(case):
    return tuple(case[k] for k in ("r1", "r2", "r3") if k in case)


# ---- the calls ----------------------------------------------------------------------

_kept = {}


def _context():
    """The handle a program keeps for all its calls."""
    if "ctx" not in _kept:
        _kept["ctx"] = cpsz_b200.Context(0)
    return _kept["ctx"]


def _proposer():
    if "mlp" not in _kept:
        _kept["mlp"] = learned.load(_context())
    return _kept["mlp"]


def _room(points, comps, **where):
    """Output buffer with room for any blob of the field; the bytes behind the blob stay zero."""
    return torch.zeros(points * comps * 8 + (64 << 20), dtype=torch.uint8, **where)


def _pinned(t):
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t).numpy()


def prepare(case, seed):
    kind, r = case["kind"], _sides(case)
    n = math.prod(r)
    s = {"kind": kind, "r": r, "eb": case.get("eb"), "ctx": _context()}
    if kind == "batch2d":
        layout = workloads.batch_layout(case["layout"], case["fields"], case["lo"], case["hi"])
        s["fields"] = [tuple(_field_2d(seed * 1000 + k, a, b, max(1, a * b // 1600), 40.0))
                       for k, (a, b, _, _) in enumerate(layout)]
        s["ebs"] = np.array([e for _, _, _, e in layout])
        s["out"] = _room(sum(a * b for a, b, _, _ in layout), 2, device="cuda")
        torch.cuda.synchronize()
        return s
    f = _case_3d(case, seed) if len(r) == 3 else _case_2d(case, seed)
    if kind in ("compress2d", "compress3d", "learned2d"):
        s["fields"], s["out"] = f, _room(n, len(f), device="cuda")
        if kind == "learned2d":
            s["mlp"] = _proposer()
    elif kind == "archive2d":
        s["fields"], s["out"] = [_pinned(a) for a in f], _room(n, 2, device="cuda")
        s["frame"] = torch.zeros(n * 8 + (16 << 20), dtype=torch.uint8, pin_memory=True).numpy()
    elif kind == "log2d":
        s["fields"], s["out"] = [a.cpu().numpy() for a in f], _room(n, 2).numpy()
    else:
        torch.cuda.synchronize()
        if kind == "decompress2d":
            s["blob"] = cpsz_b200.sz_compress_cp_preserve_2d_offline(*f, max_pwr_eb=case["eb"], ctx=s["ctx"])
        else:
            s["blob"] = cpsz_b200.sz_compress_cp_preserve_3d_offline_log(*f, max_pwr_eb=case["eb"], ctx=s["ctx"])
        s["fields"] = [torch.empty(r, dtype=torch.float32, device="cuda") for _ in f]
    torch.cuda.synchronize()
    return s


def run(s):
    kind, f, r, eb, ctx = s["kind"], s["fields"], s["r"], s["eb"], s["ctx"]
    if kind == "compress2d":
        return s["out"], cpsz_b200.compress_2d_into(*f, *r, eb, s["out"], ctx=ctx)
    if kind == "compress3d":
        return s["out"], cpsz_b200.compress_3d_into(*f, *r, eb, s["out"], ctx=ctx)
    if kind == "archive2d":
        size = cpsz_b200.compress_2d_into(*f, *r, eb, s["out"], ctx=ctx)
        return s["frame"], cpsz_b200.lossless_compress_gpu(s["out"][:size], out=s["frame"], ctx=ctx)
    if kind == "decompress2d":
        return cpsz_b200.sz_decompress_cp_preserve_2d_offline(s["blob"], *r, *f, ctx=ctx)
    if kind == "decompress3d":
        return cpsz_b200.sz_decompress_cp_preserve_3d_online_log(s["blob"], *r, *f, ctx=ctx)
    if kind == "log2d":
        size = cpsz_b200.compress_2d_log_into(*f, *r, eb, s["out"], ctx=ctx)
        back = cpsz_b200.sz_decompress_cp_preserve_2d_offline_log(s["out"][:size].tobytes(), *r, ctx=ctx)
        return s["out"], size, *back
    if kind == "batch2d":
        offsets = cpsz_b200.compress_2d_batch(f, s["ebs"], out=s["out"], ctx=ctx)
        return s["out"], offsets.astype(np.int64)
    return s["out"], *cpsz_b200.compress_2d_learned(*f, eb, mlp=s["mlp"], out=s["out"], ctx=ctx)


# Blob bytes per point, as a share of the field's, measured on these fields: each output is written once.
BLOB_SHARE = 0.2


def work(case):
    kind = case["kind"]
    if kind == "batch2d":
        layout = workloads.batch_layout(case["layout"], case["fields"], case["lo"], case["hi"])
        points, comps = sum(a * b for a, b, _, _ in layout), 2
    else:
        points, comps = math.prod(_sides(case)), len(_sides(case))
    field, blob = 4 * comps * points, 4 * comps * points * BLOB_SHARE
    if kind == "log2d":
        return {"bytes": 2 * (field + blob), "flops": 0}
    # the proposer's two hidden layers and its output, once for every vertex
    flops = 2 * (99 * 128 + 128 * 128 + 128) * points if kind == "learned2d" else 0
    return {"bytes": field + blob, "flops": flops}


def exact(case, seed):
    return None
