"""The work a user of this engine has it do, as cases that can be timed.

Sizes are the repository's own: the small 360-view scan (256 x 192 detector,
reference grid), the 512^3 and 1024^3 production scans, the 512^3 projector
pair, the uneven scans of a batch, and the tiny scan of the smoke test.

Each case is one pass through the public entry points:
  filter   ops.filter_projections       raw images -> filtered projections
  bp       ops.backproject              filtered projections -> volume slab
  fdk      both, one after the other    raw images -> volume, on the device
  fp       ops.forward_project          volume -> projections (the adjoint of bp)
  facade   CtVolume.reconstructInto     host images -> host volume
  batch    ops.Batch.run                several uneven scans in one graph

Lengths are in detector pixels at the rotation axis: D is the distance from
the focus to the axis, vs the voxel edge. `views` are spread over 360 degrees.
"""
import math
import random

import numpy as np
import torch

from ct_b200 import CtVolume, ops
from ct_b200 import _lib as L

DEVICE = "cuda"
STORE = {"fp32": L.FP32, "fp16": L.FP16, "bf16": L.BF16}
DTYPE = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
FILTER = {"ramlak": L.RAMLAK, "shepplogan": L.SHEPPLOGAN, "hann": L.HANN}
RAW = {"u8": L.U8, "u16": L.U16, "f32": L.F32}
RAW_BYTES = {"u8": 1, "u16": 2, "f32": 4}


# ------------------------------------------------------------------- cases
def _filter(W, H, views, raw, store, filt, pad):
    return {"op": "filter", "W": W, "H": H, "views": views, "D": 2.44 * W, "raw": raw, "store": store,
            "filter": filt, "pad": pad}


def _bp(W, H, views, D, X, Y, Z, vs, store, **more):
    c = {"op": "bp", "W": W, "H": H, "views": views, "D": D, "X": X, "Y": Y, "Z": Z, "vs": vs, "store": store,
         "z0": 0, "z1": Z, "x_from": 0, "y_from": 0, "full": 0, "u_offset": 0.0, "heights": False}
    c.update(more)
    return c


def _fdk(W, H, views, D, edge, vs, raw, store, filt, pad):
    return dict(_bp(W, H, views, D, edge, edge, edge, vs, store), op="fdk", raw=raw, filter=filt, pad=pad)


def _fp(W, H, views, D, X, Y, Z, vs, **more):
    return dict(_bp(W, H, views, D, X, Y, Z, vs, "fp32", **more), op="fp")


def _facade(W, H, views, D, raw, store, filt, order, zmin, zmax):
    return {"op": "facade", "W": W, "H": H, "views": views, "D": D, "raw": raw, "store": store, "filter": filt,
            "pad": 1, "order": order, "zmin": zmin, "zmax": zmax}


def _batch(scans, shapes, store, edge_max, views_max):
    return {"op": "batch", "scans": scans, "shapes": shapes, "store": store, "edge_max": edge_max,
            "views_max": views_max}


def listed():
    return [
        # the filter over a run of views of a 2048-wide detector, as the large scan is filtered chunk by chunk
        dict(_filter(2048, 2048, 144, "u16", "fp16", "hann", 1), name="filter_2048_fp16"),
        # a detector cropped to an odd width (no power of two): the circular filter through a longer transform
        dict(_filter(701, 409, 360, "u16", "fp32", "shepplogan", 1), name="filter_701_fp32"),
        # the smallest scan: a quick look or a geometry check, where latency and launches count
        dict(_fdk(32, 20, 24, 120.0, 30, 1.0, "u16", "fp32", "ramlak", 1), name="fdk_tiny"),
        # a small scan at low resolution: a preview, or one of a series of specimens
        dict(_fdk(200, 150, 120, 500.0, 96, 2.0, "u16", "fp16", "hann", 1), name="fdk_small"),
        # the 360-view 256 x 192 scan into 256^3 voxels of one pixel
        dict(_bp(256, 192, 360, 1000.0, 256, 256, 256, 1.0, "fp32"), name="bp_256_fp32"),
        # production size at full precision: 720 views of 1024^2 into 512^3
        dict(_bp(1024, 1024, 720, 2500.0, 512, 512, 512, 2.0, "fp32"), name="bp_512_fp32"),
        # the largest scan, one z-slab of it: 1440 views of 2048^2, 256 central slices of 1024^3
        dict(_bp(2048, 2048, 1440, 5000.0, 1024, 1024, 1024, 2.0, "fp16", z0=384, z1=640), name="bp_1024_slab_fp16"),
        # a region of interest off the axis, ragged sizes, a shifted detector and height offsets
        dict(_bp(1021, 777, 500, 2600.0, 333, 301, 77, 1.3, "bf16", x_from=61, y_from=190, full=600, z0=3, z1=74,
                 u_offset=7.25, heights=True), name="bp_region_bf16"),
        # the forward projector of an iterative method: 512^3 and 360 views of 512^2
        dict(_fp(512, 512, 360, 2500.0, 512, 512, 512, 1.0), name="fp_512"),
        # the same at the start of a multi-resolution scheme, sizes off any tile
        dict(_fp(161, 130, 90, 420.0, 97, 101, 83, 1.6, u_offset=-2.5, heights=True), name="fp_small"),
        # the whole path a user takes, host images to host volume in the order it is saved in
        dict(_facade(256, 192, 360, 1000.0, "u16", "fp16", "ramlak", "zfastest", 0.0, 1.0), name="facade_256_fp16"),
        # uneven scans reconstructed together
        dict(_batch(6, 5, "fp16", 320, 400), name="batch_fp16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """A case of the same ranges, at most a quarter of the largest listed one's work."""
    op = rng.choice(["filter", "filter", "bp", "bp", "bp", "fdk", "fp", "fp", "facade", "batch"])
    store = rng.choice(["fp32", "fp16", "bf16"])
    raw = rng.choice(["u16", "u16", "u8", "f32"])
    filt = rng.choice(list(FILTER))
    if op == "filter":
        W = rng.choice([256, 512, 1024, 2048]) if rng.random() < 0.4 else _log(rng, 100, 2048)
        H = _log(rng, 64, 1500)
        views = max(4, min(720, _log(rng, 4.0e5, 5.0e8) // (W * H)))
        return _filter(W, H, views, raw, store, filt, 2 if rng.random() < 0.3 else 1)
    if op == "batch":
        return _batch(rng.randint(2, 8), rng.randrange(1 << 20), store, rng.randint(120, 280), rng.randint(100, 360))
    if op == "facade":
        W = _log(rng, 48, 400)
        H = max(16, int(W * rng.uniform(0.5, 1.1)))
        zmin = rng.choice([0.0, 0.0, 0.25, 0.4])
        zmax = rng.choice([1.0, 1.0, 0.75, 0.6])
        return _facade(W, H, _log(rng, 40, 500), W * rng.uniform(1.8, 4.5), raw, store, filt,
                       rng.choice(["zfastest", "xfastest"]), zmin, zmax)
    if op == "fdk":
        W = _log(rng, 32, 512)
        edge = max(16, int(W * rng.uniform(0.4, 1.0)))
        return _fdk(W, max(16, int(W * rng.uniform(0.6, 1.0))), _log(rng, 24, 400), W * rng.uniform(1.8, 4.5), edge,
                    round(W / edge * rng.uniform(0.6, 1.0), 3), raw, store, filt, rng.choice([1, 1, 2]))
    W = _log(rng, 96, 512 if op == "fp" else 1400)
    H = max(32, int(W * rng.uniform(0.5, 1.1)))
    X = min(420, max(32, int(W * rng.uniform(0.3, 1.0))))
    Y = max(32, int(X * rng.uniform(0.8, 1.2)))
    Z = max(16, int(X * rng.uniform(0.2, 1.1)))
    views = _log(rng, 40, 720)
    views = max(24, min(views, int((2.0e10 if op == "fp" else 9.0e10) / (X * Y * Z))))
    more = {"u_offset": rng.choice([0.0, round(rng.uniform(-5.0, 5.0), 2)]), "heights": rng.random() < 0.4}
    if rng.random() < 0.4:   # a region of a larger grid
        more.update(full=int(max(X, Y) * 1.4), x_from=int(X * rng.uniform(0.0, 0.35)), y_from=int(Y * 0.1))
    if rng.random() < 0.4:   # a slab of the box
        more.update(z0=int(Z * rng.uniform(0.0, 0.4)), z1=int(Z * rng.uniform(0.6, 1.0)) + 1)
        more["z1"] = min(Z, more["z1"])
    span = more.get("full") or max(X, Y)
    vs = round(W / span * rng.uniform(0.5, 1.0), 3)
    D = W * rng.uniform(1.8, 4.5)
    return _fp(W, H, views, D, X, Y, Z, vs, **more) if op == "fp" else _bp(W, H, views, D, X, Y, Z, vs, store, **more)


# ------------------------------------------------------------------ inputs
def _gen(seed, salt=0):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(1000003 * seed + salt)
    return g


def _line_integrals(rng, gen, W, H, a, b, views, noise):
    """Views a .. b-1 of the shadows of some ellipsoids on their orbits, in [0, ~3], with noise."""
    u = torch.arange(W, device=DEVICE, dtype=torch.float32)
    v = torch.arange(H, device=DEVICE, dtype=torch.float32)
    th = torch.arange(a, b, device=DEVICE, dtype=torch.float32) * (2 * math.pi / views)
    p = torch.randn((b - a, H, W), generator=gen, device=DEVICE) * noise
    for r, ph, vc, ru, rv, dens in rng:
        uc = W * (0.5 + r * torch.cos(th - ph))
        du = ((u[None, :] - uc[:, None]) / (ru * W)) ** 2
        dv = ((v - vc * H) / (rv * H)) ** 2
        p.add_((1.0 - du[:, None, :] - dv[None, :, None]).clamp_(min=0).sqrt_(), alpha=dens)
    return p


def _objects(seed):
    r = random.Random(seed)
    body = [(0.0, 0.0, 0.5, 0.42, 0.6, 1.2)]
    return body + [(r.uniform(0, 0.3), r.uniform(0, 6.28), r.uniform(0.2, 0.8), r.uniform(0.01, 0.15),
                    r.uniform(0.02, 0.2), r.uniform(0.2, 0.8)) for _ in range(5)]


def _chunks(views, pixels):
    n = max(1, min(views, (1 << 27) // pixels))
    return [(a, min(views, a + n)) for a in range(0, views, n)]


def _raw_images(W, H, views, raw, seed, salt=0):
    """Intensity images exp(-p) with photon-like noise, as the detector delivers them (air at full scale)."""
    dt = {"u8": torch.uint8, "u16": torch.uint16, "f32": torch.float32}[raw]
    out = torch.empty((views, H, W), dtype=dt, device=DEVICE)
    gen, obj = _gen(seed, salt), _objects(1000 * seed + salt)
    for a, b in _chunks(views, H * W):
        i = torch.exp(-_line_integrals(obj, gen, W, H, a, b, views, 0.0))
        i.add_(torch.randn(i.shape, generator=gen, device=DEVICE) * i.sqrt() * 0.004).clamp_(0.0005, 1.0)
        out[a:b] = i if raw == "f32" else (i * (255.0 if raw == "u8" else 65535.0)).round_().to(torch.int32).to(dt)
    return out


def _filtered(W, H, views, store, seed):
    """Ramp-filtered noisy line integrals: what the backprojector meets."""
    out = torch.empty((views, H, W), dtype=DTYPE[store], device=DEVICE)
    gen, obj = _gen(seed, 1), _objects(seed)
    ramp = torch.arange(W // 2 + 1, device=DEVICE, dtype=torch.float32) / (W // 2 + 1)
    ramp = ramp * 0.5 * (1.0 + torch.cos(math.pi * ramp))
    for a, b in _chunks(views, H * W):
        p = _line_integrals(obj, gen, W, H, a, b, views, 0.01)
        out[a:b] = torch.fft.irfft(torch.fft.rfft(p) * ramp, n=W)
    return out


def _volume(X, Y, Zs, seed):
    """A piecewise smooth object with some noise, (Zs, Y, X)."""
    x, y, z = (torch.linspace(-1, 1, n, device=DEVICE) for n in (X, Y, Zs))
    v = torch.randn((Zs, Y, X), generator=_gen(seed, 2), device=DEVICE) * 0.01
    r = random.Random(seed)
    for k in range(6):
        c = [0.0] * 3 if k == 0 else [r.uniform(-0.5, 0.5) for _ in range(3)]
        s = [0.85] * 3 if k == 0 else [r.uniform(0.08, 0.4) for _ in range(3)]
        d = (((x - c[0]) / s[0]) ** 2)[None, None, :] + (((y - c[1]) / s[1]) ** 2)[None, :, None]
        v.add_(((d + (((z - c[2]) / s[2]) ** 2)[:, None, None]) < 1.0).to(torch.float32), alpha=0.3 if k else 1.0)
    return v


def _angles(views):
    return np.arange(views, dtype=np.float64) * (360.0 / views)


def _heights(c, seed):
    return np.random.default_rng(seed).uniform(-3.0, 3.0, c["views"]) if c.get("heights") else None


def _geometry(c):
    det, ref = ops.detector(c["W"], c["H"], c["D"], c.get("u_offset", 0.0))
    if "X" not in c:
        return det, ref
    X, Y, Z, x0, y0 = c["X"], c["Y"], c["Z"], c["x_from"], c["y_from"]
    full = (c["full"], c["full"], Z) if c["full"] else (X, Y, Z)
    return det, ops.custom_grid(det, full, c["vs"], box=(x0, x0 + X, y0, y0 + Y, 0, Z))


def _shapes(c):
    """Detector, views, volume edge and geometry of every scan of a batch."""
    r = random.Random(c["shapes"])
    out = []
    for i in range(c["scans"]):
        W, H = r.randint(128, 768), r.randint(128, 768)
        edge = r.randint(96, c["edge_max"])
        out.append({"W": W, "H": H, "views": r.randint(90, c["views_max"]), "D": W * r.uniform(1.9, 4.0), "X": edge,
                    "Y": edge, "Z": edge, "vs": round(0.9 * W / edge, 3), "z0": 0, "z1": edge, "x_from": 0,
                    "y_from": 0, "full": 0, "u_offset": 0.0, "raw": "u16", "pad": 1,
                    "filter": list(FILTER)[i % 3], "store": c["store"]})
    return out


def prepare(case, seed):
    c, s = case, {"case": case}
    if c["op"] == "batch":
        scans = []
        for i, sc in enumerate(_shapes(c)):
            det, grid = _geometry(sc)
            scans.append(dict(raw=_raw_images(sc["W"], sc["H"], sc["views"], sc["raw"], seed, i),
                              angles_deg=_angles(sc["views"]), heights_px=None, det=det, grid=grid,
                              filter=FILTER[sc["filter"]], pad=sc["pad"],
                              vol=torch.zeros((sc["Z"], sc["Y"], sc["X"]), device=DEVICE)))
        s.update(scans=scans, batch=ops.Batch(scans, STORE[c["store"]]))
        return s
    if c["op"] == "facade":
        img = _raw_images(c["W"], c["H"], c["views"], c["raw"], seed).cpu().pin_memory()
        v = CtVolume()
        v.setProjectionsPointer(img.data_ptr(), RAW[c["raw"]], c["views"], c["W"], c["H"], _angles(c["views"]),
                                pixel_size=0.5, fcd_mm=0.5 * c["D"], keep=img)
        v.setFrequencyFilterType(c["filter"])
        v.setPrecision(c["store"])
        v.setVolumeBounds(0.0, 1.0, 0.0, 1.0, c["zmin"], c["zmax"])
        x, y, z = v.grid().box
        zf = c["order"] == "zfastest"
        out = torch.zeros((x, y, z) if zf else (z, y, x), pin_memory=True)
        s.update(img=img, ct=v, out=out, order=L.Z_FASTEST if zf else L.X_FASTEST)
        return s
    s["det"], s["grid"] = _geometry(c)
    s["angles"], s["heights"] = _angles(c["views"]), _heights(c, seed)
    if c["op"] in ("filter", "fdk"):
        s["raw"] = _raw_images(c["W"], c["H"], c["views"], c["raw"], seed)
        s["filtered"] = torch.zeros(s["raw"].shape, dtype=DTYPE[c["store"]], device=DEVICE)
    if c["op"] == "bp":
        s["filtered"] = _filtered(c["W"], c["H"], c["views"], c["store"], seed)
    if c["op"] in ("bp", "fdk"):
        s["vol"] = torch.zeros((c["z1"] - c["z0"], c["Y"], c["X"]), device=DEVICE)
    if c["op"] == "fp":
        s["vol"] = _volume(c["X"], c["Y"], c["z1"] - c["z0"], seed)
        s["proj"] = torch.zeros((c["views"], c["H"], c["W"]), device=DEVICE)
    return s


def _scale(c):
    """Filtered values in 16 bits are stored near unit magnitude."""
    return 1.0 if c["store"] == "fp32" else 1.0 / c["W"]


def run(s):
    c = s["case"]
    if c["op"] == "batch":
        s["batch"].run()
        return [sc["vol"] for sc in s["scans"]]
    if c["op"] == "facade":
        s["ct"].reconstructInto(s["out"].data_ptr(), s["order"])
        return s["out"]
    if c["op"] == "filter":
        return ops.filter_projections(s["raw"], s["det"], FILTER[c["filter"]], c["pad"], STORE[c["store"]], _scale(c),
                                      out=s["filtered"])
    if c["op"] == "bp":
        return ops.backproject(s["filtered"], s["angles"], s["heights"], s["det"], s["grid"], c["z0"], c["z1"],
                               out=s["vol"])
    if c["op"] == "fp":
        return ops.forward_project(s["vol"], s["angles"], s["heights"], s["det"], s["grid"], c["z0"], c["z1"],
                                   out=s["proj"])
    f = ops.filter_projections(s["raw"], s["det"], FILTER[c["filter"]], c["pad"], STORE[c["store"]], _scale(c),
                               out=s["filtered"])
    return [f, ops.backproject(f, s["angles"], s["heights"], s["det"], s["grid"], c["z0"], c["z1"],
                               load_scale=1.0 / _scale(c), out=s["vol"])]


# ------------------------------------------------------------------- work
_UPDATE_FLOPS = 12   # a row coordinate, three linear interpolations, a weighted sum


def _box(c):
    """(full x, full y, x_from, y_from, X, Y, Z of the slab, Z of the box, first slice, vs) of a case."""
    if c["op"] == "facade":
        det, g = _facade_grid(c)
        X, Y, Z = g.box
        return g.x_size, g.y_size, g.x_from, g.y_from, X, Y, Z, g.z_size, g.z_from, 1.0
    fx = c["full"] or c["X"]
    fy = c["full"] or c["Y"]
    return fx, fy, c["x_from"], c["y_from"], c["X"], c["Y"], c["z1"] - c["z0"], c["Z"], c["z0"], c["vs"]


def _facade_grid(c):
    return ops.detector(c["W"], c["H"], c["D"], 0.0, rel=(0.0, 1.0, 0.0, 1.0, c["zmin"], c["zmax"]))


def _columns(c):
    """Voxel columns inside the reconstruction cylinder."""
    fx, fy, x0, y0, X, Y, _, _, _, vs = _box(c)
    r = _radius(c)
    x = (np.arange(X) - (fx / 2.0 - x0)) * vs
    y = (np.arange(Y) - (fy / 2.0 - y0)) * vs
    return int(((x[None, :] ** 2 + y[:, None] ** 2) < r * r).sum())


def _radius(c):
    rad = c["W"] // 2
    return float(int(math.sqrt(c["D"] ** 2 * rad ** 2 / (c["D"] ** 2 + rad ** 2))))


def work(case):
    c = case
    if c["op"] == "batch":
        w = [work(dict(sc, op="fdk")) for sc in _shapes(c)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    px = c["views"] * c["W"] * c["H"]
    by, fl = 0.0, 0.0
    if c["op"] != "fp" and c["op"] != "bp":   # raw samples in, one real transform each way per row
        by += px * RAW_BYTES[c["raw"]]
        fl += px * (5.0 * math.log2(max(2, c["W"] * c["pad"])) * c["pad"] + 4.0)
    if c["op"] in ("filter", "bp", "fdk"):
        by += px * (4 if c["store"] == "fp32" else 2)
    if c["op"] == "fp":
        by += px * 4
    if c["op"] != "filter":
        _, _, _, _, X, Y, Zs, _, _, _ = _box(c)
        by += 4.0 * X * Y * Zs
        fl += float(_UPDATE_FLOPS) * _columns(c) * Zs * c["views"]
    return {"bytes": by, "flops": fl}


# ------------------------------------------------------- values in 64 bits
def _window(name, n, nyq):
    x = torch.arange(n, device=DEVICE, dtype=torch.float64) / nyq
    if name == "shepplogan":
        return x * torch.sinc(0.5 * x)
    if name == "hann":
        return x * 0.5 * (1.0 + torch.cos(math.pi * x))
    return x


def _exact_filter(raw, c):
    """-ln of the normalised intensity, cosine weight and the row filter, all in 64 bits."""
    W, H, D = c["W"], c["H"], float(np.float32(c["D"]))
    M = W if c["pad"] == 1 else 1 << (2 * W - 1).bit_length()
    win = _window(c["filter"], M // 2 + 1, M // 2 + 1) * W
    u = torch.arange(W, device=DEVICE, dtype=torch.float64) - W / 2.0
    v = H / 2.0 - torch.arange(H, device=DEVICE, dtype=torch.float64)
    weight = D / torch.sqrt(D * D + u[None, :] ** 2 + v[:, None] ** 2)
    out = torch.empty(raw.shape, dtype=torch.float64, device=DEVICE)
    for a, b in _chunks(raw.shape[0], 4 * H * W):
        s = raw[a:b].to(torch.float64)
        if c["raw"] != "f32":
            s = s / (255.0 if c["raw"] == "u8" else 65535.0) + 1e-6
        p = -torch.log(s / (1.0 + 1e-6)) * weight
        out[a:b] = torch.fft.irfft(torch.fft.rfft(p, n=M) * win, n=M)[..., :W] * _scale(c)
    return out


def _view_columns(c, th):
    """(u0, fu, U, kept) of every voxel column (Y, X) for the view at angle th (radians)."""
    fx, fy, x0, y0, X, Y, _, _, _, vs = _box(c)
    D, W = float(np.float32(c["D"])), c["W"]
    vs = float(np.float32(vs))
    x = ((torch.arange(X, device=DEVICE, dtype=torch.float64) - (fx / 2.0 - x0)) * vs)[None, :]
    y = ((torch.arange(Y, device=DEVICE, dtype=torch.float64) - (fy / 2.0 - y0)) * vs)[:, None]
    t = -x * math.sin(th) + y * math.cos(th) + float(np.float32(c.get("u_offset", 0.0)))
    U = D / (D - (x * math.cos(th) + y * math.sin(th)))
    u = t * U + W / 2.0
    kept = (x * x + y * y < _radius(c) ** 2) & (u >= 0) & (u <= W - 1.1)
    u = torch.where(kept, u, torch.zeros_like(u))
    u0 = u.floor()
    return u0.long(), u - u0, U, kept


def _rows(c, U, kept, h, za, zb):
    """(v0, fv, kept) of the voxels of slab slices za .. zb-1."""
    _, _, _, _, _, _, _, fz, z0, vs = _box(c)
    H = c["H"]
    z = ((torch.arange(za, zb, device=DEVICE, dtype=torch.float64) + z0 - fz / 2.0) * float(np.float32(vs)))[:, None, None]
    v = H / 2.0 - (z + h) * U
    k = kept & (v >= 0) & (v <= H - 1.1)
    v = torch.where(k, v, torch.zeros_like(v))
    v0 = v.floor()
    return v0.long(), v - v0, k


def _view_angles(views):
    """Radians, rounded to single precision as the reference holds them."""
    return [float(np.float32(a / 180.0 * math.pi)) for a in _angles(views)]


def _exact_bp(p, c, heights, scale):
    _, _, _, _, X, Y, Zs, _, _, _ = _box(c)
    W = c["W"]
    out = torch.zeros((Zs, Y, X), dtype=torch.float64, device=DEVICE)
    step = max(1, (1 << 25) // (X * Y))
    for i, th in enumerate(_view_angles(c["views"])):
        u0, fu, U, kept = _view_columns(c, th)
        q = p[i].to(torch.float64).reshape(-1)
        h = 0.0 if heights is None else float(np.float32(heights[i]))
        for za in range(0, Zs, step):
            zb = min(Zs, za + step)
            v0, fv, k = _rows(c, U, kept, h, za, zb)
            j = v0 * W + u0
            top = torch.lerp(q[j], q[j + 1], fu.expand_as(fv))
            j += W
            s = torch.lerp(top, torch.lerp(q[j], q[j + 1], fu.expand_as(fv)), fv)
            out[za:zb] += torch.where(k, s * (U * U * scale), torch.zeros_like(s))
    return out


def _exact_fp(vol, c, heights):
    _, _, _, _, X, Y, Zs, _, _, _ = _box(c)
    W, H = c["W"], c["H"]
    out = torch.zeros((c["views"], H * W), dtype=torch.float64, device=DEVICE)
    vol = vol.to(torch.float64)
    step = max(1, (1 << 25) // (X * Y))
    for i, th in enumerate(_view_angles(c["views"])):
        u0, fu, U, kept = _view_columns(c, th)
        h = 0.0 if heights is None else float(np.float32(heights[i]))
        for za in range(0, Zs, step):
            zb = min(Zs, za + step)
            v0, fv, k = _rows(c, U, kept, h, za, zb)
            x = torch.where(k, vol[za:zb] * (U * U), torch.zeros_like(fv))
            j = (v0 * W + u0).reshape(-1)
            for dv, wv in ((0, 1.0 - fv), (W, fv)):
                for du, wu in ((0, 1.0 - fu), (1, fu)):
                    out[i].index_add_(0, j + (dv + du), (x * wv * wu).reshape(-1))
    return out.reshape(c["views"], H, W)


def _updates(c):
    _, _, _, _, X, Y, Zs, _, _, _ = _box(c)
    return float(X) * Y * Zs * c["views"]


def exact(case, seed):
    c = case
    if c["op"] == "batch":
        scans = _shapes(c)
        if sum(_updates(dict(sc, op="fdk")) for sc in scans) > 6.0e10:
            return None
        return [_exact_bp(_exact_filter(_raw_images(sc["W"], sc["H"], sc["views"], sc["raw"], seed, i), sc),
                          dict(sc, op="fdk"), None, 1.0 / _scale(sc)) for i, sc in enumerate(scans)]
    if c["op"] == "filter":
        return _exact_filter(_raw_images(c["W"], c["H"], c["views"], c["raw"], seed), c)
    if _updates(c) > (2.0e10 if c["op"] == "fp" else 1.0e11):
        return None
    heights = _heights(c, seed)
    if c["op"] == "fp":
        return _exact_fp(_volume(c["X"], c["Y"], c["z1"] - c["z0"], seed), c, heights)
    if c["op"] == "bp":
        return _exact_bp(_filtered(c["W"], c["H"], c["views"], c["store"], seed), c, heights, 1.0)
    f = _exact_filter(_raw_images(c["W"], c["H"], c["views"], c["raw"], seed), c)
    v = _exact_bp(f, c, heights, 1.0 / _scale(c))
    if c["op"] == "fdk":
        return [f, v]
    return v.permute(2, 1, 0).contiguous() if c["order"] == "zfastest" else v
