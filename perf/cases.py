"""Timed workloads of the registration engine, each through its public entry points.

A registration is a loop of a few operations on device images and displacement fields (see
`fastwarp_b200.syn.run_syn_ops`), so most cases are one block of that loop: the midpoint warps, the
similarity and its gradient, the regularisation of the update, the update of a transform pair. A few
are whole calls: one SyN iteration, a whole SyN stage, one step of the linear optimiser. Sizes are
those of the benchmark's configurations: 64^3, the 193 x 229 x 193 template (1 mm) and its pyramid
levels (96 x 114 x 96, 48 x 57 x 48), 160 to 240 voxels an axis for served requests, and
385 x 457 x 385 (0.5 mm).

`listed` and `draw` give cases (dicts of plain values), `prepare` the inputs and handles a user's
program has before the call, `run` one pass, `work` its bytes and operations, `tolerance` how far
another correct implementation may be off, and `exact` the outputs in 64 bits from plain torch.

Fields are (3, nz, ny, nx) in millimetres along x, y, z, images (nz, ny, nx), x fastest.
"""
import ctypes
import math

import numpy as np
import torch
import torch.nn.functional as F

from fastwarp_b200 import _native as N
from fastwarp_b200.backend import (CudaBackend, CudaLinearEngine, binning_from_ranges,
                                   linear_transform, make_affine, make_grid)
from fastwarp_b200.syn import SynRecipe, run_syn_device, syn_step

DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")
STEP = 0.1     # the recipe's gradient step (voxels)


def _case(kind, nx, ny, nz, name=None, **more):
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "mm": 1.0, "oblique": False}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the gradient at the coarsest level of a 1 mm registration: latency counts
        _case("similarity", 48, 57, 48, "similarity_coarse", mm=4.0, radius=4, masked=False),
        # the same at the finest level, where most of a registration's time goes
        _case("similarity", 193, 229, 193, "similarity_fine", radius=4, masked=False),
        # a skull-stripped scan: masked, 0.8 mm, its axes oblique to the scanner's
        _case("similarity", 181, 217, 165, "similarity_masked", mm=0.8, oblique=True, radius=3,
              masked=True),
        # a Mattes channel of a multi-contrast SyN at the finest level
        _case("mattes", 193, 229, 193, "mattes_fine", bins=32),
        # both images to the midpoint at the finest level (a coarser one reads the full-resolution
        # images through the level's fields: `shrink` in `draw`)
        _case("midpoint", 193, 229, 193, "midpoint_fine", shrink=1),
        # smoothing of one side's gradient, its largest vector and the scaling
        _case("regularise", 193, 229, 193, "regularise_fine", variance=3.0),
        # one side's composition and inversion pair, at the middle and the finest level
        _case("update", 96, 114, 96, "update_middle", mm=2.0),
        _case("update", 193, 229, 193, "update_fine"),
        # one whole SyN iteration at 0.5 mm: the largest fields a user registers
        _case("iteration", 385, 457, 385, "iteration_half_mm", mm=0.5, radius=4),
        # whole SyN stages: a small single-level pair, and the 1 mm template recipe
        _case("stage", 64, 64, 64, "stage_small", levels=1, radius=2, channels=1, step=0.25),
        _case("stage", 193, 229, 193, "stage_template", levels=3, radius=4, channels=1, step=0.1),
        # one iteration of the affine stage's optimiser: a value with its gradient, then the
        # values of a line search, on a quarter of the voxels
        _case("line_search", 193, 229, 193, "line_search_fine", affine=True, values=5),
    ]


def _dims(rng, lo, hi, most):
    while True:
        d = [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(3)]
        if d[0] * d[1] * d[2] <= most:
            return d


def draw(rng):
    kind = rng.choice(["similarity", "similarity", "mattes", "midpoint", "regularise", "update",
                       "update", "iteration", "stage", "stage", "line_search"])
    full = 193 * 229 * 193
    if kind == "iteration":
        c = _case(kind, *_dims(rng, 90, 400, 385 * 457 * 385))
        c.update(mm=rng.choice([0.5, 0.8, 1.0]), radius=rng.choice([2, 4, 4]))
    elif kind == "stage":
        levels = rng.choice([1, 2, 3, 3])
        channels = rng.choice([1, 1, 2])
        lo, hi = ((32, 80), (56, 130), (130, 215))[levels - 1]
        c = _case(kind, *_dims(rng, lo, hi, full // 2 if channels == 2 else full))
        c.update(levels=levels, channels=channels, radius=rng.choice([2, 4, 4]),
                 step=rng.choice([0.1, 0.2, 0.25]))
    else:
        c = _case(kind, *_dims(rng, 40, 240, full))
        c["mm"] = rng.choice([0.5, 0.8, 1.0, 1.0, 2.0, 4.0])
        if kind == "similarity":
            c.update(radius=rng.choice([2, 3, 4, 4, 4]), masked=rng.random() < 0.25)
        elif kind == "mattes":
            c.update(bins=rng.choice([24, 32, 32]))
        elif kind == "midpoint":
            c.update(shrink=rng.choice([1, 2, 4]) if max(c["nx"], c["ny"], c["nz"]) <= 60 else 1)
        elif kind == "regularise":
            c.update(variance=rng.choice([1.0, 3.0, 3.0, 9.0]))
        elif kind == "line_search":
            c.update(affine=rng.random() < 0.6, values=rng.choice([3, 5, 7]))
    c["oblique"] = rng.random() < 0.2
    return c


# ---- grids and interpolation ---------------------------------------------------------------------

def _geometry(case, shrink=1):
    """(size, spacing, origin, direction) of the case's level grid, or with `shrink` of the
    full-resolution grid of that many times the level's voxels."""
    size = np.array([case["nx"], case["ny"], case["nz"]]) * shrink
    sp = np.full(3, case["mm"] / shrink)
    d = np.eye(3)
    if case["oblique"]:
        a, b = 0.21, -0.13
        rz = np.array([[math.cos(a), -math.sin(a), 0], [math.sin(a), math.cos(a), 0], [0, 0, 1]])
        rx = np.array([[1, 0, 0], [0, math.cos(b), -math.sin(b)], [0, math.sin(b), math.cos(b)]])
        d = rz @ rx
    centre = np.array([4.0, -7.0, 11.0])
    return size, sp, centre - d @ (sp * (size - 1) / 2.0), d


def _grid(geo):
    size, sp, org, d = geo
    return make_grid([int(s) for s in size], sp, org, d)


def _axes(geo, dtype=torch.float64):
    nx, ny, nz = (int(s) for s in geo[0])
    z = torch.arange(nz, device=DEV, dtype=dtype)[:, None, None]
    y = torch.arange(ny, device=DEV, dtype=dtype)[None, :, None]
    x = torch.arange(nx, device=DEV, dtype=dtype)[None, None, :]
    return x, y, z


def _slabs(nz, voxels):
    step = max(1, int(4e6 * nz / voxels))
    return [(k, min(k + step, nz)) for k in range(0, nz, step)]


def _inside(c, size):
    ok = None
    for a in range(3):
        t = (c[a] >= -0.5) & (c[a] < size[a] - 0.5)
        ok = t if ok is None else ok & t
    return ok


def _corners(vols, c, size):
    """Trilinear values of (nz, ny, nx) volumes at continuous indices, neighbours clamped."""
    lo, w = [], []
    for a in range(3):
        f = torch.floor(c[a])
        w.append(c[a] - f)
        lo.append(f.nan_to_num(0.0).clamp(-2.0, size[a] + 1.0).long())
    out = [0.0] * len(vols)
    flat = [v.reshape(-1) for v in vols]
    for q in range(8):
        i = [(lo[a] + (q >> a & 1)).clamp(0, size[a] - 1) for a in range(3)]
        t = 1.0
        for a in range(3):
            t = t * (w[a] if q >> a & 1 else 1.0 - w[a])
        at = i[0] + size[0] * (i[1] + size[1] * i[2])
        out = [o + t * v[at] for o, v in zip(out, flat)]
    return out


def _index_of_step(geo):
    """3 x 3: millimetres to index steps (the cofactor inverse)."""
    m = geo[3] * geo[1][None, :]
    c = np.array([[m[(r + 1) % 3, (k + 1) % 3] * m[(r + 2) % 3, (k + 2) % 3]
                   - m[(r + 1) % 3, (k + 2) % 3] * m[(r + 2) % 3, (k + 1) % 3] for r in range(3)]
                  for k in range(3)])
    return c * (1.0 / (m[0, 0] * c[0, 0] + m[0, 1] * c[1, 0] + m[0, 2] * c[2, 0]))


def _moved(geo, u, k0, k1):
    """Continuous indices of x + u(x) on the field's own grid, for slices k0..k1."""
    x, y, z = _axes(geo)
    inv = _index_of_step(geo)
    v = [u[a, k0:k1].double() for a in range(3)]
    base = (x, y, z[k0:k1])
    return [base[r] + (inv[r, 0] * v[0] + inv[r, 1] * v[1] + inv[r, 2] * v[2]) for r in range(3)]


def _compose(geo, disp, warping):
    """warping(x) + disp(x + warping(x)), zero added outside."""
    size = [int(s) for s in geo[0]]
    disp, warping = disp.double(), warping.double()
    out = warping.clone()
    for k0, k1 in _slabs(size[2], warping[0].numel()):
        c = _moved(geo, warping, k0, k1)
        ok = _inside(c, size)
        for a, v in enumerate(_corners(list(disp), c, size)):
            out[a, k0:k1] += torch.where(ok, v, torch.zeros_like(v))
    return out


def _warp(src_geo, src, geo, u, affine=None):
    """The image through x + u(x) and the affine (matrix, offset); zero outside its buffer."""
    size, ssize = [int(s) for s in geo[0]], [int(s) for s in src_geo[0]]
    sp, org, d = geo[1:]
    ds, inv = d * sp[None, :], _index_of_step(src_geo)
    x, y, z = _axes(geo)
    out = torch.zeros(size[::-1], device=DEV, dtype=torch.float64)
    m, t = (np.eye(3), np.zeros(3)) if affine is None else affine
    for k0, k1 in _slabs(size[2], out.numel()):
        p = [org[r] + ds[r, 0] * x + ds[r, 1] * y + ds[r, 2] * z[k0:k1] + u[r, k0:k1].double()
             for r in range(3)]
        q = [m[r, 0] * p[0] + m[r, 1] * p[1] + m[r, 2] * p[2] + t[r] - src_geo[2][r] for r in range(3)]
        c = [inv[r, 0] * q[0] + inv[r, 1] * q[1] + inv[r, 2] * q[2] for r in range(3)]
        v = _corners([src], c, ssize)[0]
        out[k0:k1] = torch.where(_inside(c, ssize), v, torch.zeros_like(v))
    return out


# ---- seeded inputs -------------------------------------------------------------------------------

def _rng(seed, part):
    return torch.Generator(device="cpu").manual_seed(int(seed) * 64 + part)


def _smooth_noise(shape, seed, part, cell=14):
    """Three smooth components of unit size, zero on the faces."""
    g = _rng(seed, part)
    coarse = [max(4, -(-s // cell) + 2) for s in shape]
    u = torch.randn((1, 3, *coarse), generator=g).to(DEV)
    u = F.avg_pool3d(F.pad(u, (1,) * 6, mode="replicate"), 3, 1)
    u = F.interpolate(u, size=tuple(shape), mode="trilinear", align_corners=True)[0]
    for a, s in enumerate(shape):
        d = torch.minimum(torch.arange(s), torch.arange(s).flip(0)).to(DEV).float()
        ramp = (d / max(1.0, 0.12 * s)).clamp(max=1.0)
        u = u * (ramp * ramp * (3 - 2 * ramp)).reshape([-1 if q == a else 1 for q in range(3)])
    return u / (u * u).sum(0).sqrt().max()


def _noise(shape, seed, part):
    g = torch.Generator(device=DEV).manual_seed(int(seed) * 64 + part)
    return torch.randn(shape, generator=g, device=DEV)


def _sampled(vols, geo, u):
    """(k, nz, ny, nx) volumes at x + u(x) in float32, for making inputs."""
    size = [int(s) for s in geo[0]]
    inv = _index_of_step(geo)
    x, y, z = _axes(geo, torch.float32)
    base = (x, y, z)
    at = [2.0 * (base[r] + inv[r, 0] * u[0] + inv[r, 1] * u[1] + inv[r, 2] * u[2]) / (size[r] - 1) - 1.0
          for r in range(3)]
    return F.grid_sample(vols[None], torch.stack(at, -1)[None], mode="bilinear",
                         padding_mode="border", align_corners=True)[0]


def _head(shape, seed, part):
    """A head phantom: nested ellipsoids, small structures, a smooth bias and Rician noise."""
    g = torch.Generator().manual_seed(int(seed) * 64 + part)
    r = torch.rand(64, generator=g).tolist()
    zz, yy, xx = (torch.linspace(-1, 1, s, device=DEV).reshape([-1 if q == a else 1 for q in range(3)])
                  for a, s in enumerate(shape))
    img = torch.zeros(tuple(shape), device=DEV)
    for k, (level, rad) in enumerate(zip((0.2, 0.5, 0.8), (0.86, 0.71, 0.46))):
        c = [0.06 * (v - 0.5) for v in r[3 * k:3 * k + 3]]
        e = ((xx - c[0]) / rad) ** 2 + ((yy - c[1]) / (1.05 * rad)) ** 2 + ((zz - c[2]) / rad) ** 2
        img = torch.where(e <= 1, torch.full_like(img, level), img)
    for k in range(8):
        c = [0.7 * (v - 0.5) for v in r[10 + 4 * k:13 + 4 * k]]
        s = 0.05 + 0.08 * r[13 + 4 * k]
        e = ((xx - c[0]) ** 2 + (yy - c[1]) ** 2 + (zz - c[2]) ** 2) / (s * s)
        img = torch.where(e <= 1, torch.full_like(img, 0.2 if k % 2 else 0.5), img)
    img = img * (1.0 + 0.1 * (r[50] - 0.5) * xx + 0.2 * (r[51] - 0.5) * yy * zz + 0.1 * r[52] * xx * xx)
    return img


def _scan(clean, seed, part):
    return ((clean + 0.02 * _noise(clean.shape, seed, part)) ** 2
            + (0.02 * _noise(clean.shape, seed, part + 1)) ** 2).sqrt()


def _pair(geo, seed, amp):
    """Two float32 images of one head, `amp` voxels apart."""
    shape = [int(s) for s in geo[0][::-1]]
    clean = _head(shape, seed, 1)
    moved = _sampled(clean[None], geo, amp * float(geo[1][0]) * _smooth_noise(shape, seed, 2))[0]
    return _scan(clean, seed, 3), _scan(moved, seed, 5)


def _half_transform(geo, seed, part, amp=2.5):
    """A smooth field of at most `amp` voxels and its inverse, as a SyN stage holds them."""
    shape = [int(s) for s in geo[0][::-1]]
    u = amp * float(geo[1][0]) * _smooth_noise(shape, seed, part)
    v = torch.zeros_like(u)
    for _ in range(12):
        v = -_sampled(u, geo, v)
    for a in range(3):  # the faces are held at zero
        for f in (u, v):
            f.select(a + 1, 0).zero_()
            f.select(a + 1, f.shape[a + 1] - 1).zero_()
    return u, v


def _affine(geo, seed):
    """A small rigid and affine map about the grid's centre: (matrix, offset)."""
    r = (torch.rand(12, generator=_rng(seed, 40)).double().numpy() - 0.5) * 2
    a, b, c = 0.08 * r[:3]
    m = np.array([[math.cos(c), -math.sin(c), 0], [math.sin(c), math.cos(c), 0], [0, 0, 1]])
    m = m @ np.array([[1, 0, 0], [0, math.cos(a), -math.sin(a)], [0, math.sin(a), math.cos(a)]])
    m = m @ np.array([[math.cos(b), 0, math.sin(b)], [0, 1, 0], [-math.sin(b), 0, math.cos(b)]])
    m = m @ np.diag(1.0 + 0.04 * r[3:6])
    centre = geo[2] + geo[3] @ (geo[1] * (geo[0] - 1) / 2.0)
    return m, centre + 3.0 * float(geo[1][0]) * r[6:9] - m @ centre


def _mask(shape, seed):
    r = torch.rand(3, generator=_rng(seed, 41)).tolist()
    zz, yy, xx = (torch.linspace(-1, 1, s, device=DEV).reshape([-1 if q == a else 1 for q in range(3)])
                  for a, s in enumerate(shape))
    return (((xx / (0.65 + 0.1 * r[0])) ** 2 + (yy / (0.7 + 0.1 * r[1])) ** 2
             + (zz / (0.65 + 0.1 * r[2])) ** 2) <= 1).float()


def _inputs(case, seed):
    """The case's input tensors, from the seed alone."""
    k = case["kind"]
    geo = _geometry(case)
    shape = [int(s) for s in geo[0][::-1]]
    if k == "similarity":
        f, m = _pair(geo, seed, 2.0)
        return {"f": f, "m": m, "mask": _mask(shape, seed) if case["masked"] else None}
    if k == "mattes":
        f, m = _pair(geo, seed, 2.0)
        return {"f": f, "m": (1.0 - m).abs()}
    if k == "midpoint":
        src = _geometry(case, case["shrink"])
        f, m = _pair(src, seed, 2.0)
        return {"f": f, "m": m, "fi": _half_transform(geo, seed, 10)[1],
                "mi": _half_transform(geo, seed, 11)[1], "affine": _affine(geo, seed)}
    if k == "regularise":
        # a raw gradient: large where the images' edges are, noise elsewhere
        edge = _head(shape, seed, 1)
        g = torch.stack([edge - edge.roll(1, a) for a in (2, 1, 0)])
        return {"g": (1e-3 * (g + 0.05) * _noise((3, *shape), seed, 12))}
    if k == "update":
        u, v = _half_transform(geo, seed, 10)
        step = _smooth_noise(shape, seed, 13, 9)
        return {"u": STEP * float(geo[1][0]) * step, "field": u, "inverse": v}
    if k == "iteration":
        f, m = _pair(geo, seed, 3.0)
        a, ai = _half_transform(geo, seed, 10, 1.5)
        b, bi = _half_transform(geo, seed, 11, 1.5)
        return {"f": f, "m": m, "f2m": a, "f2m_inv": ai, "m2m": b, "m2m_inv": bi,
                "affine": _affine(geo, seed)}
    if k == "stage":
        f, m = _pair(geo, seed, 4.0)
        pairs = [(f, m)]
        if case["channels"] == 2:
            pairs.append(((0.9 - f).abs(), (0.9 - m).abs()))
        return {"pairs": pairs}
    f, m = _pair(geo, seed, 2.0)
    m = (0.9 - m).abs()
    # every fourth voxel, jittered inside its cell, with the fixed image's bin there
    n = f.numel()
    at = torch.arange(0, n, 4, device=DEV)
    nx, ny, nz = (int(s) for s in geo[0])
    jit = torch.rand((3, at.numel()), generator=torch.Generator(device=DEV).manual_seed(int(seed) * 64 + 42),
                     device=DEV, dtype=torch.float64) - 0.5
    c = [(at % nx) + jit[0], (at // nx % ny) + jit[1], (at // (nx * ny)) + jit[2]]
    c = [q.clamp(0, s - 1) for q, s in zip(c, (nx, ny, nz))]
    fv = _corners([f.double()], c, (nx, ny, nz))[0]
    bins = 32
    fr = (float(fv.min()), float(fv.max()))
    size = (fr[1] - fr[0]) / (bins - 4)
    fbin = (fv / size - (fr[0] / size - 2.0)).long().clamp(2, bins - 3)
    ds = geo[3] * geo[1][None, :]
    pts = torch.stack([geo[2][r] + ds[r, 0] * c[0] + ds[r, 1] * c[1] + ds[r, 2] * c[2] for r in range(3)], 1)
    return {"m": m, "points": pts, "fbin": fbin, "franges": fr,
            "mrange": (float(m.min()), float(m.max())), "bins": bins}


def _transforms(case, seed):
    """The linear transforms a line search visits: parameters and centre."""
    geo = _geometry(case)
    r = (torch.rand(32, generator=_rng(seed, 43)).double().numpy() - 0.5) * 2
    centre = geo[2] + geo[3] @ (geo[1] * (geo[0] - 1) / 2.0)
    mm = float(geo[1][0])
    if case["affine"]:
        start = np.concatenate([(np.eye(3) + 0.03 * r[:9].reshape(3, 3)).reshape(-1), 2.0 * mm * r[9:12]])
        step = np.concatenate([0.004 * r[12:21], 0.3 * mm * r[21:24]])
    else:
        start = np.concatenate([0.05 * r[:3], 2.0 * mm * r[3:6]])
        step = np.concatenate([0.006 * r[6:9], 0.3 * mm * r[9:12]])
    return [start + 0.618 ** k * step * (k > 0) for k in range(case["values"] + 1)], centre


# ---- the engine's side ---------------------------------------------------------------------------

_BACKEND = []


def _backend():
    if not _BACKEND:
        _BACKEND.append(CudaBackend(0))
    return _BACKEND[0]


class _View:
    """A device buffer of the engine for zero-copy interop; it keeps the buffer alive."""

    def __init__(self, owner, ptr, shape, strides):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False),
                                         "strides": strides, "version": 3}


def _field_tensor(field, shape):
    ps = ctypes.c_int64()
    ptr = N.lib().fw_field_device_ptr(field.handle, ctypes.byref(ps))
    nz, ny, nx = shape
    return torch.as_tensor(_View(field, ptr, (3, nz, ny, nx), (4 * ps.value, 4 * nx * ny, 4 * nx, 4)),
                           device=DEV)


def _image_tensor(image, shape):
    ptr = N.lib().fw_image_device_ptr(image.handle)
    return torch.as_tensor(_View(image, ptr, tuple(shape), None), device=DEV)


def _new_field(b, grid, t):
    f = b.zero_field(grid)
    _field_tensor(f, t.shape[1:]).copy_(t)
    torch.cuda.synchronize()
    return f


def _new_image(b, grid, t):
    return b.upload_image(grid, t.float().cpu().numpy())


def prepare(case, seed):
    b = _backend()
    k = case["kind"]
    geo = _geometry(case)
    g = _grid(geo)
    shape = [int(s) for s in geo[0][::-1]]
    x = _inputs(case, seed)
    s = {"case": case, "b": b, "shape": shape}
    if k in ("similarity", "mattes"):
        s["f"], s["m"] = _new_image(b, g, x["f"]), _new_image(b, g, x["m"])
        if x.get("mask") is not None:
            s["mask"] = _new_image(b, g, x["mask"])
    elif k == "midpoint":
        sg = _grid(_geometry(case, case["shrink"]))
        s["f"], s["m"] = _new_image(b, sg, x["f"]), _new_image(b, sg, x["m"])
        s["fi"], s["mi"] = _new_field(b, g, x["fi"]), _new_field(b, g, x["mi"])
        s["affine"] = make_affine(*x["affine"])
    elif k == "regularise":
        s["g"] = _new_field(b, g, x["g"])
    elif k == "update":
        for q in ("u", "field", "inverse"):
            s[q] = _new_field(b, g, x[q])
    elif k == "iteration":
        s["f"], s["m"] = _new_image(b, g, x["f"]), _new_image(b, g, x["m"])
        s["state"] = {q: _new_field(b, g, x[q]) for q in ("f2m", "f2m_inv", "m2m", "m2m_inv")}
        s["affine"] = make_affine(*x["affine"])
        s["recipe"] = SynRecipe(gradient_step=STEP, update_field_variance=3.0, cc_radius=case["radius"],
                                iterations=[1], shrink_factors=[1], smoothing_sigmas=[0.0],
                                convergence_threshold=-1.0)
    elif k == "stage":
        s["f"] = [_new_image(b, g, p[0]) for p in x["pairs"]]
        s["m"] = [_new_image(b, g, p[1]) for p in x["pairs"]]
        s["recipe"] = _recipe(case)
    else:
        binning = binning_from_ranges(x["bins"], x["franges"], x["mrange"])
        s["level"] = CudaLinearEngine(b).prepare_level(
            g, x["m"].double().cpu().numpy(), x["points"].cpu().numpy(),
            x["fbin"].cpu().numpy().astype(np.uint32), binning)
        ps, centre = _transforms(case, seed)
        s["ts"] = [linear_transform("affine" if case["affine"] else "euler", p, centre) for p in ps]
    return s


def _recipe(case):
    n = case["levels"]
    return SynRecipe(gradient_step=case["step"], update_field_variance=3.0, cc_radius=case["radius"],
                     iterations=[[30], [50, 20], [70, 50, 20]][n - 1],
                     shrink_factors=[[1], [2, 1], [4, 2, 1]][n - 1],
                     smoothing_sigmas=[[0.0], [1.0, 0.0], [2.0, 1.0, 0.0]][n - 1],
                     convergence_threshold=-1.0, channel_weights=[1.0 / case["channels"]] * case["channels"])


def run(s):
    case, b, shape = s["case"], s["b"], s["shape"]
    k = case["kind"]
    if k == "similarity":
        if case["masked"]:
            pair, norms = b.cc_value_derivative_pair_masked_with_norms(s["f"], s["m"], s["mask"], case["radius"])
        else:
            pair, norms = b.cc_value_derivative_pair_with_norms(s["f"], s["m"], case["radius"])
    elif k == "mattes":
        pair, norms = b.mi_value_derivative_pair_with_norms(s["f"], s["m"], case["bins"])
    if k in ("similarity", "mattes"):
        return {"values": [pair[0][0], pair[1][0]], "norms": list(norms),
                "d_fixed": _field_tensor(pair[0][1], shape), "d_moving": _field_tensor(pair[1][1], shape)}
    if k == "midpoint":
        f = b.warp_through_field(s["f"], s["fi"])
        m = b.warp_through_field(s["m"], s["mi"], affine=s["affine"])
        return {"fixed": _image_tensor(f, shape), "moving": _image_tensor(m, shape)}
    if k == "regularise":
        g = b.copy_field(s["g"])
        b.smooth_field(g, case["variance"])
        top = b.max_scaled_norm(g)
        b.scale(g, STEP / top)
        return {"max": top, "update": _field_tensor(g, shape)}
    if k == "update":
        field = b.compose(s["u"], s["field"])
        inverse = b.copy_field(s["inverse"])
        (inverse, _), (field, _) = b.invert_pair(field, inverse)
        return {"field": _field_tensor(field, shape), "inverse": _field_tensor(inverse, shape)}
    if k == "iteration":
        state = {q: b.copy_field(f) for q, f in s["state"].items()}
        rec, _, _ = syn_step(b, s["recipe"], [s["f"]], [s["m"]], s["affine"], state, want_updates=False)
        out = {q: _field_tensor(f, shape) for q, f in state.items()}
        out["energy"] = rec["energy"]
        return out
    if k == "stage":
        w, iw, recs = run_syn_device(b, s["recipe"], s["f"], s["m"])
        return {"warp": _field_tensor(w, shape), "inverse_warp": _field_tensor(iw, shape),
                "energies": np.array([r["energy"] for r in recs])}
    value, grad = s["level"].value_and_derivative(s["ts"][0])
    return {"value": value, "gradient": grad,
            "values": np.array([s["level"].value(t) for t in s["ts"][1:]])}


# ---- what a pass cannot do without ---------------------------------------------------------------

def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    k = case["kind"]
    if k == "similarity":
        w = 2 * case["radius"] + 1
        return {"bytes": n * (36 if case["masked"] else 32), "flops": n * (3 * 5 * w + 80)}
    if k == "mattes":  # the images once for the ranges, once for the histogram and the gradient
        return {"bytes": n * 32, "flops": n * 120}
    if k == "midpoint":
        return {"bytes": n * 32 + 8 * n * case["shrink"] ** 3, "flops": n * 2 * 40}
    if k == "regularise":
        taps = 2 * int(3.3 * math.sqrt(case["variance"]) + 1) + 1
        return {"bytes": n * 24, "flops": n * 3 * 3 * 2 * taps}
    if k == "update":  # the update, the field and its inverse in, both out
        return {"bytes": n * 60, "flops": n * 3 * 90}
    if k == "iteration":  # the images and the four fields in, the four fields out
        return {"bytes": n * 104, "flops": n * 1500}
    if k == "stage":
        its, sh = _recipe(case).iterations, _recipe(case).shrink_factors
        vox = sum(i * (n // f ** 3) for i, f in zip(its, sh))
        return {"bytes": vox * (96 + 8 * case["channels"]), "flops": vox * 1500}
    passes = case["values"] + 1
    return {"bytes": passes * (n // 4 * 16 + 4 * n), "flops": passes * (n // 4) * 120}


# About four times the error of the float32 outputs against `exact` over listed and drawn cases
# (largest seen, rel / max: similarity 8.4e-7 / 6.4e-5, mattes 5.4e-7 / 4.9e-5, midpoint 3.7e-8 /
# 2.4e-7, regularise 2.0e-7 / 2.3e-6, update and iteration 6e-8 / 3.9e-7, line_search 3.7e-7 /
# 4.8e-7). A stage runs up to 140 iterations, each on the last one's rounding: with the window
# sums in another arithmetic, 1e-10 apart, its fields move by 1.8e-7 / 6.3e-6, and the rounding of
# an update (2e-7) enters at every iteration.
_TOLERANCE = {"similarity": (4e-6, 3e-4), "mattes": (2.5e-6, 2e-4), "midpoint": (1.5e-7, 1e-6),
              "regularise": (8e-7, 1e-5), "update": (2.5e-7, 2e-6), "iteration": (3e-7, 4e-6),
              "stage": (1e-5, 1e-3), "line_search": (2e-6, 1e-5)}


def tolerance(case):
    rel, top = _TOLERANCE[case["kind"]]
    return {"rel": rel, "max": top}


# ---- the same outputs in 64 bits -----------------------------------------------------------------

def exact(case, seed):
    k = case["kind"]
    if k == "stage":
        return None
    geo = _geometry(case)
    size = [int(s) for s in geo[0]]
    x = _inputs(case, seed)
    if k == "similarity":
        return _exact_cc(geo, x["f"], x["m"], case["radius"], x["mask"])
    if k == "mattes":
        one, other = (_exact_mattes(geo, a, b, case["bins"]) for a, b in ((x["f"], x["m"]), (x["m"], x["f"])))
        return {"values": [one[0], other[0]], "norms": [one[2], other[2]], "d_fixed": one[1],
                "d_moving": other[1]}
    if k == "midpoint":
        src = _geometry(case, case["shrink"])
        return {"fixed": _warp(src, x["f"].double(), geo, x["fi"]),
                "moving": _warp(src, x["m"].double(), geo, x["mi"], x["affine"])}
    if k == "regularise":
        g = _exact_smooth(geo, x["g"], case["variance"])
        top = float((g * g).sum(0).sqrt().max()) / float(geo[1][0])
        return {"max": top, "update": g * (STEP / top)}
    if k == "update":
        field, inverse = _exact_invert_pair(geo, _compose(geo, x["u"], x["field"]), x["inverse"].double())
        return {"field": field, "inverse": inverse}
    if k == "iteration":
        if x["f"].numel() > 3e7:
            return None
        fm = _warp(geo, x["f"].double(), geo, x["f2m_inv"])
        mm = _warp(geo, x["m"].double(), geo, x["m2m_inv"], x["affine"])
        cc = _exact_cc(geo, fm, mm, case["radius"], None)
        out = {"energy": cc["values"][0]}
        for d, q in (("d_fixed", "f2m"), ("d_moving", "m2m")):
            g = _exact_smooth(geo, cc[d], 3.0)
            g = g * (STEP / (float((g * g).sum(0).sqrt().max()) / float(geo[1][0])))
            out[q], out[q + "_inv"] = _exact_invert_pair(geo, _compose(geo, g, x[q]), x[q + "_inv"].double())
        return out
    ps, centre = _transforms(case, seed)
    value, grad = _exact_sampled_mi(case, geo, x, ps[0], centre, True)
    return {"value": value, "gradient": grad,
            "values": np.array([_exact_sampled_mi(case, geo, x, p, centre, False)[0] for p in ps[1:]])}


def _gradient(geo, img):
    """Half-spacing central differences along the physical axes, zero where a probe leaves the
    buffer. The probes of a face lie on its edge, so each goes through its physical point in
    the rounding of 64 bits, as the definition has it."""
    size = [int(s) for s in geo[0]]
    sp, org, d = geo[1:]
    inv = _index_of_step(geo)
    out = torch.zeros((3, *img.shape), device=DEV, dtype=torch.float64)
    x, y, z = _axes(geo)
    for k0, k1 in _slabs(size[2], img.numel()):
        s = (x * sp[0], y * sp[1], z[k0:k1] * sp[2])
        p = [((d[r, 0] * s[0] + d[r, 1] * s[1]) + d[r, 2] * s[2]) + org[r] for r in range(3)]

        def probe(a, sign):
            e = [(p[r] + sign * (0.5 * sp[a]) if r == a else p[r]) - org[r] for r in range(3)]
            return [(inv[r, 0] * e[0] + inv[r, 1] * e[1]) + inv[r, 2] * e[2] for r in range(3)]

        for a in range(3):
            lo, hi = probe(a, -1.0), probe(a, 1.0)
            ok = _inside(lo, size) & _inside(hi, size)
            v = (_corners([img], hi, size)[0] - _corners([img], lo, size)[0]) / sp[a]
            out[a, k0:k1] = torch.where(ok, v, torch.zeros_like(v))
    return out


def _box(v, r):
    for a in range(3):
        n = v.shape[a]
        out = v.clone()
        for o in range(1, min(r, n - 1) + 1):
            out.narrow(a, 0, n - o).add_(v.narrow(a, o, n - o))
            out.narrow(a, o, n - o).add_(v.narrow(a, 0, n - o))
        v = out
    return v


def _exact_cc(geo, f, m, r, mask):
    f, m = f.double(), m.double()
    w = torch.ones_like(f) if mask is None else (mask != 0).double()
    fw, mw = f * w, m * w
    cnt, sf, sm = (_box(v, r).clamp(min=1.0) if v is w else _box(v, r) for v in (w, fw, mw))
    sff, smm, sfm = _box(fw * fw, r) - sf * sf / cnt, _box(mw * mw, r) - sm * sm / cnt, _box(fw * mw, r) - sf * sm / cnt
    fi, mi = f - sf / cnt, m - sm / cnt
    del sf, sm, cnt, fw, mw
    eps = np.finfo(np.float64).eps
    p = sff * smm
    ok = p.abs() > eps
    one = torch.ones_like(p)
    cc = torch.where(ok, sfm * sfm / torch.where(ok, p, one), one)
    value = -float((cc * w).sum() / w.sum())
    del cc
    ok = (sff > eps) & (smm > eps) & (w > 0)
    p, a, b = (torch.where(ok, v, one) for v in (p, sff, smm))
    zero = torch.zeros_like(p)
    cf = torch.where(ok, 2 * sfm / p * (fi - sfm / b * mi), zero)
    cm = torch.where(ok, 2 * sfm / p * (mi - sfm / a * fi), zero)
    df, dm = cf * _gradient(geo, m), cm * _gradient(geo, f)
    return {"values": [value, value], "norms": [float(df.norm()), float(dm.norm())], "d_fixed": df,
            "d_moving": dm}


def _spline(u):
    a = u.abs()
    return torch.where(a < 1, (4 - 6 * a * a + 3 * a ** 3) / 6, torch.where(a < 2, (2 - a) ** 3 / 6, torch.zeros_like(a)))


def _spline_slope(u):
    a = u.abs()
    s = torch.where(a < 1, -2 * a + 1.5 * a * a, torch.where(a < 2, -0.5 * (2 - a) ** 2, torch.zeros_like(a)))
    return s * torch.sign(u)


def _mutual_information(fbin, term, mbin, bins, moving_size):
    """-MI of the samples' joint Parzen histogram, and each cell's factor in the gradient."""
    joint = torch.zeros(bins * bins, device=DEV, dtype=torch.float64)
    for o in range(-1, 3):
        joint += torch.bincount(fbin * bins + mbin + o, weights=_spline(mbin + o - term), minlength=bins * bins)
    n = fbin.numel()
    total = joint.sum()
    joint = (joint / total).reshape(bins, bins)
    pf = torch.bincount(fbin, minlength=bins).double() / total
    pm = joint.sum(0)
    eps = np.finfo(np.float64).eps
    ok = (pf[:, None] > eps) & (pm[None, :] > eps) & (joint > eps)
    one = torch.ones_like(joint)
    pr = torch.log(torch.where(ok, joint / pm.clamp(min=eps)[None, :], one))
    value = -float((joint * torch.where(ok, pr - torch.log(pf.clamp(min=eps))[:, None], 0 * one)).sum())
    return value, torch.where(ok, -pr / (moving_size * n), 0 * one).reshape(-1)


def _slope_of(fbin, term, mbin, bins, ratio):
    return sum(_spline_slope(mbin + o - term) * ratio[fbin * bins + mbin + o] for o in range(-1, 3))


def _exact_mattes(geo, f, m, bins):
    f, m = f.double(), m.double()

    def terms(v):
        size = (v.max() - v.min()) / (bins - 4)
        t = (v / size - (v.min() / size - 2.0)).reshape(-1)
        return t, t.long().clamp(2, bins - 3), float(size)

    _, fbin, _ = terms(f)
    term, mbin, size = terms(m)
    value, ratio = _mutual_information(fbin, term, mbin, bins, size)
    d = _slope_of(fbin, term, mbin, bins, ratio).reshape(f.shape) * _gradient(geo, m)
    return value, d, float(d.norm())


def _taps(variance, length):
    """exp(-v) I_n(v) until all but 0.001 of the sum is there, normalised."""
    half, total, n = [], 0.0, 0
    while True:
        t = math.exp(-variance) * sum((variance / 2) ** (2 * j + n) / (math.factorial(j) * math.factorial(j + n))
                                      for j in range(60))
        half.append(t)
        total += t if n == 0 else 2 * t
        n += 1
        if n >= 2 and (total >= 0.999 or len(half) > length):
            break
    return [h / total for h in half]


def _exact_smooth(geo, g, variance):
    v = g.double()
    for a in (3, 2, 1):
        n = v.shape[a]
        taps = _taps(variance, n)
        at = torch.arange(n, device=DEV)
        out = taps[0] * v
        for o, t in enumerate(taps):
            if o:
                out += t * (v.index_select(a, (at + o).clamp(max=n - 1)) + v.index_select(a, (at - o).clamp(min=0)))
        v = out
    w = 1.0 - variance / 0.5 if variance < 0.5 else 1.0
    v = w * v + (1.0 - w) * g.double()
    for a in (1, 2, 3):
        v.select(a, 0).zero_()
        v.select(a, v.shape[a] - 1).zero_()
    return v


def _exact_invert(geo, field, psi):
    top = mean = math.inf
    for it in range(20):
        if not (top > 0.1 and mean > 0.001):
            break
        e = _compose(geo, field, psi)
        norm = (e * e).sum(0).sqrt() / float(geo[1][0])
        top, mean = float(norm.max()), float(norm.mean())
        eps = 0.75 if it == 0 else 0.5
        cut = torch.where(norm > eps * top, eps * top / norm.clamp(min=1e-300), torch.ones_like(norm))
        psi = psi - eps * cut * e
        for a in (1, 2, 3):
            psi.select(a, 0).zero_()
            psi.select(a, psi.shape[a] - 1).zero_()
    return psi


def _exact_invert_pair(geo, field, inverse):
    inverse = _exact_invert(geo, field, inverse)
    return _exact_invert(geo, inverse, field), inverse


def _rotations(p):
    """Rz Rx Ry of the angles (x, y, z), and its three derivatives."""
    def r(axis, a, slope):
        c, s = (-math.sin(a), math.cos(a)) if slope else (math.cos(a), math.sin(a))
        m = np.zeros((3, 3))
        i, j = [(1, 2), (2, 0), (0, 1)][axis]
        m[i, i] = m[j, j] = c
        m[i, j], m[j, i] = -s, s
        if not slope:
            m[axis, axis] = 1.0
        return m
    full = [[r(a, p[a], False) for a in range(3)]] + [[r(a, p[a], a == d) for a in range(3)] for d in range(3)]
    return [q[2] @ q[0] @ q[1] for q in full]


def _exact_sampled_mi(case, geo, x, p, centre, want):
    bins = x["bins"]
    size = [int(s) for s in geo[0]]
    m = x["m"].double()
    lo, hi = x["mrange"]
    width = (hi - lo) / (bins - 4)
    inv = _index_of_step(geo)
    if case["affine"]:
        mat, tr = p[:9].reshape(3, 3), p[9:]
    else:
        mat, tr = _rotations(p)[0], p[3:]
    d = [x["points"][:, r] - centre[r] for r in range(3)]
    y = [mat[r, 0] * d[0] + mat[r, 1] * d[1] + mat[r, 2] * d[2] + (tr[r] + centre[r] - geo[2][r]) for r in range(3)]

    def at(off):
        c = [inv[r, 0] * (y[0] + off[0]) + inv[r, 1] * (y[1] + off[1]) + inv[r, 2] * (y[2] + off[2]) for r in range(3)]
        return _corners([m], c, size)[0], _inside(c, size)

    mv, ok = at((0.0, 0.0, 0.0))
    term = (mv / width - (lo / width - 2.0))[ok]
    mbin = term.long().clamp(2, bins - 3)
    fbin = x["fbin"][ok]
    value, ratio = _mutual_information(fbin, term, mbin, bins, width)
    if not want:
        return value, None
    w = torch.zeros_like(mv)
    w[ok] = _slope_of(fbin, term, mbin, bins, ratio)
    g = []
    for a in range(3):
        off = [0.0, 0.0, 0.0]
        off[a] = 0.5 * float(geo[1][a])
        up, iu = at(off)
        dn, il = at([-o for o in off])
        g.append(torch.where(iu & il, (up - dn) / float(geo[1][a]), torch.zeros_like(up)) * w)
    moment = np.array([[float((g[r] * d[c]).sum()) for c in range(3)] for r in range(3)])
    shift = np.array([float(v.sum()) for v in g])
    if case["affine"]:
        return value, np.concatenate([moment.reshape(-1), shift])
    return value, np.concatenate([[float((q * moment).sum()) for q in _rotations(p)[1:]], shift])
