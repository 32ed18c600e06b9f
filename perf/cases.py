"""The calls a program makes into this library, as cases that can be timed.

Each kind below is one path through the package's public entry points
(distance-occlusion_b200/__init__.py, or the C ABI where the package has no
wrapper), over the sizes and contents its users bring.  `listed()` names one
case of each; `draw()` gives more cases of the same ranges.

  sdf      signed border field in one call: deltas and distances (the tool's -s)
  twopass  two-pass signed field: exterior and interior deltas, distances (-S)
  df       unsigned field step by step: initial deltas, a delta method, distances (-d)
  edt      exact Euclidean transform straight from the mask
  felz     DOL::Felzenszwalb on a float field: from a mask or arbitrary heights
  chamfer  Chamfer 3-4 on an integer field
  occ      direction weights and the occlusion sweep (-x)
  sites    distances to float sites and their gradient, one training step
  batch    many uneven images and volumes in one launch

A mask is what a user's program holds before these calls: packed words on the
GPU.  Everything random comes from the seed; sizes come from the case alone.
"""
import ctypes as C
import importlib.util
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    if "dol_b200" not in sys.modules:
        pkg = os.path.join(ROOT, "distance-occlusion_b200")
        spec = importlib.util.spec_from_file_location("dol_b200", os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["dol_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["dol_b200"]


dol = _package()
FLT_MAX = float(np.finfo(np.float32).max)
DEV = "cuda"


def listed():
    return [
        # a small sprite or glyph, signed, the tool's default method: the latency of a call
        {"name": "sdf_image_small", "kind": "sdf", "w": 250, "h": 180, "d": 1, "method": "danielsson",
         "content": "noise", "scale": 24},
        # the tool's default run: 1024 x 1024, 100 points, Danielsson, step by step
        {"name": "df_image_points", "kind": "df", "w": 1024, "h": 1024, "d": 1, "method": "danielsson",
         "content": "points", "scale": 100},
        # an image of no special size through the exact transform, signed
        {"name": "edt_image_odd", "kind": "edt", "w": 1501, "h": 1013, "d": 1, "form": "signed",
         "content": "noise", "scale": 48},
        # the reference's float Felzenszwalb on a field of heights, in place
        {"name": "felz_image_heights", "kind": "felz", "w": 1024, "h": 1024, "d": 1, "content": "heights",
         "scale": 32},
        # integer Chamfer, int16, the benchmark's image size
        {"name": "chamfer_image", "kind": "chamfer", "w": 1024, "h": 1024, "d": 1, "dtype": "int16",
         "content": "points", "scale": 100},
        # the 256^3 union of boxes and spheres, signed, by each delta method
        {"name": "sdf_volume_danielsson", "kind": "sdf", "w": 256, "h": 256, "d": 256, "method": "danielsson",
         "content": "shapes", "scale": 64},
        {"name": "sdf_volume_fastsweep", "kind": "sdf", "w": 256, "h": 256, "d": 256, "method": "fastsweep",
         "content": "shapes", "scale": 64},
        {"name": "sdf_volume_jumpflood", "kind": "sdf", "w": 256, "h": 256, "d": 256, "method": "jumpflood",
         "content": "shapes", "scale": 64},
        # the headline: signed exact transform of a 1024^3 volume of value noise
        {"name": "edt_volume_large", "kind": "edt", "w": 1024, "h": 1024, "d": 1024, "form": "signed",
         "content": "noise", "scale": 16},
        # occlusion of a 256^3 volume: eight octant planes
        {"name": "occ_volume", "kind": "occ", "w": 256, "h": 256, "d": 256, "content": "noise", "scale": 32},
        # one training step on 4096 float sites over a 512 x 512 grid: distances, loss, gradient
        {"name": "sites_step", "kind": "sites", "w": 512, "h": 512, "d": 1, "n": 4096, "method": "jumpflood"},
        # 4096 uneven images and 64 volumes, signed, one launch
        {"name": "batch_uneven", "kind": "batch", "images": 4096, "volumes": 64, "sizes": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sdf", "sdf", "sdf", "twopass", "df", "edt", "edt", "felz", "chamfer", "occ", "sites", "batch"])
    if kind == "batch":
        return {"kind": kind, "images": _log_int(rng, 16, 2048), "volumes": rng.randrange(0, 24),
                "sizes": rng.randrange(2, 1 << 20)}
    volume = kind in ("sdf", "twopass", "df", "edt", "occ", "sites") and rng.random() < 0.55
    if volume:
        lo, hi = {"edt": (48, 512), "sites": (24, 144), "occ": (40, 280)}.get(kind, (40, 256))
        w, h, d = (_log_int(rng, lo, hi) for _ in range(3))
    else:
        lo, hi = (64, 1600) if kind != "edt" else (64, 3000)
        w, h, d = _log_int(rng, lo, hi), _log_int(rng, lo, hi), 1
    case = {"kind": kind, "w": w, "h": h, "d": d}
    if kind == "sites":
        case["n"] = min(_log_int(rng, 64, 8192), w * h * d // 8)
        case["method"] = rng.choice(["danielsson", "jumpflood"])
        return case
    if kind in ("sdf", "twopass", "df"):
        case["method"] = rng.choice(["danielsson", "fastsweep", "jumpflood"])
    if kind == "edt":
        case["form"] = rng.choice(["signed", "signed", "dist", "squared"])
    if kind == "chamfer":
        case["dtype"] = rng.choice(["int16", "int16", "int32"])
    contents = ["noise", "noise", "points"] + (["shapes"] if d > 1 else []) + (["heights"] * 2 if kind == "felz" else [])
    case["content"] = rng.choice(contents)
    case["scale"] = {"noise": rng.randrange(8, 64), "points": _log_int(rng, 20, 2000), "shapes": rng.randrange(8, 80),
                     "heights": rng.randrange(8, 64)}[case["content"]]
    return case


# ---- inputs -----------------------------------------------------------------------------------


def _dims(case):
    return (case["w"], case["h"]) if case["d"] == 1 else (case["w"], case["h"], case["d"])


def _noise(gen, w, h, d, spacing):
    """Value noise in [0, 1): random lattice values, linear in between; slice by slice of the lattice for volumes."""
    nx, ny, nz = (s // spacing + 2 for s in (w, h, d))
    if d == 1:
        lattice = torch.rand((1, 1, ny, nx), device=DEV, generator=gen)
        full = torch.nn.functional.interpolate(lattice, size=((ny - 1) * spacing + 1, (nx - 1) * spacing + 1),
                                               mode="bilinear", align_corners=True)
        yield 0, full[0, 0, None, :h, :w]
        return
    lattice = torch.rand((1, 1, nz, ny, nx), device=DEV, generator=gen)
    step = max(1, min(nz - 1, (1 << 27) // (w * h * spacing) or 1))   # lattice cells of z at a time
    for k in range(0, nz - 1, step):
        e = min(nz - 1, k + step)
        full = torch.nn.functional.interpolate(
            lattice[:, :, k:e + 1], size=((e - k) * spacing + 1, (ny - 1) * spacing + 1, (nx - 1) * spacing + 1),
            mode="trilinear", align_corners=True)
        z = k * spacing
        n = min((e - k) * spacing, d - z)
        if n > 0:
            yield z, full[0, 0, :n, :h, :w]


def _pack(bits):
    """Booleans (..., w) to int32 words (rows padded to whole words), bit i of word j being cell 32 j + i."""
    w = bits.shape[-1]
    if w % 32:
        bits = torch.nn.functional.pad(bits, (0, 32 - w % 32))
    b = bits.reshape(-1, 4, 8).to(torch.uint8)
    weights = torch.tensor([1 << i for i in range(8)], dtype=torch.uint8, device=bits.device)
    return (b * weights).sum(-1, dtype=torch.uint8).reshape(-1).view(torch.int32)


def _unpack(mask, case):
    w, h, d = case["w"], case["h"], case["d"]
    bits = (mask.view(-1, 1) >> torch.arange(32, device=mask.device, dtype=torch.int32)) & 1
    return bits.view(d, h, -1)[:, :, :w].bool()


def _mask(case, seed):
    w, h, d = case["w"], case["h"], case["d"]
    gen = torch.Generator(device=DEV).manual_seed(seed)
    if case["content"] == "noise":
        return torch.cat([_pack(v >= 0.5) for _, v in _noise(gen, w, h, d, case["scale"])])
    bits = torch.zeros((d, h, w), dtype=torch.bool, device=DEV)
    if case["content"] == "points":
        at = torch.randint(0, w * h * d, (case["scale"],), device=DEV, generator=gen)
        bits.view(-1)[at] = True
        return _pack(bits)
    # shapes: half boxes, half spheres, sides and radii of 4 to 40 cells
    r = np.random.RandomState(seed & 0x7FFFFFFF)
    for i in range(case["scale"]):
        c = [r.randint(0, s) for s in (d, h, w)]
        if i % 2 == 0:
            half = [r.randint(4, 41) // 2 for _ in range(3)]
            bits[tuple(slice(max(0, a - b), a + b + 1) for a, b in zip(c, half))] = True
        else:
            rad = r.randint(4, 41)
            lo = [max(0, a - rad) for a in c]
            sub = bits[tuple(slice(l, a + rad + 1) for l, a in zip(lo, c))]
            ax = [(torch.arange(n, device=DEV) + l - a) ** 2 for n, l, a in zip(sub.shape, lo, c)]
            sub |= (ax[0][:, None, None] + ax[1][None, :, None] + ax[2][None, None, :]) <= rad * rad
    return _pack(bits)


class _Item(C.Structure):
    _fields_ = [("w", C.c_int), ("h", C.c_int), ("d", C.c_int), ("reserved", C.c_int),
                ("mask_word_offset", C.c_longlong), ("delta_byte_offset", C.c_longlong), ("dist_offset", C.c_longlong)]


def _batch_layout(case):
    """Image sides log-uniform in [32, 1024] with heights up to twice that, volume sides uniform in [32, 128]."""
    rng = random.Random(case["sizes"])
    n = case["images"] + case["volumes"]
    items = (_Item * n)()
    words = delta = cells = 0
    for i in range(n):
        if i < case["images"]:
            w = int(32.0 * 32.0 ** rng.random())
            h, d = int(w * (1.0 + rng.random())), 1
        else:
            w = h = d = rng.randrange(32, 129)
        items[i] = _Item(w, h, d, 0, words, delta, cells)
        words += (w + 31) // 32 * h * d
        delta += (w * h * d * (4 if d == 1 else 6) + 15) // 16 * 16
        cells += w * h * d
    return items, words, delta, cells


def _batch_masks(items, words, seed):
    """Each image one star-shaped outline of 3 to 12 corners, each volume the union of 8 spheres."""
    r = np.random.RandomState(seed & 0x7FFFFFFF)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    masks = torch.zeros(words, dtype=torch.int32, device=DEV)
    radii = 0.2 + 0.25 * torch.rand((len(items), 13), device=DEV, generator=gen)
    balls = torch.rand((len(items), 8, 4), device=DEV, generator=gen)
    line = torch.arange(2048, device=DEV, dtype=torch.float32)
    for i, it in enumerate(items):
        if it.d == 1:
            k = int(r.randint(3, 13))
            y, x = line[:it.h, None] - 0.5 * it.h, line[None, :it.w] - 0.5 * it.w
            a = (torch.atan2(y, x) + math.pi) * (k / (2 * math.pi) * 0.999999)
            f = a.floor()
            rad = radii[i, :k + 1].clone()
            rad[k] = rad[0]
            j = f.long()
            bits = torch.hypot(x, y) <= it.w * torch.lerp(rad[j], rad[j + 1], a - f)
        else:
            s = line[:it.w]
            c, q = balls[i, :, :3] * it.w, (it.w / 8 + balls[i, :, 3] * (it.w / 3 - it.w / 8)) ** 2
            e = (s[None, :, None] - c[:, None, :]) ** 2   # (ball, position, axis)
            bits = ((e[:, :, 2][:, :, None, None] + e[:, :, 1][:, None, :, None] + e[:, :, 0][:, None, None, :])
                    <= q[:, None, None, None]).any(0)
        p = _pack(bits)
        masks[it.mask_word_offset:it.mask_word_offset + p.numel()] = p
    return masks


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "batch":
        items, words, delta, cells = _batch_layout(case)
        n = len(items)
        state["masks"] = _batch_masks(items, words, seed)
        state["deltas"] = torch.zeros(delta // 2, dtype=torch.int16, device=DEV)
        state["dist"] = torch.zeros(cells, dtype=torch.float32, device=DEV)
        state["workspace"] = torch.empty(dol.lib().dol_batch_workspace_size(n), dtype=torch.uint8, device=DEV)
        dol.check(dol.lib().dol_batch_prepare(n, items, C.c_void_p(state["workspace"].data_ptr()),
                                              C.c_size_t(state["workspace"].numel()), _stream()))
        return state
    if kind == "sites":
        gen = torch.Generator(device=DEV).manual_seed(seed)
        dims = _dims(case)
        extent = torch.tensor(dims, dtype=torch.float32, device=DEV)
        unit = torch.rand((case["n"], len(dims)), device=DEV, generator=gen)
        state["sites"] = (unit * extent).requires_grad_(True)
        # the distances the step is fitted to: those of the sites moved by half a cell
        moved = unit * extent + 0.5 * torch.randn(unit.shape, device=DEV, generator=gen)
        moved = torch.minimum(moved.clamp_(min=0), extent - 0.01)
        state["target"] = dol.sites_forward(moved, dims, case["method"])[0]
        state["function"] = dol.site_distance_function()
        return state
    if kind == "felz" and case["content"] == "heights":
        gen = torch.Generator(device=DEV).manual_seed(seed)
        _, v = next(_noise(gen, case["w"], case["h"], 1, case["scale"]))
        rough = torch.rand(v.shape[1:], device=DEV, generator=gen)
        state["field"] = (v[0] * 400.0 + rough * 25.0).contiguous()
        return state
    state["mask"] = _mask(case, seed)
    return state


# ---- one pass ------------------------------------------------------------------------------------


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _tensor_ptr(t):
    return C.c_void_p(t.data_ptr())


_FORMS = {"squared": dol.EDT_SQUARED, "dist": dol.EDT_DIST, "signed": dol.EDT_SIGNED}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        dol.check(dol.lib().dol_batch_run(case["images"] + case["volumes"], _tensor_ptr(state["masks"]),
                                          _tensor_ptr(state["deltas"]), _tensor_ptr(state["dist"]),
                                          _tensor_ptr(state["workspace"]), _stream()))
        return {"deltas": state["deltas"], "dist": state["dist"]}
    dims = _dims(case)
    if kind == "sdf":
        deltas, dist = dol.sdf(state["mask"], dims, case["method"])
        return {"deltas": deltas, "dist": dist}
    if kind == "twopass":
        ext, intr, dist = dol.sdf_two_pass(state["mask"], dims, case["method"])
        return {"exterior": ext, "interior": intr, "dist": dist}
    if kind == "df":
        deltas = dol.init_deltas(state["mask"], dims)
        dol.propagate(case["method"], deltas, dims)
        return {"deltas": deltas, "dist": dol.deltas_to_dist(deltas, dims)}
    if kind == "edt":
        return {"dist": dol.edt_mask(state["mask"], dims, _FORMS[case["form"]])}
    if kind == "felz":
        dist = state["field"].clone() if "field" in state else dol.init_distances(state["mask"], dims)
        return {"dist": dol.felzenszwalb(dist, dims)}
    if kind == "chamfer":
        dist = dol.init_distances_int(state["mask"], dims, case["dtype"])
        dol.chamfer(dist, dims)
        return {"dist": dist}
    if kind == "occ":
        return {"weights": dol.occlusion_sweep(dol.init_dirw(state["mask"], dims), dims)}
    sites = state["sites"]
    sites.grad = None
    dist = state["function"].apply(sites, dims, case["method"])
    (dist - state["target"]).square().sum().backward()
    return {"dist": dist.detach(), "grad": sites.grad}


# ---- what a pass cannot do without ------------------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind == "batch":
        _, words, delta, cells = _batch_layout(case)
        return {"bytes": 4 * words + delta + 4 * cells, "flops": 0}
    w, h, d = case["w"], case["h"], case["d"]
    cells = w * h * d
    mask = 4 * ((w + 31) // 32) * h * d
    delta = 4 if d == 1 else 6
    if kind in ("sdf", "df"):
        total = mask + cells * (delta + 4)
    elif kind == "twopass":
        total = mask + cells * (2 * delta + 4)
    elif kind == "edt":
        total = mask + 4 * cells
    elif kind == "felz":
        total = 8 * cells if case["content"] == "heights" else mask + 4 * cells
    elif kind == "chamfer":
        total = mask + cells * (2 if case["dtype"] == "int16" else 4)
    elif kind == "occ":
        total = mask + cells * 4 * (4 if d == 1 else 8)
    else:   # sites: sites and target in, distances and gradient out
        total = cells * 8 + 2 * case["n"] * 4 * (2 if d == 1 else 3)
    return {"bytes": total, "flops": 0}


# ---- the same in 64 bits -------------------------------------------------------------------------------


def _min_along(f, axis, exact_ints):
    """min over q' of (q - q')^2 + f(q') along an axis, by brute force outwards; stops where no offset can win."""
    f = f.transpose(0, axis)
    best = f.clone()
    for k in range(1, f.shape[0]):
        if k % 8 == 1 and k * k >= best.max().item() - (0 if exact_ints else f.min().item()):
            break
        best[k:] = torch.minimum(best[k:], f[:-k] + k * k)
        best[:-k] = torch.minimum(best[:-k], f[k:] + k * k)
    return best.transpose(0, axis).contiguous()


def _edt_squared(bits):
    """Squared distances (int32, 1 << 30 for none) of a (d, h, w) volume to its set cells."""
    d, h, w = bits.shape
    none = 1 << 30
    out = torch.empty(bits.shape, dtype=torch.int32, device=bits.device)
    pos = torch.arange(w, device=bits.device, dtype=torch.int32)
    for z in range(d):   # along x: the nearest set cell on either side
        left = torch.where(bits[z], pos, -(1 << 15)).cummax(1).values
        right = torch.where(bits[z], -pos, -(1 << 15)).flip(1).cummax(1).values.flip(1)
        near = torch.minimum(pos - left, -right - pos)
        out[z] = torch.where(near >= 1 << 14, torch.full_like(near, none), near * near)
    out = _min_along(out, 1, True)
    return out if d == 1 else _min_along(out, 0, True)


def _root(sq, form):
    far = sq >= 1 << 30
    v = sq.double()
    if form != "squared":
        v.sqrt_()
    v[far] = FLT_MAX if form == "squared" else math.sqrt(FLT_MAX)
    return v


def _exact_occlusion(bits):
    d, h, w = bits.shape
    planes = 4 if d == 1 else 8
    out = torch.empty((planes, d, h, w), dtype=torch.float64, device=bits.device)
    flips = [[a for a, s in ((2, p & 1), (1, p & 2), (0, p & 4)) if s] for p in range(planes)]
    for p in range(planes):
        out[p] = bits.double().flip(flips[p])
    kk, jj = torch.meshgrid(torch.arange(d, device=bits.device), torch.arange(h, device=bits.device), indexing="ij")
    kk, jj = kk.reshape(-1), jj.reshape(-1)
    flat = out.view(planes, -1)
    third = float(np.float32(0.33333333))
    order = (kk + jj).argsort()
    kk, jj = kk[order], jj[order]
    first = torch.searchsorted((kk + jj), torch.arange(d + h + w + 1, device=bits.device)).tolist()
    for s in range(1, d + h + w - 2):   # cells with i + j + k = s need those of s - 1 alone
        lo, hi = first[max(0, s - w + 1)], first[min(s + 1, d + h + w)]
        k, j = kk[lo:hi], jj[lo:hi]
        i = s - k - j
        c = (k * h + j) * w + i
        zero = torch.zeros((), dtype=torch.float64, device=bits.device)
        a = torch.where(i > 0, flat[:, (c - 1).clamp(min=0)], zero)
        b = torch.where(j > 0, flat[:, (c - w).clamp(min=0)], zero)
        if d == 1:
            q = 0.75 * (a + b - a * b)
        else:
            e = torch.where(k > 0, flat[:, (c - w * h).clamp(min=0)], zero)
            q = third * (a + b + e - a * b * e)
        x = flat[:, c]
        flat[:, c] = x + (1 - x) * q
    for p in range(planes):
        out[p] = out[p].flip(flips[p])
    return out


def exact(case, seed):
    # The delta methods and the gradient over their assignment have no closed form: their
    # distances follow from whole-number deltas, which are compared as they are.
    kind = case["kind"]
    if kind not in ("edt", "felz", "occ"):
        return None
    state = prepare(case, seed)
    if kind == "felz" and case["content"] == "heights":
        f = _min_along(state["field"].double(), 0, False)
        return {"dist": _min_along(f, 1, False)}
    cells = case["w"] * case["h"] * case["d"]
    if kind == "edt" and case["content"] != "noise" and cells > 1 << 25:
        return None   # brute force over long walks
    bits = _unpack(state["mask"], case) if cells <= 1 << 28 else torch.cat(
        [_unpack(part, dict(case, d=16)) for part in state["mask"].view(case["d"] // 16, -1)])
    shape = (case["h"], case["w"]) if case["d"] == 1 else (case["d"], case["h"], case["w"])
    if kind == "occ":
        out = _exact_occlusion(bits)
        return {"weights": out.view((out.shape[0],) + shape)}
    if kind == "felz":
        return {"dist": _root(_edt_squared(bits), "squared").view(shape)}
    v = _root(_edt_squared(bits), case["form"])
    if case["form"] == "signed":
        v -= _root(_edt_squared(~bits), "signed")
    return {"dist": v.view(shape)}
