"""The work that programs built on this package have it do, as timed cases.

Every case is one pass through the public entry points on inputs that a seed
determines; `listed` names fixed ones, `draw` makes more of the same ranges.
Kinds:

  frame   one RGBA8 image of a scene (an interactive viewer's redraw)
  path    a camera path, every image read back to pinned host memory (a
          recorded fly-through)
  train   differentiable render and its adjoint (one optimisation step of the
          splat parameters, without the optimiser)
  round   every candidate view of a segmentation round scored in one call
  label   one chosen view shown to the labeller and its mask lifted to
          evidence (the per-view half of the active loop)
  sort    stable radix argsort of (key, value) pairs
  scan    gather scan of per-item counts into offsets

Scenes follow splatfield_b200/synth.py: Gaussian clusters in [-2, 2]^3 or
means uniform in [-1, 1]^3, log-scales around -4, random rotations, opacity
logits of deviation 1.5.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from splatfield_b200 import core, synth

DEG60 = math.radians(60.0)


# ------------------------------------------------------------------- cases

def listed():
    return [
        # A thumbnail of a small object: launch latency is all there is.
        {"name": "thumbnail", "kind": "frame", "scene": "uniform", "n": 3001, "sh": 1, "w": 97, "h": 61,
         "cull": 0},
        # The small workload of synth.py: one 512x512 view of a 100k-splat object.
        {"name": "object_frame", "kind": "frame", "scene": "uniform", "n": 100_000, "sh": 1, "w": 512, "h": 512,
         "cull": 0},
        # An interactive full-HD redraw of a scanned scene with view-dependent colour.
        {"name": "viewer_frame", "kind": "frame", "scene": "clustered", "n": 1_000_000, "sh": 16, "w": 1920,
         "h": 1080, "cull": 1},
        # The headline workload as its user sees it: a 30-camera orbit, each image on the host.
        {"name": "orbit_1080p", "kind": "path", "scene": "clustered", "n": 1_000_000, "sh": 16, "w": 1920,
         "h": 1080, "cull": 1, "cameras": 30},
        # One optimisation step on an odd-sized crop of a small scene.
        {"name": "train_crop", "kind": "train", "scene": "uniform", "n": 50_021, "sh": 4, "w": 333, "h": 217,
         "cull": 0},
        # One optimisation step at full size (the adjoint workload of synth.py).
        {"name": "train_1080p", "kind": "train", "scene": "clustered", "n": 1_000_000, "sh": 16, "w": 1920,
         "h": 1080, "cull": 1},
        # The segmentation round of synth.py: 20 masked candidate views.
        {"name": "round_masked", "kind": "round", "scene": "clustered", "n": 1_000_000, "sh": 16, "views": 20,
         "sides": "512", "form": "evidence", "mode": "lut", "cull": 1},
        # An early, unmasked round on a small scene at ragged view sizes, exact entropies.
        {"name": "round_small", "kind": "round", "scene": "uniform", "n": 60_000, "sh": 9, "views": 6,
         "sides": "200,317,449", "form": "responsibility", "mode": "fp64", "cull": 0},
        # The uneven round of synth.py (3M splats, sides 256 to 1024), a quarter of its views.
        {"name": "round_uneven", "kind": "round", "scene": "clustered", "n": 3_000_000, "sh": 4, "views": 16,
         "sides": "256,384,512,768,1024", "form": "adjoint", "mode": "fp64", "cull": 1},
        # The chosen view of a round: its image for the labeller, its evidence, its EIG.
        {"name": "label_view", "kind": "label", "scene": "clustered", "n": 1_000_000, "sh": 16, "w": 512, "h": 512,
         "mode": "lut", "cull": 0},
        # The depth argsort at the largest size the benchmark sweeps.
        {"name": "argsort_10m", "kind": "sort", "n": 10_000_000, "bits": 32},
        # Intersection offsets of a million splats.
        {"name": "scan_1m", "kind": "scan", "n": 1_000_003},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "path", "train", "train", "round", "round", "label", "sort", "scan"])
    if kind == "sort":
        return {"kind": kind, "n": _log_int(rng, 1000, 10_000_000), "bits": rng.choice([8, 13, 16, 24, 32])}
    if kind == "scan":
        return {"kind": kind, "n": _log_int(rng, 1000, 10_000_000)}
    case = {"kind": kind, "scene": rng.choice(["uniform", "clustered", "clustered"]),
            "n": _log_int(rng, 3000, 1_000_000), "sh": rng.choice([1, 4, 9, 16]), "cull": rng.choice([0, 1])}
    if kind == "round":
        case["views"] = rng.randint(2, 20)
        case["sides"] = ",".join(str(_log_int(rng, 128, 640)) for _ in range(rng.randint(1, 4)))
        case["form"] = rng.choice(["responsibility", "evidence", "adjoint"])
        case["mode"] = rng.choice(["lut", "fp64"])
        return case
    case["w"] = _log_int(rng, 64, 1920)
    case["h"] = _log_int(rng, 48, 1080)
    if kind == "path":
        case["cameras"] = rng.randint(2, 30)
    if kind == "label":
        case["mode"] = rng.choice(["lut", "fp64"])
    return case


# ------------------------------------------------------------------ inputs

def _gen(seed, stream):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1_000_003 + stream) & 0x7FFFFFFF)


def _scene(case, seed):
    """Field-major planes: attributes [11, n], SH [k, 3, n], float32 on the GPU."""
    n, k = case["n"], case["sh"]
    g = _gen(seed, 1)

    def normal(*shape):
        return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)

    def uniform(*shape):
        return torch.rand(shape, generator=g, device="cuda", dtype=torch.float32)

    attr = torch.empty((11, n), device="cuda", dtype=torch.float32)
    if case["scene"] == "uniform":
        attr[0:3] = uniform(3, n) * 2.0 - 1.0
    else:
        centres = uniform(3, 8) * 4.0 - 2.0
        which = torch.randint(0, 8, (n,), generator=g, device="cuda")
        attr[0:3] = (centres[:, which] + 0.3 * normal(3, n)).clamp_(-2.0, 2.0)
    q = normal(4, n)
    attr[3:7] = q / q.norm(dim=0, keepdim=True)
    attr[7:10] = -4.0 + 0.5 * normal(3, n)
    attr[10] = 1.5 * normal(n)
    sh = 0.1 * normal(k, 3, n)
    sh[0] *= 5.0
    return attr, sh


def _splats(case, seed):
    attr, sh = _scene(case, seed)
    return core.CpuSplats(attr.cpu().numpy(), sh.cpu().numpy()).upload()


def _orbit(case, seed, count):
    """Cameras around the scene, the first at an angle the seed picks."""
    radius = 3.0 if case["scene"] == "uniform" else 4.0
    w, h = case["w"], case["h"]
    t0 = 2.0 * math.pi * float(np.random.default_rng([seed, 2]).random())
    cams = []
    for i in range(count):
        t = t0 + 2.0 * math.pi * i / count
        cam = core.look_at((radius * math.cos(t), 0.0, radius * math.sin(t)), (0.0, 0.0, 0.0))
        cam.fov[0], cam.fov[1] = synth.fov_for(w, h)
        cams.append(cam)
    return cams


def _sphere(case, seed, count):
    radius = 3.0 if case["scene"] == "uniform" else 3.5
    v = np.random.default_rng([seed, 3]).standard_normal((count, 3))
    v *= radius / np.linalg.norm(v, axis=1, keepdims=True)
    cams = []
    for p in v:
        cam = core.look_at(tuple(float(x) for x in p), (0.0, 0.0, 0.0))
        cam.fov[0] = cam.fov[1] = DEG60
        cams.append(cam)
    return cams


def _ellipses(w, h, rng):
    """One to three ellipses, bytes row-major (a labeller's binary mask)."""
    x = (np.arange(w) + 0.5)[None, :]
    y = (np.arange(h) + 0.5)[:, None]
    m = np.zeros((h, w), bool)
    for _ in range(int(rng.integers(1, 4))):
        cx, cy, t = rng.random() * w, rng.random() * h, rng.random() * math.pi
        ax, ay = (0.08 + 0.22 * rng.random()) * w, (0.08 + 0.22 * rng.random()) * h
        dx, dy = x - cx, y - cy
        u, v = (math.cos(t) * dx + math.sin(t) * dy) / ax, (-math.sin(t) * dx + math.cos(t) * dy) / ay
        m |= u * u + v * v <= 1.0
    return m.astype(np.uint8).reshape(-1)


def _posterior(n, seed):
    """a, b log-uniform in [1, 1024]."""
    r = torch.rand((2, n), generator=_gen(seed, 4), device="cuda", dtype=torch.float64)
    ab = torch.exp(r * math.log(1024.0)).float()
    return ab[0], ab[1]


def _round_sizes(case):
    sides = [int(x) for x in case["sides"].split(",")]
    return [(sides[v % len(sides)],) * 2 for v in range(case["views"])]


def _eig_mode(case):
    return core.EIG_FP64 if case["mode"] == "fp64" else core.EIG_LUT_F32


def _sort_inputs(case, seed):
    """Depths of splats as float bits, cut to the sorted bits, and their ids."""
    n, bits = case["n"], case["bits"]
    z = 0.1 + 8.0 * torch.rand(n, generator=_gen(seed, 5), device="cuda", dtype=torch.float32)
    keys = z.view(torch.int32)
    if bits < 32:
        keys = (keys >> 5) & ((1 << bits) - 1)
    vals = torch.arange(n, device="cuda", dtype=torch.int32)
    return keys.contiguous(), vals


def _scan_inputs(case, seed):
    """A depth order and per-splat tile counts, most of them small."""
    n = case["n"]
    g = _gen(seed, 6)
    order = torch.randperm(n, generator=g, device="cuda").to(torch.int32)
    counts = (torch.rand(n, generator=g, device="cuda") ** 4 * 40.0).to(torch.int32)
    return order, counts


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "sort":
        st["keys"], st["vals"] = _sort_inputs(case, seed)
        st["scratch"] = core.RadixScratch(case["n"])
        return st
    if kind == "scan":
        st["order"], st["counts"] = _scan_inputs(case, seed)
        st["offsets"] = torch.zeros(case["n"], device="cuda", dtype=torch.int32)
        st["scratch"] = core.ScanScratch(case["n"])
        return st
    n = case["n"]
    splats = st["splats"] = _splats(case, seed)
    if kind == "round":
        sizes = _round_sizes(case)
        st["cams"] = _sphere(case, seed, case["views"])
        if case["form"] != "responsibility":
            rng = np.random.default_rng([seed, 7])
            st["masks"] = [core.Mask.from_bytes(s, _ellipses(*s, rng)) for s in sizes]
        a, b = _posterior(n, seed)
        st["beta"] = core.BetaState.from_host(a.cpu().numpy(), b.cpu().numpy())
        st["round"] = core.Round(n, sizes)
        st["round"].set_tuning(lanes=8, raster_cull=case["cull"])
        return st
    size = st["size"] = (case["w"], case["h"])
    scratch = st["scratch"] = core.RenderScratch(splats.n, size)
    scratch.set_tuning(raster_cull=case["cull"], raster_schedule=core.SCHEDULE_TILES)
    if kind == "path":
        st["cams"] = _orbit(case, seed, case["cameras"])
        st["images"] = torch.empty((case["cameras"], size[1], size[0]), dtype=torch.int32, pin_memory=True)
    elif kind == "label":
        st["cams"] = _sphere(case, seed, 1)
        st["mask"] = core.Mask.from_bytes(size, _ellipses(*size, np.random.default_rng([seed, 7])))
        st["acc"] = core.Accumulators(n)
        a, b = _posterior(n, seed)
        st["beta"] = core.BetaState.from_host(a.cpu().numpy(), b.cpu().numpy())
    else:
        st["cams"] = _orbit(case, seed, 1)
    if kind == "train":
        st["dl"] = _dl(case, seed)
        st["d_attr"] = torch.empty((11, n), device="cuda", dtype=torch.float32)
        st["d_sh"] = torch.empty((case["sh"], 3, n), device="cuda", dtype=torch.float32)
    return st


def _dl(case, seed):
    """dL/d(rgba) of an L2 loss at a typical residual."""
    w, h = case["w"], case["h"]
    return torch.randn((h, w, 4), generator=_gen(seed, 8), device="cuda", dtype=torch.float32) * (0.1 / (w * h))


# -------------------------------------------------------------------- pass

class _Mem:
    """Device memory that a library call returned, for torch.as_tensor."""

    def __init__(self, view, shape, typestr):
        self.view = view
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "data": (view.ptr, False),
                                         "strides": None, "version": 3}


def _tensor(view):
    typestr = "<f4" if view.dtype == np.float32 else "<i4"
    return torch.as_tensor(_Mem(view, view.shape, typestr), device="cuda")


def run(st):
    case = st["case"]
    kind = case["kind"]
    s = torch.cuda.current_stream().cuda_stream
    if kind == "sort":
        k, v = st["scratch"].argsort(st["keys"].data_ptr(), st["vals"].data_ptr(), case["n"], case["bits"],
                                     stream=s)
        return _tensor(k), _tensor(v)
    if kind == "scan":
        core.exclusive_scan_gather(st["order"].data_ptr(), st["counts"].data_ptr(), st["offsets"].data_ptr(),
                                   case["n"], st["scratch"], stream=s)
        return st["offsets"]
    splats = st["splats"]
    if kind == "round":
        rnd, mode = st["round"], _eig_mode(case)
        if case["form"] == "responsibility":
            eig = rnd.eig(splats, st["beta"], st["cams"], mode, stream=s)
            words = [_tensor(rnd.responsibility(v)[0]) for v in range(case["views"])]
        elif case["form"] == "evidence":
            eig = rnd.evidence(splats, st["beta"], st["cams"], st["masks"], mode, stream=s)
            words = [_tensor(x) for v in range(case["views"]) for x in rnd.evidence_words(v)]
        else:
            eig = rnd.evidence_adjoint(splats, st["beta"], st["cams"], st["masks"], mode, stream=s)
            words = [_tensor(x) for v in range(case["views"]) for x in rnd.adjoint_responsibility(v)]
        return eig, words
    scratch, size, cams = st["scratch"], st["size"], st["cams"]
    if kind == "frame":
        return _tensor(splats.render_with(scratch, cams[0], size, stream=s))[:, :size[0]]
    if kind == "path":
        splats.render_frames_to_host(scratch, cams, size, out=st["images"].numpy().view(np.uint32), stream=s)
        return st["images"]
    if kind == "train":
        image = _tensor(splats.render_forward(scratch, cams[0], size, stream=s))
        splats.render_backward_into(scratch, cams[0], size, st["dl"].data_ptr(), st["d_attr"].data_ptr(),
                                    st["d_sh"].data_ptr(), stream=s)
        return image, st["d_attr"], st["d_sh"]
    isects = splats.prepare_isects(scratch, cams[0], size, stream=s)
    image = _tensor(splats.finalize_rgb(scratch, isects, size, stream=s))[:, :size[0]]
    splats.accumulate_prepared(scratch, isects, size, st["acc"], st["mask"], stream=s)
    eig = st["beta"].eig(st["acc"], _eig_mode(case), stream=s)
    return image, _tensor(st["acc"].fg), _tensor(st["acc"].bg), eig


# -------------------------------------------------------------------- work

# f32 operations: a splat's projection without its colour, one multiply-add
# per SH coefficient and channel, one (pixel, splat) composite; contributing
# splats per pixel of these scenes (most pixels saturate or are empty).
PROJECT_FLOPS, COMPOSITE_FLOPS, CONTRIBUTORS = 150, 24, 12


def work(case):
    n, kind = case["n"], case["kind"]
    if kind == "sort":
        return {"bytes": 16 * n, "flops": 0}
    if kind == "scan":
        return {"bytes": 12 * n, "flops": n}
    k = case["sh"]
    used = max(d for d in (1, 4, 9, 16) if d <= k)
    colour = 12 * used * n
    if kind == "round":
        pixels = sum(w * h for w, h in _round_sizes(case))
        v = case["views"]
        words = 4 if case["form"] == "responsibility" else 8
        return {"bytes": 44 * n + 8 * n + words * n * v + pixels // 8,
                "flops": v * PROJECT_FLOPS * n + COMPOSITE_FLOPS * CONTRIBUTORS * pixels}
    pixels = case["w"] * case["h"]
    frames = case.get("cameras", 1)
    frame = PROJECT_FLOPS * n + 6 * used * n + COMPOSITE_FLOPS * CONTRIBUTORS * pixels
    if kind == "train":
        return {"bytes": 2 * (44 * n + colour) + 12 * (k - used) * n + 32 * pixels, "flops": 4 * frame}
    if kind == "label":
        return {"bytes": 44 * n + colour + 16 * n + 4 * pixels + pixels // 8, "flops": 2 * frame}
    return {"bytes": 44 * n + colour + 4 * pixels * frames, "flops": frames * frame}


# ---------------------------------------------------- the values in 64 bits

def _view64(cam, w, h):
    v = core.view_for_camera(cam, w, h)
    t = lambda x: torch.tensor([float(c) for c in x], dtype=torch.float64, device="cuda")  # noqa: E731
    return {"rot": torch.stack([t(v.rot0), t(v.rot1), t(v.rot2)]), "trans": t(v.trans),
            "focal": [float(c) for c in v.focal], "pos": t(v.world_pos)}


def _basis64(k, d):
    x, y, z = d
    b = [torch.full_like(x, 0.2820948)]
    if k >= 4:
        b += [-0.48860252 * y, 0.48860252 * z, -0.48860252 * x]
    if k >= 9:
        b += [1.09254848 * x * y, -1.0925485 * z * y, 0.9461747 * z * z - 0.31539157, -1.0925485 * z * x,
              0.54627424 * (x * x - y * y)]
    if k >= 16:
        c, s, t = x * x - y * y, 2.0 * x * y, 0.4570458 - 2.285229 * z * z
        b += [-0.5900436 * x * s + y * c, -0.5900436 * x * c - y * s, t * y, t * x,
              z * (1.8658817 * z * z - 1.119529), 1.4453057 * z * s, 1.4453057 * z * c]
    return torch.stack(b)


def _project64(attr, sh, v, w, h, colour):
    """Screen-space splats of one view: mean, conic, opacity and colour as
    differentiable planes, and (without gradient) depth, visibility, tile box."""
    cut = float(np.float32(10.0) / np.float32(255.0))
    mean, q, s = attr[0:3], attr[3:7], torch.exp(attr[7:10])
    op = torch.sigmoid(attr[10])
    cam = v["rot"] @ mean + v["trans"][:, None]
    seen = (op >= cut) & (cam[2] > 0.1)
    iz = 1.0 / torch.where(seen, cam[2], torch.ones_like(cam[2]))
    qw, qx, qy, qz = q
    r = [[1 - 2 * (qy * qy + qz * qz), 2 * (qx * qy - qw * qz), 2 * (qx * qz + qw * qy)],
         [2 * (qx * qy + qw * qz), 1 - 2 * (qx * qx + qz * qz), 2 * (qy * qz - qw * qx)],
         [2 * (qx * qz - qw * qy), 2 * (qy * qz + qw * qx), 1 - 2 * (qx * qx + qy * qy)]]
    fx, fy = v["focal"]
    lx, ly = 1.3 * w / (2 * fx), 1.3 * h / (2 * fy)
    u, vv = (cam[0] * iz).clamp(-lx, lx), (cam[1] * iz).clamp(-ly, ly)
    rot = v["rot"]
    t0 = [fx * iz * (rot[0, c] - u * rot[2, c]) for c in range(3)]
    t1 = [fy * iz * (rot[1, c] - vv * rot[2, c]) for c in range(3)]
    j0 = [sum(t0[a] * r[a][c] for a in range(3)) * s[c] for c in range(3)]
    j1 = [sum(t1[a] * r[a][c] for a in range(3)) * s[c] for c in range(3)]
    ca = sum(x * x for x in j0) + 0.3
    cb = sum(x * y for x, y in zip(j0, j1))
    cc = sum(x * x for x in j1) + 0.3
    det = (ca * cc - cb * cb).clamp_min(1e-6)
    mx, my = fx * cam[0] * iz + 0.5 * w, fy * cam[1] * iz + 0.5 * h
    planes = [mx, my, cc / det, -cb / det, ca / det, op]
    if colour:
        d = mean - v["pos"][:, None]
        d = d / d.norm(dim=0, keepdim=True)
        k = max(x for x in (1, 4, 9, 16) if x <= sh.shape[0])
        rgb = torch.einsum("kn,kcn->cn", _basis64(k, d), sh[:k]) + 0.5
        planes += list(rgb)
    with torch.no_grad():
        ext = torch.log(op.clamp_min(cut) / cut)
        ex, ey = torch.sqrt(2 * ext * ca), torch.sqrt(2 * ext * cc)
        tx, ty = (w + 15) // 16, (h + 15) // 16
        box = [((m + o * e) / 16 + a).nan_to_num().clamp(0, t).to(torch.int64) for m, e, o, a, t in
               ((mx, ex, -1, 0, tx), (my, ey, -1, 0, ty), (mx, ex, 1, 1, tx), (my, ey, 1, 1, ty))]
    return torch.stack(planes), cam[2].detach(), seen, box


def _tile_lists64(z, seen, box, w):
    """Splat ids sorted by (tile, depth, id), the tiles of the list and each tile's first entry."""
    tx = (w + 15) // 16
    bw, bh = (box[2] - box[0]).clamp_min(0), (box[3] - box[1]).clamp_min(0)
    cnt = torch.where(seen, bw * bh, torch.zeros_like(bw))
    order = torch.argsort(z, stable=True)
    c = cnt[order]
    ids = torch.repeat_interleave(order, c)
    k = torch.arange(ids.numel(), device=ids.device) - torch.repeat_interleave(c.cumsum(0) - c, c)
    wid = bw[ids].clamp_min(1)
    tile = (box[0][ids] + k % wid) + (box[1][ids] + k // wid) * tx
    tile, o = torch.sort(tile, stable=True)
    tiles, num = torch.unique_consecutive(tile, return_counts=True)
    return ids[o], tiles, num, num.cumsum(0) - num


def _composite64(planes, lists, w, h, weigh):
    """Walks the tiles in groups of like length; calls weigh(pixel rows,
    pixel columns, inside, splat ids [G, M], alpha T [G, M, 256], T [G, 256])
    for each group."""
    ids, tiles, num, first = lists
    tx = (w + 15) // 16
    order = torch.argsort(num)
    num_h = num[order].cpu().numpy()
    ly, lx = torch.meshgrid(torch.arange(16, device=ids.device), torch.arange(16, device=ids.device),
                            indexing="ij")
    lo = 0
    while lo < len(num_h):
        hi = lo + 1
        while hi < len(num_h) and (hi + 1 - lo) * int(num_h[hi]) * 256 <= 24_000_000:
            hi += 1
        sel = order[lo:hi]
        m = int(num_h[hi - 1])
        j = torch.arange(m, device=ids.device)[None, :]
        valid = j < num[sel][:, None]
        gid = ids[(first[sel][:, None] + j).clamp_max(ids.numel() - 1)]
        px = (tiles[sel] % tx)[:, None] * 16 + lx.reshape(1, 256)
        py = (tiles[sel] // tx)[:, None] * 16 + ly.reshape(1, 256)
        inside = (px < w) & (py < h)
        p = planes[:6, gid]
        dx = p[0][:, :, None] - (px + 0.5)[:, None, :]
        dy = p[1][:, :, None] - (py + 0.5)[:, None, :]
        power = 0.5 * (p[2][:, :, None] * dx * dx + p[4][:, :, None] * dy * dy) + p[3][:, :, None] * dx * dy
        alpha = (p[5][:, :, None] * torch.exp(-power)).clamp_max(0.999)
        alpha = alpha * ((alpha >= 1.0 / 255.0) & valid[:, :, None])
        step = torch.log1p(-alpha)
        after = torch.cumsum(step, 1)
        before = torch.exp(after - step)
        alpha = alpha * (before >= 1.0 / 255.0)
        vis = alpha * before
        t = torch.exp((torch.log1p(-alpha)).sum(1))
        weigh(py, px, inside, gid, vis, t)
        lo = hi


def _render64(case, seed, cam):
    """Float image and the gradients of <dl, image>."""
    w, h = case["w"], case["h"]
    attr, sh = (x.double() for x in _scene(case, seed))
    attr.requires_grad_(True)
    sh.requires_grad_(True)
    dl = _dl(case, seed).double()
    planes, z, seen, box = _project64(attr, sh, _view64(cam, w, h), w, h, True)
    leaf = planes.detach().requires_grad_(True)
    image = torch.zeros((h, w, 4), dtype=torch.float64, device="cuda")

    def weigh(py, px, inside, gid, vis, t):
        rgb = torch.einsum("cgm,gmp->gpc", leaf[6:9][:, gid], vis)
        out = torch.cat([rgb, (1.0 - t)[:, :, None]], 2)
        y, x = py[inside], px[inside]
        image[y, x] = out.detach()[inside]
        (out[inside] * dl[y, x]).sum().backward()

    _composite64(leaf, _tile_lists64(z, seen, box, w), w, h, weigh)
    planes.backward(torch.where(seen, leaf.grad, torch.zeros_like(leaf.grad)))
    return image, torch.where(seen, attr.grad, torch.zeros_like(attr.grad)), \
        torch.where(seen, sh.grad, torch.zeros_like(sh.grad))


def _entropy64(a, b):
    s = a + b
    return (torch.lgamma(a) + torch.lgamma(b) - torch.lgamma(s) - (a - 1) * torch.digamma(a)
            - (b - 1) * torch.digamma(b) + (s - 2) * torch.digamma(s))


def _eig64(case, seed, eps):
    a, b = (x.double() for x in _posterior(case["n"], seed))
    k = 1.0 + eps / (a + b)
    return float((_entropy64(a, b) - _entropy64(a * k, b * k)).clamp_min(0).sum())


def _lift64(case, seed, attr, cam, w, h, mask):
    """Real-valued (fg, bg) responsibilities of one view; no mask: all in fg."""
    with torch.no_grad():
        planes, z, seen, box = _project64(attr, None, _view64(cam, w, h), w, h, False)
        fg = torch.zeros(case["n"], dtype=torch.float64, device="cuda")
        bg = torch.zeros_like(fg)
        inside_mask = None if mask is None else torch.from_numpy(mask.reshape(h, w)).cuda().bool()

        def weigh(py, px, inside, gid, vis, t):
            vis = vis * inside[:, None, :]
            if inside_mask is None:
                fg.index_add_(0, gid.reshape(-1), vis.sum(2).reshape(-1))
                return
            m = inside_mask[py.clamp_max(h - 1), px.clamp_max(w - 1)][:, None, :]
            fg.index_add_(0, gid.reshape(-1), (vis * m).sum(2).reshape(-1))
            bg.index_add_(0, gid.reshape(-1), (vis * ~m).sum(2).reshape(-1))

        _composite64(planes, _tile_lists64(z, seen, box, w), w, h, weigh)
    return fg, bg


def exact(case, seed):
    """Images in bytes, fixed-point words, sorted keys and offsets are whole
    numbers and have no value here."""
    kind = case["kind"]
    if kind == "train":
        return _render64(case, seed, _orbit(case, seed, 1)[0])
    if kind == "round":
        attr = _scene(case, seed)[0].double()
        rng = np.random.default_rng([seed, 7])
        eig, words = [], []
        for (w, h), cam in zip(_round_sizes(case), _sphere(case, seed, case["views"])):
            mask = None if case["form"] == "responsibility" else _ellipses(w, h, rng)
            fg, bg = _lift64(case, seed, attr, cam, w, h, mask)
            eig.append(_eig64(case, seed, fg + bg))
            if case["form"] == "responsibility":
                words.append(None)
            elif case["form"] == "evidence":
                words += [None, None]
            else:
                words += [fg, bg]
        return np.array(eig), words
    if kind == "label":
        attr = _scene(case, seed)[0].double()
        fg, bg = _lift64(case, seed, attr, _sphere(case, seed, 1)[0], case["w"], case["h"], None)
        return None, None, None, _eig64(case, seed, fg + bg)
    return None
