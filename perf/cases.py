"""The work this framework is measured on: frames, batches, flushes and shaded views, each
through the entry points a program calls (rust-sloth_gb300/sloth_gpu.py, diff_render.py and,
where the binding has no method, the C ABI of include/sloth_gpu.h).

Depth buffers are returned as the bit patterns of their f32 values: the frames' contract is
bit equality, and a background of f32::MAX would hide any relative error.

A program renders on one dedicated CUDA stream, as bench.py does; every context here shares
it.  Depth and frame cells are left on the device (sloth_ctx_device_buffers) except where
the use is a host one (a terminal frame, a flush).
"""
from __future__ import annotations

import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = Path(__file__).resolve().parent.parent / "rust-sloth_gb300"
if str(_PKG) not in sys.path:
    sys.path.insert(0, str(_PKG))

import diff_render as DR  # noqa: E402
import sloth_gpu as S  # noqa: E402
import workloads as W  # noqa: E402

LIGHT = (0.577, 0.577, 0.577)


def listed():
    return [
        # The smallest call: the CLI's sphere in a 160x48 terminal-sized image, cleared, drawn
        # and read back to host arrays.  Launches and the round trip are all there is.
        {"name": "cli_sphere_160x48", "kind": "frame", "mesh": "sphere", "n": 960, "w": 160, "h": 48,
         "image": True, "direct": 0, "tpb": 256, "to": "host"},
        # One frame of the image/JS export: the same sphere at 640x360, flushed as HTML to host.
        {"name": "html_sphere_640x360", "kind": "frame", "mesh": "sphere", "n": 960, "w": 640, "h": 360,
         "image": True, "direct": 0, "tpb": 256, "to": "html"},
        # A queue of models drawn one after another into one frame (match_meshes with several
        # files): many small draws, the default settings.
        {"name": "queue_16_models_1280x720", "kind": "queue", "models": 16, "n": 1280, "w": 1280, "h": 720,
         "image": True, "direct": 0},
        # A finely tessellated indexed model at the settings its autotuner picks (direct folds).
        {"name": "ico_82k_640x360_tuned", "kind": "frame", "mesh": "ico", "n": 81920, "w": 640, "h": 360,
         "image": True, "direct": 64, "tpb": 1024, "to": "device"},
        # A soup in a terminal context (no newlines) of odd width and height, default settings:
        # the odd-width key layout and resolve.
        {"name": "soup_200k_1921x1079_odd", "kind": "frame", "mesh": "soup", "n": 200000, "w": 1921, "h": 1079,
         "image": False, "direct": 0, "tpb": 256, "to": "device"},
        # The headline frame: a million small triangles and 2,000 large ones at 3840x2160.
        {"name": "soup_1m_3840x2160", "kind": "frame", "mesh": "soup", "n": 1002000, "w": 3840, "h": 2160,
         "image": True, "direct": 0, "tpb": 256, "to": "device"},
        # The turntable export: 24 views of one model in a terminal-sized image, new angles each
        # pass.  A launch-bound batch.
        {"name": "turntable_24x160x48", "kind": "batch", "views": 24, "subdiv": 4, "w": 160, "h": 48, "soups": 0,
         "smax": 0, "direct": 0, "tpb": 256},
        # The uneven batch: views of a displaced icosphere and soups of 1k-500k triangles at
        # viewports from 80x24 to 1920x1080, at the settings the autotuner picks.
        {"name": "uneven_128_views_32_soups", "kind": "batch", "views": 128, "subdiv": 6, "w": 640, "h": 360,
         "soups": 32, "smax": 500000, "direct": 64, "tpb": 1024},
        # A host with a fixed memory budget: one soup through the no-allocation entry point.
        {"name": "noalloc_20k_640x360", "kind": "noalloc", "n": 20000, "w": 640, "h": 360, "image": True},
        # Shading with its adjoint at the smallest size in use: a coarse fit on a few small views,
        # through the autograd function.
        {"name": "fit_4x96_sub2", "kind": "shade", "views": 4, "w": 96, "h": 96, "subdiv": 2, "store": True},
        # One step of the inverse-rendering fit: 64 views at 256x256 of a subdivision-4 sphere,
        # visibility stored between forward and backward.
        {"name": "fit_64x256_sub4_stored", "kind": "shade", "views": 64, "w": 256, "h": 256, "subdiv": 4,
         "store": True},
        # The differentiable render at 512x512, 32 views of a subdivision-5 sphere, visibility
        # decoded again in the backward pass (the memory-saving setting).
        {"name": "shade_32x512_sub5_recomputed", "kind": "shade", "views": 32, "w": 512, "h": 512, "subdiv": 5,
         "store": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "queue", "batch", "batch", "noalloc", "shade", "shade"])
    if kind == "frame":
        mesh = rng.choice(["sphere", "ico", "soup", "soup"])
        h = _log(rng, 24, 2160)
        w = min(3840, max(40, int(h * rng.uniform(1.3, 3.4))))
        n = {"sphere": 960, "ico": 20 * 4 ** rng.randint(2, 6), "soup": _log(rng, 1000, 1000000)}[mesh]
        return {"kind": "frame", "mesh": mesh, "n": n, "w": w, "h": h, "image": rng.random() < 0.7,
                "direct": rng.choice([0, 0, 16, 64]), "tpb": rng.choice([128, 256, 1024, 4096]),
                "to": "device" if w * h > 300000 else rng.choice(["device", "host", "html"])}
    if kind == "queue":
        h = _log(rng, 48, 1080)
        return {"kind": "queue", "models": rng.randint(2, 24), "n": _log(rng, 320, 20000),
                "w": int(h * rng.uniform(1.3, 3.0)), "h": h, "image": rng.random() < 0.7,
                "direct": rng.choice([0, 16])}
    if kind == "batch":
        h = _log(rng, 24, 360)
        return {"kind": "batch", "views": _log(rng, 2, 96), "subdiv": rng.randint(2, 5), "w": int(h * rng.uniform(1.3, 3.4)),
                "h": h, "soups": rng.choice([0, 0, 3, 8]), "smax": _log(rng, 2000, 200000),
                "direct": rng.choice([0, 64]), "tpb": rng.choice([256, 1024])}
    if kind == "noalloc":
        h = _log(rng, 24, 480)
        return {"kind": "noalloc", "n": _log(rng, 100, 32768), "w": int(h * rng.uniform(1.2, 2.0)), "h": h,
                "image": rng.random() < 0.7}
    s = _log(rng, 48, 384)
    return {"kind": "shade", "views": _log(rng, 2, 32), "w": s, "h": max(16, int(s * rng.uniform(0.7, 1.3))),
            "subdiv": rng.randint(2, 5), "store": rng.random() < 0.5}


# ---- what a program has in hand before the call ------------------------------------------
_stream = None
_icos: dict[int, tuple] = {}


def stream() -> torch.cuda.Stream:
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream(torch.device("cuda", 0))
    return _stream


def _sphere_mesh(subdiv: int, seed: int, amplitude: float) -> dict:
    """A displaced icosphere; its undisplaced geometry is the same for every seed."""
    if subdiv not in _icos:
        _icos[subdiv] = W.icosphere(subdiv)
    v, f = _icos[subdiv]
    if amplitude:
        v = v * (1.0 + amplitude * W.value_noise3(v, seed))[:, None]
    p = np.ascontiguousarray(v.astype(np.float32).T)
    return {"x": p[0], "y": p[1], "z": p[2], "idx": f.astype(np.uint32),
            "rgb": np.tile(np.array([200, 180, 90], np.uint8), (f.shape[0], 1)),
            "bbox_max": np.maximum(p.max(1), 0.0)}


def _host_mesh(case, seed) -> dict:
    n = case["n"]
    if case["mesh"] == "sphere":
        return W.uv_sphere()
    if case["mesh"] == "ico":
        return _sphere_mesh(int(round(math.log(n / 20, 4))), seed, 0.1)
    large = max(1, n // 501)
    return W.soup(n - large, seed=seed, n_large=large)


def _upload(ctx, m) -> S.Mesh:
    return S.Mesh(ctx, m["x"], m["y"], m["z"], m["rgb"], m.get("idx"), m["bbox_max"])


def _rotation(rng) -> np.ndarray:
    a = rng.uniform(0.0, 2.0 * np.pi, 3)
    return S.euler_rotation(*W.cli_rotation(yaw=a[0], pitch=a[1], roll=a[2]))


class _Device:
    """Device memory of the library, for torch.as_tensor.  The tensor keeps this object, and
    with it the handles that own the memory, for as long as it lives."""

    def __init__(self, ptr: int, n: int, owners: tuple):
        self.owners = owners
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (ptr, False), "version": 3}


def _device_view(st, ptr: int, n: int) -> torch.Tensor:
    key = (ptr, n)
    if key not in st["views"]:
        st["views"][key] = torch.as_tensor(_Device(ptr, n, (st["ctx"], st.get("batch"))), device="cuda")
    return st["views"][key]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    s = stream()
    with torch.cuda.stream(s):
        st = {"case": case, "views": {}}
        if case["kind"] == "noalloc":
            m = W.soup(case["n"] - max(1, case["n"] // 501), seed=seed, n_large=max(1, case["n"] // 501))
            U = S.viewport_transform(case["w"], case["h"], S.scene_extent([m["bbox_max"]]))
            st["m"] = np.ascontiguousarray(S.mat4_mul(U, _rotation(rng)).reshape(16))
            st["in"] = [torch.from_numpy(np.ascontiguousarray(m[k]).reshape(-1)).cuda() for k in ("x", "y", "z", "rgb")]
            nz = case["w"] * case["h"]
            st["out"] = [torch.empty(n, dtype=torch.int32, device="cuda")
                         for n in (nz + (case["h"] if case["image"] else 0), nz, nz)]
            return st
        st["ctx"] = ctx = S.Context(0, stream=s.cuda_stream)
        if case["kind"] == "frame":
            st["meshes"] = [_upload(ctx, _host_mesh(case, seed))]
            st["R"] = [_rotation(rng)]
            ctx.set_triangles_per_block(case["tpb"])
        elif case["kind"] == "queue":
            st["meshes"], st["R"] = [], []
            for k in range(case["models"]):
                m = (_sphere_mesh(int(round(math.log(max(case["n"], 20) / 20, 4))), seed + k, 0.2) if k % 2 else
                     W.soup(case["n"], seed=seed + k, n_large=2, sigma=0.1))
                st["meshes"].append(_upload(ctx, m))
                st["R"].append(_rotation(rng))
        elif case["kind"] == "batch":
            _prepare_batch(st, case, seed, rng)
        else:
            _prepare_shade(st, case, seed)
        if case["kind"] in ("frame", "queue"):
            ctx.set_direct_samples(case["direct"])
            ctx.set_viewport(case["w"], case["h"], case["image"])
        return st


def _prepare_batch(st, case, seed, rng):
    ctx = st["ctx"]
    ctx.set_direct_samples(case["direct"])
    ico = _sphere_mesh(case["subdiv"], seed, 0.1)
    mi = _upload(ctx, ico)
    frames = []
    U = S.viewport_transform(case["w"], case["h"], S.scene_extent([ico["bbox_max"]]))
    for _ in range(case["views"]):
        R = S.euler_rotation(*W.cli_rotation(pitch=float(rng.uniform(0.0, 2.0 * np.pi))))
        frames.append({"w": case["w"], "h": case["h"], "image": True, "U": U, "draws": [(mi, R)]})
    sizes = [(80, 24), (160, 48), (640, 360), (1920, 1080)]
    for k in range(case["soups"]):
        # spread over the range on a logarithmic scale, the same sizes for every seed
        n = int(1000 * (case["smax"] / 1000) ** ((k + 0.5) / case["soups"]))
        m = W.soup(n, seed=seed + 1000 + k, n_large=max(1, n // 500))
        w, h = sizes[k % 4]
        frames.append({"w": w, "h": h, "image": True,
                       "U": S.viewport_transform(w, h, S.scene_extent([m["bbox_max"]])),
                       "draws": [(_upload(ctx, m), _rotation(rng))]})
    st["batch"] = b = S.Batch(ctx, frames)
    b.set_triangles_per_block(case["tpb"])
    st["cells"] = sum(c for c, _ in b.sizes)
    st["zs"] = sum(z for _, z in b.sizes)
    st["R"] = np.ascontiguousarray(np.stack([np.asarray(f["draws"][0][1], np.float32).reshape(16) for f in frames]))


def _shade_inputs(case, seed):
    """Host mesh, positions, vertex colours, loss gradient and views (U, R) of a shade case."""
    rng = np.random.default_rng(seed)
    m = _sphere_mesh(case["subdiv"], seed, 0.05)
    nv = m["x"].size
    pos = np.stack([m["x"], m["y"], m["z"]], 1) + rng.normal(0, 0.002, (nv, 3)).astype(np.float32)
    vrgb = rng.uniform(0.1, 0.9, (nv, 3)).astype(np.float32)
    angles = rng.uniform(0.0, 2.0 * np.pi, (case["views"], 2))
    return m, pos.astype(np.float32), vrgb, angles


def _target(case, seed, n, device):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return torch.rand(n, 3, generator=g, device=device, dtype=torch.float32)


def _prepare_shade(st, case, seed):
    m, pos, vrgb, angles = _shade_inputs(case, seed)
    U = S.viewport_transform(case["w"], case["h"], S.scene_extent([m["bbox_max"]]))
    views = [{"w": case["w"], "h": case["h"], "image": False, "U": U,
              "R": S.euler_rotation(*W.cli_rotation(pitch=a, yaw=0.3 * b))} for a, b in angles]
    st["sv"] = DR.ShadedViews(st["ctx"], m, views, stream(), store_visibility=case["store"])
    dev = torch.device("cuda", 0)
    st["pos"] = torch.from_numpy(pos).to(dev).requires_grad_(True)
    st["vrgb"] = torch.from_numpy(vrgb).to(dev).requires_grad_(True)
    st["light"] = torch.tensor(LIGHT, dtype=torch.float32, device=dev).requires_grad_(True)
    st["target"] = _target(case, seed, case["views"] * case["w"] * case["h"], dev)


# ---- one pass ----------------------------------------------------------------------------
def run(st):
    kind = st["case"]["kind"]
    if kind in ("frame", "queue"):
        return _run_frame(st)
    if kind == "batch":
        b = st["batch"]
        b.set_transforms(st["R"])
        b.render()
        c, z = ctypes.c_void_p(), ctypes.c_void_p()
        b.ctx._check(b.lib.sloth_batch_frame_buffers(b.h, 0, ctypes.byref(c), ctypes.byref(z)))
        return {"cells": _device_view(st, c.value, st["cells"]), "z": _device_view(st, z.value, st["zs"])}
    if kind == "noalloc":
        return _run_noalloc(st)
    return _run_shade(st)


def _run_frame(st):
    case, ctx = st["case"], st["ctx"]
    ctx.update(st["meshes"])
    ctx.clear()
    for m, R in zip(st["meshes"], st["R"]):
        ctx.draw_mesh(m, R)
    to = case.get("to", "device")
    if to == "host":
        cells, z, winner = ctx.read()
        return {"cells": cells.view(np.int32), "z": z.view(np.int32), "winner": winner}
    if to == "html":
        return {"text": np.frombuffer(ctx.flush(S.FLUSH_HTML), np.uint8)}
    c, z = ctx.device_buffers()
    nz = case["w"] * case["h"]
    return {"cells": _device_view(st, c, nz + (case["h"] if case["image"] else 0)), "z": _device_view(st, z, nz)}


def _run_noalloc(st):
    case = st["case"]
    x, y, z, rgb = (t.data_ptr() for t in st["in"])
    cells, zb, win = (t.data_ptr() for t in st["out"])
    e = S.load_library().sloth_render_noalloc(x, y, z, case["n"], rgb, st["m"].ctypes.data_as(S._f32p), case["w"],
                                              case["h"], 1 if case["image"] else 0, cells, zb, win,
                                              stream().cuda_stream)
    if e != S.OK:
        raise S.SlothError(e, "sloth_render_noalloc")
    return {"cells": st["out"][0], "z": st["out"][1], "winner": st["out"][2]}


def _run_shade(st):
    with torch.cuda.stream(stream()):
        rgb = DR.shade_views(st["pos"], st["vrgb"], st["light"], st["sv"])
        # the gradient of sum((rgb - target)^2), given to backward() as it is
        grad = torch.autograd.grad(rgb, (st["pos"], st["vrgb"], st["light"]), 2.0 * (rgb.detach() - st["target"]))
        return {"rgb": rgb.detach(), "pos": grad[0], "vrgb": grad[1], "light": grad[2]}


# ---- what a pass cannot do without -------------------------------------------------------
def work(case):
    """Bytes: 39 per triangle of a soup (9 floats, 3 colour bytes; an indexed mesh 12 of
    indices, 3 of colour and about 6 of shared vertices), 4 per depth cell and per frame cell
    written, the text of a flush.  Operations: about 100 per triangle (transform, edges,
    normal, ranges) and 20 per depth cell (one edge and depth evaluation of its winner)."""
    nz = case["w"] * case["h"]
    out = 8 * nz + (4 * case["h"] if case.get("image") else 0)
    if case["kind"] == "frame":
        n = case["n"]
        b = n * (39 if case["mesh"] == "soup" else 21) + (nz * 37 if case["to"] == "html" else out)
        return {"bytes": b, "flops": 100 * n + 20 * nz}
    if case["kind"] == "queue":
        n = case["models"] * case["n"]
        return {"bytes": n * 30 + out, "flops": 100 * n + 20 * nz}
    if case["kind"] == "noalloc":
        return {"bytes": case["n"] * 39 + out + 4 * nz, "flops": 100 * case["n"] + 20 * nz}
    if case["kind"] == "batch":
        tri = 20 * 4 ** case["subdiv"]
        b, fl = tri * 21 + case["views"] * (8 * nz + 4 * case["h"]), case["views"] * (100 * tri + 20 * nz)
        for k in range(case["soups"]):
            n = int(1000 * (case["smax"] / 1000) ** ((k + 0.5) / case["soups"]))
            c = (80 * 24, 160 * 48, 640 * 360, 1920 * 1080)[k % 4]
            b, fl = b + n * 39 + 8 * c, fl + 100 * n + 20 * c
        return {"bytes": b, "flops": fl}
    tri, v = 20 * 4 ** case["subdiv"], case["views"]
    # forward: the image out (12 per cell); backward: its gradient in, the gradients out
    return {"bytes": tri * 21 + v * nz * 24 + tri // 2 * 24, "flops": v * (100 * tri + 150 * nz)}


# ---- the shaded image and its gradients in 64 bits ---------------------------------------
def _rot32(roll, pitch, yaw):
    """ZYX Euler rotation from f32 angles, in f32 steps (rows of a 3x3)."""
    f = np.float32
    sr, cr, sp, cp, sy, cy = (f(g(float(f(a)))) for a in (roll, pitch, yaw) for g in (math.sin, math.cos))
    return np.array([[cy * cp, cy * sp * sr - sy * cr, cy * sp * cr + sy * sr],
                     [sy * cp, sy * sp * sr + cy * cr, sy * sp * cr - cy * sr],
                     [-sp, cp * sr, cp * cr]], np.float32)


def _view_matrix(case, extent, a, b):
    """3x4 of utransform * rotation in f32, the products summed left to right."""
    f = np.float32
    w, h = f(case["w"]), f(case["h"])
    scale = f(f(min(h, w / f(2.0)) / f(extent)) / f(2.0))
    roll, pitch = f(0.3 * b), f(f(a) + f(math.pi))
    R = _rot32(roll, pitch, f(0.0))
    D = np.array([scale, -scale, scale], np.float32)
    M = np.zeros((3, 4), np.float32)
    M[:, :3] = D[:, None] * R
    M[0, 3], M[1, 3] = w / f(4.0), h / f(2.0)
    return M


def _visible(p, f, w, h):
    """The winning (triangle, x, y) of every depth cell of one view with screen positions p
    (f32, eager torch rounds each step): the reference's loop over samples, all at once."""
    A, B, C = p[f[:, 0]], p[f[:, 1]], p[f[:, 2]]
    tri = torch.stack([A, B, C])
    mn, mx = tri.amin(0), tri.amax(0)
    x0 = torch.ceil(mn[:, 0].clamp(min=1.0)).clamp(max=w).long()
    y0 = torch.ceil(mn[:, 1].clamp(min=1.0)).clamp(max=h).long()
    x1 = torch.ceil((mx[:, 0] * 2.0).clamp(max=w - 1)).long()
    x1 = torch.minimum(x1, torch.floor(mx[:, 0]).long() + 1)   # nothing is covered right of the triangle
    y1 = torch.ceil(mx[:, 1].clamp(max=h - 1)).long()
    nx, ny = (x1 - x0).clamp(min=0), (y1 - y0).clamp(min=0)
    n = nx * ny
    t = torch.repeat_interleave(torch.arange(f.shape[0], device=p.device), n)
    k = torch.arange(t.numel(), device=p.device) - (torch.cumsum(n, 0) - n)[t]
    x, y = x0[t] + k % nx[t].clamp(min=1), y0[t] + torch.div(k, nx[t].clamp(min=1), rounding_mode="floor")
    px, py = x.float(), y.float()

    def orient(a, b, qx, qy):
        return (b[:, 0] - a[:, 0]) * (qy - a[:, 1]) - (b[:, 1] - a[:, 1]) * (qx - a[:, 0])

    a, b, c = A[t], B[t], C[t]
    w0, w1, w2 = orient(b, c, px, py), orient(c, a, px, py), orient(a, b, px, py)
    inv = 1.0 / orient(a, b, c[:, 0], c[:, 1])
    z = a[:, 2] + inv * ((w1 * (b[:, 2] - a[:, 2])) + (w2 * (c[:, 2] - a[:, 2])))
    keep = (w0 >= 0) & (w1 >= 0) & (w2 >= 0) & (z < torch.finfo(torch.float32).max)
    cell = y * w + 2 * x
    keep &= cell < w * h
    t, x, y, z, cell = t[keep], x[keep], y[keep], z[keep], cell[keep]
    # nearest first, then the earliest in (triangle, row, column): two stable sorts
    order = torch.argsort(z + 0.0, stable=True)
    order = order[torch.argsort(cell[order], stable=True)]
    cell, t, x, y = cell[order], t[order], x[order], y[order]
    first = torch.ones_like(cell, dtype=torch.bool)
    first[1:] = cell[1:] != cell[:-1]
    return cell[first], t[first], x[first], y[first]


def exact(case, seed):
    """The shaded image of sloth_batch_shade and the gradients of its adjoint in 64 bits, for
    the visibility the f32 render has; frames and text are whole numbers and have none."""
    if case["kind"] != "shade":
        return None
    dev = torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")
    m, pos, vrgb, angles = _shade_inputs(case, seed)
    w, h = case["w"], case["h"]
    extent = max(0.0, float(np.max(m["bbox_max"])))
    f = torch.from_numpy(m["idx"].astype(np.int64)).to(dev)
    p32 = torch.from_numpy(pos).to(dev)
    P = p32.double().requires_grad_(True)
    V = torch.from_numpy(vrgb).to(dev).double().requires_grad_(True)
    L = torch.tensor(LIGHT, dtype=torch.float32, device=dev).double().requires_grad_(True)
    target = _target(case, seed, case["views"] * w * h, dev).double()
    image = torch.zeros(case["views"] * w * h, 3, dtype=torch.float64, device=dev)
    loss = 0.0
    for k, (a, b) in enumerate(angles):
        M = _view_matrix(case, extent, a, b)
        rows = [[float(v) for v in r] for r in M]
        s32 = torch.stack([((r[0] * p32[:, 0] + r[1] * p32[:, 1]) + r[2] * p32[:, 2]) + r[3] for r in rows], 1)
        cell, t, x, y = _visible(s32, f, w, h)
        M64 = torch.from_numpy(M).to(dev).double()
        q = P @ M64[:, :3].T + M64[:, 3]
        i = f[t]
        A, B, C = q[i[:, 0]], q[i[:, 1]], q[i[:, 2]]
        px, py = x.double(), y.double()

        def orient(u, v, qx, qy):
            return (v[:, 0] - u[:, 0]) * (qy - u[:, 1]) - (v[:, 1] - u[:, 1]) * (qx - u[:, 0])

        o = orient(A, B, C[:, 0], C[:, 1])
        b0, b1, b2 = (orient(u, v, px, py) / o for u, v in ((B, C), (C, A), (A, B)))
        n = torch.linalg.cross(B - A, C - A)
        s = ((n / n.norm(dim=1, keepdim=True)) @ L).clamp(0.0, 1.0)
        rgb = (b0[:, None] * V[i[:, 0]] + b1[:, None] * V[i[:, 1]] + b2[:, None] * V[i[:, 2]]) * s[:, None]
        at = k * w * h + cell
        image[at] = rgb.detach()
        loss = loss + ((rgb - target[at]) ** 2).sum()
    g = torch.autograd.grad(loss, (P, V, L))
    return {"rgb": image, "pos": g[0], "vrgb": g[1], "light": g[2]}
