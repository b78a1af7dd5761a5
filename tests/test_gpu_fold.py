"""Draws without tiles (rust-sloth_gb300/csrc/fold.cuh): frames bit for bit against the
oracle at the sizes where the fold can go wrong -- one triangle to one over a block's 32,
triangles of one sample to ones the whole GPU walks, frames narrower than a tile, odd
widths, wrapped samples and hostile coordinates."""
import ctypes as C

import numpy as np
import pytest

import sloth_gpu as S
import workloads as W
from oracle import oracle as O
from gpu_helpers import oracle_render
from test_gpu_parity import hostile_soup, span_soup

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def noalloc(m, M, w, h, image):
    n = int(m["rgb"].shape[0])
    ins = [torch.from_numpy(np.ascontiguousarray(m[k]).reshape(-1)).cuda() for k in ("x", "y", "z", "rgb")]
    nz = w * h
    cells = torch.full((nz + (h if image else 0),), -1, dtype=torch.int32, device="cuda")
    z = torch.full((nz,), 7, dtype=torch.int32, device="cuda")
    win = torch.full((nz,), 7, dtype=torch.int32, device="cuda")
    mm = np.ascontiguousarray(M.reshape(16), np.float32)
    st = S.load_library().sloth_render_noalloc(*(t.data_ptr() for t in ins[:3]), n, ins[3].data_ptr(),
                                               mm.ctypes.data_as(C.POINTER(C.c_float)), w, h, int(image),
                                               cells.data_ptr(), z.data_ptr(), win.data_ptr(),
                                               C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == S.OK
    torch.cuda.synchronize()
    return cells.cpu().numpy().view(np.uint32), z.cpu().numpy(), win.cpu().numpy()


def check(got, ref, label):
    for a, b, name in zip(got, (ref.cells, ref.z.view(np.int32), ref.winner), ("cells", "z", "winner")):
        assert np.array_equal(a, b), f"{label}: {name} differ at {np.nonzero(a != b)[0][:5]}"


@pytest.mark.parametrize("w,h,image", [(1, 1, True), (7, 33, False), (161, 95, True), (640, 360, True), (2, 4096, True)])
@pytest.mark.parametrize("n,large,sigma", [(1, 0, 0.3), (31, 1, 0.01), (33, 0, 0.002), (700, 40, 0.2)])
def test_noalloc_sizes(w, h, image, n, large, sigma):
    m = W.soup(n, seed=n + w, n_large=large, sigma=sigma)
    R = O.euler_rotation(*W.cli_rotation(yaw=0.7, pitch=0.4))
    U = O.viewport_transform(w, h, 0.7)     # an extent below the soup's: wrapped samples
    check(noalloc(m, O.mat4_mul(U, R), w, h, image), oracle_render([m], R, w, h, image, U=U), f"{n}+{large} {w}x{h}")


@pytest.mark.parametrize("seed,w,h,image", [(0, 403, 150, True), (1, 512, 128, False)])
def test_noalloc_hostile(seed, w, h, image):
    eye = np.eye(4, dtype=np.float32)
    m = span_soup(seed, w, h)
    check(noalloc(m, eye, w, h, image), oracle_render([m], eye, w, h, image, U=eye), f"spans {seed} {w}x{h}")
    m = hostile_soup(seed)
    R = O.euler_rotation(*W.cli_rotation(yaw=0.4 + seed))
    U = O.viewport_transform(w, h, O.scene_extent([m["bbox_max"]]))
    check(noalloc(m, O.mat4_mul(U, R), w, h, image), oracle_render([m], R, w, h, image, U=U), f"hostile {seed}")


@pytest.mark.parametrize("w,h,image", [(160, 48, True), (161, 47, False)])
def test_context_mixes_fold_and_tiles(w, h, image):
    """Draws of one frame with and without tiles, in both orders, over frames and a resize:
    each keeps the keys of the ones before it.  The big soup (its triangles cover the frame) is
    drawn with culling off, which keeps the tiles whatever its size."""
    small, ico = W.soup(100, seed=3, sigma=0.05), W.displaced_icosphere(2, seed=5)
    big = W.soup(6000, seed=4, n_large=400, sigma=0.8)
    R = O.euler_rotation(*W.cli_rotation(yaw=0.6, pitch=0.2))
    with S.Context(0) as c:
        dev = {id(m): S.Mesh(c, m["x"], m["y"], m["z"], m["rgb"], m["idx"], m["bbox_max"]) for m in (small, ico, big)}
        for k, (order, scale) in enumerate([((small, big, ico), 40.0), ((big, small, ico, small), 40.0),
                                            ((ico, ico, small), 1.0), ((small, big, big), 40.0)]):
            ww, hh = (w, h) if k < 3 else (w + 64, h + 32)
            U = O.viewport_transform(ww, hh, O.scene_extent([m["bbox_max"] for m in order]))
            Rs = [R * np.float32(scale) if m is big else R for m in order]
            c.set_viewport(ww, hh, image)
            c.set_utransform(U)
            c.clear()
            for m, Rm in zip(order, Rs):
                c.set_depth_cull(m is not big)
                c.draw_mesh(dev[id(m)], Rm)
            check([a.view(np.int32) if a.dtype == np.float32 else a for a in c.read()],
                  oracle_render(list(order), Rs, ww, hh, image, U=U), f"mix {k} {ww}x{hh}")


@pytest.mark.parametrize("side", [3, 60, 130])
def test_context_fold_queue_classes(side):
    """A grid of right triangles of `side` samples a side: walked by their block (up to 128
    samples), by one warp (up to 4096) and by many; enough of them for the filter."""
    rng = np.random.default_rng(side)
    n = 700
    c = rng.uniform([0, 0], [256, 200], (n, 2))
    t = np.zeros((n, 3, 3), np.float32)
    t[:, :, :2] = c[:, None, :] + np.array([[0, 0], [0, side], [side, 0]])
    t[:, :, 2] = rng.uniform(-1, 1, (n, 3))
    t[::3] = t[::3, ::-1]
    v = t.reshape(-1, 3)
    m = {"x": v[:, 0].copy(), "y": v[:, 1].copy(), "z": v[:, 2].copy(), "idx": None,
         "rgb": rng.integers(0, 256, (n, 3), dtype=np.uint8), "bbox_max": np.ones(3, np.float32)}
    eye = np.eye(4, dtype=np.float32)
    with S.Context(0) as ctx:
        dm = S.Mesh(ctx, m["x"], m["y"], m["z"], m["rgb"])
        for w, h, image in ((512, 256, True), (513, 255, False)):
            ctx.set_viewport(w, h, image)
            ctx.set_utransform(eye)
            ctx.clear()
            ctx.draw_mesh(dm, eye)
            check([a.view(np.int32) if a.dtype == np.float32 else a for a in ctx.read()],
                  oracle_render([m], eye, w, h, image, U=eye), f"side {side} {w}x{h}")


@pytest.mark.parametrize("direct", [4, 16, 64])
def test_context_fold_after_direct_draw(direct):
    """A fresh context whose first draw is binned with direct samples on: that draw makes the
    tiles' keys current, and the folds after it still start from empty queue counters.  (With
    culling off a draw keeps the tiles whatever its size.)"""
    w, h = 161, 47
    big, ico = W.soup(6000, seed=4, n_large=400, sigma=0.8), W.displaced_icosphere(2, seed=5)
    R = O.euler_rotation(*W.cli_rotation(yaw=0.6, pitch=0.2))
    U = O.viewport_transform(w, h, O.scene_extent([big["bbox_max"], ico["bbox_max"]]))
    with S.Context(0) as c:
        dev = {id(m): S.Mesh(c, m["x"], m["y"], m["z"], m["rgb"], m["idx"], m["bbox_max"]) for m in (ico, big)}
        c.set_direct_samples(direct)
        c.set_viewport(w, h, False)
        c.set_utransform(U)
        for k, order in enumerate(((big, ico, ico, big), (ico, big, ico), (big, ico))):
            Rs = [R * np.float32(40.0) if m is big else R for m in order]
            c.clear()
            for m, Rm in zip(order, Rs):
                c.set_depth_cull(m is not big)
                c.draw_mesh(dev[id(m)], Rm)
            check([a.view(np.int32) if a.dtype == np.float32 else a for a in c.read()],
                  oracle_render(list(order), Rs, w, h, False, U=U), f"frame {k}")


def moved(m):
    return dict(m, x=(m["x"] * np.float32(0.8) + np.float32(0.1)).astype(np.float32))


@pytest.mark.parametrize("w,h,image", [(320, 200, True), (161, 95, False)])
def test_context_fold_draws_in_a_row(w, h, image):
    """Many folded draws in one frame: each one's setup runs beside the walk of the queue
    before, in three sets of counters and two halves of a queue that grows on the way; a mesh
    updated between its draws, and two contexts that draw in turn on one stream."""
    ms = [W.soup(40 + 90 * k * k, seed=k, n_large=3 * k, sigma=0.01 + 0.05 * (k % 3)) for k in range(7)]
    ms += [W.displaced_icosphere(3, seed=9)]
    R = O.euler_rotation(*W.cli_rotation(yaw=0.6, pitch=0.2))
    U = O.viewport_transform(w, h, O.scene_extent([m["bbox_max"] for m in ms]))
    stream = torch.cuda.Stream()
    with S.Context(0, stream=stream.cuda_stream) as a, S.Context(0, stream=stream.cuda_stream) as b:
        dev = [S.Mesh(a, m["x"], m["y"], m["z"], m["rgb"], m["idx"], m["bbox_max"]) for m in ms]
        for c in (a, b):
            c.set_viewport(w, h, image)
            c.set_utransform(U)
        for frame in range(3):
            drawn = {a: [], b: []}
            a.clear()
            b.clear()
            for k in range(2 * len(ms)):
                i = (5 * k + frame) % len(ms)
                for c in (a, b) if k % 3 == 0 else (a,):
                    c.draw_mesh(dev[i], R)
                    drawn[c].append(ms[i])
                if k == 9:
                    i = (5 * (k + 1) + frame) % len(ms)
                    ms[i] = moved(ms[i])
                    dev[i].update(ms[i]["x"], ms[i]["y"], ms[i]["z"], ms[i]["rgb"])
            for c in (a, b):
                check([v.view(np.int32) if v.dtype == np.float32 else v for v in c.read()],
                      oracle_render(drawn[c], R, w, h, image, U=U), f"frame {frame} {w}x{h}")


def test_context_fold_many_triangles():
    """More triangles than an updated mesh folds: the mesh as it was made folds, the same mesh
    after an update takes the tiles, and both frames are the oracle's."""
    m = W.soup(131100, seed=11, n_large=3, sigma=0.01)
    R = O.euler_rotation(*W.cli_rotation(yaw=0.6, pitch=0.2))
    with S.Context(0) as c:
        dm = S.Mesh(c, m["x"], m["y"], m["z"], m["rgb"], m["idx"], m["bbox_max"])
        c.set_viewport(181, 90, False)
        U = O.viewport_transform(181, 90, O.scene_extent([m["bbox_max"]]))
        c.set_utransform(U)
        for step in range(2):
            if step:
                m = moved(m)
                dm.update(m["x"], m["y"], m["z"], m["rgb"])
            c.clear()
            c.draw_mesh(dm, R)
            check([v.view(np.int32) if v.dtype == np.float32 else v for v in c.read()],
                  oracle_render([m], R, 181, 90, False, U=U), f"step {step}")
