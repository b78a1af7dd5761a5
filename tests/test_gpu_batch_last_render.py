"""What a batch hands out is its last render, also when that one outgrew the tile-entry buffer:
nothing is rendered again by a read, with transforms or positions that came after it."""
import numpy as np
import pytest

import sloth_gpu as S
import workloads as W
from oracle import oracle as O
from gpu_helpers import assert_same, oracle_render

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("after", ["transforms", "mesh"])
@pytest.mark.parametrize("ask", ["read", "flush", "fragments"])
def test_read_after_an_overflow_is_the_render_that_overflowed(after, ask):
    m, other = W.soup(3000, seed=41, n_large=10), W.soup(3000, seed=77, n_large=10)
    small = O.mat4_mul(O.euler_rotation(*W.cli_rotation()), np.diag([0.05, 0.05, 0.05, 1.0]).astype(np.float32))
    R, R2 = (O.euler_rotation(*W.cli_rotation(yaw=a)) for a in (0.3, 1.9))
    frames = []
    with S.Context(0) as c:
        c.set_depth_cull(False)             # a batch of few samples keeps its tiles
        dm = S.Mesh(c, m["x"], m["y"], m["z"], m["rgb"], None, m["bbox_max"])
        for w, h, image in ((640, 360, True), (321, 181, False)):
            frames.append({"w": w, "h": h, "image": image, "U": O.viewport_transform(w, h, 1.0), "draws": [(dm, small)]})
        b = S.Batch(c, frames)
        b.render()
        b.render()                          # the graph, with the small entry buffer
        b.set_transforms(np.stack([R] * 2))
        b.render()                          # outgrows it
        keep = (other["x"], other["y"], other["z"], np.ascontiguousarray(other["rgb"].reshape(-1)))
        if after == "transforms":
            b.set_transforms(np.stack([R2] * 2))
        else:
            dm.update(*keep)
        if ask == "flush":
            n = S.C.c_uint64()
            assert b.lib.sloth_batch_flush(b.h, 0, S.FLUSH_PLAIN, None, 0, S.C.byref(n)) == S.OK
        elif ask == "fragments":
            b.fragments()
        for rep in range(2):
            for i, f in enumerate(frames):
                assert_same((*b.read(i), None), oracle_render([m], R, f["w"], f["h"], f["image"], U=f["U"]), f"{rep}/{i}")
        m2, Rn = (m, R2) if after == "transforms" else (other, R)
        for rep in range(3):                # grows the buffer, captures, replays
            b.render()
            for i, f in enumerate(frames):
                assert_same((*b.read(i), None), oracle_render([m2], Rn, f["w"], f["h"], f["image"], U=f["U"]), f"next {rep}/{i}")
        b.close()


def test_a_batch_that_crosses_the_line_keeps_its_graphs():
    """Transforms on both sides of the line between tiles and none, render after render: every
    frame exact, from the graph of its own form, and settings that the captured renders depend
    on capture them again."""
    m = W.soup(9000, seed=6, n_large=20)
    R = O.euler_rotation(*W.cli_rotation(yaw=0.8))
    far = O.mat4_mul(R, np.diag([60.0, 60.0, 60.0, 1.0]).astype(np.float32))
    w, h = 160, 48
    U = O.viewport_transform(w, h, O.scene_extent([m["bbox_max"]]))
    refs = {id(T): oracle_render([m, m], T, w, h, True, U=U) for T in (R, far)}
    with S.Context(0) as c:
        dm = S.Mesh(c, m["x"], m["y"], m["z"], m["rgb"], None, m["bbox_max"])
        b = S.Batch(c, [{"w": w, "h": h, "image": True, "U": U, "draws": [(dm, R), (dm, R)]}])

        def across(n, label):
            for k in range(n):
                T = far if k % 2 else R
                b.set_transforms(np.stack([T, T]))
                b.render()
                assert_same((*b.read(0), None), refs[id(T)], f"{label} {k}")

        across(7, "both forms")
        for change in (lambda: c.set_depth_cull(False), lambda: c.set_depth_cull(True), lambda: b.set_direct_samples(16),
                       lambda: b.set_triangles_per_block(1024), lambda: b.set_persistent(False),
                       lambda: b.set_tile_shape(3), lambda: c.set_keep_tiles(True), lambda: c.set_keep_tiles(False)):
            change()
            across(4, "after a change of settings")
        b.close()
