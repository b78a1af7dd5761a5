"""The batch tests with depth culling off, which keeps a batch's tile raster (batches of few
samples otherwise go without tiles), and a batch that changes from one to the other."""
import numpy as np
import pytest

import sloth_gpu as S
import workloads as W
from oracle import oracle as O
from gpu_helpers import assert_same, oracle_render
from test_gpu_batch import (check_frames, dev_mesh, mixed_frames,                          # noqa: F401
                            test_batch_dense_frames_split_tiles, test_batch_entry_overflow_replans,
                            test_batch_exact_across_setting_changes, test_batch_matches_oracle_and_replays)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = S.Context(0)
    c.set_depth_cull(False)
    yield c
    c.close()


@pytest.mark.parametrize("big", [False, True])
def test_batch_changes_between_fold_and_tiles(big):
    """A batch rendered without tiles, then with (culling off, or transforms whose estimate
    is past the fold's), then without again: planned and replayed, every frame exact."""
    with S.Context(0) as c:
        m = W.soup(9000, seed=6, n_large=20)
        dm = dev_mesh(c, m)
        R = O.euler_rotation(*W.cli_rotation(yaw=0.8))
        frames = []
        for w, h, image in ((160, 48, True), (161, 47, False), (320, 180, True)):
            U = O.viewport_transform(w, h, O.scene_extent([m["bbox_max"]]))
            frames.append({"w": w, "h": h, "image": image, "U": U, "draws": [(dm, R), (dm, R)]})
        b = S.Batch(c, frames)
        # 60 times the size: most triangles cover the frame, the estimate is far past the limit
        far = O.mat4_mul(R, np.diag([60.0, 60.0, 60.0, 1.0]).astype(np.float32))
        for step, tiles in enumerate((False, True, False)):
            Rk = far if tiles and big else R
            if big:
                b.set_transforms(np.stack([Rk] * 6))
            else:
                c.set_depth_cull(not tiles)
            for rep in range(3):
                b.render()
                for i, f in enumerate(frames):
                    ref = oracle_render([m, m], Rk, f["w"], f["h"], f["image"], U=f["U"])
                    assert_same((*b.read(i), None), ref, f"step {step} render {rep} frame {i}")
        b.close()


@pytest.mark.parametrize("tpb", [128, 4096])
def test_batch_fold_of_many_triangles(tpb):
    """More than 2^18 triangles of hardly a sample each: the fold goes through the batch's setup kernel, with the
    newline rows beside it, in chunks of one and of several per block."""
    with S.Context(0) as c:
        a, s = W.displaced_icosphere(5, seed=2), W.soup(3000, seed=7, n_large=6, sigma=0.05)
        da, ds = dev_mesh(c, a), dev_mesh(c, s)
        frames, refs = [], []
        for k in range(14):
            w, h, image = ((160, 48, True), (97, 61, False))[k % 2]
            U = O.viewport_transform(w, h, O.scene_extent([a["bbox_max"], s["bbox_max"]]))
            R = O.euler_rotation(*W.cli_rotation(pitch=0.5 * k))
            frames.append({"w": w, "h": h, "image": image, "U": U, "draws": [(da, R), (ds, R)]})
            refs.append(oracle_render([a, s], R, w, h, image, U=U))
        b = S.Batch(c, frames)
        b.set_triangles_per_block(tpb)
        for rep in range(2):
            b.render()
            for i, ref in enumerate(refs):
                assert_same((*b.read(i), None), ref, f"tpb {tpb} render {rep} frame {i}")
        b.close()


@pytest.mark.parametrize("direct,persistent", [(0, True), (16, False)])
def test_batch_overflow_is_exact_on_the_device(ctx, direct, persistent):
    """A graph replay whose entries outgrow the buffer: the frames in device memory are exact
    without a read that re-plans, at odd and even widths, and so are the next renders', one
    of which grows the buffer."""
    torch = pytest.importorskip("torch")

    class Dev:
        def __init__(self, ptr, n):
            self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (ptr, False), "version": 3}

    m = W.soup(3000, seed=41, n_large=10)
    dm = dev_mesh(ctx, m)
    small = O.mat4_mul(O.euler_rotation(*W.cli_rotation()), np.diag([0.05, 0.05, 0.05, 1.0]).astype(np.float32))
    frames = []
    for w, h, image in ((640, 360, True), (321, 181, False)):
        frames.append({"w": w, "h": h, "image": image, "U": O.viewport_transform(w, h, 1.0), "draws": [(dm, small)]})
    b = S.Batch(ctx, frames)
    b.set_direct_samples(direct)
    b.set_persistent(persistent)
    b.render()
    b.render()                      # graph captured with the small entry buffer
    R = O.euler_rotation(*W.cli_rotation(yaw=0.3))
    b.set_transforms(np.stack([R] * 2))
    for rep in range(3):
        b.render()
        torch.cuda.synchronize()
        for i, f in enumerate(frames):
            ref = oracle_render([m], R, f["w"], f["h"], f["image"], U=f["U"])
            c, z = S.C.c_void_p(), S.C.c_void_p()
            assert b.lib.sloth_batch_frame_buffers(b.h, i, S.C.byref(c), S.C.byref(z)) == S.OK
            cells = torch.as_tensor(Dev(c.value, ref.cells.size), device="cuda").cpu().numpy()
            zz = torch.as_tensor(Dev(z.value, ref.z.size), device="cuda").cpu().numpy()
            assert np.array_equal(cells, ref.cells.view(np.int32)), f"render {rep} frame {i}"
            assert np.array_equal(zz, ref.z.view(np.int32)), f"render {rep} frame {i}"
    b.close()


def test_batch_fold_by_single_warps():
    """71,680 triangles of about ten samples: the fold takes 32 triangles to a block of one
    warp; then transforms a hundred times smaller, planned anew and replayed."""
    with S.Context(0) as c:
        a = W.displaced_icosphere(4, seed=2)
        da = dev_mesh(c, a)
        frames = []
        for k in range(14):
            w, h, image = ((320, 90, True), (161, 95, False))[k % 2]
            frames.append({"w": w, "h": h, "image": image, "U": O.viewport_transform(w, h, O.scene_extent([a["bbox_max"]])),
                           "draws": [(da, O.euler_rotation(*W.cli_rotation(pitch=0.5 * k)))]})
        b = S.Batch(c, frames)
        tiny = np.diag([0.01, 0.01, 0.01, 1.0]).astype(np.float32)
        for scale in (None, tiny, None):
            Rs = [f["draws"][0][1] if scale is None else O.mat4_mul(f["draws"][0][1], scale) for f in frames]
            b.set_transforms(np.stack(Rs))
            for rep in range(2):
                b.render()
                for i, f in enumerate(frames):
                    ref = oracle_render([a], Rs[i], f["w"], f["h"], f["image"], U=f["U"])
                    assert_same((*b.read(i), None), ref, f"render {rep} frame {i}")
        b.close()
