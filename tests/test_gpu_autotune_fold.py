"""Autotuning what goes without tiles: the settings that do nothing to it stay as the caller
set them, and where tiles are drawn every setting is still tried."""
import pytest

import sloth_gpu as S
import workloads as W
from oracle import oracle as O
from gpu_helpers import assert_same, oracle_render
from test_gpu_batch import dev_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("direct,tpb", [(0, 256), (16, 4096), (7, 1024)])
def test_context_keeps_what_does_nothing(direct, tpb):
    m = W.soup(3000, seed=53, n_large=20)
    R = O.euler_rotation(*W.cli_rotation(yaw=1.1))
    w, h = 320, 180
    with S.Context(0) as c:
        dm = dev_mesh(c, m)
        c.set_viewport(w, h, True)
        c.update([dm])
        c.set_direct_samples(direct)
        c.set_triangles_per_block(tpb)
        for _ in range(2):
            best = c.autotune([(dm, R), (dm, R)], reps=2)
            assert (best["direct"], best["tpb"]) == (direct, tpb) and best["ms"] > 0
        c.clear()
        for _ in range(2):
            c.draw_mesh(dm, R)
        assert_same((*c.read(), None), oracle_render([m, m], R, w, h, True), "autotuned")
        c.set_keep_tiles(True)      # with tiles: one of the candidates
        best = c.autotune([(dm, R)], reps=2)
        assert best["direct"] in (0, 4, 16, 64) and best["tpb"] in (128, 256, 1024, 4096)


def test_context_leaves_a_direct_limit_that_bars_the_fold():
    """Above 131,072 triangles a direct limit keeps the tiles: a frame that folds with limit 0
    and is the fastest then has that limit, and one found with tiles has its own."""
    m = W.displaced_icosphere(7, seed=5)
    R = O.euler_rotation(*W.cli_rotation(yaw=1.1))
    with S.Context(0) as c:
        dm = dev_mesh(c, m)
        c.set_viewport(640, 360, True)
        c.update([dm])
        c.set_direct_samples(64)
        best = c.autotune([(dm, R)], reps=3)
        c.set_timing(True)
        c.clear()
        c.draw_mesh(dm, R)
        c.synchronize()
        folds = c.kernel_time("fold")[1]
        assert folds == (1 if best["direct"] == 0 else 0)


@pytest.mark.parametrize("direct,tpb,persistent", [(16, 1024, False), (0, 256, True)])
def test_batch_keeps_what_does_nothing(direct, tpb, persistent):
    m = W.soup(3000, seed=53, n_large=20)
    R = O.euler_rotation(*W.cli_rotation(yaw=1.1))
    with S.Context(0) as c:
        dm = dev_mesh(c, m)
        U = O.viewport_transform(160, 48, O.scene_extent([m["bbox_max"]]))
        b = S.Batch(c, [{"w": 160, "h": 48, "image": True, "U": U, "draws": [(dm, R)]} for _ in range(4)])
        b.set_direct_samples(direct)
        b.set_triangles_per_block(tpb)
        b.set_persistent(persistent)
        best = b.autotune(reps=2)
        assert (best["direct"], best["tpb"], bool(best["persistent"])) == (direct, tpb, persistent)
        b.render()
        for i in range(4):
            assert_same((*b.read(i), None), oracle_render([m], R, 160, 48, True, U=U), f"frame {i}")
        b.close()
