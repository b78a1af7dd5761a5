"""The tile raster with depth culling on, which is what large frames take: the parity tests'
scenes -- hostile coordinates, odd widths, wrapped samples, every tile shape, slices, the
tuning settings, entry-buffer overflows -- with SLOTH_OPTION_KEEP_TILES, since draws and
batches of few samples otherwise go without tiles.  Which kernels ran is checked."""
import numpy as np
import pytest

import sloth_gpu as S
import workloads as W
from oracle import oracle as O
from gpu_helpers import assert_same, gpu_render, oracle_render
from test_gpu_batch import (check_frames, dev_mesh, mixed_frames,                          # noqa: F401
                            test_batch_dense_frames_split_tiles, test_batch_entry_overflow_replans,
                            test_batch_every_tile_shape_and_autotune, test_batch_exact_across_setting_changes,
                            test_batch_matches_oracle_and_replays, test_context_autotune_renders_the_same_frame,
                            test_context_every_tile_shape, test_context_tuning_settings)
from test_gpu_parity import (hostile_soup, span_soup, test_clear_redraw_and_resize,        # noqa: F401
                             test_dense_small_viewport_split_tiles, test_depth_culling_skips_hidden_fragments,
                             test_hostile_indexed, test_hostile_soups, test_indexed_icosphere_multi_mesh,
                             test_micro_cases, test_row_span_walk, test_scaled_config2_soup,
                             test_spatial_order_keeps_draw_order_ties, test_uv_sphere_config,
                             test_viewport_one_by_one_and_width_one, test_yawed_soup_wraps)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = S.Context(0)
    c.set_keep_tiles(True)
    yield c
    c.close()


@pytest.fixture(autouse=True)
def only_tiles(ctx):
    """No draw of a test's context goes without tiles."""
    ctx.set_timing(True)
    before = ctx.kernel_time("fold")[1]
    yield
    assert ctx.kernel_time("fold")[1] == before
    ctx.set_timing(False)


def test_the_option_decides(ctx):
    m = W.uv_sphere()
    dm = dev_mesh(ctx, m)
    R = O.euler_rotation(*W.cli_rotation(yaw=0.5))
    ctx.set_viewport(160, 48, True)
    ctx.update([dm])
    raster = ctx.kernel_time("raster")[1]
    ctx.clear()
    ctx.draw_mesh(dm, R)
    ctx.read()
    assert ctx.kernel_time("raster")[1] == raster + 1
    with S.Context(0) as c:
        c.set_timing(True)
        c.set_viewport(160, 48, True)
        c.update([dm])
        c.clear()
        c.draw_mesh(dm, R)
        c.read()
        assert c.kernel_time("fold")[1] == 1 and c.kernel_time("raster")[1] == 0
    for bad in (-1, 2):
        assert ctx.lib.sloth_ctx_set_option(ctx.h, S.OPTION_KEEP_TILES, bad) == 1


@pytest.mark.parametrize("shape", range(5))
@pytest.mark.parametrize("w,h,image", [(403, 150, True), (512, 128, False)])
def test_hostile_scenes_in_every_tile_shape(ctx, shape, w, h, image):
    ctx.set_tile_shape(shape)
    try:
        eye = np.eye(4, dtype=np.float32)
        m = span_soup(shape, w, h)
        assert_same(gpu_render(ctx, [m], eye, w, h, image, U=eye), oracle_render([m], eye, w, h, image, U=eye), "spans")
        ms = [hostile_soup(shape), hostile_soup(shape + 50, n=500)]
        R = O.euler_rotation(*W.cli_rotation(yaw=0.4 + shape, pitch=0.3))
        U = O.viewport_transform(w, h, 0.7)     # an extent below the soups': wrapped samples
        assert_same(gpu_render(ctx, ms, R, w, h, image, U=U), oracle_render(ms, R, w, h, image, U=U), "hostile")
    finally:
        ctx.set_tile_shape(0)


@pytest.mark.parametrize("direct", [0, 16])
@pytest.mark.parametrize("tpb", [128, 4096])
def test_overflow_with_culling(direct, tpb):
    """test_overflow_fallback_multi_draw's draws, which outgrow the entry buffer of the first,
    twice over: the second frame's buffer has grown."""
    small, big = W.soup(100, seed=7), W.soup(30000, seed=8, n_large=50)
    big2 = W.soup(20000, seed=9, n_large=30, sigma=0.04)
    R = O.euler_rotation(*W.cli_rotation(yaw=0.6))
    with S.Context(0) as c:
        c.set_keep_tiles(True)
        c.set_direct_samples(direct)
        c.set_triangles_per_block(tpb)
        dev = [dev_mesh(c, m) for m in (small, big, big2)]
        c.set_viewport(320, 180, True)
        c.update(dev[:1])
        c.clear()
        c.draw_mesh(dev[0], R)
        c.read()
        for w, h, image in ((640, 360, True), (640, 360, True), (641, 200, False)):
            c.set_viewport(w, h, image)
            c.update(dev)
            c.clear()
            for d in dev:
                c.draw_mesh(d, R)
            assert_same((*c.read(), None), oracle_render([small, big, big2], R, w, h, image), f"overflow {w}x{h}")


def test_batch_of_a_context_that_keeps_tiles():
    """A batch rendered without tiles, with, and without again as its context's option goes,
    planned and replayed."""
    with S.Context(0) as c:
        meshes, dev, frames = mixed_frames(c)
        b = S.Batch(c, frames[:10])
        for on in (False, True, False, True):
            c.set_keep_tiles(on)
            for rep in range(3):
                b.render()
                check_frames(b, meshes, frames[:10], f"keep tiles {on} render {rep}")
        b.close()
