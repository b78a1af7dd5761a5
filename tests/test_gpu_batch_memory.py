"""A batch that goes without tiles holds no fill list (20 bytes a triangle), and one that comes
to need it gets it."""
import numpy as np
import pytest

import sloth_gpu as S
import workloads as W
from oracle import oracle as O
from gpu_helpers import assert_same, oracle_render
from test_gpu_batch import dev_mesh

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_fill_list_only_with_tiles():
    m = W.displaced_icosphere(6, seed=2)            # 81,920 triangles, 24 views of 97x61
    R = O.euler_rotation(*W.cli_rotation(yaw=0.4))
    w, h, n = 97, 61, 24
    U = O.viewport_transform(w, h, O.scene_extent([m["bbox_max"]]))
    ref = oracle_render([m], R, w, h, True, U=U)
    ntri = n * m["rgb"].shape[0]
    with S.Context(0) as c:
        dm = dev_mesh(c, m)
        free0 = torch.cuda.mem_get_info()[0]
        b = S.Batch(c, [{"w": w, "h": h, "image": True, "U": U, "draws": [(dm, R)]} for _ in range(n)])
        for _ in range(2):
            b.render()
        assert_same((*b.read(n - 1), None), ref, "fold")
        held = free0 - torch.cuda.mem_get_info()[0]
        # records, rows, queue and its frames: 108 bytes a triangle; the rest is small
        assert held < 118 * ntri, held / ntri
        c.set_keep_tiles(True)
        for _ in range(3):
            b.render()
            for i in (0, n - 1):
                assert_same((*b.read(i), None), ref, f"tiles {i}")
        c.set_keep_tiles(False)
        b.render()
        assert_same((*b.read(0), None), ref, "fold again")
        b.close()
