"""A large draw's newline rows go into the frame's tree on a stream of their own; whatever
empties that tree for the next frame waits for them, also where nothing is drawn into it."""
import numpy as np
import pytest

import sloth_gpu as S
import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", ["read", "synchronize", "fragments", "read_async", "device_buffers"])
def test_blank_frame_after_a_large_draw(first):
    m = W.soup(140000, seed=3, n_large=20)      # above 2^17: the newline rows on their own stream
    R = O.euler_rotation(*W.cli_rotation(yaw=0.4))
    w, h = 320, 200
    with S.Context(0) as c:
        c.set_depth_cull(False)                 # the tile raster, whatever the estimate
        dm = S.Mesh(c, m["x"], m["y"], m["z"], m["rgb"], None, m["bbox_max"])
        c.set_viewport(w, h, True)
        c.update([dm])
        blank = np.full(w * h + h, ord(" "), np.uint32)
        for rep in range(4):
            c.clear()
            c.draw_mesh(dm, R)
            c.clear()
            if first == "read_async":
                cells = np.zeros(w * h + h, np.uint32)
                c.read_into_async(cells, None)
                c.synchronize()
                assert np.array_equal(cells, blank), rep
            elif first != "read":
                getattr(c, first)()
            cells, z, winner = c.read()
            assert np.array_equal(cells, blank) and (winner == -1).all(), rep
        dm.close()
