"""sloth_ctx_read of small frames through page-locked memory: any subset of the buffers, at
sizes around a 16-byte line and around the largest staged frame, against the oracle."""
import numpy as np
import pytest

import sloth_gpu as S
import workloads as W
from oracle import oracle as O
from gpu_helpers import oracle_render

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,image", [(1, 1, False), (3, 1, True), (5, 1, False), (160, 48, True), (256, 127, True),
                                       (256, 128, False), (257, 128, False), (255, 128, True)])
def test_read_subsets(w, h, image):
    m = W.soup(400, seed=w, n_large=4, sigma=0.1)
    R = O.euler_rotation(*W.cli_rotation(yaw=0.4))
    U = O.viewport_transform(w, h, 0.9)
    ref = oracle_render([m], R, w, h, image, U=U)
    with S.Context(0) as c:
        dm = S.Mesh(c, m["x"], m["y"], m["z"], m["rgb"])
        c.set_viewport(w, h, image)
        c.set_utransform(U)
        c.clear()
        c.draw_mesh(dm, R)
        for want in ((1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (0, 0, 0)):
            got = c.read(*(bool(k) for k in want))
            for a, b, k in zip(got, (ref.cells, ref.z, ref.winner), want):
                assert (a is None) == (not k)
                if k:
                    assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), want
