"""sloth_ctx_read into any memory the copies reach: pageable, page-locked and device buffers,
mixed, for frames read through the staging memory (up to 32768 cells) and above."""
import ctypes as C
import itertools

import numpy as np
import pytest

import sloth_gpu as S
import workloads as W
from oracle import oracle as O
from gpu_helpers import oracle_render

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("w,h", [(160, 48), (300, 200)])
def test_any_destination(w, h):
    m = W.soup(400, seed=w, n_large=4, sigma=0.1)
    R = O.euler_rotation(*W.cli_rotation(yaw=0.4))
    U = O.viewport_transform(w, h, 0.9)
    ref = oracle_render([m], R, w, h, True, U=U)
    want = [a.view(np.int32) for a in (ref.cells, ref.z, ref.winner)]
    types = (C.c_uint32, C.c_float, C.c_int32)
    with S.Context(0) as c:
        dm = S.Mesh(c, m["x"], m["y"], m["z"], m["rgb"])
        c.set_viewport(w, h, True)
        c.set_utransform(U)
        c.clear()
        c.draw_mesh(dm, R)
        for kinds in itertools.product(("host", "pinned", "device", None), repeat=3):
            bufs = [None if k is None else torch.full((a.size,), 7, dtype=torch.int32, device="cuda" if k == "device" else "cpu",
                                                      pin_memory=k == "pinned") for k, a in zip(kinds, want)]
            torch.cuda.synchronize()
            args = [None if b is None else C.cast(b.data_ptr(), C.POINTER(t)) for b, t in zip(bufs, types)]
            assert c.lib.sloth_ctx_read(c.h, *args) == S.OK, kinds
            for b, a in zip(bufs, want):
                assert b is None or np.array_equal(b.cpu().numpy(), a), kinds
