"""The flush formatter at the edges of its chunks (1024 cells), words and 16-byte lines:
frames of one cell to one past two chunks, whose text starts at every place in a line, in
every format and both modes, against the oracle's emitter; the size asked for alone; and
colours of one, two and three digits in one run."""
import numpy as np
import pytest

import sloth_gpu as S
from oracle import oracle as O
from gpu_helpers import oracle_render

pytestmark = pytest.mark.gpu


def colours(w, h, seed):
    """One triangle a cell pair over the frame, in random colours of every digit count."""
    rng = np.random.default_rng(seed)
    n = 4 * (w // 2 + 1) + 8
    x0, y0 = rng.uniform(0, max(w / 2, 1), n), rng.uniform(0, h, n)
    v = np.stack([np.stack([x0, y0], 1), np.stack([x0, y0 + h], 1), np.stack([x0 + 3, y0], 1)], 1)
    z = rng.uniform(-1, 1, (n, 3, 1))
    p = np.concatenate([v, z], 2).astype(np.float32).reshape(-1, 3)
    rgb = rng.choice([0, 5, 9, 10, 42, 99, 100, 200, 255], (n, 3)).astype(np.uint8)
    return {"x": p[:, 0].copy(), "y": p[:, 1].copy(), "z": p[:, 2].copy(), "idx": None, "rgb": rgb,
            "bbox_max": np.ones(3, np.float32)}


@pytest.mark.parametrize("w,h", [(1, 1), (3, 1), (15, 1), (31, 33), (32, 32), (1023, 1), (1025, 1), (683, 3), (160, 48)])
@pytest.mark.parametrize("image", [True, False])
def test_flush_edges(w, h, image):
    m, eye = colours(w, h, w + h), np.eye(4, dtype=np.float32)
    ref = oracle_render([m], eye, w, h, image, U=eye)
    with S.Context(0) as c:
        dm = S.Mesh(c, m["x"], m["y"], m["z"], m["rgb"])
        c.set_viewport(w, h, image)
        c.set_utransform(eye)
        c.clear()
        c.draw_mesh(dm, eye)
        for f in (O.FLUSH_PLAIN, O.FLUSH_ANSI, O.FLUSH_HTML):
            want = O.flush(ref.cells, image, f)
            assert c.flush(f) == want, f"format {f}"
            n = S.C.c_uint64()
            assert c.lib.sloth_ctx_flush(c.h, f, None, 0, S.C.byref(n)) == S.OK and n.value == len(want)
