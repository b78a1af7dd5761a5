"""A mesh that updates have made larger or smaller than it was made: the frames are exact, and
draws and batches go by the size it has, not the size it had (the sum of its edges comes back
from the device), so that one made tiny does not go without tiles for good."""
import numpy as np
import pytest

import sloth_gpu as S
import workloads as W
from oracle import oracle as O
from gpu_helpers import assert_same, oracle_render
from test_gpu_batch import dev_mesh

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def scaled(m, k):
    out = dict(m)
    for a in "xyz":
        out[a] = (m[a] * np.float32(k)).astype(np.float32)
    return out


def edges2(m):
    """Sum over the triangles of their longest edge squared."""
    v = np.stack([m["x"], m["y"], m["z"]], 1).astype(np.float64)
    t = v[m["idx"].reshape(-1, 3)] if m.get("idx") is not None else v.reshape(-1, 3, 3)
    return max(1e-30, ((t - np.roll(t, 1, axis=1)) ** 2).sum(2).max(1).sum())


class Updater:
    """Updates a mesh from host arrays, device arrays or device triples, and keeps them alive."""

    def __init__(self, dm, how):
        self.dm, self.how, self.keep = dm, how, []

    def __call__(self, m):
        rgb = np.ascontiguousarray(m["rgb"].reshape(-1))
        if self.how == "host":
            self.keep.append((m["x"], m["y"], m["z"], rgb))
            self.dm.update(*self.keep[-1])
            return
        t = torch.from_numpy(np.stack([m["x"], m["y"], m["z"]], 1 if self.how == "triples" else 0)).cuda()
        c = torch.from_numpy(rgb).cuda()
        torch.cuda.synchronize()
        self.keep.append((t, c))
        if self.how == "triples":
            self.dm.update_interleaved(t.data_ptr(), c.data_ptr())
        else:
            self.dm.update_device(*(t[k].data_ptr() for k in range(3)), c.data_ptr())


# 4 triangles, one over what the sum takes one by one, many more with every third, and indexed
MESHES = {"few": lambda: W.soup(3, seed=2, n_large=1, sigma=1.0), "step2": lambda: W.soup(4097, seed=2, n_large=0, sigma=0.5),
          "step3": lambda: W.soup(12000, seed=3, n_large=0, sigma=0.5), "indexed": lambda: W.displaced_icosphere(4, seed=5)}


@pytest.mark.parametrize("how", ["host", "device", "triples"])
@pytest.mark.parametrize("kind", sorted(MESHES))
def test_context_follows_the_size(kind, how):
    w, h = 640, 400
    full = MESHES[kind]()
    R = O.euler_rotation(*W.cli_rotation(yaw=0.5))
    U = O.viewport_transform(w, h, 1.0)
    # the viewport's scale is 160; an estimate of 1e9 samples is past the line at any depth
    sizes = {"small": scaled(full, 0.01), "full": scaled(full, (1e9 / edges2(full)) ** 0.5 / 160.0)}
    with S.Context(0) as c:
        dm = dev_mesh(c, sizes["small"])
        up = Updater(dm, how)
        c.set_timing(True)
        c.set_viewport(w, h, True)
        c.set_utransform(U)

        def draw(m, label):
            f, r = c.kernel_time("fold")[1], c.kernel_time("raster")[1]
            c.clear()
            c.draw_mesh(dm, R)
            assert_same((*c.read(), None), oracle_render([m], R, w, h, True, U=U), label)
            f, r = c.kernel_time("fold")[1] - f, c.kernel_time("raster")[1] - r
            assert f + r == 1
            return bool(f)

        assert draw(sizes["small"], "as made")
        for size in ("full", "small", "full"):
            up(sizes[size])
            c.synchronize()
            want = size == "small" or kind == "few"     # four triangles never pass the line
            assert draw(sizes[size], size) == want, size
        up(sizes["small"])
        draw(sizes["small"], "queued right behind the update")


@pytest.mark.parametrize("how", ["host", "triples"])
def test_batch_follows_the_size(how):
    """The tiles of a batch need an entry buffer, allocated by the first render that takes them."""
    small, full = scaled(W.soup(20000, seed=3, n_large=0, sigma=0.5), 0.01), scaled(W.soup(20000, seed=3, n_large=0, sigma=0.5), 3.0)
    R = O.euler_rotation(*W.cli_rotation(yaw=0.5))
    with S.Context(0) as c:
        dm = dev_mesh(c, small)
        up = Updater(dm, how)
        frames = [{"w": w, "h": h, "image": im, "U": O.viewport_transform(w, h, 1.0), "draws": [(dm, R)]}
                  for w, h, im in ((640, 360, True), (321, 181, False))]
        b = S.Batch(c, frames)

        def check(m, label):
            for i, f in enumerate(frames):
                assert_same((*b.read(i), None), oracle_render([m], R, f["w"], f["h"], f["image"], U=f["U"]), f"{label} {i}")

        for _ in range(2):
            b.render()
        check(small, "as made")
        free = torch.cuda.mem_get_info()[0]
        up(full)
        b.render()
        check(full, "queued right behind the update")
        for rep in range(3):
            b.render()
            check(full, f"full {rep}")
        assert torch.cuda.mem_get_info()[0] < free - 4 * 20000, "the batch still goes without tiles"
        up(small)
        for rep in range(3):
            b.render()
            check(small, f"small again {rep}")
        b.close()
