"""sloth_mesh_update_interleaved against sloth_mesh_update: the same frame from the same
positions and colours, at vertex and triangle counts around a block and with colours that
start at every byte of a word; and ShadedViews fed from the host, transposed and sliced."""
import numpy as np
import pytest

import sloth_gpu as S
import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,shift", [(1, 0), (85, 1), (86, 2), (700, 3), (700, 0)])
def test_same_frame_as_separate_arrays(n, shift):
    m, other = W.soup(n, seed=n, sigma=0.2), W.soup(n, seed=n + 1, sigma=0.2)
    with S.Context(0) as c:
        a, b = (S.Mesh(c, m["x"], m["y"], m["z"], m["rgb"]) for _ in range(2))
        xyz = torch.from_numpy(np.stack([other["x"], other["y"], other["z"]], 1)).cuda()
        rgb = torch.zeros(3 * n + shift, dtype=torch.uint8, device="cuda")
        rgb[shift:] = torch.from_numpy(other["rgb"].reshape(-1)).cuda()
        torch.cuda.synchronize()
        a.update(other["x"], other["y"], other["z"], np.ascontiguousarray(other["rgb"].reshape(-1)))
        b.update_interleaved(xyz.data_ptr(), rgb.data_ptr() + shift)
        out = []
        for dm in (a, b):
            c.set_viewport(120, 61, True)
            c.set_utransform(S.viewport_transform(120, 61, 1.0))
            c.clear()
            c.draw_mesh(dm, np.eye(4, dtype=np.float32))
            out.append(c.read())
        assert (out[0][2] >= 0).any() or n < 10
        for p, q in zip(*out):
            assert np.array_equal(p.view(np.uint32), q.view(np.uint32))


def test_shaded_views_take_positions_in_any_form():
    import diff_render as DR
    m = W.displaced_icosphere(2, seed=1)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = S.Context(0, stream=stream.cuda_stream)
        U = S.viewport_transform(80, 40, S.scene_extent([m["bbox_max"]]))
        sv = DR.ShadedViews(ctx, m, [{"w": 80, "h": 40, "image": False, "U": U, "R": np.eye(4, dtype=np.float32)}], stream)
        p = torch.from_numpy(np.stack([m["x"], m["y"], m["z"]], 1)).cuda()
        v = torch.rand(p.shape[0], 3, device="cuda")
        light = torch.tensor([0.0, 0.0, 1.0], device="cuda")
        want = DR.shade_views(p, v, light, sv).clone()
        assert (want > 0).any()
        wide = torch.cat([p, torch.full_like(p, 9.0)], 1)
        for q in (p.cpu(), p.double(), p.t().contiguous().t(), wide[:, :3], wide, torch.cat([p, p])):
            assert torch.equal(DR.shade_views(q, v, light, sv), want)
        torch.cuda.synchronize()
        sv.close()
        ctx.close()
