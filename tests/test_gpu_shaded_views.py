"""What a program may do with ShadedViews beyond a fit: keep one gradient and let the others
go, detach it in place, and subclass render and shade."""
import numpy as np
import pytest

import sloth_gpu as S
import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
import diff_render as DR  # noqa: E402


def views(cls):
    m = W.displaced_icosphere(2, seed=1)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = S.Context(0, stream=stream.cuda_stream)
        U = S.viewport_transform(80, 40, S.scene_extent([m["bbox_max"]]))
        sv = cls(ctx, m, [{"w": 80, "h": 40, "image": False, "U": U, "R": np.eye(4, dtype=np.float32)}], stream)
        p = torch.from_numpy(np.stack([m["x"], m["y"], m["z"]], 1)).cuda()
        v = torch.rand(p.shape[0], 3, device="cuda")
        light = torch.tensor([0.1, 0.2, 0.9], device="cuda")
    return ctx, sv, stream, [t.requires_grad_(True) for t in (p, v, light)]


def test_each_gradient_stands_by_itself():
    ctx, sv, stream, leaves = views(DR.ShadedViews)
    with torch.cuda.stream(stream):
        DR.shade_views(*leaves, sv).sum().backward()
        grads = [t.grad for t in leaves]
        assert all((g != 0).any() for g in grads)
        assert len({g.untyped_storage().data_ptr() for g in grads}) == 3
        for t, g in zip(leaves, grads):
            assert g.untyped_storage().nbytes() == 4 * t.numel() and g.shape == t.shape
            g.detach_()
            before = [o._version for o in grads if o is not g]
            g.zero_()
            assert [o._version for o in grads if o is not g] == before
        torch.cuda.synchronize()
    sv.close()
    ctx.close()


def test_a_subclass_sees_every_call():
    calls = []

    class Logged(DR.ShadedViews):
        def render(self, pos):
            calls.append("render")
            super().render(pos)

        def shade(self, vrgb, light):
            calls.append("shade")
            return super().shade(vrgb, light) * 2.0

        def shade_backward(self, vrgb, light, grad_rgb):
            calls.append("shade_backward")
            return super().shade_backward(vrgb, light, grad_rgb)

    ctx, sv, stream, leaves = views(Logged)
    with torch.cuda.stream(stream):
        rgb = DR.shade_views(*leaves, sv)
        plain = DR.ShadedViews.shade(sv, leaves[1].detach(), leaves[2].detach())
        assert torch.equal(rgb, 2.0 * plain) and (plain > 0).any()
        rgb.sum().backward()
        assert calls == ["render", "shade", "shade_backward"]
        torch.cuda.synchronize()
    sv.close()
    ctx.close()


@pytest.mark.parametrize("subdiv", [0, 2, 4])
def test_gradients_into_used_buffers(subdiv):
    """sloth_batch_shade_gradients into buffers of any content against sloth_batch_shade_backward
    into zeros, each buffer alone and together; what lies behind a buffer stays as it is."""
    m = W.displaced_icosphere(subdiv, seed=1)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = S.Context(0, stream=stream.cuda_stream)
        U = S.viewport_transform(81, 40, S.scene_extent([m["bbox_max"]]))
        sv = DR.ShadedViews(ctx, m, [{"w": 81, "h": 40, "image": False, "U": U, "R": np.eye(4, dtype=np.float32)}], stream)
        p = torch.from_numpy(np.stack([m["x"], m["y"], m["z"]], 1)).cuda()
        v, light = torch.rand(p.shape[0], 3, device="cuda"), torch.tensor([0.1, 0.2, 0.9], device="cuda")
        g = torch.rand(sv.ncells, 3, device="cuda")
        sv.render(p)
        sv.shade(v, light)
        ins = (v.data_ptr(), light.data_ptr(), g.data_ptr())
        sizes = (3 * p.shape[0], 3 * p.shape[0], 3)
        want = [torch.zeros(n, device="cuda") for n in sizes]
        sv.batch.shade_backward(*ins, *(t.data_ptr() for t in want))
        for mask in ((1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1)):
            got = [torch.full((n + 2,), 7.0, device="cuda") for n in sizes]
            sv.batch.shade_gradients(*ins, *(t.data_ptr() if k else 0 for t, k in zip(got, mask)))
            for t, w_, k in zip(got, want, mask):
                assert (t[-2:] == 7.0).all() and (k or (t == 7.0).all())
                # the same sums in another order of the atomics
                assert not k or (t[:-2] - w_).norm() <= 1e-5 * w_.norm()
                assert not k or ((t[:-2] == 0) == (w_ == 0)).all()
        torch.cuda.synchronize()
        sv.close()
        ctx.close()
