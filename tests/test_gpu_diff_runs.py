"""The backward pass's runs (rust-sloth_gb300/csrc/diff.cu): gradients against the f64
adjoint where runs are longest (a coarse mesh: rows of many samples of one triangle, runs
cut at the warp's end) and shortest (triangles below a sample), at even and odd widths, and a
gradient that is not finite, which reaches only its own triangle's vertices."""
import numpy as np
import pytest

import sloth_gpu as S
import workloads as W
from oracle import diff_shade as D
from test_gpu_diff import LIGHT, env, host_pos, oracle_views, rel, views_of               # noqa: F401

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
import diff_render as DR  # noqa: E402


def setup(env, m, specs, store):
    ctx, stream = env
    views = views_of(m, specs)
    sv = DR.ShadedViews(ctx, m, views, stream, store_visibility=store)
    rng = np.random.default_rng(3)
    vrgb = rng.uniform(0.1, 0.9, (m["x"].size, 3)).astype(np.float32)
    grad = rng.normal(size=(sv.ncells, 3)).astype(np.float32)
    return sv, views, vrgb, grad


def backward(env, sv, m, vrgb, grad):
    with torch.cuda.stream(env[1]):
        dev = torch.device("cuda", 0)
        v, L = torch.from_numpy(vrgb).to(dev), torch.tensor(LIGHT, dtype=torch.float32, device=dev)
        sv.render(torch.from_numpy(host_pos(m)).to(dev))
        sv.shade(v, L)
        out = sv.shade_backward(v, L, torch.from_numpy(grad).to(dev))
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in out]


# Tolerances (2-norm): a screen coordinate near 100 carries an f32 error of 4e-6, so an edge
# function of a triangle of size s has a relative error of about 4e-6/s: s is tens of samples
# for the coarse mesh (well below the 1e-4 of the other gradient tests).  For the fine one it
# is 0.6, and a hundredth of that for triangles edge-on at the silhouette: 1e-3 for what
# divides by the area once (colours), 1e-2 for what divides twice (positions).
@pytest.mark.parametrize("store", [True, False])
@pytest.mark.parametrize("subdiv,specs,tol", [
    (0, [(256, 128, False, 0.4), (255, 127, True, 1.1)], (1e-4, 1e-4, 1e-4)),
    (4, [(34, 17, False, 0.4), (33, 18, True, 2.0), (65, 9, False, 0.1)], (1e-2, 1e-3, 1e-3))])
def test_runs_against_the_f64_adjoint(env, subdiv, specs, tol, store):
    m = W.displaced_icosphere(subdiv, seed=3, amplitude=0.0)
    sv, views, vrgb, grad = setup(env, m, specs, store)
    got = backward(env, sv, m, vrgb, grad)
    want = [0.0, 0.0, 0.0]
    for (a, n), ov in zip(sv.cells, oracle_views(m, views)):
        part = D.shade_vjp(host_pos(m).astype(np.float64), vrgb.astype(np.float64), np.array(LIGHT), m["idx"], ov,
                           grad[a:a + n].astype(np.float64))
        want = [w_ + p for w_, p in zip(want, part)]
    for g, w_, t, name in zip(got, want, tol, ("pos", "vrgb", "light")):
        assert rel(g, np.asarray(w_)) < t, name
    sv.close()


@pytest.mark.parametrize("w,h", [(160, 80), (161, 79)])
def test_non_finite_gradient_stays_with_its_triangle(env, w, h):
    m = W.displaced_icosphere(2, seed=3, amplitude=0.0)
    sv, views, vrgb, grad = setup(env, m, [(w, h, False, 0.7)], True)
    win = oracle_views(m, views)[0].winner
    cell = int(np.nonzero(win >= 0)[0][200])
    clean = grad.copy()
    clean[cell] = 0.0
    grad[cell] = [np.inf, 1.0, np.nan]
    got, ref = backward(env, sv, m, vrgb, grad), backward(env, sv, m, vrgb, clean)
    mine = np.zeros(m["x"].size, bool)
    mine[np.asarray(m["idx"]).reshape(-1, 3)[win[cell]]] = True
    for g, r in zip(got[:2], ref[:2]):
        assert np.isfinite(g[~mine]).all() and rel(g[~mine], r[~mine]) < 1e-4
        assert not np.isfinite(g[mine]).all()
    sv.close()
