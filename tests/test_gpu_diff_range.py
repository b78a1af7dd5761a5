"""Gradients near the largest float: what each sample adds to the colours is finite, and so is
their sum, although the plain sum of the run's image gradients is not."""
import numpy as np
import pytest

import workloads as W
from oracle import diff_shade as D
from test_gpu_diff import LIGHT, env, host_pos, oracle_views                             # noqa: F401
from test_gpu_diff_runs import backward, setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("store", [True, False])
@pytest.mark.parametrize("w,h", [(256, 128), (255, 127)])
def test_large_finite_gradients(env, w, h, store):
    m = W.displaced_icosphere(1, seed=3, amplitude=0.0)
    sv, views, vrgb, grad = setup(env, m, [(w, h, False, 0.7)], store)
    ov = oracle_views(m, views)[0]
    win = ov.winner.reshape(h, w)
    # three samples in a row of one triangle: cells x, x+2, x+4 of a row, unwrapped
    rows, cols = np.nonzero((win[:, :-4] >= 0) & (win[:, :-4] == win[:, 2:-2]) & (win[:, :-4] == win[:, 4:])
                            & (np.arange(w - 4)[None, :] % 2 == 0))
    big = np.float32(1.5e38)
    checked = 0
    for k in range(0, rows.size, max(1, rows.size // 40)):
        g = np.zeros_like(grad)
        at = rows[k] * w + cols[k]
        g[[at, at + 2, at + 4], 0] = big
        want = D.shade_vjp(host_pos(m).astype(np.float64), vrgb.astype(np.float64), np.array(LIGHT), m["idx"], ov,
                           g.astype(np.float64))[1]
        if not 1e37 < np.abs(want).max() < 2e38:    # unlit, or past the largest float itself
            continue
        got = backward(env, sv, m, vrgb, g)[1]
        assert np.isfinite(got).all()
        # three terms of f32 barycentrics of triangles tens of samples wide (4e-6 of a
        # coordinate near 100 each), against the largest
        assert np.abs(got - want).max() < 1e-4 * np.abs(want).max()
        checked += 1
    assert checked > 0
    sv.close()
