"""Draws without tiles (rust-sloth_gb300/csrc/fold.cuh): frames bit for bit against the
oracle at the sizes where the fold can go wrong -- one triangle to one over a block's 32,
triangles of one sample to ones the whole GPU walks, frames narrower than a tile, odd
widths, wrapped samples and hostile coordinates."""
import ctypes as C

import numpy as np
import pytest

import sloth_gpu as S
import workloads as W
from oracle import oracle as O
from gpu_helpers import oracle_render
from test_gpu_parity import hostile_soup, span_soup

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def noalloc(m, M, w, h, image):
    n = int(m["rgb"].shape[0])
    ins = [torch.from_numpy(np.ascontiguousarray(m[k]).reshape(-1)).cuda() for k in ("x", "y", "z", "rgb")]
    nz = w * h
    cells = torch.full((nz + (h if image else 0),), -1, dtype=torch.int32, device="cuda")
    z = torch.full((nz,), 7, dtype=torch.int32, device="cuda")
    win = torch.full((nz,), 7, dtype=torch.int32, device="cuda")
    mm = np.ascontiguousarray(M.reshape(16), np.float32)
    st = S.load_library().sloth_render_noalloc(*(t.data_ptr() for t in ins[:3]), n, ins[3].data_ptr(),
                                               mm.ctypes.data_as(C.POINTER(C.c_float)), w, h, int(image),
                                               cells.data_ptr(), z.data_ptr(), win.data_ptr(),
                                               C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == S.OK
    torch.cuda.synchronize()
    return cells.cpu().numpy().view(np.uint32), z.cpu().numpy(), win.cpu().numpy()


def check(got, ref, label):
    for a, b, name in zip(got, (ref.cells, ref.z.view(np.int32), ref.winner), ("cells", "z", "winner")):
        assert np.array_equal(a, b), f"{label}: {name} differ at {np.nonzero(a != b)[0][:5]}"


@pytest.mark.parametrize("w,h,image", [(1, 1, True), (7, 33, False), (161, 95, True), (640, 360, True), (2, 4096, True)])
@pytest.mark.parametrize("n,large,sigma", [(1, 0, 0.3), (31, 1, 0.01), (33, 0, 0.002), (700, 40, 0.2)])
def test_noalloc_sizes(w, h, image, n, large, sigma):
    m = W.soup(n, seed=n + w, n_large=large, sigma=sigma)
    R = O.euler_rotation(*W.cli_rotation(yaw=0.7, pitch=0.4))
    U = O.viewport_transform(w, h, 0.7)     # an extent below the soup's: wrapped samples
    check(noalloc(m, O.mat4_mul(U, R), w, h, image), oracle_render([m], R, w, h, image, U=U), f"{n}+{large} {w}x{h}")


@pytest.mark.parametrize("seed,w,h,image", [(0, 403, 150, True), (1, 512, 128, False)])
def test_noalloc_hostile(seed, w, h, image):
    eye = np.eye(4, dtype=np.float32)
    m = span_soup(seed, w, h)
    check(noalloc(m, eye, w, h, image), oracle_render([m], eye, w, h, image, U=eye), f"spans {seed} {w}x{h}")
    m = hostile_soup(seed)
    R = O.euler_rotation(*W.cli_rotation(yaw=0.4 + seed))
    U = O.viewport_transform(w, h, O.scene_extent([m["bbox_max"]]))
    check(noalloc(m, O.mat4_mul(U, R), w, h, image), oracle_render([m], R, w, h, image, U=U), f"hostile {seed}")
