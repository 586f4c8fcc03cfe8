"""Hits do not depend on the tree: the kernels whose lanes trace closest-hit and
shadow rays side by side render the same bits over a 4-wide tree, whose traversal
takes both kinds in one loop, as over a compressed one."""
import numpy as np
import pytest
import torch

from crisoptix_b200 import Renderer, Scene, _abi, adjoint, default_params, scenes
from helpers import large_config_params, small_sphere_room

pytestmark = pytest.mark.gpu

TREES = [_abi.BVH_DEVICE, _abi.BVH_DEVICE_WIDE4]


# fewer pixels than a warp, persistent warps alone, rounds before them
@pytest.mark.parametrize("w,h", [(5, 3), (61, 47), (520, 380)])
@pytest.mark.parametrize("textured", [False, True])
@pytest.mark.parametrize("kind", [_abi.PATH_TRACER, _abi.RESTIR_PT, _abi.CONDITIONAL_RESTIR])
def test_frames(cuda_device, kind, textured, w, h):
    desc, cam = scenes.textured_cornell_box() if textured else small_sphere_room()
    got = []
    for builder in TREES:
        sc = Scene(desc, builder=builder)
        kw = {}
        if kind == _abi.RESTIR_PT:
            kw = dict(prefix_enable_spatial=1, prefix_spatial_count=2, gather_m=1)
        r = Renderer(w, h, sc, large_config_params(sc.scene_size, renderer_type=kind, gather_radius=0.3, **kw))
        out = torch.zeros(h, w, 3, device="cuda")
        for _ in range(3):
            r.launch_frame(cam, out.data_ptr())
        r.check_device_errors()
        bufs = [r.debug_read(b).tobytes() for b in (_abi.BUF_PREFIX_RES_FRONT, _abi.BUF_SUFFIX_RES_FRONT)]
        got.append((out.cpu().numpy().tobytes(), bufs))
    assert got[0] == got[1]


@pytest.mark.parametrize("res", [3, 43, 130])
def test_path_tracer_adjoint(cuda_device, res):
    desc, cam = small_sphere_room()
    imgs, grads = [], []
    for builder in TREES:
        sc = Scene(desc, builder=builder)
        adj = adjoint.PtAdjoint(sc, res, res, default_params(sc.scene_size, max_path_len=6, seed=5))
        img = adj.render([cam])
        imgs.append(img.cpu().numpy().tobytes())
        grads.append(adj.gradient([cam], torch.ones_like(img))[1].cpu().numpy().astype(np.float64))
    assert imgs[0] == imgs[1] and np.abs(grads[0]).sum() > 0
    # the emitters' terms are non-negative: two orders of a float sum of at most
    # res * res of them are each within res * res * 2^-24 of the exact one
    np.testing.assert_allclose(grads[0], grads[1], rtol=2 * (res * res + 64) * 2.0 ** -24, atol=0)
