"""Paths on persistent warps (the path tracer's frames and the path tracer's
adjoint): images with fewer pixels than lanes, with a ragged last batch and with
several pixels a lane, against the oracle and against each other."""
import numpy as np
import pytest
import torch

from crisoptix_b200 import Scene, _abi, adjoint, default_params, scenes
from helpers import make_params, scene_size_of
from test_parity_gpu import run_parity, small_sphere_room, static

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (5, 3), (31, 1), (33, 31), (641, 479)]


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("textured", [False, True])
def test_path_tracer_frames(cuda_device, w, h, textured):
    desc, cam = scenes.textured_cornell_box() if textured else small_sphere_room()
    p = make_params(scene_size_of(desc), renderer_type=_abi.PATH_TRACER, max_path_len=6)
    run_parity(desc, cam, p, w, h, 2, static)


@pytest.mark.parametrize("w,h", SIZES)
def test_frozen_path_tracer_is_the_path_tracer(cuda_device, w, h):
    """At its frozen parameters the adjoint's estimator is the path tracer's
    first frame up to the rounding of a light connection's factors."""
    from crisoptix_b200 import Renderer

    desc, cam = small_sphere_room()
    sc = Scene(desc)
    p = default_params(sc.scene_size, renderer_type=_abi.PATH_TRACER, max_path_len=6, seed=5)
    out = torch.zeros(h, w, 3, device="cuda")
    Renderer(w, h, sc, p).launch_frame(cam, out.data_ptr())
    adj = adjoint.PtAdjoint(sc, w, h, p)
    img = adj.render([cam])[0]
    np.testing.assert_allclose(img.cpu().numpy(), out.cpu().numpy(), rtol=1e-4, atol=1e-5)
    # every pixel's gradient is added once: d(sum of the image) / d(emitter colours) is linear in dl
    ones = torch.ones(1, h, w, 3, device="cuda")
    g1, e1 = adj.gradient([cam], ones)
    g2, e2 = adj.gradient([cam], 2.0 * ones)
    np.testing.assert_allclose(2.0 * e1.cpu().numpy(), e2.cpu().numpy(), rtol=1e-4, atol=1e-6)
    np.testing.assert_allclose(2.0 * g1.cpu().numpy(), g2.cpu().numpy(), rtol=1e-3, atol=1e-4)


@pytest.mark.parametrize("nee", [0.0, 1.0])
def test_ray_counts_by_kind(cuda_device, nee):
    """Lanes that trace a closest-hit and a shadow ray side by side count each as
    what it is: with NEE at every vertex a path is one closest-hit ray and at most
    one shadow ray, without NEE it traces no shadow ray."""
    from crisoptix_b200 import Renderer

    desc, cam = scenes.cornell_box()
    sc = Scene(desc)
    w, h = 97, 53
    r = Renderer(w, h, sc, default_params(sc.scene_size, renderer_type=_abi.PATH_TRACER, max_path_len=4, nee_prob=nee))
    r.set_timing(2)
    r.launch_frame(cam, torch.zeros(h, w, 3, device="cuda").data_ptr())
    torch.cuda.synchronize()
    st = r.stats()
    if nee == 1.0:
        assert st["closest_rays"] == w * h and 0 < st["shadow_rays"] <= w * h
    else:
        assert st["closest_rays"] > w * h and st["shadow_rays"] == 0
