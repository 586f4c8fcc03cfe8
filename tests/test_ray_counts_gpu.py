"""Ray statistics of the kernels whose lanes trace closest-hit and shadow rays side
by side: a path that connects to a light at its first vertex is one closest-hit ray
and at most one shadow ray, and a frame's rays are the same ones whether its jobs run
in rounds or on persistent warps."""
import pytest
import torch

from crisoptix_b200 import Renderer, Scene, _abi, default_params, scenes
from helpers import large_config_params, small_sphere_room

pytestmark = pytest.mark.gpu


# within one warp, a broken last warp, more pixels than resident lanes
@pytest.mark.parametrize("w,h", [(5, 3), (97, 53), (400, 300)])
@pytest.mark.parametrize("textured", [False, True])
def test_flow(cuda_device, w, h, textured):
    desc, cam = scenes.textured_cornell_box() if textured else scenes.cornell_box()
    sc = Scene(desc)
    r = Renderer(w, h, sc, default_params(sc.scene_size, renderer_type=_abi.RESTIR_PT, max_path_len=4, nee_prob=1.0,
                                          prefix_enable_temporal=0, prefix_enable_spatial=0))
    r.set_timing(2)
    r.launch_frame(cam, torch.zeros(h, w, 3, device="cuda").data_ptr())
    torch.cuda.synchronize()
    st = r.stats()
    assert st["closest_rays"] == w * h and 0 < st["shadow_rays"] <= w * h
    assert st["shift_closest_rays"] == 0 and st["shift_shadow_rays"] == 0 and st["shift_jobs"] == 0


# persistent warps alone, and rounds before them
@pytest.mark.parametrize("w,h", [(61, 47), (520, 380)])
def test_shift_jobs(cuda_device, w, h):
    desc, cam = small_sphere_room()
    sc = Scene(desc)
    counts = []
    for cap in (0, 1, 64):
        r = Renderer(w, h, sc, large_config_params(sc.scene_size, gather_radius=0.3))
        r.set_job_capacity(cap)
        r.set_timing(2)
        out = torch.zeros(h, w, 3, device="cuda")
        for _ in range(3):
            r.launch_frame(cam, out.data_ptr())
            torch.cuda.synchronize()
        st = r.stats()
        counts.append([st[k] for k in ("closest_rays", "shadow_rays", "shift_closest_rays", "shift_shadow_rays",
                                       "shift_jobs")])
    assert counts[0] == counts[1] == counts[2]
    assert counts[0][2] > 0 and counts[0][3] > 0 and counts[0][4] >= counts[0][3]
