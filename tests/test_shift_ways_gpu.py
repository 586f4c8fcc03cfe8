"""Shift jobs by rounds and then on persistent warps (as a batch's views run them at
every size) and on persistent warps alone (a small frame by itself), with records
for none, some and all of the list's jobs: the same frames and records."""
import numpy as np
import pytest
import torch

from crisoptix_b200 import Batch, Renderer, Scene, _abi, scenes
from helpers import large_config_params, scene_size_of
from test_parity_gpu import STATE_BUFS, small_sphere_room

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which,capacity,kw", [
    ("room", 0, {}), ("room", 1, {}), ("room", 16, dict(prefix_len=4, max_path_len=10)),
    ("textured", 1, dict(gather_n=2)),
    ("room", 1, dict(renderer_type=_abi.RESTIR_PT, prefix_enable_spatial=1, prefix_spatial_count=3))])
def test_shift_jobs_by_rounds_and_persistent(cuda_device, which, capacity, kw):
    desc, cam = small_sphere_room() if which == "room" else scenes.textured_cornell_box()
    sc = Scene(desc)
    p = large_config_params(scene_size_of(desc), gather_radius=0.3, **kw)
    w, h = 61, 37
    single, views = Renderer(w, h, sc, p), [Renderer(w, h, sc, p) for _ in range(2)]
    for v in views:
        v.set_job_capacity(capacity)
    batch = Batch(views)
    a, b = torch.zeros(h, w, 3, device="cuda"), [torch.zeros(h, w, 3, device="cuda") for _ in views]
    for _ in range(4):
        single.launch_frame(cam, a.data_ptr())
        batch.render([cam] * 2, [o.data_ptr() for o in b])
        torch.cuda.synchronize()
        for v, y in zip(views, b):
            v.check_device_errors()
            np.testing.assert_array_equal(a.cpu().numpy().view(np.uint32), y.cpu().numpy().view(np.uint32))
            for buf in STATE_BUFS:
                assert single.debug_read(buf).tobytes() == v.debug_read(buf).tobytes(), buf
