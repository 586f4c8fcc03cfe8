"""The two ways a path flow runs -- by rounds, as views in a batch do at every
size, and on persistent warps, as a small frame by itself does -- write the same
records: batched frames against single ones, at path lengths with fewer, as
many and more rays than rounds, and with prefixes kept from other lengths."""
import numpy as np
import pytest
import torch

from crisoptix_b200 import Batch, Renderer, Scene, _abi, scenes
from helpers import scene_size_of, small_config_params
from test_parity_gpu import STATE_BUFS, small_sphere_room

pytestmark = pytest.mark.gpu

COND, PT = _abi.CONDITIONAL_RESTIR, _abi.RESTIR_PT


@pytest.mark.parametrize("which,rtype,lengths,storage", [
    ("room", COND, [(1, 1), (1, 2)], 0), ("room", COND, [(2, 8), (2, 8)], 1), ("room", COND, [(5, 8), (1, 12), (3, 9)], 0),
    ("textured", COND, [(2, 6), (1, 6)], 0), ("room", PT, [(1, 1), (1, 9)], 0), ("textured", PT, [(2, 6), (2, 10)], 1)])
def test_rounds_and_persistent_paths_write_the_same(cuda_device, which, rtype, lengths, storage):
    desc, cam = small_sphere_room() if which == "room" else scenes.textured_cornell_box()
    sc = Scene(desc)
    size = scene_size_of(desc)

    def params(prefix_len, max_path_len):
        return small_config_params(size, renderer_type=rtype, prefix_len=prefix_len, max_path_len=max_path_len,
                                   gather_m=4, gather_radius=0.3, storage=storage)

    sizes = [(67, 43), (33, 9)]
    single = [Renderer(w, h, sc, params(*lengths[0])) for w, h in sizes]
    views = [Renderer(w, h, sc, params(*lengths[0])) for w, h in sizes]
    batch = Batch(views)
    a = [torch.zeros(h, w, 3, device="cuda") for w, h in sizes]
    b = [torch.zeros(h, w, 3, device="cuda") for w, h in sizes]
    for lens in lengths:
        for r in single + views:
            r.params = params(*lens)
        for _ in range(2):
            for r, o in zip(single, a):
                r.launch_frame(cam, o.data_ptr())
            batch.render([cam] * 2, [o.data_ptr() for o in b])
            torch.cuda.synchronize()
            for r, v, x, y in zip(single, views, a, b):
                r.check_device_errors()
                v.check_device_errors()
                np.testing.assert_array_equal(x.cpu().numpy().view(np.uint32), y.cpu().numpy().view(np.uint32))
                for buf in STATE_BUFS:
                    assert r.debug_read(buf).tobytes() == v.debug_read(buf).tobytes(), buf
