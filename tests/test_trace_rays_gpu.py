"""Ray queries over arrays of any alignment and length: 16-byte loads and stores
where both arrays allow them, word by word elsewhere, against the oracle."""
import ctypes

import numpy as np
import pytest
import torch

import oracle_py as op
from crisoptix_b200 import Scene, _abi
from helpers import make_params, random_rays, small_sphere_room

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 129, 4097])
@pytest.mark.parametrize("ray_off,hit_off", [(0, 0), (1, 0), (0, 2), (3, 1)])
@pytest.mark.parametrize("builder", [_abi.BVH_DEVICE, _abi.BVH_DEVICE_WIDE4])
def test_alignment_and_length(cuda_device, n, ray_off, hit_off, builder):
    desc, _ = small_sphere_room()
    sc = Scene(desc, builder=builder)
    rays = random_rays(desc, n, seed=51)
    o = op.Oracle.from_scene(desc, 4, 4, make_params(sc.scene_size), triangles=sc.read_triangles())
    buf = torch.zeros(8 * n + 4, device="cuda")
    buf[ray_off:ray_off + 8 * n] = torch.from_numpy(np.ascontiguousarray(rays, np.float32)).cuda().view(-1)
    for any_hit in (False, True):
        hits = torch.full((4 * n + 8,), -7.0, device="cuda")
        sc.trace(buf.data_ptr() + 4 * ray_off, hits.data_ptr() + 4 * hit_off, n, any_hit)
        torch.cuda.synchronize()
        h = hits.cpu().numpy()
        want = o.trace(rays, any_hit=any_hit)
        got = h[hit_off:hit_off + 4 * n].reshape(n, 4)
        assert np.array_equal(got[:, 0].view(np.uint32), want["prim"])
        for k, name in enumerate(("t", "u", "v")):
            assert np.array_equal(got[:, 1 + k].view(np.uint32), want[name].view(np.uint32)), name
        assert (h[:hit_off] == -7.0).all() and (h[hit_off + 4 * n:] == -7.0).all()
