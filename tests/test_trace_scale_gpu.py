"""A ray's direction may have any length: scaled by a power of two, a ray hits the
same triangle at the same weights, at t over that power, to the bit."""
import numpy as np
import pytest
import torch

from crisoptix_b200 import Scene, _abi
from helpers import random_rays, small_sphere_room

pytestmark = pytest.mark.gpu


def trace(sc, rays, any_hit):
    r = torch.from_numpy(rays).cuda()
    hits = torch.zeros(len(rays), 4, device="cuda")
    sc.trace(r.data_ptr(), hits.data_ptr(), len(rays), any_hit)
    return hits.cpu().numpy()


@pytest.mark.parametrize("builder", [_abi.BVH_DEVICE, _abi.BVH_DEVICE_WIDE4])
# directions of 2^-100 .. 2^100: below 2^-94 the inverse of a component reaches the
# limits of the box tests, and at 2^40 the kernel begins to rescale
@pytest.mark.parametrize("k", [-100, -99, -97, -96, -95, -94, -90, -60, -41, -40, -39, 39, 41, 60, 100])
def test_scaled_directions(cuda_device, k, builder):
    desc, _ = small_sphere_room()
    sc = Scene(desc, builder=builder)
    rays = np.ascontiguousarray(random_rays(desc, 3000, seed=7), np.float32)
    d = rays[:, 4:7]
    d[np.abs(d) < 2.0 ** -20] = 0.0  # stays exact when scaled
    d[:300] = np.eye(3, dtype=np.float32)[np.arange(300) % 3] * np.where(np.arange(300) % 2, 1, -1)[:, None]
    rays[:, 3] = 2.0 ** -10
    rays[:, 7] = np.random.default_rng(1).uniform(0.5, 20.0, len(rays))
    scaled = rays.copy()
    scaled[:, 4:7] *= np.float32(2.0 ** k)
    scaled[:, 3] *= np.float32(2.0 ** -k)
    scaled[:, 7] *= np.float32(2.0 ** -k)
    a, b = trace(sc, rays, False), trace(sc, scaled, False)
    prim = a[:, 0].view(np.uint32)
    assert (prim != 0xFFFFFFFF).sum() > 1000 and (prim == 0xFFFFFFFF).sum() > 100
    a[:, 1] *= np.float32(2.0 ** -k)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert np.array_equal(trace(sc, rays, True).view(np.uint32), trace(sc, scaled, True).view(np.uint32))
