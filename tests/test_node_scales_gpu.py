"""Compressed-node tests at the limits of their grid arithmetic: coordinates
just below the format's limit (the largest grid steps times the largest
inverse direction components) and small ones, with axis-parallel rays (zero
direction components) and rays along a box's faces, against testing every
triangle."""
import numpy as np
import pytest

import oracle_py as op
from crisoptix_b200 import Scene, _abi
from helpers import first_mismatch, make_params
from test_bvh_geometry_gpu import aimed_rays, gpu_trace, random_soup, soup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("largest", [0.5, 20.0, 1.5e7])
def test_axis_parallel_and_aimed_rays_at_scale(cuda_device, largest):
    P = random_soup()[:2000]
    P = (P / np.abs(P).max() * largest).astype(np.float32)
    desc = soup(P, f"scale_{largest:g}")
    sc = Scene(desc)
    assert sc.bvh_info()["format"] == _abi.BVH_FORMAT_COMPRESSED8
    n = 1 << 13
    rays = aimed_rays(desc, n, seed=41)
    # axis-parallel rays through vertices (box corners) and through random points
    axis = np.random.default_rng(42).integers(0, 3, n)
    side = np.random.default_rng(43).choice([-1.0, 1.0], n)
    flat = rays.copy()
    flat[:, 4:7] = 0.0
    flat[np.arange(n), 4 + axis] = side
    flat[: n // 2, :3] = P.reshape(-1, 3)[np.random.default_rng(44).integers(0, 3 * len(P), n // 2)]
    flat[: n // 2, :3][np.arange(n // 2), axis[: n // 2]] -= (side[: n // 2] * largest).astype(np.float32)
    o = op.Oracle.from_scene(desc, 4, 4, make_params(sc.scene_size), triangles=sc.read_triangles())
    hits = 0
    for r in (rays, flat):
        for any_hit in (False, True):
            g = gpu_trace(sc, r, any_hit)
            assert first_mismatch(g, o.trace(r, any_hit=any_hit, brute=True)) is None
            hits += int((g["prim"] != _abi.INVALID_PRIM).sum())
    assert hits > 0
