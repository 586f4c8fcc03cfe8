"""Every pixel's gradient is added exactly once.  A pixel's value is homogeneous of
degree one in the emitters' colours and the materials' emissions together, so over any
image the colours and emissions times their gradients add up to the image times its
adjoint.  The adjoint here is one over the image where it is lit, so that every lit
channel adds the same to that sum, and a few pixels add a hundred thousand times more:
leaving one of them out or adding it twice moves the sum by far more than the rounding
of its float terms may."""
import numpy as np
import pytest
import torch

from crisoptix_b200 import Scene, _abi, adjoint, default_params
from helpers import large_config_params, scene_size_of, small_sphere_room

pytestmark = pytest.mark.gpu

# one pixel, part of a group, whole and broken groups, groups that are all resident at
# once with a thread a pixel (740 of 128 pixels on 148 SMs) and a few more
SIZES = [(1, 1), (5, 3), (31, 1), (128, 2), (33, 31), (320, 296), (307, 309), (641, 479)]


def check_pixels(sc, desc, img, gradient):
    """gradient(d_img) -> (d materials, d emitters)"""
    mats = adjoint.get_materials(sc)
    col = np.array([c for c, _, _ in desc.emitters], np.float64)
    x = img.cpu().numpy().reshape(-1, 3)
    lit = np.flatnonzero((x > 0).all(axis=1))
    assert len(lit) > 0
    n = len(x)
    edges = [0, n - 1, 127, 128, n // 128 * 128 - 1, n // 128 * 128]
    rng = np.random.default_rng(n)
    for pick in (lit[-8:], lit[np.searchsorted(lit, edges).clip(0, len(lit) - 1)], rng.choice(lit, 8)):
        w = np.zeros(n)
        w[lit] = 1.0
        w[pick] = 2.0 ** 17
        d = (w[:, None] / np.where(w[:, None] > 0, x, 1.0)).astype(np.float32)
        g_mat, g_em = gradient(torch.from_numpy(d.reshape(img.shape)).cuda())
        got = (col * g_em.cpu().numpy().astype(np.float64)).sum()
        got += (mats["emission"].astype(np.float64) * g_mat.cpu().numpy()[:, 4:7]).sum()
        terms = x.astype(np.float64) * d
        # all terms are positive: a float sum of n of them is within n * 2^-24, a
        # product of the replay's factors within a few dozen roundings
        bound = (x.size + 64) * 2.0 ** -24 * terms.sum()
        assert abs(got - terms.sum()) <= bound
        assert bound < 0.75 * terms[pick].sum(axis=1).min()  # the check can tell one pixel


@pytest.mark.parametrize("w,h", SIZES)
def test_path_tracer_adjoint(cuda_device, w, h):
    desc, cam = small_sphere_room()
    sc = Scene(desc)
    for seed in range(64):  # one that lights the single pixel
        adj = adjoint.PtAdjoint(sc, w, h, default_params(sc.scene_size, max_path_len=6, nee_prob=0.5, seed=seed))
        img = adj.render([cam])
        if (img > 0).all(dim=-1).any():
            break
    check_pixels(sc, desc, img, lambda d: adj.gradient([cam], d))


# the sizes above, and those around the resampled adjoint's own line (592 groups)
@pytest.mark.parametrize("w,h", SIZES[:-3] + [(296, 256), (296, 257), (641, 479)])
@pytest.mark.parametrize("k", [0, 8])
def test_resampled_adjoint(cuda_device, w, h, k):
    desc, cam = small_sphere_room()
    sc = Scene(desc)
    for seed in range(64):
        p = large_config_params(scene_size_of(desc), max_path_len=6, enable_accum=0, gather_n=1, gather_m=k + 1,
                                gather_radius=0.3, storage=_abi.STORAGE_FP32, seed=seed)
        adj = adjoint.RestirAdjoint(sc, w, h, p, 1)
        frame = adj.prepare([cam], frames=3)
        img = adj.render()
        if (img > 0).all(dim=-1).any():
            break
    np.testing.assert_array_equal(img.cpu().numpy(), frame.cpu().numpy())
    check_pixels(sc, desc, img, adj.gradient)
