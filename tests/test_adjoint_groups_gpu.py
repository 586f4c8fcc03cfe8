"""The adjoints' backward kernels work through groups of 128 pixels and gather the
gradients in shared memory beside their own.  A pixel's value is homogeneous of
degree one in the emitters' colours and the materials' emissions together, so over
any image the colours and emissions times their gradients add up to the image
times its adjoint, whatever the last group holds and wherever the parameters are
gathered."""
import dataclasses

import numpy as np
import pytest
import torch

from crisoptix_b200 import Scene, _abi, adjoint, scenes
from helpers import large_config_params, scene_size_of

pytestmark = pytest.mark.gpu


def padded_scene(param_bytes):
    """A room whose parameter block (28 bytes a material, 12 an emitter) has about
    that size, through materials that no triangle has."""
    desc, cam = scenes.sphere_room(num_spheres=12, subdiv=2, num_emitters=12, seed=4)
    n = (param_bytes - 12 * len(desc.emitters)) // 28
    if n > len(desc.materials):
        mats = np.concatenate([desc.materials, np.repeat(desc.materials[:1], n - len(desc.materials))])
        desc = dataclasses.replace(desc, materials=mats)
    return desc, cam


def check_homogeneous(sc, desc, img, d_img, g_mat, g_em):
    mats = adjoint.get_materials(sc)
    col = np.array([c for c, _, _ in desc.emitters], np.float64)
    lhs = (col * g_em.cpu().numpy().astype(np.float64)).sum()
    lhs += (mats["emission"].astype(np.float64) * g_mat.cpu().numpy()[:, 4:7]).sum()
    terms = img.cpu().numpy().astype(np.float64) * d_img.cpu().numpy()
    # all terms are positive: a float sum of n of them is within n * 2^-24, a
    # product of the replay's factors within a few dozen roundings of each other
    assert terms.sum() > 0
    assert abs(lhs - terms.sum()) <= (terms.size + 64) * 2.0 ** -24 * terms.sum()


# whole and broken groups, one pixel, a warp more than a group
@pytest.mark.parametrize("width,height,k", [(1, 1, 8), (127, 1, 8), (129, 1, 0), (16, 8, 3), (43, 23, 8)])
def test_groups_of_the_resampled_adjoint(cuda_device, width, height, k):
    desc, cam = padded_scene(0)
    run_restir(desc, cam, width, height, k)


# parameter blocks around what shared memory holds beside the kernel's own, and past it
@pytest.mark.parametrize("param_bytes", [46 << 10, 48 << 10, (48 << 10) + 64])
def test_parameter_blocks_around_the_shared_memory_limit(cuda_device, param_bytes):
    desc, cam = padded_scene(param_bytes)
    run_restir(desc, cam, 43, 23, 8)
    sc = Scene(desc)
    adj = adjoint.PtAdjoint(sc, 43, 23, large_config_params(scene_size_of(desc), max_path_len=6, nee_prob=0.3))
    img = adj.render([cam])
    d = torch.rand(img.shape, generator=torch.Generator().manual_seed(1)).cuda() + 0.5
    check_homogeneous(sc, desc, img, d, *adj.gradient([cam], d))


def run_restir(desc, cam, width, height, k):
    sc = Scene(desc)
    p = large_config_params(scene_size_of(desc), max_path_len=6, enable_accum=0, gather_n=1, gather_m=k + 1,
                            storage=_abi.STORAGE_FP32)
    adj = adjoint.RestirAdjoint(sc, width, height, p, 1)
    frame = adj.prepare([cam], frames=3)
    img = adj.render()
    np.testing.assert_array_equal(img.cpu().numpy(), frame.cpu().numpy())
    d = torch.rand(img.shape, generator=torch.Generator().manual_seed(1)).cuda() + 0.5
    if not img.any():
        return
    check_homogeneous(sc, desc, img, d, *adj.gradient(d))
