"""A pass launches as many wavefront and shift rounds as its longest path or
shift traces rays, and frames without gather neighbours build no endpoint
structure: frames at the ends of those ranges, and parameters that change
under reservoirs kept from other prefix and path lengths, against the oracle."""
import pytest

from crisoptix_b200 import _abi, scenes
from helpers import scene_size_of, small_config_params
from test_parity_gpu import run_parity, small_sphere_room, static

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prefix_len,max_path_len,k,gather_n", [
    (1, 1, 0, 1), (1, 2, 4, 1), (2, 2, 0, 2), (3, 8, 4, 1), (8, 8, 0, 1), (5, 6, 4, 2)])
def test_path_and_prefix_lengths(cuda_device, prefix_len, max_path_len, k, gather_n):
    desc, cam = small_sphere_room()
    p = small_config_params(scene_size_of(desc), prefix_len=prefix_len, max_path_len=max_path_len, gather_m=k + 1,
                            gather_n=gather_n, gather_radius=0.3, prefix_enable_spatial=1, prefix_spatial_count=2)
    run_parity(desc, cam, p, 33, 31, 3, static)


def test_reservoirs_kept_from_other_lengths(cuda_device):
    desc, cam = scenes.cornell_box()
    size = scene_size_of(desc)

    def at(prefix_len, max_path_len, k):
        return small_config_params(size, prefix_len=prefix_len, max_path_len=max_path_len, gather_m=k + 1,
                                   gather_radius=0.4)

    run_parity(desc, cam, at(1, 4, 4), 40, 24, 8, static,
               change_params={2: at(3, 8, 4), 4: at(3, 8, 0), 5: at(1, 8, 4), 6: at(4, 5, 2)})


@pytest.mark.parametrize("max_path_len", [1, 2, 5])
def test_restir_pt_lengths(cuda_device, max_path_len):
    desc, cam = scenes.cornell_box()
    p = small_config_params(scene_size_of(desc), renderer_type=_abi.RESTIR_PT, max_path_len=max_path_len, prefix_len=1,
                            prefix_enable_spatial=1, prefix_spatial_count=2, prefix_spatial_rounds=2)
    run_parity(desc, cam, p, 37, 23, 3, static)
