"""The resampled estimator's replay starts from the stored primary hit and
leaves out the ray to the last prefix vertex: at every prefix length it still
gives the frame's own gather values bit for bit."""
import numpy as np
import pytest

from crisoptix_b200 import Scene, _abi, adjoint, scenes
from helpers import large_config_params, scene_size_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prefix_len,k", [(1, 8), (2, 0), (3, 8), (4, 3), (6, 8)])
def test_replay_reproduces_the_frame_at_every_prefix_length(cuda_device, prefix_len, k):
    desc, cam = scenes.sphere_room(num_spheres=12, subdiv=2, num_emitters=12, seed=4)
    sc = Scene(desc)
    p = large_config_params(scene_size_of(desc), max_path_len=6, enable_accum=0, gather_n=1, prefix_len=prefix_len,
                            gather_m=k + 1, storage=_abi.STORAGE_FP32)
    adj = adjoint.RestirAdjoint(sc, 65, 47, p, 1)
    frame = adj.prepare([cam], frames=3)
    np.testing.assert_array_equal(adj.render().cpu().numpy(), frame.cpu().numpy())
