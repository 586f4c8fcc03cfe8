"""The memory the endpoint search keeps between calls goes back on request, also for a
caller that has no scene, and searches work on after it."""
import numpy as np
import pytest
import torch

from crisoptix_b200 import _abi
from test_endpoint_search_gpu import brute_force, gpu_search
from test_search_build_gpu import case

pytestmark = pytest.mark.gpu


def free_memory():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("searches", [0, 1, 3])
def test_release(cuda_device, searches):
    _abi.check(_abi.load().crisb_endpoint_search_release())
    e, q = case(1, 600000)
    ref, rc = brute_force(e, q, 4)
    before = free_memory()
    for _ in range(searches):
        gpu_search(e, q, 4)
    held = free_memory()
    # the workspace of 600,000 entries is 100 MB and more
    assert (held <= before - (64 << 20)) == (searches > 0)
    _abi.check(_abi.load().crisb_endpoint_search_release())
    assert free_memory() >= before - (8 << 20)
    got, gc = gpu_search(e, q, 4)
    assert (gc == rc).all() and got.tobytes() == ref.tobytes()
