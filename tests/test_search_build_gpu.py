"""The endpoint search where its build and its workspace change shape: trees of
one node and of a few entries, entry counts around a sort tile and around the
grid of the bounds pass, and calls that share the kept workspace memory from
several streams and threads and inside a captured graph.  Lists must equal the
float32 brute force exactly."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from crisoptix_b200 import _abi
from test_endpoint_search_gpu import brute_force, gpu_search, make_case

pytestmark = pytest.mark.gpu

# 1024 keys and more: scan tiles and sort tiles of the digit counts; 592 * 128: the
# largest grid of the bounds pass
SIZES = [1, 2, 3, 8, 9, 17, 1023, 1025, 4095, 4097, 592 * 128 - 1, 592 * 128 + 1]


def case(seed, n, m=64):
    rng = np.random.default_rng(seed)
    e = np.concatenate([rng.uniform(-1, 1, (n, 3)), rng.uniform(0, 0.3, (n, 1))], axis=1).astype(np.float32)
    q = rng.uniform(-1, 1, (m, 3)).astype(np.float32)
    q[: min(n, m // 2)] = e[: min(n, m // 2), :3]
    return e, q


@pytest.mark.parametrize("n", SIZES)
def test_entry_counts(cuda_device, n):
    entries, queries = case(n, n)
    ref, rc = brute_force(entries, queries, 8)
    for fn in ["crisb_endpoint_search"] + (["crisb_endpoint_search_noalloc"] if n <= 4097 else []):
        got, gc = gpu_search(entries, queries, 8, fn)
        assert (gc == rc).all() and got.tobytes() == ref.tobytes()


def test_radius_at_the_ends_of_its_range(cuda_device):
    """Radii whose square underflows or overflows, and distances on the radius."""
    queries = np.array([[0, 0, 0], [1e-20, 0, 0], [3, 4, 0], [1e25, 0, 0]], np.float32)
    radii = [0.0, 1e-30, 1e-20, 1e-18, 5.0, np.float32(np.nextafter(np.float32(5), np.float32(0))), 1e20, 3e38]
    entries = np.array([[0, 0, 0, r] for r in radii], np.float32)
    with np.errstate(over="ignore"):
        ref, rc = brute_force(entries, queries, 8)
    got, gc = gpu_search(entries, queries, 8)
    assert (gc == rc).all() and got.tobytes() == ref.tobytes()


def enqueue(e, q, k, out, cnt, stream):
    _abi.check(_abi.load().crisb_endpoint_search(
        ctypes.c_void_p(e.data_ptr()), len(e), ctypes.c_void_p(q.data_ptr()), len(q), k,
        ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(cnt.data_ptr()), ctypes.c_void_p(stream.cuda_stream)))


def test_streams_and_threads_share_the_workspace_memory(cuda_device):
    """Calls in flight at once, large ones before small ones, never share a byte."""
    cases = [make_case(20 + i, n_entries=n, n_queries=200) for i, n in enumerate([60000, 500, 30000, 4000])]
    refs = [brute_force(e, q, 8) for e, q in cases]
    failures = []

    def work(i):
        e, q = cases[i]
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            ed, qd = torch.from_numpy(e).cuda(), torch.from_numpy(q).cuda()
            outs = []
            for _ in range(20):
                out = torch.empty((len(q), 8, 2), dtype=torch.int32, device="cuda")
                cnt = torch.empty(len(q), dtype=torch.int32, device="cuda")
                enqueue(ed, qd, 8, out, cnt, stream)
                outs.append((out, cnt))
            stream.synchronize()
        for out, cnt in outs:
            if out.cpu().numpy().tobytes() != refs[i][0].tobytes() or \
                    (cnt.cpu().numpy().view(np.uint32) != refs[i][1]).any():
                failures.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures


def test_captured_search_replays(cuda_device):
    """A captured call owns its workspace: replays give the same lists, with other
    searches between them."""
    e, q = make_case(31, n_entries=5000, n_queries=300)
    ref, rc = brute_force(e, q, 8)
    ed, qd = torch.from_numpy(e).cuda(), torch.from_numpy(q).cuda()
    out = torch.zeros((len(q), 8, 2), dtype=torch.int32, device="cuda")
    cnt = torch.zeros(len(q), dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        enqueue(ed, qd, 8, out, cnt, stream)
    for _ in range(3):
        out.zero_()
        cnt.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert out.cpu().numpy().tobytes() == ref.tobytes()
        assert (cnt.cpu().numpy().view(np.uint32) == rc).all()
        gpu_search(*make_case(32, n_entries=7000, n_queries=50), 8)


def test_kept_memory_goes_back_with_a_scene(cuda_device):
    """The memory kept between searches is given back when a scene is destroyed."""
    from crisoptix_b200 import Scene, scenes

    e, q = case(1, 600000)
    gpu_search(e, q, 4)
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    held = torch.cuda.mem_get_info()[0]
    sc = Scene(scenes.cornell_box()[0])
    del sc
    torch.cuda.synchronize()
    # the workspace of 600,000 entries is 100 MB and more
    assert torch.cuda.mem_get_info()[0] >= held + (64 << 20)
