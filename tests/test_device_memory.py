"""What the library only keeps (the endpoint search's workspace) never makes an
allocation fail: the allocation helper gives it back and tries once more, and every
device allocation of the library goes through the helper.  The failures are those of a
fake allocator."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "crisoptix_b200", "csrc")

PROGRAM = r"""
#include "device_memory.h"
#include <cstdio>
#include <initializer_list>
static cudaError_t last = cudaSuccess;
extern "C" cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
int main() {
    const cudaError_t oom = cudaErrorMemoryAllocation, bad = cudaErrorInvalidValue;
    for (auto first : {cudaSuccess, oom, bad})
        for (auto second : {cudaSuccess, oom}) {
            int calls = 0, trims = 0;
            last = cudaSuccess;
            const cudaError_t e = crisb::alloc_or_trim([&] { return last = ++calls == 1 ? first : second; },
                                                       [&] { ++trims; });
            std::printf("%d %d %d %d\n", int(e), calls, trims, int(last));
        }
}
"""


def cuda_include():
    from crisoptix_b200 import build

    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc_path()))), "include")


def test_failed_allocation_is_tried_again_without_what_is_kept(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-ffunction-sections", "-Wl,--gc-sections", "-I", CSRC, "-I", cuda_include(),
                    str(src), "-o", str(exe)], check=True)
    got = [tuple(map(int, l.split())) for l in subprocess.run([str(exe)], check=True, capture_output=True,
                                                              text=True).stdout.split("\n") if l]
    # result, calls, trims, error left behind; out of memory is error 2, another error 1
    assert got == [(0, 1, 0, 0), (0, 1, 0, 0), (0, 2, 1, 0), (2, 2, 1, 2), (1, 1, 0, 1), (1, 1, 0, 1)]


# the only places that may call an allocator: the helper, and the search's own pool
# with its ways round it
ALLOWED = {"device_memory.h": {"cudaMalloc"}, "search.cu": {"cudaMallocAsync", "cudaMallocFromPoolAsync"}}


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h", ".cpp"))))
def test_allocations_go_through_the_helper(name):
    with open(os.path.join(CSRC, name)) as f:
        code = re.sub(r"//[^\n]*|\"(\\.|[^\"\\\n])*\"", "", f.read())
    calls = set(re.findall(r"\b(cudaMalloc\w*)\s*\(", code)) - {"cudaMallocHost"}
    assert calls <= ALLOWED.get(name, set())
