"""The check every compressed tree passes before use asks for the slack around each
child box that the traversal's slab test may lose to rounding (2^-9 of a grid step):
one node over two triangles, its boxes on the grid with a given slack."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "crisoptix_b200", "csrc")

PROGRAM = r"""
#include "bvh_build.h"
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <stdexcept>
using namespace crisb;
int main(int argc, char** argv) {
    const double slack = std::atof(argv[1]);
    const int side = std::atoi(argv[2]);  // 0: the lower planes have it, 1: the upper ones
    // extents of 128 in x, y and z, a grid step of one
    const float c = 64.0f, margin = box_margin(c);
    const float pos[18] = {-c, -c, -c, -1, -c, -c, -c, -1, -1, c, c, c, 1, c, c, c, 1, 1};
    Bvh8QNode nd;
    std::memset(&nd, 0, sizeof nd);
    float* p[3] = {&nd.px, &nd.py, &nd.pz};
    uint8_t* lo[3] = {nd.qlo_x, nd.qlo_y, nd.qlo_z};
    uint8_t* hi[3] = {nd.qhi_x, nd.qhi_y, nd.qhi_z};
    for (int a = 0; a < 3; ++a) {
        // the plane of grid step 0 (132) lies `slack` steps outside the widened boxes
        *p[a] = static_cast<float>(side == 0 ? -c - margin - slack : c + margin + slack - 132.0);
        for (int t = 0; t < 2; ++t) {
            double l = 1e9, h = -1e9;
            for (int v = 0; v < 3; ++v) {
                l = std::fmin(l, pos[9 * t + 3 * v + a]);
                h = std::fmax(h, pos[9 * t + 3 * v + a]);
            }
            lo[a][t] = static_cast<uint8_t>(std::fmax(0.0, side == 0 && t == 0 ? 0.0 : std::floor(l - margin - *p[a]) - 1));
            hi[a][t] = static_cast<uint8_t>(side == 1 && t == 1 ? 132.0 : std::ceil(h + margin - *p[a]) + 1);
        }
    }
    for (uint32_t t = 0; t < 2; ++t) nd.meta[t] = static_cast<uint8_t>((1u << 5) | t);
    try {
        std::printf("%d\n", validate_qbvh({nd}, {0, 1}, pos, 2, margin));
    } catch (const std::runtime_error& e) {
        std::printf("%s\n", e.what());
    }
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("qbvh")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(d / "t.cpp"), os.path.join(CSRC, "bvh_build.cpp"), "-o",
                    str(d / "t")], check=True)
    return lambda *args: subprocess.run([str(d / "t"), *map(str, args)], check=True, capture_output=True,
                                        text=True).stdout.strip()


# the builder's 2^-7, more, just what the test may lose; half of that and none.  Half
# the margin, 2^-12 of a step here, is spare
@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize("slack,ok", [(0.5, True), (2.0 ** -7, True), (2.0 ** -9, True), (2.0 ** -10, False), (0.0, False)])
def test_slack(check, slack, ok, side):
    got = check(slack, side)
    assert got == ("1" if ok else "compressed bvh check: child box without slack"), got


def test_box_that_cuts_its_triangle(check):
    assert check(-0.25, 0) == "compressed bvh check: child box does not contain its subtree"
