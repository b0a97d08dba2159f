"""Division of a render call into waves (csrc/wave_plan.h, host code): no setting
and no frame size gives a launch more items than its 32-bit counter can take
together with the requests past the end, and the waves hold every pass once."""

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
INT_MAX = 2 ** 31 - 1
# every resident lane asks past the end at most once
PAST_END = 160 * 2048

MAIN = r"""
#include <cstdio>
#include "wave_plan.h"
using namespace prt_b200;
int main()
{
    int w, h, spp, setting;
    while (std::scanf("%d %d %d %d", &w, &h, &spp, &setting) == 4)
    {
        const long long per = frame_items(w, h), paths = wave_paths(setting, 1 << 24);
        const int passes = wave_passes(paths, per, spp);
        std::printf("%lld %lld %d %d %d", per, paths, passes, wave_count(spp, passes), per <= kMaxFrameItems);
        for (int mode = 0; mode < 4; ++mode) std::printf(" %d", primary_packets(mode, 148, passes * per, per));
        std::printf("\n");
    }
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src, exe = d / "main.cpp", d / "main"
    src.write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "embree-benchmark-protoray_b200", "csrc"), "-o", str(exe), str(src)], check=True)

    def run(*case):
        out = subprocess.run([str(exe)], input=" ".join(map(str, case)), capture_output=True, text=True, check=True)
        return [int(x) for x in out.stdout.split()]
    return run


@pytest.mark.parametrize("setting", [0, 1, 65536, 1 << 26, (1 << 30) - 1, 1 << 30, (1 << 30) + 1, INT_MAX])
@pytest.mark.parametrize("w,h", [(1, 1), (8, 8), (1920, 1080), (1001, 563), (16384, 16384), (1, 1 << 27), (1 << 27, 2)])
@pytest.mark.parametrize("spp", [1, 7, 1028, 1 << 20, INT_MAX])
def test_items_of_a_launch(plan, w, h, spp, setting):
    per, paths, passes, waves, frame_ok = plan(w, h, spp, setting)[:5]
    assert per == (w + 7) // 8 * ((h + 7) // 8) * 64
    assert frame_ok
    assert 1 <= passes <= spp
    assert passes * per + PAST_END <= INT_MAX
    # batches take `paths` paths at a time
    assert 0 < paths and paths + PAST_END <= INT_MAX
    assert (waves - 1) * passes < spp <= waves * passes


def test_frames_beyond_the_counter(plan):
    assert plan(1, 1 << 28, 1, 0)[4] == 0 and plan(1 << 28, 1, 1, 0)[4] == 0
    assert plan(2, 1 << 27, 1, 0)[4] == 1


def test_camera_rays_per_lane_or_packets(plan):
    """Settings 1 and 2 ask for packets, 3 for lanes, 0 leaves it to the wave's size."""
    for w, h, spp, auto in ((256, 256, 16, 0), (1920, 1080, 1, 0), (1920, 1080, 7, 0), (1920, 1080, 8, 1),
                            (1920, 1080, 64, 1), (640, 480, 64, 1), (4096, 4096, 4, 0)):
        assert plan(w, h, spp, 0)[5:] == [auto, 1, 2, 0]
