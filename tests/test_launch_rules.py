"""How the tile kernel's launch goes by a frame's size and by what bhSetTuning (and so the autotuner) has set."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "black-hole_b200", "csrc")
SRC = r"""
#include <cstdio>
#include "bh_launch_rules.h"
int main()
{
    unsigned rays; int known, kerr, fit, set; float half;
    while (std::scanf("%u %d %d %d %d %f", &rays, &known, &kerr, &fit, &set, &half) == 6)
    {
        const bool wide = bh_wide_view(half, 1.f, 0.5f, 8.f);
        const int warps = bh_warps_per_sm(rays, known != 0, kerr != 0, wide);
        std::printf("%d %d %d\n", bh_rays_per_warp(rays, known != 0, wide), warps,
                    bh_blocks_per_sm(fit, warps, kerr ? 5 : 4, set));
    }
}
"""
SIZES = [32, 288 * 32, 512 * 32, 513 * 32, 4096 * 32, 4097 * 32, 8192 * 32, 8193 * 32, 16384 * 32, 16385 * 32,
         32768 * 32, 32769 * 32, 259200 * 32]


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "r.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I" + CSRC, str(d / "r.cpp"), "-o", str(d / "r")], check=True)

    def ask(rows):
        text = "\n".join(" ".join(map(str, r)) for r in rows)
        out = subprocess.run([str(d / "r")], input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]
    return ask


@pytest.mark.parametrize("half", [1.2, 20.0])
def test_a_set_number_limits_but_does_not_turn_the_rule_off(rules, half):
    for kerr, fit in ((0, 7), (1, 5)):
        free = rules([(n, 1, kerr, fit, 0, half) for n in SIZES])
        for number in (fit, fit + 4):      # what the autotuner sets when nothing else is faster
            assert rules([(n, 1, kerr, fit, number, half) for n in SIZES]) == free
        for number in range(1, fit):
            got = rules([(n, 1, kerr, fit, number, half) for n in SIZES])
            assert [g[2] for g in got] == [min(f[2], number) for f in free]
        assert [f[2] for f in free][-1] == fit and min(f[2] for f in free) >= 1


@pytest.mark.parametrize("half, limit", [(1.2, 1024), (9.5, 1024), (9.7, 8192), (60.0, 8192)])
def test_widths_by_the_number_of_groups(rules, half, limit):
    """Close views, which the hole and its disk fill, lose up to half their speed to narrow groups."""
    for n, (width, _, _) in zip(SIZES, rules([(n, 1, 0, 7, 0, half) for n in SIZES])):
        assert width in (1, 2, 4, 8, 16, 32)
        assert width == 32 or n // width <= limit
        assert width == 1 or 2 * n // width > limit
    assert rules([(64, 0, 1, 5, 0, half)]) == [(32, 0, 5)]      # a list whose length only the device knows
