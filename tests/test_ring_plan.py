"""The depths of the rings that the dequant groups of the pair kernel share, for every token tile and both stage widths."""

import ctypes
import subprocess

import pytest

from tuna_b200 import _lib, build

PROGRAM = """
#include <cstdio>
#include "ring_plan.h"
int main()
{
    for (int t = 32; t <= 256; t += 32)
        for (int kc = 64; kc <= 128; kc += 64) {
            const tuna::PairPlan l = tuna::pair_plan(t, kc);
            std::printf("%d %d %d %d %d %d %d %d\\n", t, kc, l.stages, l.w_stages, l.nd, l.fits, tuna::pair_dequant_warps(t) / 4, kc == tuna::pair_kc(t));
        }
}
"""


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring_plan")
    (d / "plan.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{build.CSRC}", str(d / "plan.cpp"), "-o", str(d / "plan")], check=True)
    lines = subprocess.run([str(d / "plan")], check=True, capture_output=True, text=True).stdout.splitlines()
    return [tuple(map(int, line.split())) for line in lines]


def _early_pass(w_stages, a_slots, groups, units=64):
    """Whether a group can pass its parity wait for a weight stage before the unit has landed: copies may land out of order, the
    other groups may be as far behind as the rings let them."""
    for u in range(groups, units):
        # group u % groups has finished unit u - groups, so the MMAs have consumed every unit up to u - groups - a_slots
        consumed = u - groups - a_slots
        own = {v for v in range(u) if v % groups == u % groups}
        prev = u - w_stages  # the stage's use before
        if prev >= 0 and prev > consumed and prev not in own:
            return True
    return False


def test_no_group_passes_a_wait_early(plans):
    assert len(plans) == 16
    for tile, kc, stages, w_stages, nd, fits, groups, used in plans:
        assert fits or not used, f"no rings for {tile}-token tiles"
        if not fits:
            continue
        assert stages >= groups and w_stages >= 4 and nd * tile + stages * kc // 2 <= 512
        assert not _early_pass(w_stages, stages, groups), f"{tile}-token tiles in stages of {kc} columns: {w_stages} weight stages, {stages} slots, {groups} groups"


def test_plans_in_use_keep_all_their_weight_stages(plans):
    assert [p[3] for p in plans if p[7]] == [8] * 8


WARPS_PROGRAM = PROGRAM.replace("for (int kc = 64; kc <= 128; kc += 64) {", "for (int warps = 8; warps <= tuna::pair_dequant_warps(t); warps += 8) {\n            const int kc = tuna::pair_kc(t);").replace(
    "pair_plan(t, kc)", "pair_plan(t, kc, warps)").replace("tuna::pair_dequant_warps(t) / 4, kc == tuna::pair_kc(t)", "warps / 4, 1")


def test_both_numbers_of_dequant_warps_have_their_rings(tmp_path):
    (tmp_path / "plan.cpp").write_text(WARPS_PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{build.CSRC}", str(tmp_path / "plan.cpp"), "-o", str(tmp_path / "plan")], check=True)
    lines = subprocess.run([str(tmp_path / "plan")], check=True, capture_output=True, text=True).stdout.splitlines()
    plans = [tuple(map(int, line.split())) for line in lines]
    assert len(plans) == 8 + 6
    for tile, kc, stages, w_stages, nd, fits, groups, _ in plans:
        assert fits and stages >= groups and w_stages == 8 and nd * tile + stages * kc // 2 <= 512
        assert not _early_pass(w_stages, stages, groups), (tile, groups)


# 16 dequant warps pay on long tiles; short ones, uncut or cut into short segments, are done sooner with 8
@pytest.mark.parametrize("m,n,k,warps", [(12496, 738, 512, 8), (3792, 488, 512, 8), (3192, 613, 1048, 8), (2688, 746, 624, 8), (57344, 64, 8192, 16),
                                         (11000, 43, 4104, 16), (6144, 256, 4096, 16), (10240, 777, 8192, 16), (57344, 4096, 8192, 8)])
def test_dequant_warps_by_the_length_of_a_tile(m, n, k, warps):
    cfg = _lib.TunaConfig()
    assert _lib.load().tuna_lookup_config(m, n, k, ctypes.byref(cfg)) == 0
    assert cfg.path == _lib.PATH_UMMA and cfg.dequant_warps == warps
