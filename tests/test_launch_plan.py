"""Host-side launch arithmetic (tur_b200/csrc/launch_plan.h), compiled with g++ and checked on
the CPU: every tile of a weight is owned by exactly one CTA, whole-row-tile splits are what they
claim, the workspace is large enough for the grid, and the prefill GEMM's tile classes and pairs are what they claim."""
import ctypes
import os
import subprocess
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include "launch_plan.h"
extern "C" {
void plan_split(int row_tiles, int KU, int slots, int force, int* out) {
  turq::GemvSplit p = turq::plan_gemv_split(row_tiles, KU, slots, force);
  out[0] = p.grid; out[1] = p.split_q; out[2] = p.split_r; out[3] = p.aligned ? 1 : 0;
}
long long split_start(int grid, int q, int r, long long total, int b) {
  turq::GemvSplit p{grid, q, r, false};
  return turq::gemv_split_start(p, total, b);
}
int gemv_wide(int reads, int rows, int row_tiles, int KU, int slots) {
  return turq::plan_gemv_wide(static_cast<turq::GemvPlaneReads>(reads), rows, turq::plan_gemv_split(row_tiles, KU, slots),
                              (long long)row_tiles * KU, KU, slots);
}
int gemm_bn(long long n, long long m, int sms) { return turq::plan_gemm_bn(n, m, sms); }
int gemm_pairs(long long tiles, int sms) { return turq::plan_gemm_pairs(tiles, sms); }
}
"""


@pytest.fixture(scope="module")
def plan():
    with tempfile.TemporaryDirectory() as d:
        src, so = os.path.join(d, "shim.cpp"), os.path.join(d, "shim.so")
        open(src, "w").write(SHIM)
        subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "tur_b200", "csrc"),
                        src, "-o", so], check=True)
        lib = ctypes.CDLL(so)
        lib.split_start.restype = ctypes.c_longlong
        lib.split_start.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_int]
        lib.gemm_bn.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int]
        lib.gemm_pairs.argtypes = [ctypes.c_longlong, ctypes.c_int]
        yield lib


SLOTS = 296  # two CTAs on each of 148 SMs
# (rows, K tiles per row-tile): the benchmark shapes plus ragged and tiny ones
SHAPES = [(1024, 16), (4096, 16), (5120, 16), (12288, 16), (24576, 16), (4096, 48), (151936, 16), (8192, 20),
          (5120, 32), (5120, 100), (25600, 20), (2560, 10), (640, 10), (2048, 8), (3072, 8), (1, 1), (3, 2),
          (17, 5), (49155, 10), (300, 25), (9500, 1), (4737, 7)]


@pytest.mark.parametrize("force", [-1, 0, 1])
@pytest.mark.parametrize("rows,ku", SHAPES)
def test_every_unit_has_exactly_one_owner(plan, rows, ku, force):
    row_tiles = (rows + 15) // 16
    out = (ctypes.c_int * 4)()
    plan.plan_split(row_tiles, ku, SLOTS, force, out)
    grid, q, r, aligned = out[0], out[1], out[2], out[3]
    total = row_tiles * ku
    assert 1 <= grid <= SLOTS
    starts = [plan.split_start(grid, q, r, total, b) for b in range(grid + 1)]
    assert starts[0] == 0 and starts[-1] == total
    assert all(a <= b for a, b in zip(starts, starts[1:]))
    assert all(b > a for a, b in zip(starts, starts[1:])), "no CTA without work"
    if aligned:
        assert all(s % ku == 0 for s in starts), "whole row-tiles only"
        per = q // ku
        assert per == -(-row_tiles // SLOTS)
    else:
        sizes = [b - a for a, b in zip(starts, starts[1:])]
        assert max(sizes) - min(sizes) <= 1, "even split"
    # hand-over workspace: one flag and one partial-sum slot per CTA, sized for 4 CTAs per SM
    assert grid <= 148 * 4


def test_split_choice_follows_the_stated_rule(plan):
    out = (ctypes.c_int * 4)()
    plan.plan_split(768, 16, SLOTS, -1, out)       # ffn_gate 12288 rows: 3 row-tiles per CTA, 256 CTAs (86 %)
    assert (out[0], out[1], out[3]) == (256, 48, 1)
    plan.plan_split(320, 32, SLOTS, -1, out)       # 5120 x 8192: 160 CTAs would idle 46 % of the slots, large -> even split
    assert out[3] == 0 and out[0] == SLOTS
    plan.plan_split(64, 16, SLOTS, -1, out)        # 1024 rows: small -> whole row-tiles on 64 CTAs
    assert (out[0], out[3]) == (64, 1)


Q8_0, Q6_K, Q45_K = 0, 1, 2      # how the MMA loop reads the planes


@pytest.mark.parametrize("reads,unit,n,k,narrow,wide", [
    (Q8_0, 128, 512, 8192, (), (8, 12, 16)), (Q8_0, 128, 5120, 25600, (), (3, 4, 5)),
    (Q6_K, 256, 4096, 12288, (), (4, 8)), (Q6_K, 256, 640, 6144, (), (8, 12)),
    (Q6_K, 256, 5120, 25600, (2, 3), (4,)),                          # cut shares of about one row-tile
    (Q45_K, 256, 4096, 12288, (), (6, 8, 9)), (Q45_K, 256, 25600, 5120, (), (12, 16)), (Q45_K, 256, 9600, 8192, (), (8, 14)),
    (Q45_K, 256, 5120, 8192, (8, 9, 12), ()), (Q45_K, 256, 6144, 6144, (9, 11, 16), ()), (Q45_K, 256, 5120, 25600, (3, 5), ()),
    (Q45_K, 256, 640, 8192, (8, 14), ()), (Q45_K, 256, 128, 16384, (4, 8), ()),      # no more shares than SMs
    (Q45_K, 256, 2560, 8192, (7, 8), (9, 12)),                       # a share for a little more than every SM
])
def test_wide_launches_where_they_are_faster(plan, reads, unit, n, k, narrow, wide):
    """The lines of the rule, drawn where both forms were measured with row-major planes; what is measured now stands beside it."""
    for rows in narrow + wide:
        assert bool(plan.gemv_wide(reads, rows, -(-n // 16), k // unit, SLOTS)) == (rows in wide), rows


def test_gemm_activation_tile_choice(plan):
    sms = 148
    assert plan.gemm_bn(12288, 2048, sms) == 256
    assert plan.gemm_bn(4096, 512, sms) == 128      # 32 x 2 tiles: doubling still fits one wave
    assert plan.gemm_bn(2560, 1024, sms) == 256     # 20 x 4 tiles: doubling would spill into a second wave
    assert plan.gemm_bn(1024, 2048, sms) == 128


@pytest.mark.parametrize("n", [8192, 1024, 5120, 2560, 640, 12288, 4096, 151936, 272, 1, 9700, 40000])
def test_gemm_pairs_cover_the_work(plan, n):
    """No more pairs than SMs for two CTAs each, nor than tiles."""
    tiles = 4 * -(-n // 256)
    assert plan.gemm_pairs(tiles, 148) == min(74, tiles)
    assert plan.gemm_pairs(tiles, 1) == 1
