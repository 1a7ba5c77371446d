"""Cluster sizes of the decode-batch GEMM and tile heights of the prefill GEMM (plan_batch_cluster and plan_gemm_rows in
tur_b200/csrc/launch_plan.h), compiled with g++ and checked on the CPU: every CTA of a cluster has units of its own, the measured
choices are the ones taken, the weights of a transformer layer that share an activation agree on a cluster size, so that
they go out as one launch, and a tile height is a legal one that needs no more time by the plan's measure than 256 rows."""
import ctypes
import os
import subprocess
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include "launch_plan.h"
extern "C" int batch_cluster(int tiles, int KU, const int* resident) { return turq::plan_batch_cluster(tiles, KU, resident); }
extern "C" int gemm_rows(long long call_tiles, long long m, int sms) { return turq::plan_gemm_rows(call_tiles, m, sms); }
extern "C" int batch_tile(long long tiles, long long call_tiles, long long m, long long resident, int sms) {
  return turq::plan_batch_tile(tiles, call_tiles, m, resident, sms);
}
"""
B200 = [0, 148, 74, 45, 33, 26, 22]     # clusters of 1..6 CTAs that are resident at once


@pytest.fixture(scope="module")
def lib():
    with tempfile.TemporaryDirectory() as d:
        src, so = os.path.join(d, "shim.cpp"), os.path.join(d, "shim.so")
        open(src, "w").write(SHIM)
        subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "tur_b200", "csrc"), src, "-o", so], check=True)
        lib = ctypes.CDLL(so)
        lib.gemm_rows.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int]
        lib.batch_tile.argtypes = [ctypes.c_longlong] * 4 + [ctypes.c_int]
        yield lib


@pytest.fixture(scope="module")
def cluster(lib):
    def call(n, k, resident=B200):
        return lib.batch_cluster(-(-n // 128), -(-k // 256), (ctypes.c_int * 7)(*resident))
    return call


def test_every_cta_has_units(cluster):
    for resident in (B200, [0, 16, 8, 5, 4, 3, 2], [0, 1, 1, 1, 1, 1, 1]):
        for n in (1, 128, 129, 640, 2560, 4096, 5120, 12288, 25600, 151936):
            for k in (64, 256, 320, 512, 768, 1024, 2560, 4096, 6144, 8192, 25600):
                c = cluster(n, k, resident)
                assert 1 <= c <= 6 and c <= -(-k // 256), (n, k, c)
                ku = -(-k // 256)
                shares = [ku * (r + 1) // c - ku * r // c for r in range(c)]
                assert min(shares) >= 1 and sum(shares) == ku


@pytest.mark.parametrize("n,k,want", [(8192, 2560, 1), (12288, 4096, 2), (25600, 5120, 1), (3072, 1024, 2), (4096, 4096, 4), (2560, 2560, 4),
                                      (5120, 25600, 3), (5120, 8192, 3), (2560, 8192, 6), (1024, 2048, 4)])
def test_measured_choices(cluster, n, k, want):
    assert cluster(n, k) == want


@pytest.mark.parametrize("hidden,q,kv", [(1024, 2048, 1024), (2560, 2560, 640), (4096, 4096, 1024), (5120, 8192, 1024), (4096, 4096, 4096)])
def test_projections_of_a_layer_share_a_launch(cluster, hidden, q, kv):
    assert cluster(q, hidden) == cluster(kv, hidden)


@pytest.mark.parametrize("rows,m,tiles", [((4096, 1024, 1024), 512, 3), ((4096,), 512, 4), ((12288, 12288), 512, 2), ((2560, 640, 640), 1000, 4),
                                          ((2560,), 1000, 7), ((8192, 8192), 1000, 4), ((4096,), 2048, 9), ((12288, 12288), 2048, 8),
                                          ((5120,), 4096, 18), ((25600, 25600), 4096, 16), ((12288, 12288), 128, 1)])
def test_tile_heights_that_were_measured_best(lib, rows, m, tiles):
    assert -(-m // lib.gemm_rows(sum(-(-n // 256) for n in rows), m, 148)) == tiles


def test_tile_heights_are_legal_and_no_worse_than_the_largest(lib):
    def cost(call, m, b, slots):
        return -(-call * -(-m // b) // slots) * max(b + 110, 260)
    for sms in (148, 132, 16, 2, 1):
        for call in (1, 3, 10, 24, 74, 200, 1187):
            for m in (65, 80, 129, 255, 256, 257, 999, 2048, 2999, 65535, 2 ** 30):
                b = lib.gemm_rows(call, m, sms)
                assert b % 16 == 0 and 16 <= b <= 256, (call, m, b)
                whole = -(-(-(-m // -(-m // 256))) // 16) * 16
                slots = max(1, sms // 2)
                assert cost(call, m, b, slots) <= cost(call, m, whole, slots)


def test_tiles_of_short_prompts(lib):
    """A tile is a legal one, no call outside 65..1024 rows is taken, and the measured choices are the ones taken."""
    def tile(n, m, resident=148, sms=148):
        return lib.batch_tile(-(-n // 128), -(-n // 256), m, resident, sms)
    for n in (0, 1, 128, 1000, 4096, 25600, 151936, 2 ** 31):
        for m in (1, 64, 65, 66, 127, 128, 129, 511, 1000, 1024, 1025, 8192):
            for resident, sms in ((148, 148), (16, 16), (1, 1)):
                bn = tile(n, m, resident, sms)
                assert bn == 0 or (bn % 16 == 0 and 16 <= bn <= 128 and 64 < m <= 1024), (n, m, bn)
    assert tile(0, 128) == 0
    for n, m in ((4096, 65), (4096, 128), (4096, 512), (2560, 768), (12288, 128), (12288, 384), (1024, 1000), (25600, 65)):
        assert tile(n, m) > 0, (n, m)
    for n, m in ((4096, 1000), (12288, 768), (25600, 256), (25600, 512), (151936, 512)):
        assert tile(n, m) == 0, (n, m)
