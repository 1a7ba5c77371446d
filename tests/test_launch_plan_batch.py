"""Cluster sizes of the decode-batch GEMM and tile heights of the prefill GEMM (plan_batch_cluster and plan_gemm_rows in
tur_b200/csrc/launch_plan.h), compiled with g++ and checked on the CPU: every CTA of a cluster has units of its own, the measured
choices are the ones taken, the weights of a transformer layer that share an activation agree on a cluster size, so that
they go out as one launch, a cluster size goes by the weight's shape and by nothing that a device answers, and a tile height
is a legal one that needs no more time by the plan's measure than 256 rows."""
import ctypes
import os
import subprocess
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include "launch_plan.h"
extern "C" int batch_cluster(int tiles, int KU) { return turq::plan_batch_cluster(tiles, KU); }
extern "C" int prep_cluster(long long m, long long k, int sms) { return turq::plan_prep_cluster(m, k, sms); }
// asks three times: answers[i] is what the device would say, errors[i] the status that it returns
extern "C" void ask_three_times(const int* answers, const int* errors, int* asked, int* status, int* out) {
  std::atomic<int> known{0};
  for (int i = 0; i < 3; i++) {
    out[i] = -1;
    status[i] = turq::ask_once(known, [&](int* n) { ++*asked; *n = answers[i]; return errors[i]; }, &out[i]);
  }
}
extern "C" int gemm_rows(long long call_tiles, long long m, int sms) { return turq::plan_gemm_rows(call_tiles, m, sms); }
extern "C" int batch_tile(long long tiles, long long call_tiles, long long m, int sms) {
  return turq::plan_batch_tile(tiles, call_tiles, m, sms);
}
"""


@pytest.fixture(scope="module")
def lib():
    with tempfile.TemporaryDirectory() as d:
        src, so = os.path.join(d, "shim.cpp"), os.path.join(d, "shim.so")
        open(src, "w").write(SHIM)
        subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "tur_b200", "csrc"), src, "-o", so], check=True)
        lib = ctypes.CDLL(so)
        lib.gemm_rows.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int]
        lib.batch_tile.argtypes = [ctypes.c_longlong] * 3 + [ctypes.c_int]
        lib.prep_cluster.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int]
        yield lib


@pytest.fixture(scope="module")
def cluster(lib):
    def call(n, k):
        return lib.batch_cluster(-(-n // 128), -(-k // 256))
    return call


def test_every_cta_has_units(cluster):
    for n in (1, 128, 129, 640, 2560, 4096, 5120, 12288, 25600, 151936):
        for k in (64, 256, 320, 512, 768, 1024, 2560, 4096, 6144, 8192, 25600):
            c = cluster(n, k)
            assert 1 <= c <= 6 and c <= -(-k // 256), (n, k, c)
            ku = -(-k // 256)
            shares = [ku * (r + 1) // c - ku * r // c for r in range(c)]
            assert min(shares) >= 1 and sum(shares) == ku


@pytest.mark.parametrize("n,k,want", [(28672, 8192, 2), (3584, 18944, 4), (3072, 8192, 5)])
def test_cluster_sizes_do_not_follow_the_device(cluster, n, k, want):
    """Shapes whose size was another one where the device held 48, 36, 28, 24 clusters of 3 to 6 CTAs instead of 45, 33, 26, 22:
    the size cuts the K loop, so the bits of 17 to 64 rows went with the device. The rule has no such argument now."""
    assert cluster(n, k) == want


def test_a_failed_question_to_the_device_is_returned_and_asked_again(lib):
    asked, status, out = ctypes.c_int(0), (ctypes.c_int * 3)(), (ctypes.c_int * 3)()
    lib.ask_three_times((ctypes.c_int * 3)(37, 33, 44), (ctypes.c_int * 3)(1, 0, 0), ctypes.byref(asked), status, out)
    assert list(status) == [1, 0, 0] and list(out) == [-1, 33, 33] and asked.value == 2


@pytest.mark.parametrize("n,k,want", [(8192, 2560, 1), (12288, 4096, 2), (25600, 5120, 1), (3072, 1024, 2), (4096, 4096, 4), (2560, 2560, 4),
                                      (5120, 25600, 3), (5120, 8192, 3), (2560, 8192, 6), (1024, 2048, 4)])
def test_measured_choices(cluster, n, k, want):
    assert cluster(n, k) == want


@pytest.mark.parametrize("hidden,q,kv", [(1024, 2048, 1024), (2560, 2560, 640), (4096, 4096, 1024), (5120, 8192, 1024), (4096, 4096, 4096)])
def test_projections_of_a_layer_share_a_launch(cluster, hidden, q, kv):
    assert cluster(q, hidden) == cluster(kv, hidden)


@pytest.mark.parametrize("rows,m,tiles", [((4096, 1024, 1024), 512, 3), ((4096,), 512, 4), ((12288, 12288), 512, 2), ((2560, 640, 640), 1000, 4),
                                          ((2560,), 1000, 7), ((8192, 8192), 1000, 4), ((4096,), 2048, 9), ((12288, 12288), 2048, 8),
                                          ((5120,), 4096, 18), ((25600, 25600), 4096, 16), ((12288, 12288), 128, 1),
                                          # a last wave that is nearly empty costs less than a whole one
                                          ((8192, 8192), 1300, 6), ((8192, 8192), 1500, 6), ((12288, 12288), 1700, 7), ((12288,), 1700, 7),
                                          ((25600,), 768, 3), ((13824, 13824), 700, 3), ((28672,), 1300, 6), ((1024,), 1300, 17)])
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
    def tile(n, m, sms=148):
        return lib.batch_tile(-(-n // 128), -(-n // 256), m, sms)
    for n in (0, 1, 128, 1000, 4096, 25600, 151936, 2 ** 31):
        for m in (1, 64, 65, 66, 127, 128, 129, 511, 1000, 1024, 1025, 8192):
            for sms in (148, 16, 1):
                bn = tile(n, m, sms)
                assert bn == 0 or (bn % 16 == 0 and 16 <= bn <= 128 and 64 < m <= 1024), (n, m, bn)
    assert tile(0, 128) == 0
    for n, m in ((4096, 65), (4096, 128), (4096, 512), (2560, 768), (12288, 128), (12288, 384), (1024, 1000), (25600, 65)):
        assert tile(n, m) > 0, (n, m)
    for n, m in ((4096, 1000), (12288, 768), (25600, 256), (25600, 512), (151936, 512)):
        assert tile(n, m) == 0, (n, m)


def test_rows_are_converted_by_clusters_where_they_are_long_and_few(lib):
    """Clusters that all fit the GPU at once, none for rows that four CTAs' worth of registers hold or for prompts (25600 values: 177
    us a call of 4096 rows without, 265 with them)."""
    for m in (1, 32, 64, 65, 96, 105, 106, 128, 148, 149, 512, 1024, 4096, 2 ** 30):
        for k in (64, 4096, 16384, 16448, 17408, 25600, 32768, 49152, 2 ** 31 - 64):
            for sms in (148, 16, 1):
                c = lib.prep_cluster(m, k, sms)
                assert 1 <= c <= 8 and (c == 1 or (k > 16384 and c == min(8, -(-k // 4096)) and m * c <= 5 * sms)), (m, k, sms, c)
    for m, k, c in ((32, 25600, 7), (96, 25600, 7), (128, 25600, 1), (4096, 25600, 1), (64, 17408, 5), (256, 17408, 1), (64, 49152, 8), (64, 16384, 1)):
        assert lib.prep_cluster(m, k, 148) == c, (m, k)
