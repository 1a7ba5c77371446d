"""The launch arithmetic of tur_b200/csrc/launch_plan.h for tests that claim which kernel a case reaches: compiled with g++, asked
with the SM count of a B200."""
import ctypes
import os
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMS = 148
SHIM = r"""
#include "launch_plan.h"
extern "C" int batch_cluster(int tiles, int KU) { return turq::plan_batch_cluster(tiles, KU); }
extern "C" int batch_tile(long long tiles, long long call_tiles, long long m, int sms) { return turq::plan_batch_tile(tiles, call_tiles, m, sms); }
extern "C" int gemm_rows(long long call_tiles, long long m, int sms) { return turq::plan_gemm_rows(call_tiles, m, sms); }
"""
_lib = None


def _load():
    global _lib
    if _lib is None:
        with tempfile.TemporaryDirectory() as d:
            src, so = os.path.join(d, "shim.cpp"), os.path.join(d, "shim.so")
            with open(src, "w") as f:
                f.write(SHIM)
            subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "tur_b200", "csrc"), src, "-o", so], check=True)
            _lib = ctypes.CDLL(so)
            _lib.batch_tile.argtypes = [ctypes.c_longlong] * 3 + [ctypes.c_int]
            _lib.gemm_rows.argtypes = [ctypes.c_longlong] * 2 + [ctypes.c_int]
    return _lib


def cluster(n, k):
    """CTAs that share the K loop of a decode batch."""
    return _load().batch_cluster(-(-n // 128), -(-k // 256))


def tile(ns, m):
    """Activation rows of a tile where a call of these weights goes to the decode-batch kernel in tiles, else 0."""
    return _load().batch_tile(sum(-(-n // 128) for n in ns), sum(-(-n // 256) for n in ns), m, SMS)


def pair_rows(ns, m):
    """Activation rows of a pair tile of the prefill kernel."""
    return _load().gemm_rows(sum(-(-n // 256) for n in ns), m, SMS)


def kernel(ns, m):
    """batch: decode-batch kernel, K loops shared; tiles: the same kernel, short prompts; pairs: prefill kernel."""
    return "batch" if m <= 64 else "tiles" if tile(ns, m) else "pairs"
