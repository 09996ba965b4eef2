"""Positions of buckets in a list whose total exceeds 2^31 - 1 (bucket_math.h,
compiled for the host): they saturate, every bucket's range stays inside the
list, and a list that fits is unaffected."""
import ctypes
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "universal-beta-splatting_gb300", "csrc")
SRC = """
#include "bucket_math.h"
extern "C" int32_t start(int64_t at) { return ubs::bucket_start(at); }
extern "C" int32_t scan32(int64_t v) { return ubs::scan_value<int32_t>(v); }
extern "C" int64_t scan64(int64_t v) { return ubs::scan_value<int64_t>(v); }
extern "C" void bounds(int32_t s, int32_t e, int64_t T, int64_t *lo, int64_t *hi) {
    ubs::bucket_bounds(s, e, T, *lo, *hi);
}
"""
MAX = 2 ** 31 - 1


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("bucket_math")
    (d / "m.cpp").write_text(SRC)
    subprocess.run(["g++", "-shared", "-fPIC", "-std=c++17", "-I", CSRC, str(d / "m.cpp"), "-o",
                    str(d / "m.so")], check=True)
    L = ctypes.CDLL(str(d / "m.so"))
    for f in (L.start, L.scan32, L.scan64):
        f.argtypes = [ctypes.c_int64]
    L.start.restype = L.scan32.restype = ctypes.c_int32
    L.scan64.restype = ctypes.c_int64
    L.bounds.argtypes = [ctypes.c_int32, ctypes.c_int32, ctypes.c_int64] + [
        ctypes.POINTER(ctypes.c_int64)] * 2
    return L


def _range(L, s, e, T):
    lo, hi = ctypes.c_int64(), ctypes.c_int64()
    L.bounds(s, e, T, ctypes.byref(lo), ctypes.byref(hi))
    return lo.value, hi.value


@pytest.mark.parametrize("per_bucket, buckets", [(3, 1000), (1_000_000, 8160), (MAX, 5),
                                                 (2 ** 30, 8), (70_000, 65_536)])
def test_every_bucket_stays_in_the_list(lib, per_bucket, buckets):
    rng = random.Random(per_bucket)
    counts = [rng.randint(0, per_bucket) for _ in range(buckets)]
    exact, at = [], 0
    for c in counts:
        exact.append(at)
        at += c
    stored = [lib.start(x) for x in exact]
    assert stored == [min(x, MAX) for x in exact]
    assert [lib.scan32(x) for x in exact] == stored and lib.scan64(at) == at
    for cap in (1 << 16, 100_000_000, MAX):
        T = min(at, cap)
        for b in range(0, buckets, max(1, buckets // 500)):
            end = stored[b + 1] if b + 1 < buckets else MAX
            assert _range(lib, stored[b], end, T) == (min(exact[b], T), min(exact[b] + counts[b], T))


def test_any_stored_word_gives_a_range_of_the_list(lib):
    words = [-2 ** 31, -1, 0, 1, 1000, MAX - 1, MAX]
    for T in (0, 1, 500, MAX):
        for s in words:
            for e in words:
                lo, hi = _range(lib, s, e, T)
                assert 0 <= lo <= hi <= T


def test_cursors_of_a_bucket_stay_at_the_end(lib):
    # replica cursors: the bucket's start plus the counts before the replica
    o, got = lib.start(MAX - 10), []
    for c in [7, 7, 2 ** 30, 5]:
        got.append(o)
        o = lib.start(o + c)
    assert got == [MAX - 10, MAX - 3, MAX, MAX] and o == MAX
