"""The divisions by constants of the ray caster (csrc/exact_math.cuh) over the range
that the header states for them, on the CPU: quotients equal the IEEE division from
kDivExactLowest on, and the smallest samples lie above it."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cmath>
#include <cstdint>
#include <cstring>
#define __device__
#define __forceinline__ inline
static inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
static inline float __fmul_rn(float a, float b) { return a * b; }
#include "exact_math.cuh"
template <uint32_t D>
static long wrong(int e, uint32_t step) {
    long n = 0;
    for (uint32_t m = 0; m < (1u << 23); m += step) {
        const uint32_t b = static_cast<uint32_t>(127 + e) << 23 | m;
        float x;
        std::memcpy(&x, &b, 4);
        volatile float d = static_cast<float>(D);
        n += gc::div_exact<D>(x) != x / d;
    }
    return n;
}
extern "C" long wrong_quotients(uint32_t d, int e, uint32_t step) {
    return d == 255 ? wrong<255>(e, step) : d == 65535 ? wrong<65535>(e, step)
         : d == 2040 ? wrong<2040>(e, step) : wrong<524280>(e, step);
}
extern "C" float lowest() { return gc::kDivExactLowest; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact_math")
    src, so = d / "range.cpp", d / "librange.so"
    src.write_text(SOURCE)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                        os.path.join(ROOT, "gpu-out-of-core-volume-data_gb300", "csrc"), str(src), "-o", str(so)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(str(so))
    lib.wrong_quotients.restype = ctypes.c_long
    lib.lowest.restype = ctypes.c_float
    return lib


@pytest.mark.parametrize("d", [255, 65535, 2040, 524280])
def test_quotients_from_the_stated_bound_on(lib, d):
    bound = lib.lowest()
    e = -140
    while 2.0 ** e < bound:
        e += 1
    for exponent in (e, e + 1, -72, -48, -24, 0, 19):
        assert lib.wrong_quotients(d, exponent, 37) == 0, exponent


def test_smallest_sample_lies_above_the_bound(lib):
    # one step between two voxels at the smallest weight on each of the three axes
    assert 0.0 < lib.lowest() <= 2.0 ** -72


def test_the_bound_is_needed(lib):
    """Far below it quotients do come out wrong, so the bound is no formality."""
    assert lib.wrong_quotients(524280, -110, 37) > 0
