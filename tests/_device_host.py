"""The device arithmetic of ``solvcon_gb300/csrc`` compiled for the host, so
that its very source can be compared with exact arithmetic without a GPU.

The headers are taken as they are but for the two approximate instructions
that only the GPU has: ``seed_rcp`` and ``seed_rsqrt`` stand for them, the
correctly rounded FP32 value moved by a given number of FP32 ulps."""

import ctypes
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "solvcon_gb300", "csrc")

SHIM = r"""
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
using std::max;
using std::min;
inline int seed_shift = 0;
template <typename T, typename F> T bits_as(F f)
{
    static_assert(sizeof(T) == sizeof(F), "size");
    T t;
    std::memcpy(&t, &f, sizeof(t));
    return t;
}
inline float __uint_as_float(unsigned u) { return bits_as<float>(u); }
inline unsigned __float_as_uint(float f) { return bits_as<unsigned>(f); }
inline double __longlong_as_double(long long b) { return bits_as<double>(b); }
inline long long __double_as_longlong(double d) { return bits_as<long long>(d); }
inline int __double2hiint(double d) { return static_cast<int>(__double_as_longlong(d) >> 32); }
inline int __double2loint(double d) { return static_cast<int>(__double_as_longlong(d)); }
inline double __hiloint2double(int hi, int lo)
{
    return __longlong_as_double((static_cast<long long>(hi) << 32) | static_cast<unsigned>(lo));
}
inline unsigned __umulhi(unsigned a, unsigned b) { return static_cast<unsigned>(static_cast<uint64_t>(a) * b >> 32); }
inline int __clzll(long long v) { return v == 0 ? 64 : __builtin_clzll(static_cast<unsigned long long>(v)); }
inline unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned s) { return hi << s | lo >> (32 - s); }
inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double rsqrt(double x) { return 1.0 / std::sqrt(x); }
inline float rsqrtf(float x) { return static_cast<float>(1.0 / std::sqrt(static_cast<double>(x))); }
inline float __fdividef(float a, float b) { return a / b; }
template <typename T> inline T __ldg(T const * p) { return *p; }
struct double2 { double x, y; };
inline double2 make_double2(double x, double y) { return {x, y}; }
inline float seed_rcp(float x) { return __uint_as_float(__float_as_uint(1.0f / x) + seed_shift); }
inline float seed_rsqrt(float x) { return __uint_as_float(__float_as_uint(rsqrtf(x)) + seed_shift); }
"""

SEED = re.compile(r'asm\("(\w+)\.approx\.ftz\.f32 %0, %1;" : "=f"\((\w+)\) : "f"\((.*)\)\);')


def library(tmp_path, code, headers=("divide.cuh",)):
    """A shared library of ``code``, which includes the given headers."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = str(tmp_path)
    for name in ("divide.cuh", "euler_device.cuh", "euler_fp64.cuh"):
        with open(os.path.join(CSRC, name)) as f:
            text, count = SEED.subn(r"\2 = seed_\1(\3);", f.read())
        if name == "divide.cuh":
            assert count == 2 and "asm" not in text
        with open(os.path.join(src, name), "w") as f:
            f.write(text)
    with open(os.path.join(src, "cuda_runtime.h"), "w") as f:
        f.write(SHIM)
    main = os.path.join(src, "main.cpp")
    with open(main, "w") as f:
        f.write("".join('#include "%s"\n' % h for h in headers) + code +
                '\nextern "C" void set_seed_shift(int s) { seed_shift = s; }\n')
    out = os.path.join(src, "main.so")
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC",
                    "-shared", "-I" + src, main, "-o", out], check=True)
    return ctypes.CDLL(out)
