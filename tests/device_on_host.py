"""Compiles device headers of ibtfo_gb300/csrc for the host: the same
expressions in IEEE arithmetic, with the hardware's FP32 estimates stood in for
by rounded values and its rare-argument operations by the host's own."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = r"""
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>
#include <vector>
#include <cuda_runtime.h>
#include <cuda.h>
#define IBTFO_DEVICE static inline
#ifndef __noinline__
#define __noinline__
#endif
#define asm(...) y = 1 / x
static inline long long __double_as_longlong(double x) { long long i; memcpy(&i, &x, 8); return i; }
static inline double __longlong_as_double(long long i) { double x; memcpy(&x, &i, 8); return x; }
static inline int __double2hiint(double x) { return (int)((unsigned long long)__double_as_longlong(x) >> 32); }
static inline int __double2loint(double x) { return (int)__double_as_longlong(x); }
static inline double __hiloint2double(int h, int l) { return __longlong_as_double((long long)((unsigned long long)(unsigned)h << 32 | (unsigned)l)); }
namespace ibtfo {
IBTFO_DEVICE uint64_t double_bits(double x) { uint64_t i; memcpy(&i, &x, 8); return i; }
IBTFO_DEVICE double bits_double(uint64_t i) { double x; memcpy(&x, &i, 8); return x; }
IBTFO_DEVICE uint32_t float_bits(float x) { uint32_t i; memcpy(&i, &x, 4); return i; }
IBTFO_DEVICE float bits_float(uint32_t i) { float x; memcpy(&x, &i, 4); return x; }
IBTFO_DEVICE float rcp_estimate(float x) { return 1.0f / x; }
IBTFO_DEVICE float rsqrt_estimate(float x) { return (float)(1.0 / sqrt((double)x)); }
IBTFO_DEVICE int round_int(float x) { return (int)rintf(x); }
IBTFO_DEVICE uint64_t mul_high(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a * b) >> 64); }
IBTFO_DEVICE double divide_hardware(double a, double b) { return a / b; }
IBTFO_DEVICE double sqrt_hardware(double x) { return sqrt(x); }
IBTFO_DEVICE double sqrt_rn(double x) { return sqrt(x); }
IBTFO_DEVICE double widen_hardware(float f) { return (double)f; }
IBTFO_DEVICE float2 split_hardware(double v) { const float h = (float)v; return float2{h, (float)(v - (double)h)}; }
}
"""


def build(folder, program, *flags):
    """PRELUDE + program, compiled into `folder`."""
    cxx, nvcc = shutil.which("g++"), shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not cxx or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no host compiler or CUDA headers")
    src, exe = folder / "t.cpp", folder / "t"
    src.write_text(PRELUDE + program)
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-w", *flags, "-I", cuda, "-I",
                    os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "ibtfo_gb300", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    return str(exe)


def run(exe, *args):
    return subprocess.run([exe, *map(str, args)], stdout=subprocess.PIPE, check=True).stdout
