"""The FP64 <-> FP32 conversions by integer arithmetic (bcfd_convert.cuh),
compiled for the host, against the casts: bit for bit, at rounding ties in both
directions, where the rounding carries into the exponent, at the ends of FP32's
range, for subnormals, zeros of both signs, infinities and NaN, and for random
bit patterns of every exponent."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "bio-cfd_gb300" / "csrc"
SHIM = r"""
#include <cstdint>
#include <cstring>
#define __device__
#define __forceinline__ inline
template <class T, class F> static T cast(F x) { T r; static_assert(sizeof(T) == sizeof(F), ""); std::memcpy(&r, &x, sizeof r); return r; }
static int __double2hiint(double x) { return (int)(cast<uint64_t>(x) >> 32); }
static int __double2loint(double x) { return (int)(uint32_t)cast<uint64_t>(x); }
static double __hiloint2double(int h, int l) { return cast<double>((uint64_t)(uint32_t)h << 32 | (uint32_t)l); }
static unsigned __float_as_uint(float x) { return cast<unsigned>(x); }
static float __uint_as_float(unsigned x) { return cast<float>(x); }
#include "bcfd_convert.cuh"
extern "C" void to_f32s(const double* x, float* y, int64_t n) { for (int64_t i = 0; i < n; ++i) y[i] = bcfd::to_f32(x[i]); }
extern "C" void to_f64s(const float* x, double* y, int64_t n) { for (int64_t i = 0; i < n; ++i) y[i] = bcfd::to_f64(x[i]); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("convert")
    (d / "shim.cpp").write_text(SHIM)
    so = d / "convert.so"
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC), str(d / "shim.cpp"),
                           "-o", str(so)])
    return ctypes.CDLL(str(so))


def _equal(got, ref, bits):
    nan = np.isnan(ref)
    np.testing.assert_array_equal(np.isnan(got), nan)
    np.testing.assert_array_equal(got.view(bits)[~nan], ref.view(bits)[~nan])


def test_to_f32(lib):
    rng = np.random.default_rng(7)
    f = np.frombuffer(rng.bytes(4 * 400_000), np.uint32).view(np.float32)
    f = np.concatenate([f, np.float32([0, 1, 2 ** -126, 2 ** -127, 2 ** -149, np.finfo(np.float32).max, 3.4e38])])
    f = np.abs(f[np.isfinite(f)])
    with np.errstate(over="ignore"):
        up = np.nextafter(f, np.float32(np.inf)).astype(np.float64)
    up[np.isinf(up)] = 2.0 ** 128
    low = f.astype(np.float64)
    tie = 0.5 * (low + up)  # exact; half of them round down, half up, some into the next exponent
    x = np.concatenate([low, tie, np.nextafter(tie, 0), np.nextafter(tie, np.inf),
                        np.frombuffer(rng.bytes(8 * 1_000_000), np.uint64).view(np.float64),
                        rng.normal(size=200_000) * 2.0 ** rng.integers(-160, 140, 200_000),
                        [0.0, np.inf, np.nan, 2.0 ** 128, 2.0 ** 128 - 2.0 ** 103, 2.0 ** -150, 5e-324, 1.7e308]])
    x = np.concatenate([x, -x])
    y = np.empty(x.size, np.float32)
    lib.to_f32s(x.ctypes.data_as(ctypes.c_void_p), y.ctypes.data_as(ctypes.c_void_p), ctypes.c_int64(x.size))
    with np.errstate(over="ignore", invalid="ignore", under="ignore"):
        _equal(y, x.astype(np.float32), np.uint32)


def test_to_f64(lib):
    exponents = np.arange(512, dtype=np.uint32) << 23  # both signs
    mantissas = np.uint32([0, 1, 2, 3, 7, 8, 0x400000, 0x7ffff8, 0x7ffffe, 0x7fffff])
    x = (exponents[:, None] | mantissas).ravel().view(np.float32)
    x = np.concatenate([x, np.frombuffer(np.random.default_rng(8).bytes(4 * 1_000_000), np.uint32).view(np.float32)])
    y = np.empty(x.size, np.float64)
    lib.to_f64s(x.ctypes.data_as(ctypes.c_void_p), y.ctypes.data_as(ctypes.c_void_p), ctypes.c_int64(x.size))
    with np.errstate(invalid="ignore"):
        _equal(y, x.astype(np.float64), np.uint64)
