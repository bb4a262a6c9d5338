"""Division of any numerator by a verified divisor (div_any) against IEEE division, compiled for the host: every
denormal of up to twelve bits and random numerators of every exponent, both signs, zeros, infinities,
for divisors the size of a grid spacing squared and of a face's denominator."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "shg_focused_gaussian_beams_gb300", "csrc")
CUDA_INCLUDE = "/usr/local/cuda/include"

PROGRAM = r"""
#include <cuda_runtime.h>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
template <class T> T __ldg(const T *p) { return *p; }
inline void __syncthreads() {}
inline void __syncwarp() {}
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fdiv_rn(float a, float b) { return a / b; }
inline float __fdividef(float a, float b) { return a / b; }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline float __double2float_rn(double a) { return (float)a; }
inline unsigned __float_as_uint(float a) { unsigned u; std::memcpy(&u, &a, 4); return u; }
inline float __uint_as_float(unsigned u) { float a; std::memcpy(&a, &u, 4); return a; }
#define __noinline__
#include "shg_thermal.cuh"
using namespace shg;

// The corrected product equals IEEE division on a whole binade of numerators (as the library
// establishes for each divisor before it is used).
static bool verified(float d, float r) {
    for (unsigned i = 0; i < (1u << 23); ++i) {
        const float a = __uint_as_float((127u << 23) + i), q = a * r;
        if (std::fma(std::fma(-q, d, a), r, q) != a / d) return false;
    }
    return true;
}

int main() {
    std::mt19937_64 gen(11);
    std::vector<float> divs = {1.0f, 3.0f, 0.75f, 90.702944f, 22500.0f, 1.0009766f, 2.6666667f};
    std::uniform_real_distribution<double> e(-19.0, 19.9);
    while (divs.size() < 14) divs.push_back((float)std::exp2(e(gen)));
    long bad = 0, n = 0, used = 0;
    for (float d : divs) {
        const float r = 1.0f / d;
        if (!verified(d, r)) continue;
        ++used;
        auto check = [&](float a) {
            const float want = a / d, got = div_any(a, d, r, 1);
            ++n;
            if (std::memcmp(&want, &got, 4) != 0 && !(want != want && got != got) && ++bad <= 10)
                std::printf("%a / %a: %a, not %a\n", a, d, got, want);
        };
        for (unsigned sign : {0u, 0x80000000u}) {
            for (unsigned i = 0; i < 4096; ++i)
                for (int k = 0; k < 23; ++k) check(__uint_as_float(sign | (i << k)));
            for (unsigned ex = 0; ex < 256; ++ex)
                for (int i = 0; i < 4000; ++i) check(__uint_as_float(sign | ex << 23 | (unsigned)(gen() & 0x7fffffu)));
            check(__uint_as_float(sign | 0x7f800000u));
        }
    }
    const float a = 3e-39f;  // without a verified divisor: IEEE division
    bad += div_any(a, 7.0f, 1.0f / 7.0f, 0) != a / 7.0f;
    bad += div_any(a, 0x1p30f, 0x1p-30f, 1) != a / 0x1p30f;
    std::printf("%ld of %ld differ, %ld divisors\n", bad, n, used);
    return bad != 0 || used < 10;
}
"""


def test_div_any_is_ieee_division(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("no host compiler or CUDA headers")
    src, exe = tmp_path / "div.cpp", tmp_path / "div"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", CUDA_INCLUDE, "-I", CSRC, "-o", str(exe), str(src)],
                   check=True, capture_output=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
