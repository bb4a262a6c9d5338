"""The heat sweep's edge formula in pairs of floats (edge_round) against the doubles it stands for, compiled
for the host: (float)(((double)s + K) D) bit for bit over magnitudes from the smallest denormal to the
largest, both signs, K zero, tiny, ordinary and close to -s, and factors D as the faces have them."""
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

int main() {
    std::mt19937_64 gen(3);
    std::uniform_real_distribution<double> mant(1.0, 2.0), dfac(0.05, 1.0);
    auto value = [&](int e) { return (float)std::ldexp((gen() & 1 ? 1.0 : -1.0) * mant(gen), e); };
    long bad = 0, n = 0;
    for (int e = -149; e <= 126; ++e)
        for (int i = 0; i < 40000; ++i) {
            const float s = value(e), D = (float)dfac(gen);
            double K = 0.0;
            switch (i & 7) {
                case 0: case 1: case 2: break;                                  // T_inf = 0
                case 3: K = value(std::max(-149, e - (int)(gen() % 40))); break;  // below s
                case 4: K = 0.5 * 25.0 * (double)value(-8); break;                // as faces have it
                case 5: K = -(double)s * (1.0 + std::ldexp(mant(gen), -(int)(gen() % 40))); break;
                case 6: K = value(std::min(126, e + (int)(gen() % 40))); break;
                case 7: K = 1e-3 * (double)s; break;
            }
            const float kh = (float)K, kl = (float)(K - (double)kh);
            const float want = (float)(((double)s + K) * (double)D), got = edge_round(s, K, kh, kl, D);
            ++n;
            if (std::memcmp(&want, &got, 4) != 0 && ++bad <= 5)
                std::printf("s=%a K=%a D=%a: %a, not %a\n", s, K, D, got, want);
        }
    for (float s : {0.0f, -0.0f, INFINITY, -INFINITY})
        for (double K : {0.0, 1.0, -1.0}) {
            const float want = (float)(((double)s + K) * 0.25), got = edge_round(s, K, (float)K, 0.0f, 0.25f);
            ++n;
            if (std::memcmp(&want, &got, 4) != 0 && ++bad <= 12) std::printf("s=%a K=%a: %a, not %a\n", s, K, got, want);
        }
    std::printf("%ld of %ld differ\n", bad, n);
    return bad != 0;
}
"""


def test_edge_round_is_the_double_formula(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("no host compiler or CUDA headers")
    src, exe = tmp_path / "edge.cpp", tmp_path / "edge"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", CUDA_INCLUDE, "-I", CSRC, "-o", str(exe), str(src)],
                   check=True, capture_output=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
