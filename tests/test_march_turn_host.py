"""Rounding of the marched frame, compiled for the host: the RK4 calls of a chain of slices at single points (no
diffraction), by the scaled and turning fields and by the fields themselves with the slice's coupling
constants, each against the same map in doubles. The turn from slice to slice has to add no error of
its own: two roundings of the SH per slice either way. (Turned and rounded by itself, the SH's error is
1.10 to 1.31 times the other form's.)"""
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
#include <complex>
#include <cstdio>
#include <random>
template <class T> T __ldg(const T *p) { return *p; }
inline void __syncthreads() {}
inline void __syncwarp() {}
#include "shg_march.cuh"
using namespace shg;
typedef std::complex<double> Z;

// one RK4 call of the coupled equations in doubles, fields themselves
static void call(Z &P, Z &S, Z a, Z b, double hp, double hs, double dz) {
    auto f = [&](Z p, Z s, Z &kp, Z &ks) { kp = a * s * std::conj(p) - hp * p, ks = b * p * p - hs * s; };
    Z p1, s1, p2, s2, p3, s3, p4, s4;
    f(P, S, p1, s1), f(P + 0.5 * p1, S + 0.5 * s1, p2, s2), f(P + 0.5 * p2, S + 0.5 * s2, p3, s3), f(P + p3, S + s3, p4, s4);
    P += dz / 6 * (p1 + 2.0 * p2 + 2.0 * p3 + p4);
    S += dz / 6 * (s1 + 2.0 * s2 + 2.0 * s3 + s4);
}

int main() {
    std::mt19937_64 gen(5);
    std::normal_distribution<double> nrm;
    int bad = 0;
    for (const double step : {0.004, 0.03, 0.2, -0.03}) {
        InstDesc d{};
        d.kp = d.ks = 0x1p-17f;  // scales of 2^-17: exact
        d.sp = d.ss = 0x1p-17f, d.isp = d.iss = 0x1p17f;
        d.hp = 1e-6f, d.tpa0 = 2e-6f, d.tpa1 = d.tpa1s = 0.0f;
        d.dz6 = 75.0f / 6.0f;
        const int K = 200;
        double turned = 0, plain = 0;
        for (int i = 0; i < 3000; ++i) {
            float2 P = make_float2(4.0 * nrm(gen), 4.0 * nrm(gen)), S = make_float2(nrm(gen), nrm(gen));
            Z zp(P.x, P.y), zs(S.x, S.y);
            float2 p = P, s = S;
            march_enter(p, s, d);
            float4 c{};
            float before = 0.0f;
            for (int k = 0; k < K; ++k) {
                const float arg = (float)k * 75.0f * (float)(step / 75.0), turn = arg - before;
                before = arg;
                const double h = std::sin(0.5 * turn);
                c = make_float4(-2.0 * h * h, std::sin((double)turn), std::cos((double)arg), std::sin((double)arg));
                if (k == 0) rk4_march(p, s, d);
                else rk4_turned(p, s, c, d);
                rk4_march(p, s, d);
                const float4 q = make_float4(d.kp * std::sin(arg), d.kp * std::cos(arg), -d.ks * std::sin(arg), d.ks * std::cos(arg));
                const Z e = std::polar(1.0, -(double)arg), I(0, 1);
                for (int two = 0; two < 2; ++two) {
                    rk4_point(P, S, q, d);
                    call(zp, zs, I * (double)d.kp * e, I * (double)d.ks * std::conj(e), d.hp, d.tpa0, 6.0 * d.dz6);
                }
            }
            march_leave(p, s, c, d);
            turned += std::norm(Z(s.x, s.y) - zs) / std::norm(zs);
            plain += std::norm(Z(S.x, S.y) - zs) / std::norm(zs);
        }
        const double r = std::sqrt(turned / plain);
        std::printf("turn %g: error of the SH %.3e, untouched fields %.3e, ratio %.3f\n", step, std::sqrt(turned / 3000),
                    std::sqrt(plain / 3000), r);
        bad += !(r < 1.1);
    }
    return bad;
}
"""


def test_turning_frame_adds_no_rounding(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("no host compiler or CUDA headers")
    src, exe = tmp_path / "turn.cpp", tmp_path / "turn"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", CUDA_INCLUDE, "-I", CSRC, "-o", str(exe), str(src)],
                   check=True, capture_output=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
