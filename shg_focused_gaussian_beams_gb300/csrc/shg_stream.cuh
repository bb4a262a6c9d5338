// Row and column pass of the plain march on fields in global memory: the bodies of the streaming
// launches (k_rows, k_cols in shg_march.cu) and of the persistent groups (k_march_group in
// shg_group.cu), which therefore give the same fields bit for bit.
#pragma once

#include <cuda_runtime.h>

#include "shg_march.cuh"

namespace shg {

__device__ __forceinline__ void block_add_double(double v, double *dst) {
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
        v = (l < (int)(blockDim.x >> 5)) ? red[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (l == 0 && v != 0.0) atomicAdd(dst, v);
    }
}

// A field value; from L2 (CG) where another SM wrote it earlier in the same launch.
template <bool CG>
__device__ __forceinline__ float2 ld_field(const float2 *p) {
    return CG ? __ldcg(p) : *p;
}

// Row pass. Block = 256 threads = 256/G lines of one solve; mode from the stage s:
//   s == 0           : RK4(z_0), backward transform along x, store in frequency order;
//   0 < s < nsteps   : forward transform along x, RK4(z_{s-1}), RK4(z_s), backward;
//   s == nsteps      : forward transform along x, RK4(z_{s-1}), capture, power sums.
template <int N>
struct RowShape {
    static constexpr int G = LineShape<N>::G;
    static constexpr int TPB = (N * G < 256) ? N * G : 256;  // threads per block
    static constexpr int LPB = TPB / G;                      // lines per block
    static constexpr int BPI = N / LPB;                      // blocks per solve
};

// CG: the persistent groups' form (fields read from L2, tab a copy of the split's twiddle pairs
// in shared memory).
template <int N, bool CG = false>
__device__ __forceinline__ void rows_body(const InstDesc &d, int line, int t, int s, float2 *sc, const float2 *tab) {
    constexpr int G = LineShape<N>::G, E = N / G;
    constexpr size_t NN = (size_t)N * N;
    const size_t base = (size_t)line * N;
    float2 vp[E], vs[E];
#pragma unroll
    for (int j = 0; j < E; ++j) {
        vp[j] = ld_field<CG>(&SHG_AT(d.P, base + t + G * j, NN, kChkRowsGlobal));
        vs[j] = ld_field<CG>(&SHG_AT(d.S, base + t + G * j, NN, kChkRowsGlobal));
    }
    if (s == 0) {
#pragma unroll
        for (int j = 0; j < E; ++j) {
            march_enter(vp[j], vs[j], d);
            rk4_march(vp[j], vs[j], d);
        }
        fft_nat_to_spec<N, G, +1, false, 1, G + 1, CG>(vp, t, sc, tab);
        fft_nat_to_spec<N, G, +1, false, 1, G + 1, CG>(vs, t, sc, tab);
#pragma unroll
        for (int r = 0; r < E; ++r) {
            const int k = spec_index<N, G>(t, r);
            SHG_AT(d.P, base + k, NN, kChkRowsGlobal) = vp[r];
            SHG_AT(d.S, base + k, NN, kChkRowsGlobal) = vs[r];
        }
        return;
    }
    fft_nat_to_spec<N, G, -1, false, 1, G + 1, CG>(vp, t, sc, tab);
    fft_nat_to_spec<N, G, -1, false, 1, G + 1, CG>(vs, t, sc, tab);
    const float4 c1 = d.stepc[s - 1];
#pragma unroll
    for (int r = 0; r < E; ++r) rk4_march(vp[r], vs[r], d);
    if (d.slices && s < d.nz) {
        float2 *sl = d.slices + (size_t)s * 2 * N * N;
#pragma unroll
        for (int r = 0; r < E; ++r) {
            const int k = spec_index<N, G>(t, r);
            float2 op = vp[r], os = vs[r];
            march_leave(op, os, c1, d);
            SHG_AT(sl, base + k, 2 * NN, kChkSlices) = op;
            SHG_AT(sl, NN + base + k, 2 * NN, kChkSlices) = os;
        }
    }
    if (s == d.nsteps) {
        double aS = 0.0, aP = 0.0;
#pragma unroll
        for (int r = 0; r < E; ++r) {
            const int k = spec_index<N, G>(t, r);
            march_leave(vp[r], vs[r], c1, d);
            SHG_AT(d.Pout, base + k, NN, kChkRowsGlobal) = vp[r];
            SHG_AT(d.Sout, base + k, NN, kChkRowsGlobal) = vs[r];
            aS += (double)vs[r].x * vs[r].x + (double)vs[r].y * vs[r].y;
            aP += (double)vp[r].x * vp[r].x + (double)vp[r].y * vp[r].y;
        }
        block_add_double(aS, d.acc + 1);
        block_add_double(aP, d.acc + 2);
        return;
    }
    const float4 c2 = d.stepc[s];
#pragma unroll
    for (int r = 0; r < E; ++r) {
        march_turn(vs[r], c2);
        rk4_march(vp[r], vs[r], d);
    }
    fft_spec_to_nat<N, G, +1, false, 1, G + 1, CG>(vp, t, sc, tab);
    fft_spec_to_nat<N, G, +1, false, 1, G + 1, CG>(vs, t, sc, tab);
#pragma unroll
    for (int j = 0; j < E; ++j) {
        SHG_AT(d.P, base + t + G * j, NN, kChkRowsGlobal) = vp[j];
        SHG_AT(d.S, base + t + G * j, NN, kChkRowsGlobal) = vs[j];
    }
}

// The column pass of k_cols for column x of field f (0 pump, 1 SH) of solve d, lane t of the
// column's G lanes; the TC columns of a group transpose through sc (interleaved, stride TC)
// and synchronise the block (BS) or, when the group is one warp, the warp.
struct NoWait {
    __device__ void operator()() const {}
};
template <int N, int TC, bool BS, bool CG = false, class Wait = NoWait>
__device__ __forceinline__ void cols_body(const InstDesc &d, int x, int f, int t, float2 *sc, const float2 *tab,
                                          Wait wait = Wait()) {
    constexpr int G = LineShape<N>::G, E = N / G;
    float2 *F = f == 0 ? d.P : d.S;
    const float2 *__restrict__ H = f == 0 ? d.Hp : d.Hs;
    constexpr size_t NN = (size_t)N * N;
    // propagator values first: their latency overlaps the transform
    float2 h[E];
    hprop_load<N>(H, x, t, h);
    wait();
    float2 v[E];
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = ld_field<CG>(&SHG_AT(F, (size_t)(t + G * j) * N + x, NN, kChkColsGlobal));
    fft_nat_to_spec<N, G, +1, BS, TC, G, CG>(v, t, sc, tab);
#pragma unroll
    for (int r = 0; r < E; ++r) v[r] = c_mul(v[r], h[r]);
    fft_spec_to_nat<N, G, -1, BS, TC, G, CG>(v, t, sc, tab);
#pragma unroll
    for (int j = 0; j < E; ++j) SHG_AT(F, (size_t)(t + G * j) * N + x, NN, kChkColsGlobal) = v[j];
}

}  // namespace shg
