// Persistent cooperative grid of one solve: the bounded grid-wide barrier, the grid's
// row-unit / column-group shape and the column pass with the propagator values held in
// registers. Shared by the plain march (k_march_coop, shg_march.cu) and the THERMAL march
// (k_march_coop_th, shg_thermal.cu); the row passes are those of the streaming kernels
// with one thread per point, so a run gives their results bit for bit.
#pragma once

#include <cuda_runtime.h>

#include "shg_march.cuh"

namespace shg {

// Poll limit of a grid-barrier wait (about a second).
constexpr long long kGridWaitLimit = 1ll << 22;

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release_gpu(unsigned *p, unsigned v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Grid-wide barrier of a cooperative launch on a monotonic arrival counter (zeroed before
// the launch): barrier number e of the run completes once e * gridDim.x arrivals are in.
// Thread 0 of each block arrives with a release add (ordering the block's writes, which the
// block barrier made its own, before the arrival) and polls with acquire loads (ordering
// the other blocks' writes before this block's later loads). No reset step: a waiter reads
// one word. Every wait is bounded: on timeout `code` is or-ed into *err and false is
// returned (the caller leaves the kernel), and a wait also ends once *err is non-zero (looked at on
// every 32nd poll: read on each, it doubled the interval between polls; one 128 x 128 x 200 march
// 1.19 -> 1.13 ms without).
__device__ __forceinline__ bool grid_barrier(unsigned *count, unsigned target, int *err, int code = 1) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        red_release_gpu(count, 1u);
        int good = 1;
        for (long long it = 0; ld_acquire_gpu(count) < target; ++it) {
            if ((it & 31) != 31) continue;
            if (it >= kGridWaitLimit || *(volatile int *)err) {
                atomicOr(err, code);
                good = 0;
                break;
            }
            if (it >= 127) __nanosleep(1000);
        }
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

template <int N>
struct CoopShape {
    static constexpr int G = LineShape<N>::G, E = N / G;
    static constexpr int LPB = (512 / N < N) ? 512 / N : N;  // lines per row unit
    static constexpr int TPB = LPB * N;                     // one thread per point of a unit
    static constexpr int TC = 32 / G;                    // columns per column group
    static constexpr int ROW_UNITS = N / LPB;            // groups of LPB lines
    static constexpr int COL_UNITS = 2 * (N / TC);       // column groups of both fields
    // Columns of 16 x 8 points are split over two warps. Where both DFTs are of 16 points (N = 256) each warp of a
    // pair needs all inputs of both and the pair's outputs besides, which costs more than the shorter chain gives:
    // one 256 x 256 x 400 march 2.87 ms, split 3.16 (its THERMAL march in a run of two 12.7, 13.3); 128 x 128 x 200
    // 1.19, split 1.10 (3.73, 3.53).
    static constexpr bool SPLIT = RowLanes<N, true>::SPLIT && E != G;
    static constexpr int GW = SPLIT ? 2 : 1;             // warps of a column group
    static constexpr int OUT = E / GW;                   // spectrum values per thread
    static_assert(TC * G == 32, "a column group is one warp, two of split lanes");
};

// Column group of a block: TC columns of one field on one warp, or split on two (warp h of the pair
// computes the outputs 2 r + h; a named barrier of their own synchronises them). The columns'
// propagator values stay in registers for the whole run. Block b of B holds groups b, b + B, ...
template <int N>
struct CoopColumn {
    using C = CoopShape<N>;
    static constexpr int G = C::G, E = C::E, TC = C::TC, OUT = C::OUT;
    struct PairSync {
        int id;
        __device__ void operator()() const { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }
    };
    bool active;
    int g, h, f, x, t;
    __device__ CoopColumn(int block, int blocks, int groups) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        g = warp / C::GW;
        h = warp % C::GW;
        const int u = block + blocks * g;
        active = g < groups && u < C::COL_UNITS;
        f = u / (N / TC);
        x = (u % (N / TC)) * TC + lane % TC;
        t = lane / TC;
    }
    __device__ __forceinline__ void load(const InstDesc &d, float2 (&hp)[OUT]) const {
        const float2 *H = f == 0 ? d.Hp : d.Hs;
        if constexpr (C::SPLIT) split_hprop_load<N>(H, x, t, h, hp);
        else hprop_load<N>(H, x, t, hp);
    }
    // scr: TC * N float2 per group; tab: the split's twiddle pairs in shared memory
    __device__ __forceinline__ void run(const InstDesc &d, float2 *scr, const float2 (&hp)[OUT], const float2 *tab) const {
        float2 *const F = f == 0 ? d.P : d.S, *const sc = scr + (size_t)g * TC * N + threadIdx.x % TC;
        [[maybe_unused]] constexpr size_t NN = (size_t)N * N;
        float2 v[E];
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = SHG_AT(F, (size_t)(t + G * j) * N + x, NN, kChkCoop);
        if constexpr (C::SPLIT) {
            float2 o[OUT];
            column_split<N, TC, true>(v, o, t, h, sc, tab, PairSync{g + 1},
                                      [&](int r, float2 a) { return c_mul(a, hp[r]); });
#pragma unroll
            for (int r = 0; r < OUT; ++r) {
                const size_t y = SplitLine<N, G>::nat(t, h, r);
                SHG_AT(F, y * N + x, NN, kChkCoop) = o[r];
            }
        } else {
            fft_nat_to_spec<N, G, +1, false, TC, G, true>(v, t, sc, tab);
#pragma unroll
            for (int r = 0; r < E; ++r) v[r] = c_mul(v[r], hp[r]);
            fft_spec_to_nat<N, G, -1, false, TC, G, true>(v, t, sc, tab);
#pragma unroll
            for (int j = 0; j < E; ++j) SHG_AT(F, (size_t)(t + G * j) * N + x, NN, kChkCoop) = v[j];
        }
    }
};

}  // namespace shg
