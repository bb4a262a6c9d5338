// Persistent groups: the plain march of a size class of a batch in one cooperative launch. The
// blocks form groups of BPI = N / LPB; a group takes solves of the class from a queue (longest
// first) and marches each with the streaming row and column passes (shg_stream.cuh, the same
// arithmetic), separated by barriers among its own blocks instead of kernel boundaries.
//
// Against the streaming launches a group never waits for the other groups' solves, so the row
// pass of one group (FMA issue) overlaps the column pass and barriers of the group that shares
// its SMs, and only the solves being marched are touched at a time: their fields and propagators
// stay in L2 (38 MB for 19 solves of 256 x 256), where the streaming passes go to HBM from about
// 60 such solves on. Against the cluster-resident march (shg_resident.cuh) columns cross SMs
// through L2 instead of distributed shared memory, which bounds that march from two CTAs per
// solve on (13 % fewer instructions left its 256 x 256 class at 78 ms), and every SM holds
// blocks, where sixteen-CTA clusters leave a quarter of the slots empty. Measured, 198 solves of
// 256 x 256: streaming 75.8 ms, sixteen-CTA clusters 78.5, groups 52.8 (1.21 us per solve and z
// step); 141 of 128 x 128: 13.4, 9.8, 9.4; 64 x 64 solves fit one CTA's
// shared memory and stay there (3.4 ms against 6.2). The 512-solve sweep 85.2 -> 66.3 ms. Its
// 179 solves of 256 x 256 now: groups 47.3 ms, streaming 67.8, clusters 71.1; 406 instructions per grid point and z
// step, 0.57 of the issue slots, the rest mostly barriers.
#include <cuda_runtime.h>

#include "shg_internal.h"
#include "shg_coop.cuh"
#include "shg_group_queue.cuh"
#include "shg_stream.cuh"

namespace shg {

const float2 *twiddle_symbol_address_group() {
    void *p = nullptr;
    cudaGetSymbolAddress(&p, g_twiddle);
    return static_cast<const float2 *>(p);
}
SHG_CHECK_TU(group)

namespace {

template <int N>
struct GroupShape {
    static constexpr int G = LineShape<N>::G, E = N / G;
    static constexpr int TPB = RowShape<N>::TPB, LPB = RowShape<N>::LPB, BPI = RowShape<N>::BPI;
    static constexpr int TC = 16;                       // columns of a tile (128-byte runs)
    static constexpr int TILES = TPB / (TC * G);        // tiles a block transforms at once
    static constexpr int UNITS = 2 * (N / TC);          // tiles of both fields
    static constexpr int ROW_SCR = LPB * LineScratch<N, G>::SIZE, COL_SCR = TILES * TC * N;
    static constexpr int SCR = ROW_SCR > COL_SCR ? ROW_SCR : COL_SCR;
    static constexpr size_t SMEM = (size_t)(SCR + N) * sizeof(float2);  // scratch, twiddle pairs
    static_assert(TILES >= 1 && UNITS % (TILES * BPI) == 0, "every block transforms the same number of tiles");
};

}  // namespace

// words: [0] job counter, [1 + 2 g] job of group g, [2 + 2 g] its arrival counter (all zeroed);
// err: the run's error word.
template <int N>
__global__ void __launch_bounds__(GroupShape<N>::TPB, N >= 128 ? 2 : 3)
    k_march_group(const InstDesc *__restrict__ inst, const int *__restrict__ list, int njobs, unsigned *words, int *err) {
    using Sh = GroupShape<N>;
    constexpr int G = Sh::G, BPI = Sh::BPI, LPB = Sh::LPB, TC = Sh::TC;
    extern __shared__ __align__(16) float2 gsm[];
    float2 *const scr = gsm, *const tws = gsm + Sh::SCR;
    {
        const float2 *src = twiddle_split<N, G>(g_twiddle + N);
        for (int i = threadIdx.x; i < N; i += Sh::TPB) tws[i] = src[i];
    }
    const int group = blockIdx.x / BPI, rank = blockIdx.x % BPI, tid = threadIdx.x;
    unsigned *const slot = words + 1 + 2 * group, *const bar = slot + 1;
    unsigned target = 0;
    auto meet = [&]() -> bool {  // barrier among the group's blocks
        target += BPI;
        return grid_barrier(bar, target, err);
    };
    auto take = [&] {
        if (rank == 0 && tid == 0) *(volatile unsigned *)slot = atomicAdd(words, 1u);
    };
    auto read = [&] { return ld_acquire_gpu(slot); };
    // a bad descriptor skips the solve
    auto good = [&](unsigned j) {
        const InstDesc &d = inst[list[j]];
        return SHG_REQUIRE(d.n == N && d.nsteps < d.nz && d.nsteps >= 1, kChkDescriptor, j);
    };
    unsigned job;
    while (group_next(job, (unsigned)njobs, take, meet, read, good)) {
        const InstDesc &d = inst[list[job]];
        const int K = d.nsteps;
        for (int s = 0; s <= K; ++s) {
            rows_body<N, true>(d, rank * LPB + tid / G, tid % G, s, scr + (tid / G) * LineScratch<N, G>::SIZE, tws);
            if (s == K) break;
            if (!meet()) return;
            // tiles rank * TILES + i, ... of this block: field u / (N / TC), columns of tile u % (N / TC)
            const int tile = tid / (TC * G), c = tid % TC, t = (tid % (TC * G)) / TC;
#pragma unroll 1
            for (int u = rank * Sh::TILES + tile; u < Sh::UNITS; u += BPI * Sh::TILES) {
                cols_body<N, TC, true, true>(d, (u % (N / TC)) * TC + c, u / (N / TC), t, scr + tile * TC * N + c, tws);
                __syncthreads();  // the scratch is the next tile's (or the row pass's)
            }
            if (!meet()) return;
        }
        __syncthreads();  // the scratch is the next solve's
    }
}

template <int N>
static cudaError_t launch_group_t(const InstDesc *inst, const int *list, int njobs, unsigned *words, int *err,
                                  cudaStream_t st, int *max_groups) {
    using Sh = GroupShape<N>;
    auto k = k_march_group<N>;
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::SMEM)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, Sh::TPB, Sh::SMEM)) != cudaSuccess) return e;
    int groups = per_sm * sms / Sh::BPI;
    if (groups > kMaxGroups) groups = kMaxGroups;
    if (max_groups) *max_groups = groups;
    if (!inst) return groups > 0 ? cudaSuccess : cudaErrorCooperativeLaunchTooLarge;
    if (groups > njobs) groups = njobs;
    if (groups < 1) return cudaErrorCooperativeLaunchTooLarge;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(groups * Sh::BPI, 1, 1);
    cfg.blockDim = dim3(Sh::TPB, 1, 1);
    cfg.dynamicSmemBytes = Sh::SMEM;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, inst, list, njobs, words, err);
}

cudaError_t launch_group(int n, const InstDesc *inst, const int *list, int njobs, unsigned *words, int *err,
                         cudaStream_t st, int *max_groups) {
    switch (n) {
        case 64: return launch_group_t<64>(inst, list, njobs, words, err, st, max_groups);
        case 128: return launch_group_t<128>(inst, list, njobs, words, err, st, max_groups);
        case 256: return launch_group_t<256>(inst, list, njobs, words, err, st, max_groups);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace shg
