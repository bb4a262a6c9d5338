// Adjoint of the THERMAL z-march with the temperature field held fixed, batched over solves.
//
// With T fixed, step s of Solver::CWES (-DTHERMAL, Solver.h:245-276) maps
//   X_s -> RK4_th(X_s; s) -> D -> RK4_th(.; s) = X_{s+1},
// where RK4_th is Solver.h:193-233 with the per-pixel coupling of Solver.h:44-63: n_p, n_s
// from T(x,y,s) and the phase DKint_s*(dz*inc + (s+1)*dz)/(s+1), DKint_s the running sum of
// delta-k(T) over slices 0..s (PhaseMatching.h:12-38), inc = 0, 0.25, 0.25, 0.5 per stage.
// Both RK4 calls of step s use slice s. Per voxel the solve keeps a float4 table
// (kp, ks, tpa1, DKint) built once from T; the stage constants are re-derived from it on
// the fly (th_coef_fixed).
//
// Batch layout: solve b owns states X + b*2*nn (pump then SH), tables coef + b*K*nn (slice
// s at s*nn); one launch covers every solve (blockIdx.y = b).
#include <cuda_runtime.h>

#include "shg_adjoint.cuh"
#include "shg_adjoint_th.h"
#include "shg_thermal.cuh"

namespace shg {

const float2 *twiddle_symbol_address_adjoint_th() {
    void *p = nullptr;
    cudaGetSymbolAddress(&p, g_twiddle);
    return static_cast<const float2 *>(p);
}
SHG_CHECK_TU(adjoint_th)

// coef[s*nn + i] = (kp, ks, tpa1, DKint_s) of pixel i for s < K; the running sum follows
// the order of the thermal row pass (DKint_0 = DK_0, DKint_s = DKint_{s-1} + DK_s).
__global__ void k_th_coef_table(const float *__restrict__ NP, const float *__restrict__ NS,
                                const float *__restrict__ DK, float4 *coef, int nn, int K, const ThermDesc th) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
        float dk = 0.0f;
        for (int s = 0; s < K; ++s) {
            const size_t j = (size_t)s * nn + i;
            dk = s == 0 ? DK[j] : dk + DK[j];
            const float np = NP[j], ns = NS[j];
            coef[j] = make_float4(th_kp(th, np), th_ks(th, ns), th.tpa_c * ns, dk);
        }
    }
}

__device__ __forceinline__ ThCoef th_coef_of(float4 cf, int s, float dz) {
    return th_coef_fixed(cf.x, cf.y, cf.z, cf.w, s, dz);
}

// RK4_th^T of one point at the base state (P, S) with stage constants k: (cp, cs) hold the
// cotangent of the RK4 output on entry and of its input on exit (stages 1..4 use the
// constants c0, c1, c1, c2).
__device__ __forceinline__ void th_vjp_point(const float2 P, const float2 S, float2 &cp, float2 &cs, const ThCoef &k,
                                             float hp, float t0, float w6) {
    const float t1 = k.tpa1;
    float unused[5];  // parameter sensitivities are not needed here
    float2 k1p, k1s, k2p, k2s, k3p, k3s;
    dadz_point(P, S, k.c0, hp, t0, t1, k1p, k1s);
    const float2 B2p = make_float2(fmaf(0.5f, k1p.x, P.x), fmaf(0.5f, k1p.y, P.y));
    const float2 B2s = make_float2(fmaf(0.5f, k1s.x, S.x), fmaf(0.5f, k1s.y, S.y));
    dadz_point(B2p, B2s, k.c1, hp, t0, t1, k2p, k2s);
    const float2 B3p = make_float2(fmaf(0.5f, k2p.x, P.x), fmaf(0.5f, k2p.y, P.y));
    const float2 B3s = make_float2(fmaf(0.5f, k2s.x, S.x), fmaf(0.5f, k2s.y, S.y));
    dadz_point(B3p, B3s, k.c1, hp, t0, t1, k3p, k3s);
    const float2 B4p = c_add(P, k3p), B4s = c_add(S, k3s);
    const float2 op = cp, os = cs;
    float2 cap = op, cas = os;
    float2 ck3p = make_float2(2.0f * w6 * op.x, 2.0f * w6 * op.y), ck3s = make_float2(2.0f * w6 * os.x, 2.0f * w6 * os.y);
    float2 ck2p = ck3p, ck2s = ck3s;
    float2 ck1p = make_float2(w6 * op.x, w6 * op.y), ck1s = make_float2(w6 * os.x, w6 * os.y);
    const float2 ck4p = ck1p, ck4s = ck1s;
    float2 bp = make_float2(0.f, 0.f), bs = make_float2(0.f, 0.f);
    dadz_vjp(B4p, B4s, ck4p, ck4s, k.c2, hp, t0, t1, bp, bs, unused);
    cap = c_add(cap, bp);
    cas = c_add(cas, bs);
    ck3p = c_add(ck3p, bp);
    ck3s = c_add(ck3s, bs);
    bp = bs = make_float2(0.f, 0.f);
    dadz_vjp(B3p, B3s, ck3p, ck3s, k.c1, hp, t0, t1, bp, bs, unused);
    cap = c_add(cap, bp);
    cas = c_add(cas, bs);
    ck2p = make_float2(fmaf(0.5f, bp.x, ck2p.x), fmaf(0.5f, bp.y, ck2p.y));
    ck2s = make_float2(fmaf(0.5f, bs.x, ck2s.x), fmaf(0.5f, bs.y, ck2s.y));
    bp = bs = make_float2(0.f, 0.f);
    dadz_vjp(B2p, B2s, ck2p, ck2s, k.c1, hp, t0, t1, bp, bs, unused);
    cap = c_add(cap, bp);
    cas = c_add(cas, bs);
    ck1p = make_float2(fmaf(0.5f, bp.x, ck1p.x), fmaf(0.5f, bp.y, ck1p.y));
    ck1s = make_float2(fmaf(0.5f, bs.x, ck1s.x), fmaf(0.5f, bs.y, ck1s.y));
    bp = bs = make_float2(0.f, 0.f);
    dadz_vjp(P, S, ck1p, ck1s, k.c0, hp, t0, t1, bp, bs, unused);
    cp = c_add(cap, bp);
    cs = c_add(cas, bs);
}

// Fused row passes. Between two column passes a step boundary finishes one diffraction along x,
// applies the pointwise RK4_th (or its transpose) of the boundary and starts the next diffraction
// along x, so a z step is one row and one column launch and the state crosses memory once per
// launch. A block transforms LPB lines of the pump and of the SH at once, every thread E = N / G
// points of one line in registers; between the transforms the lines lie in shared memory (in the
// transforms' own scratch) and all threads take the points in turn, a point's coefficients and
// stored states being fetched one point ahead. Instruction issue bounds the pass (69 % of the issue
// slots at 16 x 256 x 256 points, 1.9 TB/s from HBM). Against separate transform and pointwise
// passes, four launches per z step, each with the state through memory, us per z step forward /
// gradient: 16 x 256 x 256 49/133 -> 34/103, 64 x 64 x 64 16/42 -> 12.6/32. The whole pass in
// one cooperative launch with barriers among each solve's blocks was slower at every size (41/131
// and 13.3/39.5; 7.3/19.9 against 5.4/11.2 for one 64 x 64 solve).
//
// SHAPE 0: 128 threads, which all transform; 1: the same lines with 256 threads; 2: half the lines
// with 256 threads. 1 and 2 shorten the chain of points that a thread works through, for batches
// that leave the SMs room (row_shape).
template <int N, int SHAPE>
struct ThPassShape {
    static constexpr int G = LineShape<N>::G, E = N / G;
    static constexpr int LMAX = (SHAPE == 2 ? 32 : 64) / G, LPB = LMAX < N ? LMAX : N;  // lines per field
    static constexpr int FT = LPB * G;                                           // transform threads per field
    static constexpr int TPB = SHAPE && LPB * N >= 256 ? 256 : 2 * FT;
    static constexpr int BPI = N / LPB, PTS = LPB * N / TPB;                     // blocks per solve, points per thread
    static constexpr int SC = LineScratch<N, G>::SIZE;
    static constexpr int BLOCKS = 512 / TPB;  // resident blocks per SM (128 registers)
    static_assert(FT % 32 == 0 && 2 * FT <= TPB && N % LPB == 0 && LPB * N % TPB == 0 && SC >= N, "row pass shape");
};

// Roles of a thread: transform role (line of field f, lane t) and point role (points i of the
// block's LPB * N, consecutive threads consecutive points).
template <int N, int SHAPE>
struct ThPassRow {
    using Sh = ThPassShape<N, SHAPE>;
    static constexpr int G = Sh::G, E = Sh::E, LPB = Sh::LPB, SC = Sh::SC;
    float2 *sm;
    __device__ ThPassRow(float2 *s) : sm(s) {}
    __device__ static bool transforms() { return threadIdx.x < 2 * Sh::FT; }
    __device__ float2 *line() const { return sm + (threadIdx.x / G) * SC; }  // lines [0, LPB) pump, then SH
    __device__ static size_t row() {  // this thread's row in the solve's state (pump, then SH)
        const int fl = threadIdx.x / G, f = fl / LPB;
        return ((size_t)f * N + blockIdx.x * LPB + fl % LPB) * N;
    }
    __device__ float2 &at(int f, int i) const { return sm[(f * LPB + i / N) * SC + i % N]; }
    // rows of A (natural frequency order) -> lines in real space
    __device__ void finish(const float2 *A, const float2 *tab) const {
        if (!transforms()) return;
        const int t = threadIdx.x % G;
        const size_t r0 = row();
        float2 v[E];
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = SHG_AT(A, r0 + t + G * j, (size_t)2 * N * N, kChkAdjoint);
        fft_nat_to_spec<N, G, -1>(v, t, line(), tab);
        __syncwarp();  // the line's lanes have read the scratch that it overwrites
#pragma unroll
        for (int r = 0; r < E; ++r) line()[spec_index<N, G>(t, r)] = v[r];
    }
    // lines in real space -> rows of A (natural frequency order)
    __device__ void start(float2 *A, const float2 *tab) const {
        if (!transforms()) return;
        const int t = threadIdx.x % G;
        const size_t r0 = row();
        float2 v[E];
#pragma unroll
        for (int r = 0; r < E; ++r) v[r] = line()[spec_index<N, G>(t, r)];
        fft_spec_to_nat<N, G, +1>(v, t, line(), tab);
#pragma unroll
        for (int j = 0; j < E; ++j) SHG_AT(A, r0 + t + G * j, (size_t)2 * N * N, kChkAdjoint) = v[j];
    }
};

// Forward boundary of every solve: with sp >= 0 the end of the diffraction of step sp in A, whose
// result W_sp goes to save_w, and RK4_th of step sp (its second call); otherwise the state at
// (inP, inS), `stride` apart from solve to solve (inS null: no SH yet). The state X_{sp+1} goes to
// save_x. With sn >= 0 RK4_th of step sn (its first call) and the start of its diffraction in A;
// otherwise the state to out. Null pointers skip their stores, and the RK4 that nothing reads.
template <int N, int SHAPE>
__global__ void __launch_bounds__(ThPassShape<N, SHAPE>::TPB, ThPassShape<N, SHAPE>::BLOCKS)
    k_th_rows_fwd(float2 *A0, const float2 *inP, const float2 *inS, size_t stride, float2 *save_w, float2 *save_x,
                  float2 *out, const float4 *__restrict__ coef, int K, int sp, int sn,
                  const InstDesc *__restrict__ dd) {
    using Sh = ThPassShape<N, SHAPE>;
    __shared__ float2 sm[2 * Sh::LPB * Sh::SC];
    constexpr int NN = N * N, P = Sh::LPB * N;
    const int b = blockIdx.y, base = blockIdx.x * P;  // this block's points of a field
    const InstDesc &d = dd[b];
    const float2 *__restrict__ tab = g_twiddle + N;
    const ThPassRow<N, SHAPE> rw(sm);
    float2 *A = A0 + (size_t)b * 2 * NN;
    const size_t o = (size_t)b * 2 * NN + base;
    const float4 *__restrict__ cp = coef + ((size_t)b * K + (sp < 0 ? 0 : sp)) * NN + base;
    const float4 *__restrict__ cn = coef + ((size_t)b * K + (sn < 0 ? 0 : sn)) * NN + base;
    const bool second = sp >= 0 && (save_x || out || sn >= 0);
    int i = threadIdx.x;
    float4 vp = make_float4(0.f, 0.f, 0.f, 0.f), vn = vp;
    if (second) vp = cp[i];
    if (sn >= 0) vn = cn[i];
    grid_dependency_wait();
    if (sp >= 0) {
        rw.finish(A, tab);
        __syncthreads();
    }
    const float dz = d.dz;
#pragma unroll 1
    for (int j = 0; j < Sh::PTS; ++j, i += Sh::TPB) {
        const float4 fp = vp, fn = vn;
        if (j + 1 < Sh::PTS) {
            if (second) vp = cp[i + Sh::TPB];
            if (sn >= 0) vn = cn[i + Sh::TPB];
        }
        float2 p, q;
        if (sp >= 0) {
            p = rw.at(0, i);
            q = rw.at(1, i);
            if (save_w) {
                save_w[o + i] = p;
                save_w[o + NN + i] = q;
            }
            if (second) rk4_point_th(p, q, th_coef_of(fp, sp, dz), d);
        } else {
            p = inP[b * stride + base + i];
            q = inS ? inS[b * stride + base + i] : make_float2(0.f, 0.f);
        }
        if (save_x) {
            save_x[o + i] = p;
            save_x[o + NN + i] = q;
        }
        if (sn >= 0) {
            rk4_point_th(p, q, th_coef_of(fn, sn, dz), d);
            rw.at(0, i) = p;  // each thread rewrites only the points it read
            rw.at(1, i) = q;
        } else if (out) {
            out[o + i] = p;
            out[o + NN + i] = q;
        }
    }
    if (sn >= 0) {
        __syncthreads();
        rw.start(A, tab);
    }
}

// Reverse boundary of every solve's cotangent C: with sa >= 0 the end of the adjoint diffraction
// of step sa and RK4_th^T at its first call's input Xa, otherwise C as it is; with sb >= 0
// RK4_th^T of step sb at its second call's input Wb and the start of its adjoint diffraction in C,
// otherwise the cotangent to C.
template <int N, int SHAPE>
__global__ void __launch_bounds__(ThPassShape<N, SHAPE>::TPB, ThPassShape<N, SHAPE>::BLOCKS)
    k_th_rows_bwd(float2 *C0, const float2 *__restrict__ Xa, const float2 *__restrict__ Wb,
                  const float4 *__restrict__ coef, int K, int sa, int sb, const InstDesc *__restrict__ dd) {
    using Sh = ThPassShape<N, SHAPE>;
    __shared__ float2 sm[2 * Sh::LPB * Sh::SC];
    constexpr int NN = N * N, P = Sh::LPB * N;
    const int b = blockIdx.y, base = blockIdx.x * P;
    const InstDesc &d = dd[b];
    const float2 *__restrict__ tab = g_twiddle + N;
    const ThPassRow<N, SHAPE> rw(sm);
    float2 *C = C0 + (size_t)b * 2 * NN;
    const size_t o = (size_t)b * 2 * NN + base;
    const float4 *__restrict__ ca = coef + ((size_t)b * K + (sa < 0 ? 0 : sa)) * NN + base;
    const float4 *__restrict__ cb = coef + ((size_t)b * K + (sb < 0 ? 0 : sb)) * NN + base;
    int i = threadIdx.x;
    float4 va = make_float4(0.f, 0.f, 0.f, 0.f), vb = va;
    float2 xp = make_float2(0.f, 0.f), xs = xp, wp = xp, ws = xp;
    auto fetch_coef = [&](int k) {
        if (sa >= 0) va = ca[k];
        if (sb >= 0) vb = cb[k];
    };
    auto fetch_state = [&](int k) {
        if (sa >= 0) {
            xp = Xa[o + k];
            xs = Xa[o + NN + k];
        }
        if (sb >= 0) {
            wp = Wb[o + k];
            ws = Wb[o + NN + k];
        }
    };
    fetch_coef(i);
    grid_dependency_wait();
    fetch_state(i);
    if (sa >= 0) {
        rw.finish(C, tab);
        __syncthreads();
    }
    const float dz = d.dz, hp = d.hp, t0 = d.tpa0, w6 = d.dz6;
#pragma unroll 1
    for (int j = 0; j < Sh::PTS; ++j, i += Sh::TPB) {
        const float4 fa = va, fb = vb;
        const float2 gp = xp, gs = xs, hw = wp, hs = ws;
        if (j + 1 < Sh::PTS) {
            fetch_coef(i + Sh::TPB);
            fetch_state(i + Sh::TPB);
        }
        float2 p, q;
        if (sa >= 0) {
            p = rw.at(0, i);
            q = rw.at(1, i);
            th_vjp_point(gp, gs, p, q, th_coef_of(fa, sa, dz), hp, t0, w6);
        } else {
            p = C[base + i];
            q = C[NN + base + i];
        }
        if (sb >= 0) {
            th_vjp_point(hw, hs, p, q, th_coef_of(fb, sb, dz), hp, t0, w6);
            rw.at(0, i) = p;  // each thread rewrites only the points it read
            rw.at(1, i) = q;
        } else {
            C[base + i] = p;
            C[NN + base + i] = q;
        }
    }
    if (sb >= 0) {
        __syncthreads();
        rw.start(C, tab);
    }
}

// out[b] += sum |field|^2 of solve b's field at X + b*stride (FP64).
__global__ void k_abs2_sum_b(const float2 *__restrict__ X, int nn, size_t stride, double *out) {
    const float2 *A = X + blockIdx.y * stride;
    double a[1] = {0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
        const float2 v = A[i];
        a[0] += (double)v.x * v.x + (double)v.y * v.y;
    }
    block_sum_doubles(a, 1, out + blockIdx.y);
}

// Cotangent of L_b = seed_b/2 * sum |S_b|^2: c_S = seed_b * S_b, c_P = 0.
__global__ void k_seed_b(const float2 *__restrict__ X, float2 *cot, int nn, const double *__restrict__ seed) {
    const size_t o = (size_t)blockIdx.y * 2 * nn;
    const float g = (float)seed[blockIdx.y];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
        const float2 v = X[o + nn + i];
        cot[o + nn + i] = make_float2(g * v.x, g * v.y);
        cot[o + i] = make_float2(0.f, 0.f);
    }
}

static dim3 grid_b(int nn, int solves) { return dim3((unsigned)((nn + 255) / 256 < 64 ? (nn + 255) / 256 : 64), solves); }

cudaError_t launch_th_coef_table(const float *NP, const float *NS, const float *DK, float4 *coef, int nn, int K,
                                 const ThermDesc &th, cudaStream_t st) {
    k_th_coef_table<<<(nn + 255) / 256, 256, 0, st>>>(NP, NS, DK, coef, nn, K, th);
    return cudaGetLastError();
}

// Row pass shape by the number of shape-0 blocks: us per z step, forward / gradient with 10
// checkpoints, of shape 0, 1, 2 (GB300, 40 steps):
//    < 1 per SM    64^2 x 4    6.6/14.8   6.0/13.2   5.4/11.7     256^2 x 2   12.5/31.6  10.7/27.7  10.1/27.6
//    < 2 per SM   128^2 x 16  15.3/38.4  13.6/35.5  15.3/39.6     256^2 x 4   15.3/38.6  13.8/36.5  15.1/40.2
//    more          64^2 x 64  12.8/32.2  13.4/34.4  12.5/34.1     256^2 x 8   21.1/58.4  22.2/62.6  24.4/69.9
template <int N>
static int row_shape(int solves, int sms) {
    const int blocks = solves * ThPassShape<N, 0>::BPI;
    return blocks < sms ? 2 : blocks < 2 * sms ? 1 : 0;
}

template <int N, int SHAPE>
static cudaError_t launch_rows_fwd_s(float2 *A, const float2 *inP, const float2 *inS, size_t stride, float2 *save_w,
                                     float2 *save_x, float2 *out, const float4 *coef, int K, int sp, int sn,
                                     const InstDesc *d, int solves, cudaStream_t st) {
    using Sh = ThPassShape<N, SHAPE>;
    return launch_dependent(k_th_rows_fwd<N, SHAPE>, dim3(Sh::BPI, solves), Sh::TPB, st, A, inP, inS, stride, save_w,
                            save_x, out, coef, K, sp, sn, d);
}

template <int N>
static cudaError_t launch_rows_fwd_t(float2 *A, const float2 *inP, const float2 *inS, size_t stride, float2 *save_w,
                                     float2 *save_x, float2 *out, const float4 *coef, int K, int sp, int sn,
                                     const InstDesc *d, int solves, int sms, cudaStream_t st) {
    const int shape = row_shape<N>(solves, sms);
    auto launch = shape == 0   ? launch_rows_fwd_s<N, 0>
                  : shape == 1 ? launch_rows_fwd_s<N, 1>
                               : launch_rows_fwd_s<N, 2>;
    return launch(A, inP, inS, stride, save_w, save_x, out, coef, K, sp, sn, d, solves, st);
}

template <int N, int SHAPE>
static cudaError_t launch_rows_bwd_s(float2 *C, const float2 *Xa, const float2 *Wb, const float4 *coef, int K, int sa,
                                     int sb, const InstDesc *d, int solves, cudaStream_t st) {
    using Sh = ThPassShape<N, SHAPE>;
    return launch_dependent(k_th_rows_bwd<N, SHAPE>, dim3(Sh::BPI, solves), Sh::TPB, st, C, Xa, Wb, coef, K, sa, sb, d);
}

template <int N>
static cudaError_t launch_rows_bwd_t(float2 *C, const float2 *Xa, const float2 *Wb, const float4 *coef, int K, int sa,
                                     int sb, const InstDesc *d, int solves, int sms, cudaStream_t st) {
    const int shape = row_shape<N>(solves, sms);
    auto launch = shape == 0   ? launch_rows_bwd_s<N, 0>
                  : shape == 1 ? launch_rows_bwd_s<N, 1>
                               : launch_rows_bwd_s<N, 2>;
    return launch(C, Xa, Wb, coef, K, sa, sb, d, solves, st);
}

cudaError_t launch_th_rows_fwd(int n, float2 *A, const float2 *inP, const float2 *inS, size_t stride, float2 *save_w,
                               float2 *save_x, float2 *out, const float4 *coef, int K, int sp, int sn,
                               const InstDesc *d, int solves, int sms, cudaStream_t st) {
    if (sp >= K || sn >= K || (sp < 0 && !inP)) return cudaErrorInvalidValue;
    switch (n) {
        case 16: return launch_rows_fwd_t<16>(A, inP, inS, stride, save_w, save_x, out, coef, K, sp, sn, d, solves, sms, st);
        case 32: return launch_rows_fwd_t<32>(A, inP, inS, stride, save_w, save_x, out, coef, K, sp, sn, d, solves, sms, st);
        case 64: return launch_rows_fwd_t<64>(A, inP, inS, stride, save_w, save_x, out, coef, K, sp, sn, d, solves, sms, st);
        case 128: return launch_rows_fwd_t<128>(A, inP, inS, stride, save_w, save_x, out, coef, K, sp, sn, d, solves, sms, st);
        case 256: return launch_rows_fwd_t<256>(A, inP, inS, stride, save_w, save_x, out, coef, K, sp, sn, d, solves, sms, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_th_rows_bwd(int n, float2 *C, const float2 *Xa, const float2 *Wb, const float4 *coef, int K, int sa,
                               int sb, const InstDesc *d, int solves, int sms, cudaStream_t st) {
    if (sa >= K || sb >= K || (sa >= 0 && !Xa) || (sb >= 0 && !Wb)) return cudaErrorInvalidValue;
    switch (n) {
        case 16: return launch_rows_bwd_t<16>(C, Xa, Wb, coef, K, sa, sb, d, solves, sms, st);
        case 32: return launch_rows_bwd_t<32>(C, Xa, Wb, coef, K, sa, sb, d, solves, sms, st);
        case 64: return launch_rows_bwd_t<64>(C, Xa, Wb, coef, K, sa, sb, d, solves, sms, st);
        case 128: return launch_rows_bwd_t<128>(C, Xa, Wb, coef, K, sa, sb, d, solves, sms, st);
        case 256: return launch_rows_bwd_t<256>(C, Xa, Wb, coef, K, sa, sb, d, solves, sms, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_abs2_sum_b(const float2 *X, int nn, size_t stride, double *out, int solves, cudaStream_t st) {
    k_abs2_sum_b<<<grid_b(nn, solves), 256, 0, st>>>(X, nn, stride, out);
    return cudaGetLastError();
}

cudaError_t launch_seed_b(const float2 *X, float2 *cot, int nn, const double *seed, int solves, cudaStream_t st) {
    k_seed_b<<<grid_b(nn, solves), 256, 0, st>>>(X, cot, nn, seed);
    return cudaGetLastError();
}

}  // namespace shg
