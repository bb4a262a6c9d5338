// One or two Jacobi sweeps of the heat stencil (Tfield.h:113-258) in one pass over memory,
// bit-identical to single sweeps of the other kernels.
//
// A block owns an (x, y) tile with a halo of K rows (and, where a tile does not span the grid
// in x, four columns) and marches z with K sweeps in flight. A thread holds two rows of four
// adjacent columns: x neighbours come from the adjacent lanes by shuffle, the y neighbours
// outside its rows and the older z neighbour from shared memory (16-byte reads). At step p the
// input plane p arrives (cp.async, two planes ahead) and level t = 1..K computes plane p - t
// from level t-1's planes p-t-1, p-t (written in earlier steps) and p-t+1 (its own value of this
// step), so one block barrier per step orders all levels. Every voxel of every level runs the
// float operations of a single sweep; sums and products of two columns share one packed
// instruction (f32x2: the same IEEE rounding per lane), and the divisions are corrected products
// (div_const) for as long as every value lies where they equal IEEE division, which the block
// checks on the values it holds (the single-sweep kernels check every numerator).
//
// Why this split: the single-sweep kernel issues 77 thread instructions per voxel (seven shared
// loads among them) at 80 % issue, above its memory time; four columns per thread and packed
// arithmetic take 18. What each kernel measured, and when two sweeps per launch pay, stands at
// heat_block_plan.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>

#include "shg_internal.h"
#include "shg_thermal.cuh"

namespace shg {

SHG_CHECK_TU(heat_block)

namespace {

constexpr int kAhead = 2;  // planes in flight
constexpr int kRing = 4;   // slots of the input and Q/k rings: planes p-1, p and those in flight
// A shared plane holds every thread's R rows of four columns.
__host__ __device__ constexpr int plane_floats(int threads, int R) { return 4 * R * threads; }
__host__ __device__ constexpr int shared_planes(int K) { return 2 * kRing + 2 * (K - 1); }
constexpr int kRows = 2;   // rows per thread
constexpr int kMaxLevels = 2;

typedef unsigned long long u64;

__device__ __forceinline__ u64 pack2(float x, float y) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(u64 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// Four adjacent columns of one row.
struct V4 {
    u64 a, b;
};
__device__ __forceinline__ V4 ld4(const float *p) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p);
    return {v.x, v.y};
}
__device__ __forceinline__ void st4(float *p, V4 v) { *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(v.a, v.b); }
__device__ __forceinline__ void cp_async16(float *dst, const float *src, bool ok) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst), n = ok ? 16u : 0u;  // 0: zero fill
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ u64 div2(u64 s, u64 r, u64 nd) {
    const u64 q = mul2(s, r);
    return fma2(fma2(q, nd, s), r, q);
}

// Smallest and largest magnitude of an accumulator and two values (a NaN is passed over: both
// division paths give NaN for it).
__device__ __forceinline__ float min_abs3(float a, float b, float c) {
    float r;
    asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max_abs3(float a, float b, float c) {
    float r;
    asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// Range of the magnitudes seen. While all lie in [2^-60, 2^99), the sum of two values is 0 or at
// least 2^-83 in magnitude and below 2^100, where the corrected products equal IEEE division (a
// zero sum of such values is +0, and gives +0 either way).
struct Range {
    float lo, hi;
    __device__ __forceinline__ void add(V4 v) {
        const float2 a = unpack2(v.a), b = unpack2(v.b);
        lo = min_abs3(min_abs3(lo, a.x, a.y), b.x, b.y);
        hi = max_abs3(max_abs3(hi, a.x, a.y), b.x, b.y);
    }
    __device__ __forceinline__ bool out() const { return !(lo >= 0x1p-60f && hi < 0x1p99f); }
};

__device__ __forceinline__ u64 div2_any(u64 s, float d, float r, int fast) {
    const float2 v = unpack2(s);
    return pack2(div_any(v.x, d, r, fast), div_any(v.y, d, r, fast));
}
// Magnitudes seen where zeros may be among them: with the sign rotated to the bottom and less one, +0
// is the largest of unsigned values, -0 the smallest (its quotient is -0, that of a corrected product
// +0).
struct RangeZero {
    unsigned lo;
    float hi;
    __device__ __forceinline__ void add(u64 s) {
        const float2 v = unpack2(s);
        const unsigned a = __float_as_uint(v.x), b = __float_as_uint(v.y);
        lo = min(lo, min(__funnelshift_l(a, a, 1) - 1u, __funnelshift_l(b, b, 1) - 1u));
        hi = max_abs3(hi, v.x, v.y);
    }
    __device__ __forceinline__ void add(V4 v) { add(v.a), add(v.b); }
    // +0 or a magnitude in [2^(elo - 127), top)
    __device__ __forceinline__ bool in(unsigned elo, float top) const { return lo >= (elo << 24) - 1u && hi < top; }
    // Temperatures: sums of two are +0 or in [2^-100, 2^100).
    __device__ __forceinline__ bool out() const { return !in(50u, 0x1p99f); }
    // Numerators: as the corrected products were verified for.
    __device__ __forceinline__ bool ok() const { return in(kDivExpLo, 0x1p101f); }
};

struct DivConst {  // reciprocals, negated divisors and the final factor, both halves alike
    u64 rx, ndx, ry, ndy, rz, ndz, l2;
};
__device__ __forceinline__ u64 twice(float v) { return pack2(v, v); }

// Sums of the x and y neighbours of four voxels.
struct Sums {
    u64 xa, xb, ya, yb;
};
__device__ __forceinline__ Sums lateral_sums(V4 cc, V4 ym, V4 yp, float xl, float xr) {
    const float2 c01 = unpack2(cc.a), c23 = unpack2(cc.b);
    return {pack2(__fadd_rn(c01.y, xl), __fadd_rn(c23.x, c01.x)), pack2(__fadd_rn(c23.y, c01.y), __fadd_rn(xr, c23.x)),
            add2(yp.a, ym.a), add2(yp.b, ym.b)};
}

// Interior formula (Tfield.h:132) for four voxels with the divisions as corrected products.
__device__ __forceinline__ V4 interior4(const DivConst &d, const Sums &s, V4 sz, V4 q) {
    V4 o;
    o.a = mul2(d.l2, add2(add2(add2(div2(s.xa, d.rx, d.ndx), div2(s.ya, d.ry, d.ndy)),
                               div2(sz.a, d.rz, d.ndz)), q.a));
    o.b = mul2(d.l2, add2(add2(add2(div2(s.xb, d.rx, d.ndx), div2(s.yb, d.ry, d.ndy)),
                               div2(sz.b, d.rz, d.ndz)), q.b));
    return o;
}

// The same for numerators of any magnitude, out of line: only values below 2^-77 (a Gaussian's
// underflowing tails beside zeros), infinities and -0 come here.
__device__ __noinline__ V4 interior4_any(const HeatCoef &c, Sums s, V4 sz, V4 q) {
    auto half = [&](u64 x, u64 y, u64 z, u64 q2) {
        return mul2(twice(c.L2), add2(add2(add2(div2_any(x, c.dx2, c.rdx2, c.fast_div),
                                                div2_any(y, c.dy2, c.rdy2, c.fast_div)),
                                           div2_any(z, c.dz2, c.rdz2, c.fast_div)), q2));
    };
    return {half(s.xa, s.ya, sz.a, q.a), half(s.xb, s.yb, sz.b, q.b)};
}

// The z faces' formula for four voxels: (n + az s1 + bz s2 + t) / den_z, n the inward neighbour, s1
// and s2 the sums of the x and y neighbours. Scalar products and sums: the packed forms carry no
// promise against contraction. ANY: numerators of any magnitude.
template <bool ANY>
__device__ __forceinline__ V4 face4(const HeatCoef &c, V4 n, const Sums &s) {
    auto f = [&](u64 n2, u64 s1, u64 s2) {
        const float2 m = unpack2(n2), u = unpack2(s1), w = unpack2(s2);
        auto g = [&](float n1, float u1, float w1) {
            return __fadd_rn(__fadd_rn(__fadd_rn(n1, __fmul_rn(c.az, u1)), __fmul_rn(c.bz, w1)), c.tinfBiz);
        };
        const u64 v = pack2(g(m.x, u.x, w.x), g(m.y, u.y, w.y));
        return ANY ? div2_any(v, c.den_z, c.rden_z, c.fast_face) : div2(v, twice(c.rden_z), twice(-c.den_z));
    };
    return {f(n.a, s.xa, s.ya), f(n.b, s.xb, s.yb)};
}

// mask ? a : b, bitwise (masks all ones or zero)
__device__ __forceinline__ float blend(unsigned m, float a, float b) {
    unsigned r;
    asm("lop3.b32 %0, %1, %2, %3, 0xca;" : "=r"(r) : "r"(m), "r"(__float_as_uint(a)), "r"(__float_as_uint(b)));
    return __uint_as_float(r);
}

// BC 0: the voxel of the four that lies on the face x = 0 (left) or x = NX-1, of a row inside
// the grid in y: the face formula away from the z faces (zs: sums of the z neighbours), else
// the vertical edge's (zs: the inward z neighbours). ANY: numerators of any magnitude.
template <bool ZFACE, bool ANY = false>
__device__ __forceinline__ float x_face(const HeatCoef &c, V4 cc, const Sums &s, V4 zs, bool left) {
    const float2 zl = unpack2(zs.a), zr = unpack2(zs.b), yl = unpack2(s.ya), yr = unpack2(s.yb);
    const float tx = left ? unpack2(cc.a).y : unpack2(cc.b).x;  // inward x neighbour
    const float yy = left ? yl.x : yr.y, zz = left ? zl.x : zr.y;
    if (ZFACE)
        return edge_round(__fadd_rn(__fadd_rn(__fmul_rn(c.av, tx), __fmul_rn(c.bv, zz)), __fmul_rn(c.cv, yy)), c.KV, c.KVh,
                          c.KVl, c.V);
    float f = __fadd_rn(tx, __fmul_rn(c.ax, yy));
    f = __fadd_rn(f, __fmul_rn(c.bx, zz));
    f = __fadd_rn(f, c.tinfBix);
    if (ANY) return div_any(f, c.den_x, c.rden_x, c.fast_face);
    const float w = f * c.rden_x;
    return fmaf(fmaf(-w, c.den_x, f), c.rden_x, w);
}

// BC 0: four voxels of the top face y = NY-1, its edges and corners included (zs as above).
template <bool ZFACE, bool ANY = false>
__device__ __forceinline__ V4 top_row(const HeatCoef &c, V4 cc, const Sums &s, V4 ym, V4 zs, bool left, bool right) {
    const float2 c01 = unpack2(cc.a), c23 = unpack2(cc.b), m01 = unpack2(ym.a), m23 = unpack2(ym.b);
    const float2 x01 = unpack2(s.xa), x23 = unpack2(s.xb), z01 = unpack2(zs.a), z23 = unpack2(zs.b);
    const float m[4] = {m01.x, m01.y, m23.x, m23.y}, sx[4] = {x01.x, x01.y, x23.x, x23.y};
    const float z[4] = {z01.x, z01.y, z23.x, z23.y};
    const float tx = left ? c01.y : c23.x, me = left ? m[0] : m[3], ze = left ? z[0] : z[3];
    float o[4], e;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (ZFACE) {
            const float f = __fadd_rn(__fadd_rn(__fmul_rn(c.ah, m[i]), __fmul_rn(c.bh, z[i])), __fmul_rn(c.ch, sx[i]));
            o[i] = edge_round(f, c.KH, c.KHh, c.KHl, c.H);
        } else {
            float f = __fadd_rn(m[i], __fmul_rn(c.ay, sx[i]));
            f = __fadd_rn(f, __fmul_rn(c.by, z[i]));
            f = __fadd_rn(f, c.tinfBiy);
            const float w = f * c.rden_y;
            o[i] = ANY ? div_any(f, c.den_y, c.rden_y, c.fast_face) : fmaf(fmaf(-w, c.den_y, f), c.rden_y, w);
        }
    }
    if (ZFACE) {
        const float f = __fadd_rn(__fmul_rn(c.AV, tx), __fmul_rn(c.BV, me));
        e = __fmul_rn(__fadd_rn(__fadd_rn(f, __fmul_rn(c.CV, ze)), c.tinfBiD), c.GV);
    } else {
        const float f = __fadd_rn(__fadd_rn(__fmul_rn(c.ad, me), __fmul_rn(c.bd, tx)), __fmul_rn(c.cd, ze));
        e = edge_round(f, c.KD, c.KDh, c.KDl, c.D);
    }
    return {pack2(left ? e : o[0], o[1]), pack2(o[2], right ? e : o[3])};
}

// Planes [z0, z1) of a block's tile. vx (a power of two, at most 32) vectors per region row: rows start at warp
// boundaries or share a warp, so x neighbours across a row's ends belong to no stored voxel.
// ORDINARY: returns the first plane that is not stored, z1 unless a value was out of range (then with no
// copy in flight). Otherwise values of any kind.
template <int BC, int K, int THREADS, bool ORDINARY>
__device__ __forceinline__ int heat_chunk(float *__restrict__ Tf, const float *__restrict__ Ti,
                                          const float *__restrict__ QK, const HeatCoef &c, const HeatBlockGrid &g,
                                          const int z0, const int z1) {
    static_assert(K <= kMaxLevels && K <= kRing - kAhead, "the Q/k ring holds the planes of K levels");
    constexpr int R = kRows, PL = plane_floats(THREADS, R);
    extern __shared__ __align__(16) float hb_smem[];
    const int vx = g.vx, rows = R * (THREADS / vx), row = 4 * vx;
    const int v = threadIdx.x & (vx - 1), r = R * (threadIdx.x / vx);
    const int x = (int)blockIdx.x * g.txi - g.xh + 4 * v, y = (int)blockIdx.y * g.tyi - g.yh + r;
    const size_t sxy = (size_t)g.nx * g.ny;
    // a shared plane holds the region's rows, and the grid a vector at least (block-uniform)
    if (!SHG_REQUIRE(rows * row == PL && (vx & (vx - 1)) == 0 && g.nx % 4 == 0 && g.nx >= 8, kChkHeatVoxel, vx)) return z1;
    // this thread's first vector in shared plane 0, and the rows above and below its own;
    // planes: input ring, Q/k ring, levels 1..K-1
    float *const sm = hb_smem + (r * vx + v) * 4, *const sm1 = sm + row;
    const float *const smm = r > 0 ? sm - row : sm, *const smp = r + R < rows ? sm + R * row : sm1;
    const bool xin = x >= 0 && x < g.nx;
    const bool xst = xin && x >= (int)blockIdx.x * g.txi && x < ((int)blockIdx.x + 1) * g.txi;
    const int ylo = (int)blockIdx.y * g.tyi, yhi = min(g.ny, ylo + g.tyi);
    bool in[R], st[R];
    bool top[R];                     // BC 0: the row is on the top face
    unsigned keep[R], kl[R], kr[R];  // voxels that are kept: the middle two, the first, the last
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int yk = y + k;
        in[k] = xin && yk >= 0 && yk < g.ny;
        st[k] = xst && yk >= ylo && yk < yhi;
        const bool kept = !in[k] || yk == 0 || (BC != 0 && yk == g.ny - 1);
        keep[k] = kept ? 0xffffffffu : 0u;
        kl[k] = kept || (BC != 0 && x == 0) ? 0xffffffffu : 0u;
        kr[k] = kept || (BC != 0 && x + 4 == g.nx) ? 0xffffffffu : 0u;
        top[k] = BC == 0 && in[k] && yk == g.ny - 1;
    }

    const bool xface = x == 0 || x + 4 == g.nx;

    const int plo = max(0, z0 - K), pin = min(g.nz, z1 + K);  // input planes [plo, pin)
    const int pend = z1 - 1 + K;                              // last step
    int fp = plo;                                             // plane of the next fetch
    // source and destination rows, held to the grid where the thread's own are not in it
    const int xc = min(max(x, 0), g.nx - 4), yc0 = min(max(y, 0), g.ny - 1), yc1 = min(max(y + 1, 0), g.ny - 1);
    const int dy1 = (yc1 - yc0) * g.nx;
    const float *srcT = Ti + plo * sxy + yc0 * g.nx + xc, *srcQ = QK + plo * sxy + yc0 * g.nx + xc;
    float *dst = Tf + z0 * sxy + yc0 * g.nx + xc;
    auto held = [&](long long o) { return SHG_REQUIRE(o >= 0 && o + 3 < (long long)(sxy * g.nz), kChkHeatVoxel, o); };
    auto fetch = [&](int slot) {  // plane fp, and Q/k of plane fp - 1 (first used when plane fp has arrived)
        if (fp < pin) {
            cp_async16(sm + slot * PL, srcT, in[0] && held(srcT - Ti));
            cp_async16(sm1 + slot * PL, srcT + dy1, in[1] && held(srcT + dy1 - Ti));
            if (fp > plo) {
                cp_async16(sm + (kRing + slot) * PL, srcQ, in[0] && held(srcQ - QK));
                cp_async16(sm1 + (kRing + slot) * PL, srcQ + dy1, in[1] && held(srcQ + dy1 - QK));
                srcQ += sxy;
            }
            srcT += sxy;
        }
        cp_async_commit();
        ++fp;
    };

    // Planes that are read before they are written hold ones (any finite values would do: they
    // reach no stored voxel, but could be reported as out of range).
    const V4 ones = {twice(1.0f), twice(1.0f)};
#pragma unroll
    for (int i = 0; i < shared_planes(K); ++i)
        if (i == 2 || i == 3 || i == kRing || i == kRing + 3 || i >= 2 * kRing) {
            st4(sm + i * PL, ones);
            st4(sm1 + i * PL, ones);
        }
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the launch before this one has finished
    fetch(0);
    fetch(1);

    // plane p - t of level t = 0..K-1, and plane p, p - 2 of level 0. Rows outside the grid hold
    // ones throughout.
    V4 cc[K][R], cur[R], zm0[R];
#pragma unroll
    for (int k = 0; k < R; ++k)
#pragma unroll
        for (int t = 0; t < K; ++t) cc[t][k] = ones;
    const DivConst d = {twice(c.rdx2), twice(-c.dx2), twice(c.rdy2), twice(-c.dy2), twice(c.rdz2), twice(-c.dz2),
                        twice(c.L2)};
    // Q/k is checked against 2^60 beside the temperatures, so that a value computed in the
    // running step, whose range the others learn at the next barrier, is below 2^100 too
    auto verified = [&] { return c.fast_div && c.fast_face && c.L2 < 0x1p30f; };
    Range seen{verified() ? 1.0f : 0.0f, 1.0f};         // of the ordinary chunk
    RangeZero seen0{verified() ? ~0u : 0u, 1.0f};  // of the other
    float qhi = 0.0f;

    // Arrival of plane p (ring slot s): this thread's values, then the barrier that orders the
    // previous step's level planes and plane p - 1, and tells every thread whether a value it
    // may read was out of range.
    auto arrive = [&](auto Mode, int s) -> bool {
        constexpr bool ZEROS = decltype(Mode)::value > 0;
        cp_async_wait<kAhead - 1>();
        const V4 q[R] = {ld4(sm + (kRing + s) * PL), ld4(sm1 + (kRing + s) * PL)};
        cur[0] = ld4(sm + s * PL);
        cur[1] = ld4(sm1 + s * PL);
        zm0[0] = ld4(sm + (s + 2) % kRing * PL);  // before the barrier: the fetch below reuses the slot
        zm0[1] = ld4(sm1 + (s + 2) % kRing * PL);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if (!in[k]) cur[k] = zm0[k] = ones;
            if (ZEROS) seen0.add(cur[k]);
            else seen.add(cur[k]);
            const float2 a = unpack2(q[k].a), b = unpack2(q[k].b);
            qhi = max_abs3(max_abs3(qhi, a.x, a.y), b.x, b.y);
        }
        const bool bad = __syncthreads_or((ZEROS ? seen0.out() : seen.out()) || !(qhi < 0x1p60f));
        fetch((s + kAhead) % kRing);
        return bad;
    };
    // end of a step: the new planes of levels 1..K-1 (plane p - t of level t), read from the
    // next step on
    auto leave = [&](int s) {
#pragma unroll
        for (int t = 1; t < K; ++t) {
            st4(sm + (2 * kRing + (t - 1) * 2 + ((s - t + 8) & 1)) * PL, cc[t][0]);
            st4(sm1 + (2 * kRing + (t - 1) * 2 + ((s - t + 8) & 1)) * PL, cc[t][1]);
        }
    };
    auto store = [&](int z, const V4 (&w)[R]) {
        if (z >= z0) {
            const size_t o = dst - Tf;
            if (st[0] && SHG_REQUIRE(o + 3 < sxy * g.nz, kChkHeatVoxel, o)) st4(dst, w[0]);
            if (st[1] && SHG_REQUIRE(o + dy1 + 3 < sxy * g.nz, kChkHeatVoxel, o)) st4(dst + dy1, w[1]);
            dst += sxy;
        }
    };
    // Shared plane that holds plane z = p - t of level t - 1 (before), and z - 1 (older; the one
    // that this step's value replaces), at a step with slot s.
    auto before = [](int s, int t) { return t == 1 ? (s + kRing - 1) % kRing : 2 * kRing + (t - 2) * 2 + ((s - t + 8) & 1); };
    auto older = [](int s, int t) { return 2 * kRing + (t - 2) * 2 + ((s - t + 9) & 1); };
    // Q/k of plane p - t: fetched with plane p - t + 1
    auto heat = [](int s, int t) { return kRing + (s - t + 1 + kRing) % kRing; };

    // Step p: with all values in range (MODE 0), zeros among them (1), or values of any kind (2). Levels
    // outside their range of planes compute on what they have; no stored voxel sees the result.
    auto body = [&](auto Mode, int s, int p) {
        constexpr int MODE = decltype(Mode)::value;
        sfor<K>([&](auto T) {
            constexpr int t = decltype(T)::value + 1;
            const int z = p - t;
            const int pl = before(s, t) * PL;
            const V4 ym = ld4(smm + pl), yp = ld4(smp + pl);
            const V4 zm[R] = {t == 1 ? zm0[0] : ld4(sm + older(s, t) * PL), t == 1 ? zm0[1] : ld4(sm1 + older(s, t) * PL)};
            Sums sums[R];
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const V4 w = cc[t - 1][k];
                const float xl = __shfl_up_sync(0xffffffffu, unpack2(w.b).y, 1);
                const float xr = __shfl_down_sync(0xffffffffu, unpack2(w.a).x, 1);
                sums[k] = lateral_sums(w, k == 0 ? ym : cc[t - 1][0], k == 0 ? cc[t - 1][1] : yp, xl, xr);
            }
            V4 nw[R];
            // the voxels of BC 0's lateral faces among this thread's, instead of what nw holds
            auto lateral = [&](auto Z, int k, V4 zs) {
                constexpr bool ZF = decltype(Z)::value;
                if (xface) {
                    const float e = x_face<ZF, (MODE > 0)>(c, cc[t - 1][k], sums[k], zs, x == 0);
                    const float2 o01 = unpack2(nw[k].a), o23 = unpack2(nw[k].b);
                    nw[k] = {pack2(x == 0 ? e : o01.x, o01.y), pack2(o23.x, x == 0 ? o23.y : e)};
                }
                if (top[k])
                    nw[k] = top_row<ZF, (MODE > 0)>(c, cc[t - 1][k], sums[k], k == 0 ? ym : cc[t - 1][0], zs, x == 0, x + 4 == g.nx);
            };
            if (z != 0 && z != g.nz - 1) {
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    const V4 sz = {add2(cur[k].a, zm[k].a), add2(cur[k].b, zm[k].b)};
                    const V4 q = ld4((k ? sm1 : sm) + heat(s, t) * PL);
                    bool ok = true;
                    // this thread's own value of the level below, of this step, may be of any kind: the
                    // others learn of it at the next barrier
                    if (MODE == 1 && t > 1) ok = !seen0.out();
                    if (MODE == 2) {
                        RangeZero n{verified() ? ~0u : 0u, 0.0f};
                        n.add(sums[k].xa), n.add(sums[k].xb), n.add(sums[k].ya), n.add(sums[k].yb);
                        n.add(sz);
                        ok = n.ok();
                    }
                    nw[k] = ok ? interior4(d, sums[k], sz, q) : interior4_any(c, sums[k], sz, q);
                    if (BC == 0) lateral(std::false_type{}, k, sz);
                }
            } else {
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    const V4 zn = z == 0 ? cur[k] : zm[k];
                    nw[k] = face4<(MODE > 0)>(c, zn, sums[k]);
                    if (BC == 0) lateral(std::true_type{}, k, zn);
                }
            }
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const float2 w01 = unpack2(cc[t - 1][k].a), w23 = unpack2(cc[t - 1][k].b);
                const float2 o01 = unpack2(nw[k].a), o23 = unpack2(nw[k].b);
                nw[k].a = pack2(blend(kl[k], w01.x, o01.x), blend(keep[k], w01.y, o01.y));
                nw[k].b = pack2(blend(keep[k], w23.x, o23.x), blend(kr[k], w23.y, o23.y));
                if (t < K && MODE == 0) seen.add(nw[k]);
                if (t < K && MODE == 1) seen0.add(nw[k]);
            }
            if (t == K) store(z, nw);
#pragma unroll
            for (int k = 0; k < R; ++k) {
                cc[t - 1][k] = cur[k];
                cur[k] = nw[k];
            }
        });
        leave(s);
    };
    // A step whose levels have nothing to compute yet: plane p only moves into place.
    auto skip = [&](int s) {
#pragma unroll
        for (int k = 0; k < R; ++k) cc[0][k] = cur[k];
        leave(s);
    };
    // The first step is one, and so is the second unless the chunk starts at the first slice: up to
    // half of the steps of the two- and four-plane chunks that small grids are cut into.
    constexpr std::integral_constant<int, 0> in_range{};
    constexpr std::integral_constant<int, 1> zeros{};
    constexpr std::integral_constant<int, 2> any{};
    int p = plo;
    if constexpr (ORDINARY) {
        bool good = !arrive(in_range, 0);
        if (good) {
            skip(0);
            ++p;
            good = !arrive(in_range, 1);
        }
        if (good) {
            if (plo > 0)
                skip(1);
            else
                body(in_range, 1, p);
            if (++p > pend) return z1;
            for (;;) {  // slots as constants: four steps to an iteration
                if (arrive(in_range, 2)) break;
                body(in_range, 2, p);
                if (++p > pend) return z1;
                if (arrive(in_range, 3)) break;
                body(in_range, 3, p);
                if (++p > pend) return z1;
                if (arrive(in_range, 0)) break;
                body(in_range, 0, p);
                if (++p > pend) return z1;
                if (arrive(in_range, 1)) break;
                body(in_range, 1, p);
                if (++p > pend) return z1;
            }
        }
        cp_async_wait<0>();
        __syncthreads();
        return max(z0, p - K);
    } else {
        int s = 0;
        auto step = [&](auto Mode) {
            if (p < plo + (plo > 0 ? 2 : 1))
                skip(s);
            else
                body(Mode, s, p);
            s = (s + 1) % kRing;
            return ++p > pend;
        };
        // zeros and values down to 2^-77 first: the same step (the faces test their numerators); from the
        // first value below that every numerator is tested
        while (!arrive(zeros, s))
            if (step(zeros)) return z1;
        for (;;) {
            if (step(any)) return z1;
            arrive(any, s);
        }
    }
}

template <int BC, int K, int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS)
    k_heat_block(float *__restrict__ Tf, const float *__restrict__ Ti, const float *__restrict__ QK,
                 const __grid_constant__ HeatCoef c, const __grid_constant__ HeatBlockGrid g) {
    // Short chunks: the next sweep's blocks may start as soon as all of these have, so that their
    // set-up up to their own wait overlaps this launch's last planes. Of long ones it takes SM
    // slots for nothing (256x256x400 oven 48.4 us per sweep with it, 47.8 without).
    if (g.zc <= 16) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int z0 = (int)blockIdx.z * g.zc, z1 = min(g.nz, z0 + g.zc);
    const int z = heat_chunk<BC, K, THREADS, true>(Tf, Ti, QK, c, g, z0, z1);
    // The planes from a value out of range on. A crystal at 0 C has them: it holds zeros for good on the
    // faces that are never written, and heat spreads into the rest in small values. us per sweep with
    // heat down to 1e-20 from a zero crystal, open top / oven, ordinary temperatures in brackets:
    // 64x64x200 8.2 (5.1) / 5.4 (3.8), 128x128x200 11.8 (8.8) / 7.8 (6.3), 256x256x400 74 (60) / 52 (45.6). With
    // the heat of a Gaussian that underflows to denormals a launch waits for its blocks in the corners:
    // 64x64x200 8.4 / 6.0, 128x128x200 19 / 13, 256x256x400 265 / 215 (the single-sweep kernels: 17 / 11, 23 / 16,
    // 95 / 83). In line: as a function called here it cost the ordinary chunk registers that are kept
    // across calls (256x256x400 oven 45.9; 77 / 56 from a zero crystal, 274 / 233 with denormals).
    if (z < z1) heat_chunk<BC, K, THREADS, false>(Tf, Ti, QK, c, g, z, z1);
}

typedef void (*HeatBlockKernel)(float *, const float *, const float *, const HeatCoef, const HeatBlockGrid);

template <int BC, int THREADS>
HeatBlockKernel kernel_k(int K) {
    switch (K) {
        case 1: return k_heat_block<BC, 1, THREADS>;
        default: return k_heat_block<BC, 2, THREADS>;
    }
}

HeatBlockKernel kernel_of(int bc, int K, int threads) {
    if (threads == 256) return bc == 0 ? kernel_k<0, 256>(K) : kernel_k<1, 256>(K);
    return bc == 0 ? kernel_k<0, 512>(K) : kernel_k<1, 512>(K);
}

}  // namespace

bool heat_block_supported(int nx, int ny, int nz) {
    return nx % 4 == 0 && nx >= 8 && ny >= 2 && nz >= 2 && (long long)nx * ny * nz < (1ll << 31);
}

// Tiling and sweeps per launch for a grid: the candidate whose modelled time per sweep is
// least. The model (cycles at 1.92 GHz, fitted to the sweeps measured below): 4300 cycles per wave
// of blocks (launch, set-up, first planes), then per z step that computes 1500 (2500 with two
// sweeps in flight) at 16 warps per SM, a third of which is latency; with the open top's lateral
// faces 1700 + 70000 / NX (their lanes' share of a warp falls with NX), 1.65 times that with two
// sweeps. A launch that leaves slots free is marked up by a third: the next launch's early blocks
// crowd onto the same SMs. A sweep that does not fit L2 cannot beat 2600 bytes per cycle. Two
// sweeps per launch halve the memory traffic and the launches but add two rows of halo on each
// side and two planes at each chunk's ends; three and four were built too and lost (their state
// spills at the 128 registers of two 256-thread blocks per SM). us per sweep on GB300, the
// TMA-staged sweep (shg_heat_tma.cu) -> one / two sweeps per launch here:
//   32x32x50    open top 14.8 -> 4.4 / 4.8,   oven 10.6 -> 2.6 / 2.6
//   64x64x200   open top 14.7 -> 5.6 / 6.4,   oven 10.6 -> 4.2 / 4.2
//   100x100x75  open top 16.8 -> 4.7 / 5.8,   oven 11.6 -> 4.1 / 4.0
//   128x128x200 open top 21.0 -> 9.6 / 9.8,   oven 14.8 -> 7.6 / 6.7
//   200x200x150 open top 32.5 -> 19.5 / 19.4, oven 25.4 -> 16.6 / 14.2
//   256x256x400 open top 86.2 -> 69.2 / 65.9, oven 71.4 -> 64.8 / 48.4
// (47 us is the HBM copy rate for one sweep's 12 bytes per voxel.) The plan's choice now, same grids, open top /
// oven: 3.9 / 2.3, 5.1 / 3.8, 4.4 / 3.6, 8.8 / 6.3, 17.8 / 13.3, 59.7 / 45.6. At 256x256x400 oven with two sweeps
// per launch: 73 warp instructions per four voxels and level of a warp, 46 % issue, FMA pipe 22 % (the packed
// forms take it for two cycles), shared-memory latency the top stall.
// The plan of one tiling: regions of vx vectors by kRows threads / vx rows (a whole row, or tiles with a
// halo vector on each side), chunks of zc planes. False for what is none.
static bool tile_plan(int nx, int ny, int nz, int levels, int threads, int vx, int zc, HeatBlockPlan *out) {
    if (levels < 1 || levels > kMaxLevels || (threads != 256 && threads != 512) || vx < 2 || vx > 32 || (vx & (vx - 1)) ||
        zc < 1 || zc > nz)
        return false;
    const int vecs = nx / 4, rows = kRows * (threads / vx);
    const bool whole_x = vx >= vecs, whole_y = rows >= ny;
    if ((!whole_x && vx < 8) || (!whole_y && rows <= 2 * levels)) return false;
    const int ti = whole_x ? vecs : vx - 2, tyi = whole_y ? ny : rows - 2 * levels;
    out->g = HeatBlockGrid{nx, ny, nz, vx, 4 * ti, tyi, whole_x ? 0 : 4, whole_y ? 0 : levels, zc};
    out->grid = dim3((vecs + ti - 1) / ti, (ny + tyi - 1) / tyi, (nz + zc - 1) / zc);
    out->threads = threads;
    out->levels = levels;
    out->smem = (size_t)shared_planes(levels) * plane_floats(threads, kRows) * sizeof(float);
    return true;
}

static cudaError_t allow_shared(const HeatBlockPlan &p, int bc) {
    return cudaFuncSetAttribute(kernel_of(bc, p.levels, p.threads), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)p.smem);
}

static cudaError_t search_plan(int dev, int nx, int ny, int nz, int bc, int levels, HeatBlockPlan *out) {
    int sms = 0;
    cudaError_t e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    constexpr double kWave = 4300, kBytesPerCycle = 2600, kL2 = 100e6;
    const double bytes = 12.0 * nx * ny * nz;
    const int vecs = nx / 4;
    double best = 1e300;
    for (int K = levels ? levels : 1; K <= (levels ? levels : kMaxLevels); ++K)
        for (int threads = 256; threads <= 512; threads *= 2)
            for (int vx = 2; vx <= 32; vx *= 2) {
                HeatBlockPlan t;
                if (!tile_plan(nx, ny, nz, K, threads, vx, nz, &t)) continue;
                const int bps = 512 / threads, warps = threads / 128;  // blocks per SM, warps per scheduler of one
                const long long slots = (long long)bps * sms, tiles = (long long)t.grid.x * t.grid.y;
                for (int nc = 1; nc <= nz; ++nc) {
                    const int zc = (nz + nc - 1) / nc;
                    const long long blocks = tiles * ((nz + zc - 1) / zc), waves = (blocks + slots - 1) / slots;
                    const double w = warps * (waves > 1 ? (double)bps : (double)((blocks + sms - 1) / sms));
                    const double full = bc == 0 ? (1700 + 70000.0 / nx) * (K == 1 ? 1.0 : 1.65) : K == 1 ? 1500 : 2500;
                    double cost = waves * (kWave + (zc + 2 * K - 2) * full * (0.35 + 0.65 * w / 4));
                    if (waves == 1 && 5 * blocks < 4 * slots) cost *= 1.35;
                    if (bytes > kL2) cost = std::max(cost, bytes / kBytesPerCycle);
                    if (cost / K < best) {
                        best = cost / K;
                        tile_plan(nx, ny, nz, K, threads, vx, zc, out);
                    }
                    if (blocks > 8 * slots) break;
                }
                if (vx >= vecs) break;
            }
    if (best == 1e300) return cudaErrorInvalidConfiguration;
    return allow_shared(*out, bc);
}

cudaError_t heat_block_tiling(int nx, int ny, int nz, int bc, int levels, int threads, int vx, int zc, HeatBlockPlan *out) {
    if (!heat_block_supported(nx, ny, nz) || !tile_plan(nx, ny, nz, levels, threads, vx, zc, out)) return cudaErrorInvalidValue;
    return allow_shared(*out, bc);
}

cudaError_t heat_block_plan(int nx, int ny, int nz, int bc, int levels, HeatBlockPlan *out) {
    if (!heat_block_supported(nx, ny, nz) || levels < 0 || levels > kMaxLevels) return cudaErrorInvalidValue;
    // the search is tens of microseconds, as long as a few sweeps: kept per device and grid
    static std::mutex mu;
    static std::map<std::tuple<int, int, int, int, int, int>, HeatBlockPlan> plans;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const auto key = std::make_tuple(dev, nx, ny, nz, bc != 0, levels);
    std::lock_guard<std::mutex> lock(mu);
    const auto it = plans.find(key);
    if (it != plans.end()) {
        *out = it->second;
        return cudaSuccess;
    }
    if ((e = search_plan(dev, nx, ny, nz, bc, levels, out)) != cudaSuccess) return e;
    if (plans.size() >= 256) plans.clear();
    plans[key] = *out;
    return cudaSuccess;
}

cudaError_t launch_heat_block(float *Tf, const float *Ti, const float *QK, const HeatCoef &c, int bc,
                              const HeatBlockPlan &p, cudaStream_t st) {
    // programmatic serialisation (the kernel waits for the launch before it): a plain chain of
    // launches takes 4.1 us each on GB300 and grows in steps of 2.05 us with the kernels' time,
    // this one 1.4 us and the kernels' time
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = p.grid;
    cfg.blockDim = dim3(p.threads, 1, 1);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel_of(bc, p.levels, p.threads), Tf, Ti, QK, c, p.g);
}

}  // namespace shg
