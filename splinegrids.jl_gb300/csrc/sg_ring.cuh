// sg_ring.cuh -- per-grid adjoint passes: an axis k >= 1 as warp-private cp.async rings or columns,
// axis 0 as shared-memory tiles, and one thread per output for short sums and small passes.
// (Which runs, and where the warp tasks of sg_warp.cuh do: adj_axis_kernel, adj_axis0_kernel.)
//
// Unless said otherwise they sum the samples of a control point from zero in increasing
// view order, one FMA per sample: the order (and so the bits) of the other adjoint kernels.
#pragma once

#include <cooperative_groups.h>

#include "sg_warp.cuh"

namespace sg {

// ---------------------------------------------------------------------------------
// Axis k >= 1 (the map of adj_axis_warp): Y[m, c, q] = sum_j B[j, c - b(j)] X[m, j, q].
// The pass streams X, the largest array of the adjoint, and is bound by the bytes in
// flight.  Unit = one warp x 32*VEC consecutive m x CC control points x one column; a
// CTA is one warp, so units start and end on their own.  Each lane keeps a ring of
// kRingRows rows of its own 16 bytes in shared memory, filled by cp.async kRingGroup
// rows per commit group: 16 KB in flight per warp without a register or a barrier (a
// lane reads only what it copied itself).  A few warps per SM already cover the memory
// latency, so units can be long, and the d spans a unit shares with the next one (its
// halo, read twice) stay a small part of it.  Support starts come from the support
// table (the position where the next control point completes is a register compare per
// row); basis rows are staged 32 at a time, one per lane.
// Measured on (256, 256) -> (4096, 4096), 3 channels, Float32 (201 MB): 42 us, 5.4 TB/s with
// the halo's 12 % (the 1024-wide stream tiles of the batch queue: 56 us; a copy: 30 us).
// What is left is the rows around completed control points and the halo.
// ---------------------------------------------------------------------------------
constexpr int kRingRows = 32;      // rows of the ring
constexpr int kRingGroup = 8;      // rows per commit group (a wait costs ~100 cycles: 4-row groups were slower)

// Values as the kernel computes with them: Float32 pairs use the packed FMA, with the
// basis values staged as (b, b) pairs.
template <typename T>
struct RingV;
template <>
struct RingV<float> {
    using V = float2;
    static __device__ __forceinline__ V zero() { return make_float2(0.f, 0.f); }
    static __device__ __forceinline__ V bcast(float b) { return make_float2(b, b); }
    static __device__ __forceinline__ V fma(V b, V x, V c) { return __ffma2_rn(b, x, c); }
    template <int H>
    static __device__ __forceinline__ void ld(const void *p, V (&v)[H]) {
        if constexpr (H == 2) {
            const float4 t = *reinterpret_cast<const float4 *>(p);
            v[0] = make_float2(t.x, t.y);
            v[1] = make_float2(t.z, t.w);
        } else {
            v[0] = *reinterpret_cast<const float2 *>(p);
        }
    }
    template <int H>
    static __device__ __forceinline__ void st(float *p, const V (&v)[H]) {
        if constexpr (H == 2) *reinterpret_cast<float4 *>(p) = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
        else *reinterpret_cast<float2 *>(p) = v[0];
    }
};
template <>
struct RingV<double> {
    using V = double;
    static __device__ __forceinline__ V zero() { return 0.0; }
    static __device__ __forceinline__ V bcast(double b) { return b; }
    static __device__ __forceinline__ V fma(V b, V x, V c) { return ::fma(b, x, c); }
    template <int H>
    static __device__ __forceinline__ void ld(const void *p, V (&v)[H]) {
        if constexpr (H == 2) {
            const double2 t = *reinterpret_cast<const double2 *>(p);
            v[0] = t.x;
            v[1] = t.y;
        } else {
            v[0] = *reinterpret_cast<const double *>(p);
        }
    }
    template <int H>
    static __device__ __forceinline__ void st(double *p, const V (&v)[H]) {
        if constexpr (H == 2) *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
        else *p = v[0];
    }
};
template <int D>
__host__ __device__ constexpr int ring_row_vals() { return (D + 1) / 2 * 2; }  // staged rows of 16-byte multiples
template <int D, typename T>
__host__ __device__ constexpr int ring_smem() {
    return kRingRows * 512 + 32 * ring_row_vals<D>() * (int)sizeof(typename RingV<T>::V);
}

template <int D, typename T>
__global__ void __launch_bounds__(32)
k_adj_ring(const int32_t *__restrict__ perm, const int32_t *__restrict__ lb, const T *__restrict__ B, int64_t ns,
           const T *__restrict__ X, int64_t M, int64_t n, int CC, int64_t gxw, int64_t chunks, T *__restrict__ Y) {
    constexpr int d = D - 1;
    constexpr int VEC = 16 / (int)sizeof(T);  // values per lane
    constexpr int RV = ring_row_vals<D>();
    constexpr int G = kRingGroup, NG = kRingRows / G;
    constexpr int RB = 512;                   // bytes of a ring row
    using RT = RingV<T>;
    using V = typename RT::V;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x;
    unsigned char *const ring = smem + lane * 16, *const ring_end = ring + kRingRows * RB;
    V *s_B = reinterpret_cast<V *>(smem + kRingRows * RB);
    const int64_t unit = blockIdx.x + grid_start();
    const int64_t mw = unit % gxw, rest = unit / gxw;
    const int64_t chunk = rest % chunks, q = rest / chunks;
    const int c0 = (int)(chunk * CC);
    const int c1 = (c0 + CC < n) ? c0 + CC : (int)n;
    const int s_lo = lb[c0], s_hi = lb[c1 + d];  // support starts c0 - d .. c1 - 1
    const int64_t m0 = (mw * 32 + lane) * VEC;
    const bool act = m0 < M;
    const T *xq = X + m0 + M * ns * q;

    const T *src = xq + M * (int64_t)s_lo;  // next row to copy (sorted axis)
    int next = s_lo;
    unsigned char *ip = ring;               // where it goes
    auto issue = [&]() {                    // the next G rows
        if (act) {
            if (!perm && next + G <= s_hi) {
                const T *p = src;
#pragma unroll
                for (int u = 0; u < G; ++u) {
                    cp_async<16>(ip + u * RB, p);
                    p += M;
                }
                src = p;
            } else {
                for (int u = 0; u < G && next + u < s_hi; ++u)
                    cp_async<16>(ip + u * RB, xq + M * (int64_t)(perm ? perm[next + u] : next + u));
            }
        }
        next += G;
        ip += G * RB;
        if (ip == ring_end) ip = ring;
        cp_async_commit();
    };
#pragma unroll
    for (int g = 0; g + 1 < NG; ++g) issue();

    T nb[D];  // the next 32 rows' basis values, one row per lane
    auto fetch = [&](int r0) {
        const int s = r0 + lane;
        if (s < s_hi) {
            const int64_t j = perm ? perm[s] : s;
#pragma unroll
            for (int i = 0; i < D; ++i) nb[i] = B[j + ns * i];
        }
    };
    fetch(s_lo);

    V acc[D][2];
#pragma unroll
    for (int i = 0; i < D; ++i) acc[i][0] = acc[i][1] = RT::zero();
    int cur = c0 - d;                     // control point of acc[0]
    int bd = lb[c0 + 1];                  // cur is complete at this position: lb[cur + 1 + d]
    int bdn = lb[(c0 + 2 <= n + d) ? c0 + 2 : (int)n + d];
    T *y = Y + m0 + M * (n * q + c0);     // control point max(cur, c0)
    auto flush = [&]() {
        if (cur >= c0) {
            if (act) RT::template st<2>(y, acc[0]);
            y += M;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int i = 0; i + 1 < D; ++i) acc[i][h] = acc[i + 1][h];
            acc[D - 1][h] = RT::zero();
        }
        ++cur;
        bd = bdn;
        const int64_t nx = (int64_t)cur + 2 + d;
        bdn = lb[nx <= n + d ? nx : n + d];
    };
    const unsigned char *xr = ring;
    for (int s = s_lo; s < s_hi; s += G) {
        const int in = (s - s_lo) & 31;
        if (in == 0) {  // a new batch of 32 basis rows
            __syncwarp();
#pragma unroll
            for (int i = 0; i < D; ++i) s_B[lane * RV + i] = RT::bcast(nb[i]);
            __syncwarp();
            fetch(s + 32);
        }
        const V *br = s_B + in * RV;
        cp_async_wait<NG - 2>();  // the group has landed (each lane reads what it copied)
#pragma unroll 1
        for (int t = s; t < s + G && t < s_hi; t += 4) {  // four rows in registers
            V x[4][2], b[4][RV];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                RT::template ld<2>(xr + u * RB, x[u]);
#pragma unroll
                for (int i = 0; i < RV; i += 2) {
                    V h[2];
                    RT::template ld<2>(br + u * RV + i, h);
                    b[u][i] = h[0];
                    b[u][i + 1] = h[1];
                }
            }
            xr += 4 * RB;
            br += 4 * RV;
            auto add = [&](int u) {
#pragma unroll
                for (int i = 0; i < D; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) acc[i][h] = RT::fma(b[u][i], x[u][h], acc[i][h]);
            };
            // segments of the four rows between completed control points
            const int lim = s_hi - t < 4 ? s_hi - t : 4;
            for (int lo = 0;;) {
                const int hi = bd - t < lim ? bd - t : lim;
                if (lo == 0 && hi == 4) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) add(u);
                } else {
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (u >= lo && u < hi) add(u);
                }
                lo = hi;
                if (bd - t > lim || cur >= c1) break;
                flush();
            }
        }
        if (xr == ring_end) xr = ring;
        issue();  // into the group consumed one step ago
    }
    cp_async_wait<0>();
    while (cur < c1) flush();
}

// ---------------------------------------------------------------------------------
// Axis k >= 1, medium sizes and rows that are not 16-byte multiples: unit = one warp x 32
// consecutive m (one value per lane, any alignment) x CC control points x one column.
// Rows are loaded straight into registers, two groups of U in flight per warp.  Also every
// Float64 pass: those are bound by the FP64 pipe (D FMAs per value, 64 cycles per warp
// instruction and SM sub-partition), so what counts is even work per sub-partition.
// Measured: (1999, 1501) x 3 Float32 16 us (warp tasks with strided 16-byte lanes: 47);
// (4096, 4096) x 3 Float64, degree 3: 430 us, 1.0 of 1.2 TFLOP/s (fused tiles: 527).
// ---------------------------------------------------------------------------------
constexpr int kColsWarps = 4;  // units per CTA, neighbours along m

template <int D, typename T, int U>
__global__ void __launch_bounds__(32 * kColsWarps)
k_adj_cols(const int32_t *__restrict__ perm, const int32_t *__restrict__ lb, const T *__restrict__ B, int64_t ns,
           const T *__restrict__ X, int64_t M, int64_t n, int CC, int64_t gxw, int64_t chunks, int64_t units,
           T *__restrict__ Y) {
    constexpr int d = D - 1;
    constexpr int RV = ring_row_vals<D>();
    static_assert(32 % U == 0, "groups divide the staged batch");
    __shared__ __align__(16) T sh[kColsWarps][32 * RV];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t unit = (int64_t)blockIdx.x * kColsWarps + w + grid_start();
    if (unit >= units) return;
    T *s_B = sh[w];
    const int64_t mw = unit % gxw, rest = unit / gxw;
    const int64_t chunk = rest % chunks, q = rest / chunks;
    const int c0 = (int)(chunk * CC);
    const int c1 = (c0 + CC < n) ? c0 + CC : (int)n;
    const int s_lo = lb[c0], s_hi = lb[c1 + d];
    const int64_t m0 = mw * 32 + lane;
    const bool act = m0 < M;
    const T *xq = X + m0 + M * ns * q;
    T *yq = Y + m0 + M * n * q;
    auto load = [&](T (&x)[U], int r0) {
        if (act) {
            if (!perm && r0 + U <= s_hi) {
                const T *p = xq + M * (int64_t)r0;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    x[u] = __ldg(p);
                    p += M;
                }
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (r0 + u < s_hi) x[u] = __ldg(xq + M * (int64_t)(perm ? perm[r0 + u] : r0 + u));
            }
        }
    };
    T nb[D];
    auto fetch = [&](int r0) {
        const int s = r0 + lane;
        if (s < s_hi) {
            const int64_t j = perm ? perm[s] : s;
#pragma unroll
            for (int i = 0; i < D; ++i) nb[i] = B[j + ns * i];
        }
    };
    T xa[U], xb[U];
#pragma unroll
    for (int u = 0; u < U; ++u) xa[u] = xb[u] = T(0);
    load(xa, s_lo);
    fetch(s_lo);
    T acc[D];
#pragma unroll
    for (int i = 0; i < D; ++i) acc[i] = T(0);
    int cur = c0 - d, bd = lb[c0 + 1];
    int bdn = lb[(c0 + 2 <= n + d) ? c0 + 2 : (int)n + d];
    auto flush = [&]() {
        if (cur >= c0 && act) yq[M * cur] = acc[0];
#pragma unroll
        for (int i = 0; i + 1 < D; ++i) acc[i] = acc[i + 1];
        acc[D - 1] = T(0);
        ++cur;
        bd = bdn;
        const int64_t nx = (int64_t)cur + 2 + d;
        bdn = lb[nx <= n + d ? nx : n + d];
    };
    auto row = [&](T x, const T *b) {
        T bv[RV];
        if constexpr (sizeof(T) == 4 && RV % 4 == 0) {
#pragma unroll
            for (int i = 0; i < RV; i += 4) {
                const float4 t = *reinterpret_cast<const float4 *>(b + i);
                bv[i] = t.x; bv[i + 1] = t.y; bv[i + 2] = t.z; bv[i + 3] = t.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < RV; i += 2) {
                if constexpr (sizeof(T) == 4) {
                    const float2 t = *reinterpret_cast<const float2 *>(b + i);
                    bv[i] = t.x; bv[i + 1] = t.y;
                } else {
                    const double2 t = *reinterpret_cast<const double2 *>(b + i);
                    bv[i] = t.x; bv[i + 1] = t.y;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < D; ++i) acc[i] = ::fma(bv[i], x, acc[i]);
    };
    auto group = [&](const T (&x)[U], int s) {
        const T *br = s_B + ((s - s_lo) & 31) * RV;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (s + u < s_hi) {
                while (s + u == bd) flush();
                row(x[u], br + u * RV);
            }
        }
    };
    for (int s = s_lo; s < s_hi; s += 2 * U) {
        if (((s - s_lo) & 31) == 0) {
            __syncwarp();
#pragma unroll
            for (int i = 0; i < D; ++i) s_B[lane * RV + i] = nb[i];
            __syncwarp();
            fetch(s + 32);
        }
        if (s + U < s_hi) load(xb, s + U);
        group(xa, s);
        if (s + U < s_hi) {
            if (s + 2 * U < s_hi) load(xa, s + 2 * U);
            group(xb, s + U);
        }
    }
    while (cur < c1) flush();
}

// ---------------------------------------------------------------------------------
// Axis 0 (M = 1): Y[c, q] = sum_j B[j, c - b(j)] X[j, q], X [ns, Q], Y [n, Q].
// CTA = 32 columns x kA0Cp control points.  The samples of their supports are staged in
// shared memory in segments (cp.async, coalesced along the samples; the CTAs of an SM
// overlap one another's waits); lane = column (odd row stride: no bank conflicts), warp =
// control point.  Results leave through shared memory, eight consecutive control points
// of a column at a time: a warp's own 32 results lie n apart.  ((1999, 131) x 3: warp
// tasks with transpose tiles 18 us, these tiles 8.)
// ---------------------------------------------------------------------------------
constexpr int kA0Warps = 8;
constexpr int kA0Cp = kA0Warps;  // control points per CTA, one per warp
template <typename T>
__host__ __device__ constexpr int a0_seg() { return sizeof(T) == 4 ? 192 : 96; }  // samples per segment
// Row stride of the staged columns: odd for single values; 4 past a multiple of 32 banks for
// 16-byte loads (eight lanes of a load then cover all banks).
template <typename T, bool V4>
__host__ __device__ constexpr int a0_stride() { return a0_seg<T>() + (V4 ? 4 : 1); }
template <int D, typename T, bool V4>
__host__ __device__ constexpr int a0_smem() {
    return (int)(align16(32 * a0_stride<T, V4>() * (int64_t)sizeof(T)) + align16(a0_seg<T>() * D * (int64_t)sizeof(T)));
}

// V4 (Float32, sorted samples, ns a multiple of 4, X and B on 16-byte boundaries): samples are
// copied and read four at a time, from the multiple of 4 at or before the first.  The tiles are
// bound by the issue of their instructions: 256 control points, 4096 samples, 768 columns, degree
// 3: 1063 a warp and 12.3 us with single values, 767 and 9.3 us so.
template <int D, typename T, bool V4>
__global__ void __launch_bounds__(32 * kA0Warps)
k_adj0_tile(const int32_t *__restrict__ perm, const int32_t *__restrict__ lb, const T *__restrict__ B, int64_t ns,
            const T *__restrict__ X, int64_t n, int64_t Q, int64_t groups, T *__restrict__ Y) {
    static_assert(!V4 || sizeof(T) == 4, "16-byte groups of four");
    constexpr int d = D - 1;
    constexpr int SEG = a0_seg<T>(), STR = a0_stride<T, V4>();
    extern __shared__ __align__(16) unsigned char smem[];
    T *xs = reinterpret_cast<T *>(smem);  // [32][STR]
    T *bs = reinterpret_cast<T *>(smem + align16(32 * STR * (int64_t)sizeof(T)));  // [D][SEG]
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t tile = blockIdx.x + grid_start();
    const int64_t q0 = (tile % groups) * 32;
    const int c0 = (int)(tile / groups) * kA0Cp;
    const int c1 = c0 + kA0Cp < n ? c0 + kA0Cp : (int)n;
    const int c = c0 + w;  // this warp's control point
    const int s_hi = lb[c1 + d], s_lo = V4 ? lb[c0] & ~3 : lb[c0];
    int bd[D + 1];  // support starts c - d .. c, one span each: span i holds the samples whose
                    // basis value i belongs to c, [bd[d - i], bd[d - i + 1])
#pragma unroll
    for (int i = 0; i <= D; ++i) bd[i] = c < c1 ? lb[c + i] : 0;
    T acc = T(0);
    for (int sb = s_lo; sb < s_hi; sb += SEG) {
        const int nb = s_hi - sb < SEG ? s_hi - sb : SEG;
        if (sb != s_lo) __syncthreads();
        for (int k = w; k < 32; k += kA0Warps) {
            if (q0 + k < Q) {
                const T *xc = X + ns * (q0 + k);
                T *xd = xs + k * STR;
                if constexpr (V4) {  // whole groups: the last may end past s_hi, not past ns
                    for (int t = 4 * lane; t < nb; t += 128) cp_async<16>(xd + t, xc + sb + t);
                } else {
                    for (int t = lane; t < nb; t += 32)
                        cp_async<(int)sizeof(T)>(xd + t, xc + (perm ? perm[sb + t] : sb + t));
                }
            }
        }
        if constexpr (V4) {
            for (int t = 4 * lane; w < D && t < nb; t += 128) cp_async<16>(bs + w * SEG + t, B + ns * w + sb + t);
        } else {
            for (int t = threadIdx.x; t < nb; t += 32 * kA0Warps) {
                const int64_t j = perm ? perm[sb + t] : sb + t;
#pragma unroll
                for (int i = 0; i < D; ++i) cp_async<(int)sizeof(T)>(bs + i * SEG + t, B + j + ns * i);
            }
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        const T *xl = xs + lane * STR - sb;
#pragma unroll
        for (int i = D - 1; i >= 0; --i) {
            const int a = bd[d - i] > sb ? bd[d - i] : sb;
            const int z = bd[d - i + 1] < sb + nb ? bd[d - i + 1] : sb + nb;
            const T *bi = bs + i * SEG - sb;
            if constexpr (V4) {
                int g = a & ~3;
                auto part = [&]() {  // the samples of group g inside [a, z)
                    const float4 x = *reinterpret_cast<const float4 *>(xl + g);
                    const float4 v = *reinterpret_cast<const float4 *>(bi + g);
                    if (g >= a) acc = ::fma(v.x, x.x, acc);  // (g < z)
                    if (g + 1 >= a && g + 1 < z) acc = ::fma(v.y, x.y, acc);
                    if (g + 2 >= a && g + 2 < z) acc = ::fma(v.z, x.z, acc);
                    if (g + 3 < z) acc = ::fma(v.w, x.w, acc);  // (g + 3 >= a)
                    g += 4;
                };
                if (a < z && g < a) part();
#pragma unroll 4
                for (; g + 4 <= z; g += 4) {
                    const float4 x = *reinterpret_cast<const float4 *>(xl + g);
                    const float4 v = *reinterpret_cast<const float4 *>(bi + g);
                    acc = ::fma(v.x, x.x, acc);
                    acc = ::fma(v.y, x.y, acc);
                    acc = ::fma(v.z, x.z, acc);
                    acc = ::fma(v.w, x.w, acc);
                }
                if (a < z && g < z) part();
            } else {
#pragma unroll 8
                for (int s = a; s < z; ++s) acc = ::fma(bi[s], xl[s], acc);
            }
        }
    }
    // out through shared memory: kA0Cp consecutive control points of a column per store group
    __syncthreads();
    xs[lane * (kA0Cp + 1) + w] = acc;
    __syncthreads();
    for (int t = threadIdx.x; t < 32 * kA0Cp; t += 32 * kA0Warps) {
        const int k = t / kA0Cp, c = c0 + t % kA0Cp;
        if (c < c1 && q0 + k < Q) Y[c + n * (q0 + k)] = xs[k * (kA0Cp + 1) + t % kA0Cp];
    }
}

// ---------------------------------------------------------------------------------
// Nin = 1 with long supports: Y[c, q] = sum over the support of c.  A curve has few
// control points and no other axis to spread over, so a sequential sum per control point is
// one chain of thousands of FMAs on a handful of SMs.  Here a cluster of S CTAs shares
// one control point: every thread sums each (S * kLineThreads)th part of its CTA's
// stretch of the support, the threads' sums are added in a fixed tree and the CTAs' in
// rank order (through distributed shared memory).  Deterministic; the order depends on the
// grid's sizes only, and the batch runs such grids through this kernel too, so both give
// the same bits.  QT columns per CTA share the basis values.
// Measured on 200 control points, 100001 samples, 2 columns, Float32: 353 -> 4 us.
// ---------------------------------------------------------------------------------
constexpr int kLineThreads = 256;
constexpr int64_t kLineSupport = 256;  // supports longer than this: below, one thread per output is as fast

template <int D, typename T, int QT>
__global__ void __launch_bounds__(kLineThreads)
k_adj_line(const int32_t *__restrict__ perm, const int32_t *__restrict__ lb, const T *__restrict__ B, int64_t ns,
           const T *__restrict__ X, int64_t n, int64_t Q, int S, T *__restrict__ Y) {
    __shared__ T part[kLineThreads / 32][QT];
    __shared__ T total[QT];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t block = blockIdx.x + grid_start();
    const int64_t unit = block / S;
    const int rank = (int)(block % S);
    const int64_t c = unit % n, q0 = (unit / n) * QT;
    const int64_t lo = lb[c], len = lb[c + D] - lo;
    const int64_t per = (len + S - 1) / S;
    const int64_t a = lo + rank * per, z = a + per < lo + len ? a + per : lo + len;
    T acc[QT];
#pragma unroll
    for (int q = 0; q < QT; ++q) acc[q] = T(0);
#pragma unroll
    for (int k = 0; k < D; ++k) {  // the samples with support start c - d + k
        const int64_t b0 = lb[c + k], b1 = lb[c + k + 1];
        const int64_t s1 = z < b1 ? z : b1;
        const T *bk = B + ns * (D - 1 - k);
#pragma unroll 4
        for (int64_t s = (a > b0 ? a : b0) + threadIdx.x; s < s1; s += kLineThreads) {
            const int64_t j = perm ? perm[s] : s;
            const T b = bk[j];
#pragma unroll
            for (int q = 0; q < QT; ++q)
                if (q0 + q < Q) acc[q] = ::fma(b, X[j + ns * (q0 + q)], acc[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < QT; ++q) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
        if (lane == 0) part[w][q] = acc[q];
    }
    __syncthreads();
    if (threadIdx.x < QT) {
        T t = part[0][threadIdx.x];
#pragma unroll
        for (int i = 1; i < kLineThreads / 32; ++i) t += part[i][threadIdx.x];
        total[threadIdx.x] = t;
    }
    if (S > 1) {
        cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
        cl.sync();
        if (rank == 0 && threadIdx.x < QT) {
            T t = total[threadIdx.x];
            for (int r = 1; r < S; ++r) t += *cl.map_shared_rank(&total[threadIdx.x], r);
            if (q0 + threadIdx.x < Q) Y[c + n * (q0 + threadIdx.x)] = t;
        }
        cl.sync();  // the other CTAs' sums have been read
    } else if (threadIdx.x < QT && q0 + threadIdx.x < Q) {
        Y[c + n * (q0 + threadIdx.x)] = total[threadIdx.x];
    }
}

// ---------------------------------------------------------------------------------
// One thread per output: no staging, no windows, every load independent.  With few outputs the
// warp tasks of sg_warp.cuh leave most SMs idle and each warp is a chain of dependent steps; with
// short sums or short rows there is little for any staging to share.  The adjoint form takes any axis (M = 1 for axis 0).
// Measured on the (10, 10, 5) -> (50, 50, 25) x 4 volume, Float64: forward 24 -> 7 us, adjoint
// 50 -> 24 us (three passes each).
// ---------------------------------------------------------------------------------
constexpr int kThreadBlock = 128;

template <int D, typename T>
__global__ void __launch_bounds__(kThreadBlock)
k_adj_thread(const int32_t *__restrict__ perm, const int32_t *__restrict__ lb, const T *__restrict__ B, uint32_t ns,
             const T *__restrict__ X, uint32_t M, uint32_t n, uint32_t total, T *__restrict__ Y) {
    constexpr int d = D - 1;
    const uint32_t lin = blockIdx.x * kThreadBlock + threadIdx.x + grid_start();
    if (lin >= total) return;
    const uint32_t r = lin / M, m = lin - r * M;
    const uint32_t q = r / n, c = r - q * n;
    const T *x = X + m + (int64_t)M * ns * q;
    int bd[D + 1];  // spans c - d .. c of the view: [bd[k], bd[k + 1]) has support start c - d + k
#pragma unroll
    for (int k = 0; k <= D; ++k) bd[k] = lb[c + k];
    T acc = T(0);
    constexpr int U = 8;
    for (int s0 = bd[0]; s0 < bd[D]; s0 += U) {
        T b[U], v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {  // independent loads
            const int s = s0 + u;
            if (s < bd[D]) {
                int i = d;
#pragma unroll
                for (int k = 1; k < D; ++k) i -= s >= bd[k];
                const int64_t j = perm ? perm[s] : s;
                b[u] = B[j + (int64_t)ns * i];
                v[u] = x[M * j];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (s0 + u < bd[D]) acc = ::fma(b[u], v[u], acc);
    }
    Y[lin] = acc;
}

template <int D, typename T>
__global__ void __launch_bounds__(kThreadBlock)
k_fwd_thread(const int32_t *__restrict__ idx, const T *__restrict__ B, uint32_t ns, const T *__restrict__ X, uint32_t M,
             uint32_t n, uint32_t total, T *__restrict__ Y) {
    const uint32_t lin = blockIdx.x * kThreadBlock + threadIdx.x + grid_start();
    if (lin >= total) return;
    const uint32_t r = lin / M, m = lin - r * M;
    const uint32_t q = r / ns, j = r - q * ns;
    const int64_t b = support_start(idx[j], D - 1, n);
    const T *x = X + m + (int64_t)M * (b + (int64_t)n * q);
    T a = T(0);
#pragma unroll
    for (int i = 0; i < D; ++i) a = ::fma(B[j + (int64_t)ns * i], x[(int64_t)M * i], a);
    Y[lin] = a;
}

}  // namespace sg
