// sg_refine.cu -- refinement-matrix application (mult!, mult_adjoint!) and the
// local-refinement overwrite (and its adjoint) that build the finest-level control
// points of LocallyRefinedControlPoints (src/control_points.jl:319-349,
// src/adjoint.jl:85-205, src/refinement_matrix.jl:365-445).
#include "sg_common.cuh"

namespace sg {

constexpr int kMaxDims = SG_MAX_NIN + 1;  // control-point dims + the Nout dim

// The banded matrices of one mult!/mult_adjoint! call, by value in kernel parameters.
struct MultArgs {
    int ndims;
    int64_t size_Y[kMaxDims];
    int64_t size_B[kMaxDims];
    int32_t rm_of_dim[kMaxDims];  // index into the arrays below, -1 when not refined
    const int32_t *rp[kMaxDims];  // row_pointer (1-based)
    const int32_t *cs[kMaxDims];  // column_start (1-based)
    const void *nz[kMaxDims];
    int64_t m[kMaxDims], n[kMaxDims], nnz[kMaxDims];
};

// Row i (0-based) of a banded matrix: 0-based first column, column count, 0-based
// nzval offset (get_column_range, src/refinement_matrix.jl:101-125).
__device__ __forceinline__ void row_extent(const MultArgs &a, int r, int64_t i, int64_t &c0,
                                           int64_t &nc, int64_t &z0) {
    const int64_t next = (i == a.m[r] - 1) ? a.nnz[r] + 1 : (int64_t)a.rp[r][i + 1];
    nc = next - a.rp[r][i];
    c0 = (int64_t)a.cs[r][i] - 1;
    z0 = (int64_t)a.rp[r][i] - 1;
}

// Entry `lin` of Y = mult!(B), any dimension count and band width: the sum over the
// product of the row bands in the reference's order (first dim fastest) with the factors
// multiplied in dim order.
template <typename T>
__device__ __forceinline__ T mult_entry(const MultArgs &a, const T *__restrict__ B, int64_t lin) {
    int64_t c0[kMaxDims], nc[kMaxDims], z0[kMaxDims], Jb[kMaxDims];
    int64_t rem = lin, tot = 1;
    for (int dd = 0; dd < a.ndims; ++dd) {
        const int64_t I = rem % a.size_Y[dd];
        rem /= a.size_Y[dd];
        const int r = a.rm_of_dim[dd];
        if (r < 0) { c0[dd] = I; nc[dd] = 1; z0[dd] = 0; }
        else row_extent(a, r, I, c0[dd], nc[dd], z0[dd]);
        if (nc[dd] < 0) nc[dd] = 0;
        tot *= nc[dd];
        Jb[dd] = 0;
    }
    T out = T(0);
    for (int64_t t = 0; t < tot; ++t) {
        int64_t off = 0, stride = 1;
        bool ok = true;
        for (int dd = 0; dd < a.ndims; ++dd) {
            const int64_t J = Jb[dd] + c0[dd];
            ok = ok && J >= 0 && J < a.size_B[dd];
            off += J * stride;
            stride *= a.size_B[dd];
        }
        if (ok) {
            T contrib = B[off];
            for (int dd = 0; dd < a.ndims; ++dd) {
                const int r = a.rm_of_dim[dd];
                if (r >= 0) contrib *= ((const T *)a.nz[r])[z0[dd] + Jb[dd]];
            }
            out += contrib;
        }
        for (int dd = 0; dd < a.ndims; ++dd) {  // odometer, first dim fastest
            if (++Jb[dd] < nc[dd]) break;
            Jb[dd] = 0;
        }
    }
    return out;
}

// The same as a call: what a kernel falls back on costs it no registers.
template <typename T>
__device__ __noinline__ T mult_entry_call(const MultArgs &a, const T *__restrict__ B, int64_t lin) {
    return mult_entry(a, B, lin);
}

// refinement_matrix_array_mul_kernel (src/refinement_matrix.jl:365-403): one thread per
// entry of Y.
template <typename T>
__global__ void k_mult(MultArgs a, const T *__restrict__ B, T *__restrict__ Y, int64_t NY) {
    grid_start(B);
    for (int64_t lin = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; lin < NY;
         lin += (int64_t)gridDim.x * blockDim.x)
        Y[lin] = mult_entry(a, B, lin);
}

// Rows [lo, hi) of a banded matrix whose band covers column j.  column_start and the
// row ends are non-decreasing in a valid RefinementMatrix (the row checks of
// src/refinement_matrix.jl:163-178), so both bounds are binary searches.
__device__ __forceinline__ void rows_covering(const MultArgs &a, int r, int64_t j, int64_t &lo,
                                              int64_t &hi) {
    int64_t l = 0, h = a.m[r];
    while (l < h) {  // first row with column_start > j
        const int64_t mid = (l + h) >> 1;
        if ((int64_t)a.cs[r][mid] - 1 > j) h = mid; else l = mid + 1;
    }
    hi = l;
    l = 0;
    h = a.m[r];
    while (l < h) {  // first row whose last column >= j
        const int64_t mid = (l + h) >> 1;
        int64_t c0, nc, z0;
        row_extent(a, r, mid, c0, nc, z0);
        if (c0 + nc - 1 < j) l = mid + 1; else h = mid;
    }
    lo = l;
}

// Entry `lin` of B = mult_adjoint!(Y), any dimension count and band width: the sum of
// Y[I] prod A[I_d, J_d] over the rows I whose bands cover J, in a fixed order (first dim
// fastest).
template <typename T>
__device__ __forceinline__ T mult_adjoint_entry(const MultArgs &a, const T *__restrict__ Y, int64_t lin) {
    int64_t J[kMaxDims], lo[kMaxDims], cnt[kMaxDims], Ib[kMaxDims];
    int64_t rem = lin, tot = 1;
    for (int dd = 0; dd < a.ndims; ++dd) {
        J[dd] = rem % a.size_B[dd];
        rem /= a.size_B[dd];
        const int r = a.rm_of_dim[dd];
        if (r < 0) { lo[dd] = J[dd]; cnt[dd] = 1; }
        else {
            int64_t l, h;
            rows_covering(a, r, J[dd], l, h);
            lo[dd] = l;
            cnt[dd] = h > l ? h - l : 0;
        }
        tot *= cnt[dd];
        Ib[dd] = 0;
    }
    T acc = T(0);
    for (int64_t t = 0; t < tot; ++t) {
        int64_t off = 0, stride = 1;
        for (int dd = 0; dd < a.ndims; ++dd) {
            off += (lo[dd] + Ib[dd]) * stride;
            stride *= a.size_Y[dd];
        }
        T contrib = Y[off];
        for (int dd = 0; dd < a.ndims; ++dd) {
            const int r = a.rm_of_dim[dd];
            if (r >= 0) {
                int64_t c0, nc, z0;
                row_extent(a, r, lo[dd] + Ib[dd], c0, nc, z0);
                contrib *= ((const T *)a.nz[r])[z0 + (J[dd] - c0)];
            }
        }
        acc += contrib;
        for (int dd = 0; dd < a.ndims; ++dd) {
            if (++Ib[dd] < cnt[dd]) break;
            Ib[dd] = 0;
        }
    }
    return acc;
}

// mult_adjoint! (src/adjoint.jl:85-152) in gather form: one thread per entry of B.
// Deterministic and without atomics.
template <typename T>
__global__ void k_mult_adjoint(MultArgs a, const T *__restrict__ Y, T *__restrict__ B,
                               int64_t NB) {
    grid_start(Y);
    for (int64_t lin = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; lin < NB;
         lin += (int64_t)gridDim.x * blockDim.x)
        B[lin] = mult_adjoint_entry(a, Y, lin);
}

// ---------------------------------------------------------------------------------
// mult! and mult_adjoint! of arrays with ND = 2..4 dimensions (curves, surfaces and
// volumes with their Nout dimension), every index array unrolled.  The kernels above are
// bound by latency: their nine-entry index arrays live in local memory, and an odometer
// re-reads row pointers, column starts and band values for every term, so a thread is one
// chain of dependent loads.  Here a thread finds each dimension's band once, and the sum is
// the unrolled one for the widest band of its warp (2 to 5 terms a dimension, factors in
// registers, independent loads) or plain loops for wider ones: bound by the terms'
// instructions, so one sum for all widths up to 5, 25 predicated terms a plane, took 2 to 4
// times as long.  Terms, factors and roundings are those of the general kernels.  Measured, us,
// general kernels / one sum for all / now: (58, 58, 26) -> (114, 114, 50), bands of 2, Float32:
// mult! 46 / 22 / 11.8, mult_adjoint! 79 / 17 / 12.6; bands of 3: 122 / - / 15, 231 / 286 / 39;
// (257, 257) x 3 -> (511, 511) x 3, bands of 3, Float64, general / now: 51 / 39, 56 / 41.
// ---------------------------------------------------------------------------------
constexpr int kMultThreads = 128;

template <int ND>
struct MultNd {
    int64_t sY[ND], sB[ND];
    const int32_t *rp[ND], *cs[ND];  // NULL: dimension not refined
    const void *nz[ND];
    int64_t m[ND], nnz[ND];
};

template <int ND>
__device__ __forceinline__ void nd_row(const MultNd<ND> &p, int d, int64_t i, int64_t &c0, int64_t &nc, int64_t &z0) {
    const int64_t r0 = p.rp[d][i];
    const int64_t next = (i == p.m[d] - 1) ? p.nnz[d] + 1 : (int64_t)p.rp[d][i + 1];
    nc = next - r0;
    c0 = (int64_t)p.cs[d][i] - 1;
    z0 = r0 - 1;
}

template <int ND>
__device__ __forceinline__ void nd_decode(const int64_t (&size)[ND], int64_t lin, bool small, int64_t (&I)[ND]) {
    if (small) {  // 32-bit division
        uint32_t rem = (uint32_t)lin;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const uint32_t q = d + 1 < ND ? rem / (uint32_t)size[d] : 0u;
            I[d] = d + 1 < ND ? rem - q * (uint32_t)size[d] : rem;
            rem = q;
        }
    } else {
        int64_t rem = lin;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const int64_t q = d + 1 < ND ? rem / size[d] : 0;
            I[d] = d + 1 < ND ? rem - q * size[d] : rem;
            rem = q;
        }
    }
}

// a + b, not contracted with the product b may be: the bits of the general function.
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }

// The sum of x at k_d < n[d], stride st[d] (0 fastest), times the factors f(d, k) of dimension d at
// term k, over the first NR dimensions.  n[d] <= C: the factors sit in registers, the loads of a
// k2 are independent.
template <int C, int NR, typename T, int ND, typename F>
__device__ __forceinline__ T nd_sum_c(const T *__restrict__ x, const int (&n)[ND], const int64_t (&st)[ND], F f) {
    constexpr int C1 = NR > 1 ? C : 1;
    T w[NR][C];
#pragma unroll
    for (int d = 0; d < NR; ++d)
#pragma unroll
        for (int k = 0; k < C; ++k) w[d][k] = k < n[d] ? f(d, k) : T(1);
    T acc = T(0);
#pragma unroll(C == 2 ? 2 : 1)
    for (int k2 = 0; k2 < (NR > 2 ? C : 1); ++k2) {
        T w2 = T(1);
        if constexpr (NR > 2) {
            if (k2 >= n[2]) break;
#pragma unroll
            for (int k = 0; k < C; ++k) w2 = k == k2 ? w[2][k] : w2;
        }
        T v[C1][C];
#pragma unroll
        for (int k1 = 0; k1 < C1; ++k1)
#pragma unroll
            for (int k0 = 0; k0 < C; ++k0)
                if ((NR < 2 || k1 < n[1]) && k0 < n[0]) v[k1][k0] = x[k0 + (NR > 1 ? k1 * st[1] : 0)];
#pragma unroll
        for (int k1 = 0; k1 < C1; ++k1)
#pragma unroll
            for (int k0 = 0; k0 < C; ++k0)
                if ((NR < 2 || k1 < n[1]) && k0 < n[0]) {
                    T t = v[k1][k0] * w[0][k0];
                    if constexpr (NR > 1) t = t * w[1][k1];
                    if constexpr (NR > 2) t = t * w2;
                    acc = add_rn(acc, t);
                }
        if constexpr (NR > 2) x += st[2];
    }
    return acc;
}

// Bands of any width, the first NR dimensions.
template <int NR, typename T, int ND, typename F>
__device__ __forceinline__ T nd_sum_any(const T *__restrict__ X, const int (&n)[ND], const int64_t (&st)[ND], F f) {
    T acc = T(0);
    const int n1 = NR > 1 ? n[1] : 1, n2 = NR > 2 ? n[NR > 2 ? 2 : 0] : 1, n3 = NR > 3 ? n[NR > 3 ? 3 : 0] : 1;
    for (int k3 = 0; k3 < n3; ++k3) {
        const T w3 = NR > 3 ? f(3, k3) : T(1);
        for (int k2 = 0; k2 < n2; ++k2) {
            const T w2 = NR > 2 ? f(2, k2) : T(1);
            for (int k1 = 0; k1 < n1; ++k1) {
                const T w1 = NR > 1 ? f(1, k1) : T(1);
                const T *x = X + k1 * st[1] + (NR > 2 ? k2 * st[NR > 2 ? 2 : 0] : 0) + (NR > 3 ? k3 * st[NR > 3 ? 3 : 0] : 0);
#pragma unroll 4
                for (int k0 = 0; k0 < n[0]; ++k0) {
                    T t = x[k0] * f(0, k0);
                    if constexpr (NR > 1) t = t * w1;
                    if constexpr (NR > 2) t = t * w2;
                    if constexpr (NR > 3) t = t * w3;
                    acc = add_rn(acc, t);
                }
            }
        }
    }
    return acc;
}

// The narrowest of the unrolled sums that holds every band of the warp's threads, or the loops (the
// vote keeps the warp in one of them).  A row of a bisected dimension has degree / 2 + 1 columns at
// most, a column degree + 2 rows.
//  * Float32: unrolled, also where bands of other widths leave terms out ((50, 40, 54) x 2, degrees 2, 3,
//    2: 30 us, loops 45).
//  * Float64: a term that a thread does not have costs it as much as one it has, on a pipe that is the
//    bound.  mult! (ROWS) takes the loops ((33, 55, 50) x 3, degrees 1, 0, 4: 114 us, unrolled 407;
//    equal bands of 2 and 3: 8 and 8); mult_adjoint!, whose factors' look-ups are longer, the unrolled
//    sums while at most half of their terms are missing ((32, 59, 65) x 2, degrees 0, 1, 3: loops 74,
//    unrolled 240; (12, 12, 12) x 2, degrees 2, 3, 3: 44 and 27).
// last: the last dimension is refined (Nout is not: no factors of one are multiplied); that takes
// the loops, for the unrolled sums of ND dimensions as well would cost the kernel registers.
template <int NR, bool ROWS, typename T, int ND, typename F>
__device__ __forceinline__ T nd_sum_n(const T *__restrict__ x, const int (&n)[ND], const int64_t (&st)[ND], F f) {
    if constexpr (sizeof(T) == 8 && ROWS) {
        return nd_sum_any<NR>(x, n, st, f);
    } else {
        unsigned widest = n[0], terms = n[0];
#pragma unroll
        for (int d = 1; d < NR; ++d) {
            widest = (unsigned)n[d] > widest ? n[d] : widest;
            terms *= n[d];
        }
        const unsigned cap = __reduce_max_sync(__activemask(), widest);
        if constexpr (sizeof(T) == 8) {
            unsigned all = cap;
#pragma unroll
            for (int d = 1; d < NR; ++d) all *= cap;
            if (cap > 5 || all > 2 * __reduce_max_sync(__activemask(), terms)) return nd_sum_any<NR>(x, n, st, f);
        }
        if (cap <= 2) return nd_sum_c<2, NR>(x, n, st, f);
        if (cap <= 3) return nd_sum_c<3, NR>(x, n, st, f);
        if (cap <= 4) return nd_sum_c<4, NR>(x, n, st, f);
        if (cap <= 5) return nd_sum_c<5, NR>(x, n, st, f);
        return nd_sum_any<NR>(x, n, st, f);
    }
}
template <bool ROWS, typename T, int ND, typename F>
__device__ __forceinline__ T nd_sum(const T *__restrict__ X, const int64_t (&lo)[ND], const int (&n)[ND],
                                    const int64_t (&st)[ND], bool last, F f) {
    const T *x = X;
#pragma unroll
    for (int d = 0; d < ND; ++d) x += lo[d] * st[d];
    if (!last) return nd_sum_n<ND - 1, ROWS>(x, n, st, f);
    return nd_sum_any<ND>(x, n, st, f);
}

template <typename T, int ND>
__global__ void __launch_bounds__(kMultThreads, 6)
k_mult_nd(MultNd<ND> p, MultArgs a, const T *__restrict__ B, T *__restrict__ Y, int64_t NY, bool small) {
    const int64_t lin = blockIdx.x * (int64_t)kMultThreads + threadIdx.x + grid_start();
    if (lin >= NY) return;
    int64_t I[ND], c0[ND], st[ND], z0[ND];
    int n[ND];
    nd_decode<ND>(p.sY, lin, small, I);
    bool fits = true;
    int64_t acc = 1;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        st[d] = acc;
        acc *= p.sB[d];
        c0[d] = I[d];
        z0[d] = 0;
        n[d] = 1;
        if (p.rp[d]) {
            int64_t nc;
            nd_row(p, d, I[d], c0[d], nc, z0[d]);
            fits = fits && (nc <= 0 || (c0[d] >= 0 && c0[d] + nc <= p.sB[d]));
            n[d] = nc < 0 ? 0 : (int)nc;
        }
    }
    if (!fits) {
        Y[lin] = mult_entry_call(a, B, lin);
        return;
    }
    auto f = [&](int d, int k) {
        T r = T(1);
#pragma unroll
        for (int e = 0; e < ND; ++e)
            if (e == d && p.rp[e]) r = ((const T *)p.nz[e])[z0[e] + k];
        return r;
    };
    Y[lin] = nd_sum<true>(B, c0, n, st, p.rp[ND - 1] != nullptr, f);
}

template <typename T, int ND>
__global__ void __launch_bounds__(kMultThreads, 6)
k_mult_adjoint_nd(MultNd<ND> p, const T *__restrict__ Y, T *__restrict__ B, int64_t NB, bool small) {
    const int64_t lin = blockIdx.x * (int64_t)kMultThreads + threadIdx.x + grid_start();
    if (lin >= NB) return;
    int64_t J[ND], lo[ND], hi[ND], st[ND];
    int n[ND];
    nd_decode<ND>(p.sB, lin, small, J);
    int64_t acc = 1;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        st[d] = acc;
        acc *= p.sY[d];
        lo[d] = J[d];
        n[d] = 1;
    }
    // rows covering column J[d] (the binary searches of rows_covering, all dimensions
    // side by side so that their loads overlap)
    int64_t l0[ND], h0[ND], l1[ND], h1[ND];
    bool more = false;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        l0[d] = l1[d] = 0;
        h0[d] = h1[d] = p.rp[d] ? p.m[d] : 0;
        more = more || h0[d] > 0;
    }
    while (more) {
        more = false;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            if (l0[d] < h0[d]) {  // first row with column_start > J
                const int64_t mid = (l0[d] + h0[d]) >> 1;
                if ((int64_t)p.cs[d][mid] - 1 > J[d]) h0[d] = mid; else l0[d] = mid + 1;
                more = more || l0[d] < h0[d];
            }
            if (l1[d] < h1[d]) {  // first row whose last column >= J
                const int64_t mid = (l1[d] + h1[d]) >> 1;
                int64_t c0, nc, z0;
                nd_row(p, d, mid, c0, nc, z0);
                if (c0 + nc - 1 < J[d]) l1[d] = mid + 1; else h1[d] = mid;
                more = more || l1[d] < h1[d];
            }
        }
    }
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        if (p.rp[d]) {
            lo[d] = l1[d];
            hi[d] = l0[d];
            const int64_t c = hi[d] > lo[d] ? hi[d] - lo[d] : 0;
            n[d] = (int)c;
        }
    }
    auto f = [&](int d, int k) {  // A_d[lo + k, J]
        T r = T(1);
#pragma unroll
        for (int e = 0; e < ND; ++e)
            if (e == d && p.rp[e]) {
                int64_t c0, nc, z0;
                nd_row(p, e, lo[e] + k, c0, nc, z0);
                r = ((const T *)p.nz[e])[z0 + (J[e] - c0)];
            }
        return r;
    };
    B[lin] = nd_sum<false>(Y, lo, n, st, p.rp[ND - 1] != nullptr, f);
}

struct RefIdx {
    int nin;
    int64_t cp_size[SG_MAX_NIN];
};

// Set by the overwrite kernels when a refinement index lies outside the control-point
// grid (that entry is skipped, so no access leaves the array).  The Python and Julia
// wrappers validate indices at set-up; this flag is a last line of defence.
__device__ int g_bad_refinement_index = 0;

__device__ __forceinline__ bool ref_linear(const RefIdx &r, const int32_t *ridx, int64_t n_ref,
                                           int64_t i, int64_t &lin) {
    lin = 0;
    int64_t stride = 1;
    for (int dd = 0; dd < r.nin; ++dd) {
        const int64_t c = (int64_t)ridx[i + n_ref * dd] - 1;
        if (c < 0 || c >= r.cp_size[dd]) return false;
        lin += c * stride;
        stride *= r.cp_size[dd];
    }
    return true;
}

// local_refinement_kernel (src/control_points.jl:296-311)
template <typename T>
__global__ void k_local_refinement(RefIdx r, int nout, int64_t n_ref, const int32_t *ridx,
                                   const T *vals, T *cp, int64_t ncp) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x + grid_start();
    if (i >= n_ref) return;
    int64_t lin;
    if (!ref_linear(r, ridx, n_ref, i, lin)) { g_bad_refinement_index = 1; return; }
    for (int o = 0; o < nout; ++o) cp[lin + ncp * o] = vals[i + n_ref * o];
}

// local_refinement_adjoint_kernel (src/adjoint.jl:154-170)
template <typename T>
__global__ void k_local_refinement_adjoint(RefIdx r, int nout, int64_t n_ref,
                                           const int32_t *ridx, T *vals, T *cp, int64_t ncp) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x + grid_start();
    if (i >= n_ref) return;
    int64_t lin;
    if (!ref_linear(r, ridx, n_ref, i, lin)) { g_bad_refinement_index = 1; return; }
    for (int o = 0; o < nout; ++o) {
        vals[i + n_ref * o] = cp[lin + ncp * o];
        cp[lin + ncp * o] = T(0);
    }
}

}  // namespace sg

using namespace sg;

static int build_mult_args(int32_t dtype, int32_t ndims, const int64_t *size_Y,
                           const int64_t *size_B, int32_t n_refmat, const sg_refmat *As,
                           const int32_t *dims_refinement, MultArgs &a, const char *who) {
    if (dtype != SG_F32 && dtype != SG_F64)
        return set_error(SG_ERR_INVALID_ARGUMENT, "%s: dtype must be F32 or F64", who);
    if (ndims < 1 || ndims > kMaxDims || !size_Y || !size_B)
        return set_error(SG_ERR_INVALID_ARGUMENT, "%s: ndims %d outside 1..%d", who, ndims, kMaxDims);
    if (n_refmat < 0 || n_refmat > ndims || (n_refmat > 0 && (!As || !dims_refinement)))
        return set_error(SG_ERR_INVALID_ARGUMENT, "%s: bad refinement matrix list", who);
    memset(&a, 0, sizeof(a));
    a.ndims = ndims;
    for (int d = 0; d < ndims; ++d) {
        a.size_Y[d] = size_Y[d];
        a.size_B[d] = size_B[d];
        a.rm_of_dim[d] = -1;
        if (size_Y[d] < 0 || size_B[d] < 0)
            return set_error(SG_ERR_INVALID_ARGUMENT, "%s: negative size", who);
    }
    // validate_mult_input, src/validation.jl:90-107
    for (int r = 0; r < n_refmat; ++r) {
        const int d = dims_refinement[r];
        if (d < 0 || d >= ndims)
            return set_error(SG_ERR_INVALID_ARGUMENT, "%s: refinement dimension %d out of range", who, d);
        if (a.rm_of_dim[d] >= 0)
            return set_error(SG_ERR_INVALID_ARGUMENT, "Refinement dimensions must be unique.");
        if (As[r].m != size_Y[d] || As[r].n != size_B[d])
            return set_error(SG_ERR_INVALID_ARGUMENT,
                             "Size of refinement matrix does not match `B` and `Y` along "
                             "refinement dimension %d.", d + 1);
        if (As[r].m > 0 && (!As[r].row_pointer || !As[r].column_start || !As[r].nzval))
            return set_error(SG_ERR_INVALID_ARGUMENT, "%s: NULL refinement matrix array", who);
        a.rm_of_dim[d] = r;
        a.rp[r] = As[r].row_pointer;
        a.cs[r] = As[r].column_start;
        a.nz[r] = As[r].nzval;
        a.m[r] = As[r].m;
        a.n[r] = As[r].n;
        a.nnz[r] = As[r].nnz;
    }
    for (int d = 0; d < ndims; ++d)
        if (a.rm_of_dim[d] < 0 && size_Y[d] != size_B[d])
            return set_error(SG_ERR_INVALID_ARGUMENT,
                             "`B` and `Y` don't have the same size along dimension %d.", d + 1);
    return SG_OK;
}

static unsigned grid_for(int64_t n, int bs) {
    int64_t g = (n + bs - 1) / bs;
    if (g > 152 * 64) g = 152 * 64;  // grid-stride beyond this
    return (unsigned)(g < 1 ? 1 : g);
}

// Launches the unrolled kernels (ND = 2..4) or the general ones.
template <typename T, int ND, bool ADJ>
static void launch_mult_nd(const MultArgs &a, const void *X, void *Y, int64_t N, cudaStream_t s) {
    MultNd<ND> p;
    for (int d = 0; d < ND; ++d) {
        const int r = a.rm_of_dim[d];
        p.sY[d] = a.size_Y[d];
        p.sB[d] = a.size_B[d];
        p.rp[d] = r >= 0 ? a.rp[r] : nullptr;
        p.cs[d] = r >= 0 ? a.cs[r] : nullptr;
        p.nz[d] = r >= 0 ? a.nz[r] : nullptr;
        p.m[d] = r >= 0 ? a.m[r] : 0;
        p.nnz[d] = r >= 0 ? a.nnz[r] : 0;
    }
    const unsigned blocks = (unsigned)((N + kMultThreads - 1) / kMultThreads);
    const bool small = N <= 0xffffffffLL;
    if (ADJ) launch(k_mult_adjoint_nd<T, ND>, blocks, kMultThreads, 0, s, p, (const T *)X, (T *)Y, N, small);
    else launch(k_mult_nd<T, ND>, blocks, kMultThreads, 0, s, p, a, (const T *)X, (T *)Y, N, small);
}

template <typename T, bool ADJ>
static void launch_mult(const MultArgs &a, const void *X, void *Y, int64_t N, cudaStream_t s) {
    const bool one_launch = (N + kMultThreads - 1) / kMultThreads <= 0x7fffffffLL;
    if (a.ndims == 2 && one_launch) launch_mult_nd<T, 2, ADJ>(a, X, Y, N, s);
    else if (a.ndims == 3 && one_launch) launch_mult_nd<T, 3, ADJ>(a, X, Y, N, s);
    else if (a.ndims == 4 && one_launch) launch_mult_nd<T, 4, ADJ>(a, X, Y, N, s);
    else if (ADJ) launch(k_mult_adjoint<T>, grid_for(N, 256), 256, 0, s, a, (const T *)X, (T *)Y, N);
    else launch(k_mult<T>, grid_for(N, 256), 256, 0, s, a, (const T *)X, (T *)Y, N);
}

extern "C" int sg_mult(int32_t dtype, int32_t ndims, const int64_t *size_Y,
                       const int64_t *size_B, int32_t n_refmat, const sg_refmat *As,
                       const int32_t *dims_refinement, const void *B, void *Y,
                       sg_stream_t stream) {
    MultArgs a;
    int rc = build_mult_args(dtype, ndims, size_Y, size_B, n_refmat, As, dims_refinement, a,
                             "sg_mult");
    if (rc) return rc;
    int64_t NY = 1;
    for (int d = 0; d < ndims; ++d) NY *= size_Y[d];
    if (NY == 0) return SG_OK;
    if (!B || !Y) return set_error(SG_ERR_INVALID_ARGUMENT, "sg_mult: NULL array");
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == SG_F32) launch_mult<float, false>(a, B, Y, NY, s);
    else launch_mult<double, false>(a, B, Y, NY, s);
    return cuda_check(cudaGetLastError(), "k_mult launch");
}

extern "C" int sg_mult_adjoint(int32_t dtype, int32_t ndims, const int64_t *size_Y,
                               const int64_t *size_B, int32_t n_refmat, const sg_refmat *As,
                               const int32_t *dims_refinement, const void *Y, void *B,
                               sg_stream_t stream) {
    MultArgs a;
    int rc = build_mult_args(dtype, ndims, size_Y, size_B, n_refmat, As, dims_refinement, a,
                             "sg_mult_adjoint");
    if (rc) return rc;
    int64_t NB = 1;
    for (int d = 0; d < ndims; ++d) NB *= size_B[d];
    if (NB == 0) return SG_OK;
    if (!B || !Y) return set_error(SG_ERR_INVALID_ARGUMENT, "sg_mult_adjoint: NULL array");
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == SG_F32) launch_mult<float, true>(a, Y, B, NB, s);
    else launch_mult<double, true>(a, Y, B, NB, s);
    return cuda_check(cudaGetLastError(), "k_mult_adjoint launch");
}

static int overwrite_common(int32_t dtype, int32_t nin, int32_t nout, const int64_t *cp_size,
                            int64_t n_refined, const int32_t *ridx, const void *vals, void *cp,
                            RefIdx &r, int64_t &ncp, const char *who) {
    if (dtype != SG_F32 && dtype != SG_F64)
        return set_error(SG_ERR_INVALID_ARGUMENT, "%s: dtype must be F32 or F64", who);
    if (nin < 1 || nin > SG_MAX_NIN || nout < 1 || !cp_size || n_refined < 0)
        return set_error(SG_ERR_INVALID_ARGUMENT, "%s: bad dimensions", who);
    r.nin = nin;
    ncp = 1;
    for (int d = 0; d < nin; ++d) {
        r.cp_size[d] = cp_size[d];
        ncp *= cp_size[d];
    }
    if (n_refined > 0 && (!ridx || !vals || !cp))
        return set_error(SG_ERR_INVALID_ARGUMENT, "%s: NULL array", who);
    return SG_OK;
}

extern "C" int sg_local_refinement(int32_t dtype, int32_t nin, int32_t nout,
                                   const int64_t *cp_size, int64_t n_refined,
                                   const int32_t *refinement_indices,
                                   const void *refinement_values, void *control_points,
                                   sg_stream_t stream) {
    RefIdx r;
    int64_t ncp;
    int rc = overwrite_common(dtype, nin, nout, cp_size, n_refined, refinement_indices,
                              refinement_values, control_points, r, ncp, "sg_local_refinement");
    if (rc || n_refined == 0) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned g = (unsigned)((n_refined + 255) / 256);
    if (dtype == SG_F32)
        launch(k_local_refinement<float>, g, 256, 0, s, r, nout, n_refined, refinement_indices,
               (const float *)refinement_values, (float *)control_points, ncp);
    else
        launch(k_local_refinement<double>, g, 256, 0, s, r, nout, n_refined, refinement_indices,
               (const double *)refinement_values, (double *)control_points, ncp);
    return cuda_check(cudaGetLastError(), "k_local_refinement launch");
}

extern "C" int sg_local_refinement_adjoint(int32_t dtype, int32_t nin, int32_t nout,
                                           const int64_t *cp_size, int64_t n_refined,
                                           const int32_t *refinement_indices,
                                           void *refinement_values, void *control_points,
                                           sg_stream_t stream) {
    RefIdx r;
    int64_t ncp;
    int rc = overwrite_common(dtype, nin, nout, cp_size, n_refined, refinement_indices,
                              refinement_values, control_points, r, ncp,
                              "sg_local_refinement_adjoint");
    if (rc || n_refined == 0) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned g = (unsigned)((n_refined + 255) / 256);
    if (dtype == SG_F32)
        launch(k_local_refinement_adjoint<float>, g, 256, 0, s, r, nout, n_refined, refinement_indices,
               (float *)refinement_values, (float *)control_points, ncp);
    else
        launch(k_local_refinement_adjoint<double>, g, 256, 0, s, r, nout, n_refined, refinement_indices,
               (double *)refinement_values, (double *)control_points, ncp);
    return cuda_check(cudaGetLastError(), "k_local_refinement_adjoint launch");
}
