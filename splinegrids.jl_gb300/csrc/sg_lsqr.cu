// sg_lsqr.cu -- matrix-free LSQR on the device, for least-squares fits of spline grids.
//
// The reference fits control points by handing `LinearMap(spline_grid)`
// (ext/SplineGridsLinearMapsExt.jl:5-52: forward = evaluate!(control_points) then
// evaluate!(grid), adjoint = evaluate_adjoint!(grid) then evaluate_adjoint!(control_points))
// to IterativeSolvers.jl's `lsqr` (Project.toml compat 0.9; test/test_LinearMapsExt.jl).
// IterativeSolvers is not part of the reference tree; its `lsqr` is the published LSQR
// of Paige & Saunders (ACM TOMS 8(1):43-71, 1982, "LSQR: An algorithm for sparse linear
// equations and sparse least squares"), restated here from that paper: Golub-Kahan
// bidiagonalisation, a Givens QR update of the bidiagonal system, and the paper's stopping
// rules 1-3 with the estimates of ||A||, cond(A), ||r||, ||A'r|| and ||x||.
//
// Layout of one iteration on the device (vectors stay in HBM, scalars in a device struct):
//   F = A V                      (caller: the grid's forward evaluation)
//   U = F/alpha - (alpha/beta) U ; partial sums of U^2;
//   beta = ||U||, ||A|| estimate                              k_lsqr_axpby (phase U)
//   G = A' U                     (caller: the grid's adjoint)
//   V = G/beta - (beta/alpha) V ; partial sums of V^2, W^2;
//   alpha = ||V||, Givens rotation                            k_lsqr_axpby (phase V)
//   X += t1 W ; W = V/alpha + t2 W ; beside it (block 0) the
//   estimates and stopping rules                              k_lsqr_xw
// The last block of a vector pass to finish sums the partials and does the scalar step.
// U and V are kept unnormalised (u = U/beta, v = V/alpha), so no pass over a vector only
// rescales it: the scale is folded into the next pass that reads it.  Every reduction is a
// fixed-order two-level sum (per-block partials, then one block), so a solve is bitwise
// reproducible.  The iteration can be captured once into a CUDA graph whose body runs in a
// device-side `while` conditional node: the x/w pass sets the loop condition after
// every step (open while no stopping rule holds, closed when one does, and maxiter is one
// of the rules), so a whole solve is one graph launch with no host round trip.
#include <math.h>

#include <type_traits>

#include "sg_common.cuh"

namespace sg {
namespace {

constexpr int kLsqrThreads = 256;
// Grid of the vector passes: two blocks per SM at most.  (Every block ends with a Float64
// reduction: 12 iterations of a (2048, 2048) Float32 fit take 653 us with 304 blocks, 712 with
// 608, 774 with 912.)
constexpr int kLsqrMaxBlocks = 2 * 152;

struct LsqrState {
    // Golub-Kahan scalars of the current iteration
    double alpha, beta;
    // QR recurrence (paper section 4.1) and the norm / condition estimates (section 5)
    double rhobar, phibar, anorm, acond, ddnorm, res2, xnorm, xxnorm, z, cs2, sn2;
    double bnorm, rnorm, arnorm;
    // coefficients of the vector passes, written by the scalar step
    double cu_a, cu_b, cv_a, cv_b, t1, t2, inv_alpha;
    // parameters
    double damp, atol, btol, ctol, eps;
    // between the two parts of a step (the scalar step and its estimates)
    double theta, tau, gambar, rhs, zbar;
    long long itn, maxiter;
    int istop, done, estimate;
};

int n_blocks(int64_t n) {
    int64_t b = (n + (int64_t)kLsqrThreads * 4 - 1) / ((int64_t)kLsqrThreads * 4);
    return (int)(b < 1 ? 1 : (b > kLsqrMaxBlocks ? kLsqrMaxBlocks : b));
}

// Block-wide sum of one double, fixed order (warp shuffles, then warp 0 over the warps).
__device__ __forceinline__ double block_sum(double v, double *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (w == 0) {
        r = l < (int)(blockDim.x >> 5) ? sh[l] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    }
    return r;  // valid in thread 0
}

// Sum of squares.  Float64 values: Float64 FMAs.  Float32 values: the Float64 pipe (two
// lanes per SM and clock, conversions included) would be the bound of the whole pass, so the
// squares are summed without error in three Float32 words: r^2 = p + e exactly (FMA), and
// each addition keeps its rounding error in the next word (TwoSum, Knuth, TAOCP 4.2.2).  The
// three words carry about 70 bits, more than the Float64 sum they replace (53).  Groups of
// values whose squares or errors could leave Float32's range go the Float64 way.
// Measured on 4.2 M Float32 values (the pass U = a F + b U with its sum): 24.6 -> 10.3 us.
template <typename T>
struct SumSq {
    double s = 0.0;
    template <int N>
    __device__ __forceinline__ void add(const T (&v)[N]) {
#pragma unroll
        for (int k = 0; k < N; ++k) s += (double)v[k] * (double)v[k];
    }
    __device__ __forceinline__ double get() const { return s; }
};
template <>
struct SumSq<float> {
    double s = 0.0;
    float w0 = 0.f, w1 = 0.f, w2 = 0.f;
    static __device__ __forceinline__ float two_sum(float a, float b, float &err) {
        const float r = __fadd_rn(a, b), bb = __fsub_rn(r, a);
        err = __fadd_rn(__fsub_rn(a, __fsub_rn(r, bb)), __fsub_rn(b, bb));
        return r;
    }
    template <int N>
    __device__ __forceinline__ void add(const float (&v)[N]) {
        // the errors of squares far below the group's largest may be lost: they are below
        // 2^-65 of the sum
        float m = 0.f;
#pragma unroll
        for (int k = 0; k < N; ++k) m = fmaxf(m, fabsf(v[k]));
        if ((m >= 0x1p-40f && m <= 0x1p50f) || m == 0.f) {  // (a NaN stays one in p)
#pragma unroll
            for (int k = 0; k < N; ++k) {
                const float p = __fmul_rn(v[k], v[k]), e = __fmaf_rn(v[k], v[k], -p);
                float t, u, x;
                w0 = two_sum(w0, p, t);
                t = two_sum(t, e, u);
                w1 = two_sum(w1, t, x);
                w2 = __fadd_rn(w2, __fadd_rn(u, x));
            }
        } else {
#pragma unroll
            for (int k = 0; k < N; ++k) s += (double)v[k] * (double)v[k];
        }
    }
    __device__ __forceinline__ double get() const { return ((double)w2 + (double)w1) + (double)w0 + s; }
};

enum { kPhaseStart = 0, kPhaseU = 1, kPhaseV = 2 };

// What the vector passes share: the state, the blocks' partial sums and the counter of
// blocks that have finished.
struct LsqrShared {
    LsqrState *st;
    double *part, *part2;  // [kLsqrMaxBlocks] each
    unsigned *count;       // zero between passes
    int *skip_xw;
    cudaGraphConditionalHandle cond;
    int has_cond;
};

template <typename T>
__device__ void lsqr_scalar(const LsqrShared &sh, double s, double s2, int phase);

// End of a vector pass: the block's sums go to part / part2; the last block to finish adds
// all of them in a fixed order and does the pass' scalar step.
template <typename T>
__device__ __forceinline__ void lsqr_finish(const LsqrShared &L, double s, double s2, bool two, int phase) {
    __shared__ double sh[kLsqrThreads / 32];
    __shared__ int last;
    s = block_sum(s, sh);
    if (two) s2 = block_sum(s2, sh);
    if (threadIdx.x == 0) {
        L.part[blockIdx.x] = s;
        if (two) L.part2[blockIdx.x] = s2;
        __threadfence();
        last = atomicAdd(L.count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) {
        a += __ldcg(L.part + i);
        if (two) b += __ldcg(L.part2 + i);
    }
    a = block_sum(a, sh);
    if (two) b = block_sum(b, sh);
    if (threadIdx.x == 0) *L.count = 0;
    if (threadIdx.x < 32) {  // block_sum's result is thread 0's
        a = __shfl_sync(0xffffffffu, a, 0);
        b = __shfl_sync(0xffffffffu, b, 0);
        lsqr_scalar<T>(L, a, b, phase);
    }
}

// Calls step(V, G, i, gap) for the thread's share of n values: G groups of V consecutive ones at
// i, i + gap, ...  16-byte groups where every pointer allows it (two in flight for each
// operand), else four single values: the passes wait for memory, so bytes in flight count
// (12 iterations of a (2048, 2048) Float32 fit: 687 us with single values, 649 with groups).
template <int V> using Count = std::integral_constant<int, V>;
template <typename T, typename F>
__device__ __forceinline__ void lsqr_each(int64_t n, bool packed, int64_t i0, int64_t stride, F step) {
    constexpr int V = 16 / (int)sizeof(T);
    int64_t i = i0;
    if (packed) {
        const int64_t np = n / V;
        for (; i + stride < np; i += 2 * stride) step(Count<V>{}, Count<2>{}, i * V, stride * V);
        if (i < np) step(Count<V>{}, Count<1>{}, i * V, (int64_t)0);
        if (np * V + i0 < n) step(Count<1>{}, Count<1>{}, np * V + i0, (int64_t)0);
    } else {
        for (; i + 3 * stride < n; i += 4 * stride) step(Count<1>{}, Count<4>{}, i, stride);
        for (; i < n; i += stride) step(Count<1>{}, Count<1>{}, i, (int64_t)0);
    }
}
template <typename... P>
__device__ __forceinline__ bool aligned16(const P *...p) {
    return (((uintptr_t)p | ...) & 15) == 0;
}

// U = b, and (n-space) X = 0, W = 0; the sum of b^2 and the start of the recurrence.
template <typename T>
__global__ void __launch_bounds__(kLsqrThreads) k_lsqr_start(const T *__restrict__ b, T *__restrict__ U, int64_t m,
                                                T *__restrict__ X, T *__restrict__ W, int64_t n,
                                                LsqrShared L) {
    grid_start(b);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    SumSq<T> s;
    lsqr_each<T>(m, aligned16(b, U), (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride,
                 [&](auto vc, auto gc, int64_t i, int64_t gap) {
        constexpr int V = decltype(vc)::value, G = decltype(gc)::value;
        Pack<T, V> v[G];
#pragma unroll
        for (int g = 0; g < G; ++g) v[g] = ldp<T, V>(b + i + g * gap);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            stp<T, V>(U + i + g * gap, v[g]);
            s.add(v[g].v);
        }
    });
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        X[i] = T(0);
        W[i] = T(0);
    }
    lsqr_finish<T>(L, s.get(), 0.0, false, kPhaseStart);
}

// Y = a * Xin + b * Y with (a, b) the state's coefficients of the phase; the sums of the new
// Y^2 and (phase V) of W^2, then the phase's scalar step.
template <typename T>
__global__ void __launch_bounds__(kLsqrThreads) k_lsqr_axpby(const T *__restrict__ Xin, T *__restrict__ Y, int64_t n,
                                                const T *__restrict__ W, int phase, LsqrShared L) {
    grid_start(Xin, Y, W);
    const LsqrState *st = L.st;
    if (st->done) {  // the solve has stopped: leave every vector as it is
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            *L.skip_xw = 1;
            if (L.has_cond) cudaGraphSetConditional(L.cond, 0);
        }
        return;
    }
    const T a = (T)(phase == kPhaseU ? st->cu_a : st->cv_a), bb = (T)(phase == kPhaseU ? st->cu_b : st->cv_b);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    SumSq<T> s, s2;
    lsqr_each<T>(n, aligned16(Xin, Y, W), i0, stride, [&](auto vc, auto gc, int64_t i, int64_t gap) {
        constexpr int V = decltype(vc)::value, G = decltype(gc)::value;
        Pack<T, V> x[G], y[G], w[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            x[g] = ldp<T, V>(Xin + i + g * gap);
            y[g] = ldp<T, V>(Y + i + g * gap);
            if (W) w[g] = ldp<T, V>(W + i + g * gap);
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
#pragma unroll
            for (int k = 0; k < V; ++k)
                y[g].v[k] = bb == T(0) ? a * x[g].v[k] : fma(a, x[g].v[k], bb * y[g].v[k]);
            stp<T, V>(Y + i + g * gap, y[g]);
            s.add(y[g].v);
            if (W) s2.add(w[g].v);
        }
    });
    lsqr_finish<T>(L, s.get(), s2.get(), W != nullptr, phase);
}

template <typename T>
__device__ bool one_plus_is_one(double t) {
    return (T)1 + (T)t <= (T)1;
}

// One Float64 division or square root is a chain of dozens of dependent operations on a
// slow pipe, and a step has about thirty of them.  The warp does the independent ones of
// a level together, one per lane, and every lane gets all results.
struct Lanes {
    int lane;
    // r[i] = n_i / d_i
    __device__ __forceinline__ void div(double n0, double d0, double n1, double d1, double n2, double d2, double n3,
                                        double d3, double n4, double d4, double n5, double d5, double n6, double d6,
                                        double (&r)[7]) const {
        const double n = lane == 0 ? n0 : lane == 1 ? n1 : lane == 2 ? n2 : lane == 3 ? n3 : lane == 4 ? n4
                                                                          : lane == 5 ? n5 : n6;
        const double d = lane == 0 ? d0 : lane == 1 ? d1 : lane == 2 ? d2 : lane == 3 ? d3 : lane == 4 ? d4
                                                                          : lane == 5 ? d5 : d6;
        const double v = n / d;
#pragma unroll
        for (int i = 0; i < 7; ++i) r[i] = __shfl_sync(0xffffffffu, v, i);
    }
    __device__ __forceinline__ void root(double a, double b, double c, double (&r)[4], double d = 1.0) const {
        const double v = sqrt(lane == 0 ? a : lane == 1 ? b : lane == 2 ? c : d);
#pragma unroll
        for (int i = 0; i < 4; ++i) r[i] = __shfl_sync(0xffffffffu, v, i);
    }
};

// The scalar step of a phase, by one warp (every lane holds every value).  Phase start: beta =
// ||b||.  Phase U: beta = ||U||.  Phase V: alpha = ||V||, the QR step, estimates and stopping
// rules (first call: the initialisation).  s, s2: the pass' sums of squares.
template <typename T>
__device__ void lsqr_scalar(const LsqrShared &L, double s, double s2, int phase) {
    LsqrState S = *L.st;
    const Lanes W{(int)(threadIdx.x & 31)};
    double q[7], r[4];
    int skip = 1;
    if (phase == kPhaseStart) {
        // a new solve: the recurrence starts afresh, the parameters stay
        S.alpha = S.rhobar = S.phibar = S.anorm = S.acond = S.ddnorm = S.res2 = 0.0;
        S.xnorm = S.xxnorm = S.z = S.sn2 = S.rnorm = S.arnorm = 0.0;
        S.cs2 = -1.0;  // c_0 of the rotation behind the ||x|| estimate
        S.t1 = S.t2 = S.inv_alpha = S.cu_a = S.cu_b = 0.0;
        S.istop = 0;
        S.done = 0;
        S.estimate = 0;
        S.beta = sqrt(s);
        S.bnorm = S.beta;
        S.cv_a = S.beta > 0.0 ? 1.0 / S.beta : 0.0;  // V = A'u = G / beta
        S.cv_b = 0.0;
        S.itn = 0;
    } else if (phase == kPhaseU) {
        const double beta = sqrt(s);
        // paper section 5.1: ||B_k||_F accumulates alpha_k^2 + beta_{k+1}^2 (+ damp^2)
        if (beta > 0.0) {
            S.anorm = sqrt(S.anorm * S.anorm + S.alpha * S.alpha + beta * beta + S.damp * S.damp);
            W.div(1.0, beta, -beta, S.alpha, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, q);
            S.cv_a = q[0];                            // A'u = G / beta
            S.cv_b = S.alpha > 0.0 ? q[1] : 0.0;      // - beta v = -(beta/alpha) V
        } else {
            S.cv_a = 0.0;  // u is zero: v keeps its value (the paper's "if beta > 0")
            S.cv_b = 1.0;
        }
        S.beta = beta;
    } else if (S.itn == 0) {
        // initialisation (paper section 4.1, step 1): alpha_1 v_1 = A' u_1, w_1 = v_1
        const double alpha = sqrt(s);
        W.div(1.0, alpha, -alpha, S.beta, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, q);
        S.alpha = alpha;
        S.rhobar = alpha;
        S.phibar = S.beta;
        S.rnorm = S.beta;
        S.arnorm = alpha * S.beta;
        S.inv_alpha = alpha > 0.0 ? q[0] : 0.0;
        S.t1 = 0.0;
        S.t2 = 0.0;
        S.cu_a = S.inv_alpha;  // A v = F / alpha
        S.cu_b = S.beta > 0.0 ? q[1] : 0.0;
        skip = 0;
        if (S.arnorm == 0.0) {  // x = 0 solves the problem exactly
            S.istop = 0;
            S.done = 1;
        }
        S.itn = 1;
    } else {
        const double beta = S.beta;
        // the damped system's extra rotation (paper section 4.3)
        const double rho1sq = S.rhobar * S.rhobar + S.damp * S.damp;
        W.root(s, rho1sq, rho1sq + beta * beta, r);
        // with beta == 0 the previous v was kept, so alpha is unchanged
        const double alpha = beta > 0.0 ? r[0] : S.alpha;
        const double rhobar1 = r[1], rho = r[2];
        W.div(S.rhobar, rhobar1, S.damp, rhobar1, 1.0, alpha, -alpha, beta, rhobar1, rho, beta, rho, s2, rho * rho, q);
        const double cs1 = q[0], sn1 = q[1];
        S.inv_alpha = alpha > 0.0 ? q[2] : 0.0;
        S.cu_a = S.inv_alpha;
        S.cu_b = beta > 0.0 ? q[3] : 0.0;
        const double psi = sn1 * S.phibar;
        const double phibar0 = cs1 * S.phibar;
        // plane rotation eliminating beta (section 4.1, step 4)
        const double cs = q[4], sn = q[5];
        const double theta = sn * alpha;
        const double phi = cs * phibar0;
        S.rhobar = -cs * alpha;
        S.phibar = sn * phibar0;
        S.tau = sn * phi;
        // estimates (section 5): ||D_k||_F from ||w_k||^2 / rho_k^2, ||x|| via the
        // rotation of the lower bidiagonal factor
        S.ddnorm += q[6];
        S.res2 += psi * psi;
        S.theta = theta;
        S.gambar = -S.cs2 * rho;
        S.rhs = phi - S.sn2 * rho * S.z;
        // x and w update coefficients (step 5)
        W.div(phi, rho, -theta, rho, S.rhs, S.gambar, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, q);
        S.t1 = q[0];
        S.t2 = q[1];
        S.zbar = q[2];
        S.alpha = alpha;
        S.estimate = 1;  // the x/w pass does the rest beside its vectors
        skip = 0;
    }
    if (W.lane != 0) return;
    *L.st = S;
    *L.skip_xw = skip;
    // The loop handle starts each launch at 0 (no iteration): the initialisation opens
    // the loop, the step that meets a stopping rule closes it.
    if (L.has_cond && phase == kPhaseV && !S.estimate) cudaGraphSetConditional(L.cond, S.done ? 0u : 1u);
}

// The rest of phase V, by one warp: the norm and condition estimates and the stopping rules.
// Nothing in the x/w update waits for them.
template <typename T>
__device__ void lsqr_estimate(const LsqrShared &L) {
    LsqrState S = *L.st;
    const Lanes W{(int)(threadIdx.x & 31)};
    double q[7], r[4];
    W.root(S.gambar * S.gambar + S.theta * S.theta, S.phibar * S.phibar + S.res2, S.xxnorm + S.zbar * S.zbar, r,
           S.ddnorm);
    const double gamma = r[0];
    S.rnorm = r[1];
    S.xnorm = r[2];
    S.acond = S.anorm * r[3];
    S.arnorm = S.alpha * fabs(S.tau);
    W.div(S.gambar, gamma, S.theta, gamma, S.rhs, gamma, S.rnorm, S.bnorm, S.arnorm, S.anorm * S.rnorm + S.eps, 1.0,
          S.acond + S.eps, S.anorm * S.xnorm, S.bnorm, q);
    S.cs2 = q[0];
    S.sn2 = q[1];
    S.z = q[2];
    S.xxnorm += S.z * S.z;
    // stopping rules (section 6); the later assignment wins, as in the paper's order
    const double test1 = q[3], test2 = q[4], test3 = q[5];
    W.div(test1, 1.0 + q[6], S.atol * S.anorm * S.xnorm, S.bnorm, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, 1.0, q);
    const double t1s = q[0], rtol = S.btol + q[1];
    int istop = 0;
    if (S.itn >= S.maxiter) istop = 7;
    if (one_plus_is_one<T>(test3)) istop = 6;
    if (one_plus_is_one<T>(test2)) istop = 5;
    if (one_plus_is_one<T>(t1s)) istop = 4;
    if (test3 <= S.ctol) istop = 3;
    if (test2 <= S.atol) istop = 2;
    if (test1 <= rtol) istop = 1;
    if (!(isfinite(S.alpha) && isfinite(S.beta) && isfinite(S.rnorm))) istop = -1;
    S.istop = istop;
    if (istop != 0) S.done = 1;
    else S.itn += 1;
    S.estimate = 0;
    if (W.lane != 0) return;
    *L.st = S;
    if (L.has_cond) cudaGraphSetConditional(L.cond, S.done ? 0u : 1u);
}

// X += t1 W ; W = inv_alpha V + t2 W; block 0 first completes the scalar step.
template <typename T>
__global__ void __launch_bounds__(kLsqrThreads) k_lsqr_xw(const T *__restrict__ V, T *__restrict__ W, T *__restrict__ X,
                                             int64_t n, LsqrShared L) {
    grid_start(V, W, X);
    if (*L.skip_xw) return;
    const T t1 = (T)L.st->t1, t2 = (T)L.st->t2, ia = (T)L.st->inv_alpha;
    const int64_t stride = (int64_t)(gridDim.x - 1) * blockDim.x;
    if (blockIdx.x == 0) {  // this block's own work
        if (threadIdx.x < 32 && L.st->estimate) lsqr_estimate<T>(L);
        return;
    }
    lsqr_each<T>(n, aligned16(V, W, X), (int64_t)(blockIdx.x - 1) * blockDim.x + threadIdx.x, stride,
                 [&](auto vc, auto gc, int64_t i, int64_t gap) {
        constexpr int N = decltype(vc)::value, G = decltype(gc)::value;
        Pack<T, N> w[G], x[G], v[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            w[g] = ldp<T, N>(W + i + g * gap);
            x[g] = ldp<T, N>(X + i + g * gap);
            v[g] = ldp<T, N>(V + i + g * gap);
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
#pragma unroll
            for (int k = 0; k < N; ++k) {
                x[g].v[k] = fma(t1, w[g].v[k], x[g].v[k]);
                w[g].v[k] = fma(ia, v[g].v[k], t2 * w[g].v[k]);
            }
            stp<T, N>(X + i + g * gap, x[g]);
            stp<T, N>(W + i + g * gap, w[g]);
        }
    });
}

}  // namespace
}  // namespace sg

using namespace sg;

struct sg_lsqr {
    int32_t dtype = SG_F32;
    int64_t m = 0, n = 0;
    void *U = nullptr, *V = nullptr, *W = nullptr, *X = nullptr, *F = nullptr, *G = nullptr;
    LsqrState *st = nullptr;  // device
    double *part = nullptr;   // 2 * kLsqrMaxBlocks partial sums
    int *skip = nullptr;      // device flag: skip the x/w pass of this iteration; [1]: finished blocks
    cudaGraphConditionalHandle cond = 0;
    int has_cond = 0;
    cudaStream_t body = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int capture = 0;  // 0 none, 1 prologue, 2 body
};

namespace {

LsqrShared lsqr_shared(const sg_lsqr *h) {
    return LsqrShared{h->st, h->part, h->part + kLsqrMaxBlocks, (unsigned *)(h->skip + 1), h->skip, h->cond,
                      h->has_cond};
}

int lsqr_launch_axpby(sg_lsqr *h, const void *Xin, void *Y, int64_t len, int phase, const void *Wn,
                      cudaStream_t s) {
    const int nb = n_blocks(len);
    if (h->dtype == SG_F64)
        launch(k_lsqr_axpby<double>, nb, kLsqrThreads, 0, s, (const double *)Xin, (double *)Y, len,
               (const double *)Wn, phase, lsqr_shared(h));
    else
        launch(k_lsqr_axpby<float>, nb, kLsqrThreads, 0, s, (const float *)Xin, (float *)Y, len,
               (const float *)Wn, phase, lsqr_shared(h));
    return cuda_check(cudaGetLastError(), "k_lsqr_axpby launch");
}

bool vec_ok(const void *p) { return p && ((uintptr_t)p % 8) == 0; }

}  // namespace

extern "C" int sg_lsqr_create(int32_t dtype, int64_t m, int64_t n, void *U, void *V, void *W,
                              void *X, void *F, void *G, double damp, double atol, double btol,
                              double conlim, int64_t maxiter, sg_lsqr **out) {
    if (!out) return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_create: NULL out");
    *out = nullptr;
    if (dtype != SG_F32 && dtype != SG_F64)
        return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_create: dtype must be F32 or F64");
    if (m < 1 || n < 1 || maxiter < 1)
        return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_create: sizes and maxiter must be >= 1");
    if (!vec_ok(U) || !vec_ok(V) || !vec_ok(W) || !vec_ok(X) || !vec_ok(F) || !vec_ok(G))
        return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_create: NULL or misaligned vector");
    if (!(damp >= 0.0) || !(atol >= 0.0) || !(btol >= 0.0) || !(conlim >= 0.0))
        return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_create: tolerances must be >= 0");
    sg_lsqr *h = new sg_lsqr;
    h->dtype = dtype;
    h->m = m;
    h->n = n;
    h->U = U; h->V = V; h->W = W; h->X = X; h->F = F; h->G = G;
    int rc = dev_alloc((void **)&h->st, sizeof(LsqrState), "lsqr: state");
    if (!rc) rc = dev_alloc((void **)&h->part, 2 * kLsqrMaxBlocks * sizeof(double), "lsqr: partials");
    if (!rc) rc = dev_alloc((void **)&h->skip, 2 * sizeof(int), "lsqr: flag");
    if (!rc) rc = cuda_check(cudaMemset(h->skip, 0, 2 * sizeof(int)), "lsqr: flag");
    if (!rc) {
        LsqrState S = {};
        S.damp = damp;
        S.atol = atol;
        S.btol = btol;
        S.ctol = conlim > 0.0 ? 1.0 / conlim : 0.0;
        S.eps = dtype == SG_F64 ? 2.220446049250313e-16 : 1.1920928955078125e-07;
        S.maxiter = maxiter;
        S.done = 1;  // nothing to do before sg_lsqr_start
        rc = cuda_check(cudaMemcpy(h->st, &S, sizeof(S), cudaMemcpyHostToDevice), "lsqr: init");
    }
    if (rc) {
        sg_lsqr_destroy(h);
        return rc;
    }
    *out = h;
    return SG_OK;
}

extern "C" int sg_lsqr_destroy(sg_lsqr *h) {
    if (!h) return SG_OK;
    if (h->exec) cudaGraphExecDestroy(h->exec);
    if (h->graph) cudaGraphDestroy(h->graph);
    if (h->body) cudaStreamDestroy(h->body);
    dev_free(h->st);
    dev_free(h->part);
    dev_free(h->skip);
    delete h;
    return SG_OK;
}

extern "C" int sg_lsqr_start(sg_lsqr *h, const void *b, sg_stream_t stream) {
    if (!h || !vec_ok(b)) return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_start: NULL argument");
    cudaStream_t s = (cudaStream_t)stream;
    const int nb = n_blocks(h->m > h->n ? h->m : h->n);
    if (h->dtype == SG_F64)
        launch(k_lsqr_start<double>, nb, kLsqrThreads, 0, s, (const double *)b, (double *)h->U, h->m,
               (double *)h->X, (double *)h->W, h->n, lsqr_shared(h));
    else
        launch(k_lsqr_start<float>, nb, kLsqrThreads, 0, s, (const float *)b, (float *)h->U, h->m,
               (float *)h->X, (float *)h->W, h->n, lsqr_shared(h));
    return cuda_check(cudaGetLastError(), "k_lsqr_start launch");
}

extern "C" int sg_lsqr_after_forward(sg_lsqr *h, sg_stream_t stream) {
    if (!h) return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_after_forward: NULL handle");
    return lsqr_launch_axpby(h, h->F, h->U, h->m, kPhaseU, nullptr, (cudaStream_t)stream);
}

extern "C" int sg_lsqr_after_adjoint(sg_lsqr *h, sg_stream_t stream) {
    if (!h) return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_after_adjoint: NULL handle");
    cudaStream_t s = (cudaStream_t)stream;
    int rc = lsqr_launch_axpby(h, h->G, h->V, h->n, kPhaseV, h->W, s);
    if (rc) return rc;
    const int nb = n_blocks(h->n) + 1;
    if (h->dtype == SG_F64)
        launch(k_lsqr_xw<double>, nb, kLsqrThreads, 0, s, (const double *)h->V, (double *)h->W,
               (double *)h->X, h->n, lsqr_shared(h));
    else
        launch(k_lsqr_xw<float>, nb, kLsqrThreads, 0, s, (const float *)h->V, (float *)h->W, (float *)h->X,
               h->n, lsqr_shared(h));
    return cuda_check(cudaGetLastError(), "k_lsqr_xw launch");
}

extern "C" int sg_lsqr_capture_begin(sg_lsqr *h, sg_stream_t stream) {
    if (!h) return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_capture_begin: NULL handle");
    if (h->capture) return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_capture_begin: already capturing");
    cudaStream_t s = (cudaStream_t)stream;
    int rc = SG_OK;
    if (!h->body)
        rc = cuda_check(cudaStreamCreateWithFlags(&h->body, cudaStreamNonBlocking), "lsqr: body stream");
    if (rc) return rc;
    if (h->exec) { cudaGraphExecDestroy(h->exec); h->exec = nullptr; }
    if (h->graph) { cudaGraphDestroy(h->graph); h->graph = nullptr; }
    rc = cuda_check(cudaStreamBeginCapture(s, cudaStreamCaptureModeRelaxed), "lsqr: begin capture");
    if (rc) return rc;
    h->capture = 1;
    cudaStreamCaptureStatus cs;
    cudaGraph_t g = nullptr;
    rc = cuda_check(cudaStreamGetCaptureInfo(s, &cs, nullptr, &g, nullptr, nullptr, nullptr),
                    "lsqr: capture info");
    // the loop runs while the handle is non-zero; every launch of the graph starts it at 0
    // and the prologue's initialisation step opens it, so the loop never runs unless a
    // kernel of this solve set it
    if (!rc) rc = cuda_check(cudaGraphConditionalHandleCreate(&h->cond, g, 0, cudaGraphCondAssignDefault),
                             "lsqr: conditional handle");
    if (!rc) h->has_cond = 1;
    return rc;
}

extern "C" int sg_lsqr_capture_body(sg_lsqr *h, sg_stream_t stream, sg_stream_t *body) {
    if (!h || !body) return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_capture_body: NULL argument");
    if (h->capture != 1) return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_capture_body: not in the prologue");
    cudaStream_t s = (cudaStream_t)stream;
    cudaStreamCaptureStatus cs;
    cudaGraph_t g = nullptr;
    const cudaGraphNode_t *deps = nullptr;
    size_t ndeps = 0;
    int rc = cuda_check(cudaStreamGetCaptureInfo(s, &cs, nullptr, &g, &deps, nullptr, &ndeps),
                        "lsqr: capture info");
    if (rc) return rc;
    cudaGraphNodeParams p = {};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h->cond;
    p.conditional.type = cudaGraphCondTypeWhile;
    p.conditional.size = 1;
    cudaGraphNode_t node;
    rc = cuda_check(cudaGraphAddNode(&node, g, deps, nullptr, ndeps, &p), "lsqr: while node");
    if (!rc) rc = cuda_check(cudaStreamUpdateCaptureDependencies(s, &node, nullptr, 1,
                                                                 cudaStreamSetCaptureDependencies),
                             "lsqr: capture dependencies");
    if (!rc) rc = cuda_check(cudaStreamBeginCaptureToGraph(h->body, p.conditional.phGraph_out[0],
                                                           nullptr, nullptr, 0,
                                                           cudaStreamCaptureModeRelaxed),
                             "lsqr: begin body capture");
    if (rc) return rc;
    h->capture = 2;
    *body = (sg_stream_t)h->body;
    return SG_OK;
}

extern "C" int sg_lsqr_capture_end(sg_lsqr *h, sg_stream_t stream) {
    if (!h) return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_capture_end: NULL handle");
    cudaStream_t s = (cudaStream_t)stream;
    int rc = SG_OK;
    if (h->capture == 2) {
        cudaGraph_t bg = nullptr;
        rc = cuda_check(cudaStreamEndCapture(h->body, &bg), "lsqr: end body capture");
    }
    cudaGraph_t g = nullptr;
    if (h->capture >= 1) {
        const int rc2 = cuda_check(cudaStreamEndCapture(s, &g), "lsqr: end capture");
        if (!rc) rc = rc2;
    }
    const int complete = h->capture == 2;
    h->capture = 0;
    h->has_cond = 0;
    if (!rc && !complete)
        rc = set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_capture_end: the loop body was not captured");
    if (!rc) rc = cuda_check(cudaGraphInstantiate(&h->exec, g, 0), "lsqr: instantiate");
    if (rc) {
        if (g) cudaGraphDestroy(g);
        return rc;
    }
    h->graph = g;
    return SG_OK;
}

extern "C" int sg_lsqr_launch(sg_lsqr *h, sg_stream_t stream) {
    if (!h || !h->exec) return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_launch: no captured solve");
    return cuda_check(cudaGraphLaunch(h->exec, (cudaStream_t)stream), "lsqr: graph launch");
}

extern "C" int sg_lsqr_info(sg_lsqr *h, sg_stream_t stream, int64_t *counts, double *norms) {
    if (!h || !counts || !norms) return set_error(SG_ERR_INVALID_ARGUMENT, "sg_lsqr_info: NULL argument");
    LsqrState S;
    cudaStream_t s = (cudaStream_t)stream;
    int rc = cuda_check(cudaMemcpyAsync(&S, h->st, sizeof(S), cudaMemcpyDeviceToHost, s), "lsqr: read state");
    if (!rc) rc = cuda_check(cudaStreamSynchronize(s), "lsqr: sync");
    if (rc) return rc;
    counts[0] = S.itn;
    counts[1] = S.istop;
    counts[2] = S.done;
    norms[0] = S.anorm;
    norms[1] = S.acond;
    norms[2] = S.rnorm;
    norms[3] = S.arnorm;
    norms[4] = S.xnorm;
    norms[5] = S.bnorm;
    return SG_OK;
}
