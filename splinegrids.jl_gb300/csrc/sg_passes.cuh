// sg_passes.cuh -- host launchers of the separable passes (instantiated per value type
// in sg_passes_f32.cu / sg_passes_f64.cu so the translation units build in parallel).
#pragma once

#include <type_traits>

#include "sg_contract.cuh"
#include "sg_warp.cuh"
#include "sg_ring.cuh"

namespace sg {

// One contraction pass over one input axis (see sg_contract.cuh for the index maps).
struct AxisPass {
    const int32_t *idx = nullptr;   // sample indices of the axis (1-based)
    const int32_t *perm = nullptr;  // sorted view of the samples, or NULL when sorted
    const int32_t *lb = nullptr;    // support table of the axis (adjoint), or NULL
    const void *B = nullptr;        // basis table block of the derivative order: B[j + ns*i]
    int64_t ns = 0;                 // samples along the axis
    int d = 0;                      // degree
    int64_t n = 0;                  // control points along the axis
    int64_t M = 1;                  // product of the axes before this one
    int64_t Q = 1;                  // product of the axes after (axis-0 kHomog: without channels)
    const void *X = nullptr;
    void *Y = nullptr;
    const void *w = nullptr;        // NURBS weights (axis-0 forward pass only)
    int nch = 0;                    // output channels (Nout)
    int mode = kPlain;
    bool final_pass = false;        // writes eval
    int x_dtype = SG_F32;           // element type of X on the axis-0 forward pass
    int cc = 0;                     // adjoint: control points per chunk (0: heuristic)
    int64_t support = 0;            // Nin = 1 adjoint: samples in the longest support (adj_line_*)
};

int fwd_axis0_f32(const AxisPass &p, cudaStream_t s);
int fwd_axis0_f64(const AxisPass &p, cudaStream_t s);
int fwd_axis_f32(const AxisPass &p, cudaStream_t s);
int fwd_axis_f64(const AxisPass &p, cudaStream_t s);
int adj_axis_f32(const AxisPass &p, cudaStream_t s);
int adj_axis_f64(const AxisPass &p, cudaStream_t s);
int adj_axis0_f32(const AxisPass &p, cudaStream_t s);
int adj_axis0_f64(const AxisPass &p, cudaStream_t s);
// Nin = 1 with supports longer than kLineSupport, degrees 0..5 (p.support set)
int adj_line_f32(const AxisPass &p, cudaStream_t s);
int adj_line_f64(const AxisPass &p, cudaStream_t s);
// Samples in the longest support of an axis (lb: its support table).
inline int64_t longest_support(const int32_t *lb, int64_t n, int d) {
    int64_t m = 0;
    for (int64_t c = 0; c < n; ++c) m = lb[c + 1 + d] - lb[c] > m ? lb[c + 1 + d] - lb[c] : m;
    return m;
}

constexpr int64_t kMaxGridYZ = 65535;
constexpr int64_t kNumSMs = 152;                 // GB300
constexpr int64_t kTargetCtas = kNumSMs * 8;     // grid size aimed at by sized launches

inline unsigned gdim(int64_t v, int64_t cap) { return (unsigned)(v < 1 ? 1 : (v > cap ? cap : v)); }

template <typename T>
inline int vec_width(const AxisPass &p) {
    // 16-byte accesses along m need M to be a multiple of the vector width and all
    // base pointers 16-byte aligned (every row start is then aligned too).
    constexpr int V = 16 / (int)sizeof(T);
    const bool ok = (p.M % V == 0) && ((uintptr_t)p.X % 16 == 0) && ((uintptr_t)p.Y % 16 == 0);
    return ok ? V : 1;
}

// ------------------------------------------------------------------ forward axis 0
template <typename T, typename TX, int D, int MODE>
inline void launch_fwd_axis0_t(const AxisPass &p, cudaStream_t s) {
    // kHomog: a short axis 0 takes blocks of its length, and as many more of them (16 samples, 504900
    // columns, Float32: 404 us with whole blocks, 116 so)
    const unsigned block = MODE == kHomog && p.ns < kThreads ? (unsigned)((p.ns + 31) / 32 * 32) : kThreads;
    const unsigned gx = (unsigned)((p.ns + kThreads - 1) / kThreads);
    int64_t Qy = (MODE == kHomog) ? p.Q : (MODE == kRational ? 1 : p.Q * p.nch);
    // each thread walks Qy/gridDim.y columns with its basis values in registers; size
    // grid.y for ~32 CTAs per SM (a few columns per thread: more loads in flight per SM)
    // rather than one output per thread
    const int64_t want_y = (kTargetCtas * (MODE == kHomog ? 2 * (kThreads / block) : 4) + gx - 1) / gx;
    dim3 grid(gx, gdim(Qy < want_y ? Qy : want_y, kMaxGridYZ));
    if (MODE == kHomog) {  // channels in turn by one thread unless that leaves too few blocks
        const int64_t z = want_y / grid.y;
        grid.z = gdim(z < p.nch + 1 ? z : p.nch + 1, kMaxGridYZ);
    }
    launch(k_fwd_axis0<D, TX, T, MODE>, grid, block, 0, s, p.idx, (const T *)p.B, p.ns, p.d, (const TX *)p.X,
           (const T *)p.w, p.n, p.Q, p.nch, (T *)p.Y);
}

template <typename T, typename TX, int MODE>
inline void launch_fwd_axis0_d(const AxisPass &p, cudaStream_t s) {
    switch (p.d) {
        case 0: launch_fwd_axis0_t<T, TX, 1, MODE>(p, s); break;
        case 1: launch_fwd_axis0_t<T, TX, 2, MODE>(p, s); break;
        case 2: launch_fwd_axis0_t<T, TX, 3, MODE>(p, s); break;
        case 3: launch_fwd_axis0_t<T, TX, 4, MODE>(p, s); break;
        default: launch_fwd_axis0_t<T, TX, 0, MODE>(p, s); break;
    }
}

// Warp tasks of the axis-0 passes: enough for ~16 warps per SM.
constexpr int64_t kAxis0Tasks = (int64_t)kNumSMs * 16;

// kPlain, degrees <= 3, same-type input: warp tasks of 32 columns x a chunk of samples
// (sg_warp.cuh); few columns get short chunks (at least 32 samples) so the tasks still
// fill the GPU
template <typename T, int D>
inline void launch_fwd0_warp(const AxisPass &p, cudaStream_t s) {
    const int64_t Qy = p.Q * p.nch;
    const int64_t groups = (Qy + 31) / 32;
    if (groups == 0 || p.ns == 0) return;
    const int64_t want = (kAxis0Tasks + groups - 1) / groups;  // sample chunks wanted
    int64_t SC = (p.ns + want - 1) / want;
    SC = SC < 32 ? 32 : SC;
    const int64_t tasks = groups * ((p.ns + SC - 1) / SC);
    const int64_t blocks = (tasks + kWarpsPerBlock - 1) / kWarpsPerBlock;
    launch(k_fwd0_warp<D, T>, (unsigned)blocks, 32 * kWarpsPerBlock, 0, s, p.idx, (const T *)p.B, p.ns, p.d,
           (const T *)p.X, p.n, Qy, SC, (T *)p.Y);
}

template <typename T, typename TX>
inline void launch_fwd_axis0_m(const AxisPass &p, cudaStream_t s) {
    if constexpr (std::is_same<T, TX>::value) {
        // warp tasks when their columns alone fill the GPU; fewer columns run faster as
        // the CTA kernel (each thread keeps one sample's basis row for many columns)
        if (p.mode == kPlain && p.d <= 3 && (p.Q * p.nch + 31) / 32 >= kAxis0Tasks) {
            switch (p.d) {
                case 0: launch_fwd0_warp<T, 1>(p, s); return;
                case 1: launch_fwd0_warp<T, 2>(p, s); return;
                case 2: launch_fwd0_warp<T, 3>(p, s); return;
                default: launch_fwd0_warp<T, 4>(p, s); return;
            }
        }
    }
    if (p.mode == kPlain) launch_fwd_axis0_d<T, TX, kPlain>(p, s);
    else if (p.mode == kHomog) launch_fwd_axis0_d<T, TX, kHomog>(p, s);
    else launch_fwd_axis0_d<T, TX, kRational>(p, s);
}


// ------------------------------------------------------------------ forward axis k
template <typename T, int D, int VEC, bool FINAL, bool ST>
inline void launch_fwd_axis_t(const AxisPass &p, cudaStream_t s) {
    const int64_t per_cta = (int64_t)kThreads * VEC;
    const unsigned gx = (unsigned)((p.M + per_cta - 1) / per_cta);
    const int64_t chunks = (p.ns + kChunk - 1) / kChunk;
    // grid.y addresses sample chunks; an axis longer than 65535 chunks is launched in
    // slices, each on bases shifted by the slice's first sample.
    for (int64_t c0 = 0; c0 < chunks; c0 += kMaxGridYZ) {
        const int64_t cn = (chunks - c0 < kMaxGridYZ) ? chunks - c0 : kMaxGridYZ;
        const int64_t jb = c0 * kChunk;
        const int64_t jcount = (p.ns - jb < cn * kChunk) ? p.ns - jb : cn * kChunk;
        dim3 grid(gx, (unsigned)cn, gdim(p.Q, kMaxGridYZ));
        launch(k_fwd_axis<D, T, VEC, FINAL, ST>, grid, kThreads, 0, s, p.idx + jb, (const T *)p.B + jb, p.ns,
               jcount, p.d, (const T *)p.X, p.M, p.n, p.Q, (T *)p.Y + p.M * jb);
    }
}

// kPlain passes of degree <= 5 run as warp tasks (sg_warp.cuh), or one thread per output up
// to kThreadFwdValues outputs, where the tasks leave most of the GPU idle ((50, 50, 25) x 4,
// Float64, all three axes: 6.7 us against 24.5; at 6 M outputs the threads take 35 against 19)
constexpr int64_t kThreadFwdValues = 1 << 19;
// Samples of a warp task: kFwdRowsMax, halved down to kFwdRowsMin while that leaves fewer than
// 16 tasks an SM (Float64, whose rows take longer: 27).  A task runs its samples one after
// the other, so few long tasks leave most of the chip idle; short ones load their windows
// more often.  With 32 samples a task and with this rule, all passes: (64, 64) NURBS, (1024,
// 1024) x 3 samples 20.9 and 8.9 us; (100, 100, 100) x 3 17.7 and 10.6; (200, 160, 120) Float64 54.7
// and 44.6; with twice the tasks wanted (200, 300) NURBS, (2000, 3000) takes 15.5 for 12.5.
constexpr int kFwdRowsMax = 32, kFwdRowsMin = 4;
template <typename T>
constexpr int64_t fwd_tasks() { return (int64_t)kNumSMs * (sizeof(T) == 4 ? 16 : 27); }
template <typename T, int D, bool ST, bool FINAL, int NC = 0>
inline void launch_fwd_warp(const AxisPass &p, cudaStream_t s) {
    const int64_t gxw = (p.M + warp_width<T>() - 1) / warp_width<T>();
    const int64_t Q = NC > 0 ? 1 : p.Q;  // rational: a task holds all channels
    int rows = kFwdRowsMax;
    while (rows > kFwdRowsMin && gxw * ((p.ns + rows - 1) / rows) * Q < fwd_tasks<T>()) rows /= 2;
    const int64_t tasks = gxw * ((p.ns + rows - 1) / rows) * Q;
    const int64_t blocks = (tasks + kWarpsPerBlock - 1) / kWarpsPerBlock;
    if (blocks == 0) return;
    const int64_t total = p.M * p.ns * Q;
    if (NC == 0 && total <= kThreadFwdValues) {
        launch(k_fwd_thread<D, T>, (unsigned)((total + kThreadBlock - 1) / kThreadBlock), kThreadBlock, 0, s,
               p.idx, (const T *)p.B, (uint32_t)p.ns, (const T *)p.X, (uint32_t)p.M, (uint32_t)p.n,
               (uint32_t)total, (T *)p.Y);
        return;
    }
    launch(k_fwd_warp<D, T, ST, FINAL, NC>, (unsigned)blocks, 32 * kWarpsPerBlock, 0, s, p.idx, (const T *)p.B,
           p.ns, p.d, (const T *)p.X, p.M, p.n, Q, NC > 0 ? (int)p.nch : 0, gxw, (p.ns + rows - 1) / rows, rows,
           (T *)p.Y);
}

template <typename T, int D, int VEC, bool ST>
inline void launch_fwd_axis_v(const AxisPass &p, cudaStream_t s) {
    if (p.mode == kRational) {
        if (p.nch + 1 <= 2) launch_fwd_warp<T, D, ST, true, 2>(p, s);
        else launch_fwd_warp<T, D, ST, true, 4>(p, s);
    } else if (p.final_pass) {
        launch_fwd_warp<T, D, ST, true>(p, s);
    } else {
        launch_fwd_warp<T, D, ST, false>(p, s);
    }
}

// aligned rows: contiguous 16-byte accesses; otherwise the same VEC values per thread
// strided by the block width
template <typename T, int D>
inline void launch_fwd_axis_d(const AxisPass &p, cudaStream_t s) {
    constexpr int V = 16 / (int)sizeof(T);
    if (vec_width<T>(p) == V) launch_fwd_axis_v<T, D, V, false>(p, s);
    else launch_fwd_axis_v<T, D, V, true>(p, s);
}

// degrees 4 and 5 (NURBS take the generic rational kernel)
template <typename T, int D>
inline void launch_fwd_axis_plain(const AxisPass &p, cudaStream_t s) {
    constexpr int V = 16 / (int)sizeof(T);
    if (vec_width<T>(p) == V) {
        if (p.final_pass) launch_fwd_warp<T, D, false, true>(p, s);
        else launch_fwd_warp<T, D, false, false>(p, s);
    } else {
        if (p.final_pass) launch_fwd_warp<T, D, true, true>(p, s);
        else launch_fwd_warp<T, D, true, false>(p, s);
    }
}

template <typename T>
inline void launch_fwd_axis(const AxisPass &p, cudaStream_t s) {
    if (p.mode == kRational && (p.nch + 1 > 4 || p.d > 3)) {
        dim3 grid((unsigned)((p.M + kThreads - 1) / kThreads), gdim(p.ns, kMaxGridYZ));
        launch(k_fwd_axis_rational_generic<T>, grid, kThreads, 0, s, p.idx, (const T *)p.B, p.ns, p.d,
               (const T *)p.X, p.M, p.n, p.nch, (T *)p.Y);
        return;
    }
    switch (p.d) {
        case 0: launch_fwd_axis_d<T, 1>(p, s); break;
        case 1: launch_fwd_axis_d<T, 2>(p, s); break;
        case 2: launch_fwd_axis_d<T, 3>(p, s); break;
        case 3: launch_fwd_axis_d<T, 4>(p, s); break;
        case 4: launch_fwd_axis_plain<T, 5>(p, s); break;
        case 5: launch_fwd_axis_plain<T, 6>(p, s); break;
        default:  // any degree: runtime-degree kernel, scalar accesses
            if (p.final_pass) launch_fwd_axis_t<T, 0, 1, true, false>(p, s);
            else launch_fwd_axis_t<T, 0, 1, false, false>(p, s);
    }
}

// ------------------------------------------------------------------ adjoint axis k
template <typename T, int D, int VEC, bool ST>
inline void launch_adj_axis_t(const AxisPass &p, cudaStream_t s) {
    // Control points per CTA: as wide as possible (the halo of d knot spans shared
    // with the neighbour chunk is re-read) while the grid still gives every SM ~4 CTAs.
    const int64_t per_cta = (int64_t)kThreads * VEC;
    const unsigned gx = (unsigned)((p.M + per_cta - 1) / per_cta);
    const int64_t gz = p.Q < kMaxGridYZ ? p.Q : kMaxGridYZ;
    const int64_t want_chunks = (kNumSMs * 4 + gx * gz - 1) / (gx * gz);
    int64_t CC = (p.n + want_chunks - 1) / want_chunks;
    CC = CC < 8 ? 8 : (CC > 64 ? 64 : CC);
    if ((p.n + CC - 1) / CC > kMaxGridYZ) CC = (p.n + kMaxGridYZ - 1) / kMaxGridYZ;
    const int64_t chunks = (p.n + CC - 1) / CC;
    dim3 grid(gx, (unsigned)chunks, (unsigned)gz);
    const int smem = (int)adj_axis_smem_bytes<D, T, VEC>(kThreads);
    static bool attr_set = false;  // one instance per template instantiation
    if (!attr_set) {
        cudaFuncSetAttribute(k_adj_axis<D, T, VEC, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem);
        attr_set = true;
    }
    launch(k_adj_axis<D, T, VEC, ST>, grid, kThreads, smem, s, p.idx, p.perm, p.lb, (const T *)p.B, p.ns, p.d,
           (const T *)p.X, p.M, p.n, p.Q, (int)CC, (T *)p.Y);
}

// One thread per output (sg_ring.cuh).
template <typename T, int D>
inline void launch_adj_thread(const AxisPass &p, cudaStream_t s) {
    const int64_t total = p.M * p.n * p.Q;
    if (total == 0) return;
    launch(k_adj_thread<D, T>, (unsigned)((total + kThreadBlock - 1) / kThreadBlock), kThreadBlock, 0, s, p.perm,
           p.lb, (const T *)p.B, (uint32_t)p.ns, (const T *)p.X, (uint32_t)p.M, (uint32_t)p.n, (uint32_t)total,
           (T *)p.Y);
}

// Control points per chunk of an adjoint pass whose units are warps (k_adj_ring,
// k_adj_cols): per_chunk units per chunk.  A unit walks the rows of CC + d knot spans (the
// d last ones are read again by the next chunk), every row costs it at least `lat` cycles,
// and `per` cycles of its SM sub-partition (each has its own FP64 pipe and a quarter of the
// SM's share of the memory bandwidth), where ceil(units / sub-partitions) units share it.
// The chunk count with the smallest (CC + d) * max(lat, units per sub-partition * per); beyond
// 512 chunks in steps of 3 %.  cost_out: that product.
inline int64_t adj_chunk(const AxisPass &p, int64_t per_chunk, int64_t lat, int64_t per, int64_t *cost_out = nullptr) {
    int64_t best = p.n, best_cost = INT64_MAX, prev = 0;
    for (int64_t k = 1; k <= p.n; k += k < 512 ? 1 : k / 32) {
        const int64_t CC = (p.n + k - 1) / k;
        if (CC == prev) continue;
        prev = CC;
        const int64_t units = per_chunk * ((p.n + CC - 1) / CC);
        const int64_t share = (units + kNumSMs * 4 - 1) / (kNumSMs * 4);
        const int64_t cost = (CC + p.d) * (lat > share * per ? lat : share * per);
        if (cost < best_cost && units <= INT32_MAX) {
            best_cost = cost;
            best = CC;
        }
    }
    if (cost_out) *cost_out = best_cost;
    return p.cc > 0 && per_chunk * ((p.n + p.cc - 1) / p.cc) <= INT32_MAX ? p.cc : best;  // cc: measured by sg_grid_plan_tune
}
// Cycles of adj_chunk's model, fitted to sweeps on (256, 256) x (4096, 4096) x 3,
// (2048, 2048) and (1999, 1501) x 3 (each within 5 % of its best chunk count).
constexpr int64_t kRingLat = 170, kRingPer = 60;
constexpr int64_t kColsLat = 120, kColsPer = 12;

template <typename T, int D>
inline void launch_adj_ring(const AxisPass &p, cudaStream_t s) {
    constexpr int64_t W = warp_width<T>();
    const int64_t gxw = (p.M + W - 1) / W, per_chunk = gxw * p.Q;
    if (per_chunk == 0) return;
    const int64_t CC = adj_chunk(p, per_chunk, kRingLat, kRingPer);
    const int64_t chunks = (p.n + CC - 1) / CC;
    launch(k_adj_ring<D, T>, (unsigned)(per_chunk * chunks), 32, (ring_smem<D, T>()), s, p.perm, p.lb,
           (const T *)p.B, p.ns, (const T *)p.X, p.M, p.n, (int)CC, gxw, chunks, (T *)p.Y);
}
template <typename T, int D>
inline void launch_adj_cols(const AxisPass &p, cudaStream_t s) {
    const int64_t gxw = (p.M + 31) / 32, per_chunk = gxw * p.Q;
    if (per_chunk == 0) return;
    // Float64: a warp FMA holds a sub-partition's FP64 pipe for 64 cycles
    const int64_t CC = sizeof(T) == 4 ? adj_chunk(p, per_chunk, kColsLat, kColsPer)
                                      : adj_chunk(p, per_chunk, 64 * D + kColsLat, 64 * D);
    const int64_t chunks = (p.n + CC - 1) / CC, units = per_chunk * chunks;
    launch(k_adj_cols<D, T, 8>, (unsigned)((units + kColsWarps - 1) / kColsWarps), 32 * kColsWarps, 0, s, p.perm,
           p.lb, (const T *)p.B, p.ns, (const T *)p.X, p.M, p.n, (int)CC, gxw, chunks, units, (T *)p.Y);
}

// Warp tasks of 128 (Float64: 64) values of m x CC control points (sg_warp.cuh).
template <typename T, int D, bool ST>
inline void launch_adj_warp(const AxisPass &p, cudaStream_t s) {
    const int64_t gxw = (p.M + warp_width<T>() - 1) / warp_width<T>();
    const int64_t per_chunk = gxw * p.Q;  // tasks per chunk
    if (per_chunk == 0) return;
    const int64_t want_chunks = (kNumSMs * 32 * 2 + per_chunk - 1) / per_chunk;
    int64_t CC = (p.n + want_chunks - 1) / want_chunks;
    CC = CC < 8 ? 8 : (CC > 64 ? 64 : CC);
    const int64_t chunks = (p.n + CC - 1) / CC;
    const int64_t blocks = (per_chunk * chunks + kWarpsPerBlock - 1) / kWarpsPerBlock;
    launch(k_adj_warp<D, T, ST>, (unsigned)blocks, 32 * kWarpsPerBlock, 0, s, p.idx, p.perm, p.lb, (const T *)p.B,
           p.ns, p.d, (const T *)p.X, p.M, p.n, p.Q, (int)CC, gxw, chunks, (T *)p.Y);
}

// The kernel of an adjoint pass over an axis k >= 1, degrees 0 to 5; all give the same bits.  S:
// samples a control point sums.  The lines were drawn through 4500 measured passes (0.5 to 80
// samples a control point, 2^13 to 2^25 values, rows of 1 to 10^7); us, Float32 unless said:
//  * Rows below 24 values leave a quarter of a warp's lanes and more idle in every other kernel: one
//    thread per output ((8, 1104301) x 2, 361168 control points, degree 3: 122, rings 299).  But a
//    few thousand outputs with long sums leave the SMs idle: rings ((16, 5104), 112, degree 4: 21,
//    threads 47).  And where a control point has hardly a sample, threads read each row d + 1
//    times from far apart: warp tasks ((16, 1339501), 1079800, degree 2: 172, threads 185; (24,
//    1068033), 1087384: 150 and 241).
//  * Short sums (S < 9) never make up for the ring's 800 cycles a completed control point: warp tasks
//    ((1104, 17941), 33274, degree 1: 41, rings 56; (51332, 141) x 4 Float64, 94, degree 0: 80,
//    columns 293), or, small, one thread per output.
//  * Float64, up to 2^13 values a row and 2^23 in all, or few values: one thread per output fills the
//    FP64 pipe more evenly than units do ((40, 39431), 1287, degree 2: 28, columns 41).
//  * Many columns of few samples: four warp tasks a CTA start faster than rings ((268872, 11) x 4, 4,
//    degree 3: 19 and 23).
//  * Unsorted samples leave rows in no order that caches like: warp tasks, which keep more of them in
//    flight ((4792, 5542) Float64, 454, degree 1: 125, columns 418).
//  * The others: rings (Float32 rows of 16-byte multiples; (220, 74811), 1273, degree 1: 22, warp
//    tasks 79), columns.
enum AdjKernel { kAdjThread, kAdjWarp, kAdjLong, kAdjGeneric };
template <typename T>
inline AdjKernel adj_axis_kernel(const AxisPass &p) {
    constexpr bool f64 = sizeof(T) == 8;
    const double S = (double)p.ns * (p.d + 1) / (double)p.n;
    const int64_t MQ = p.M * p.Q, O = MQ * p.n, V = MQ * p.ns;
    const bool warp = p.d <= 3, rings = !f64 && vec_width<T>(p) == 16 / (int)sizeof(T);
    if (O > INT32_MAX || p.ns > INT32_MAX) return kAdjLong;  // k_adj_thread counts in 32 bits
    if (p.M < 24) {
        if (O < 12288 && S >= 32) return kAdjLong;
        if (warp && p.M >= 8 && (f64 ? S < 2 && O >= 1 << 18 : S < 4 && O >= 1 << 20)) return kAdjWarp;
        return kAdjThread;
    }
    if (S < 9) {
        if (O < 1 << 18 && MQ < 1 << 16) return kAdjThread;
        return warp ? kAdjWarp : kAdjLong;
    }
    if (f64 && (V < 1 << 18 || (MQ < 1 << 13 && V < 1 << 23))) return kAdjThread;
    if (warp && MQ >= 1 << 18 && p.ns < 24) return kAdjWarp;
    if (warp && !f64 && !rings && MQ >= 1 << 14 && S < 16) return kAdjWarp;
    if (warp && p.perm && (f64 ? V >= 1 << 22 : O >= 3 << 19)) return kAdjWarp;
    return kAdjLong;
}

template <typename T, int D>
inline void launch_adj_axis_d(const AxisPass &p, cudaStream_t s) {
    if constexpr (D == 0) {
        launch_adj_axis_t<T, D, 1, false>(p, s);  // runtime degree: one value a thread
    } else {
        const bool aligned = vec_width<T>(p) == 16 / (int)sizeof(T);
        const AdjKernel k = adj_axis_kernel<T>(p);
        if (k == kAdjThread) {
            launch_adj_thread<T, D>(p, s);
            return;
        }
        if constexpr (D <= 4) {
            if (k == kAdjWarp) {
                if (aligned) launch_adj_warp<T, D, false>(p, s);
                else launch_adj_warp<T, D, true>(p, s);
                return;
            }
        }
        if constexpr (sizeof(T) == 4) {
            // rings copy 16 bytes per lane; Float64 passes are bound by the FP64 pipe, which
            // the finer units of k_adj_cols fill more evenly
            if (aligned) {
                launch_adj_ring<T, D>(p, s);
                return;
            }
        }
        launch_adj_cols<T, D>(p, s);
    }
}

template <typename T>
inline void launch_adj_axis(const AxisPass &p, cudaStream_t s) {
    switch (p.d) {
        case 0: launch_adj_axis_d<T, 1>(p, s); break;
        case 1: launch_adj_axis_d<T, 2>(p, s); break;
        case 2: launch_adj_axis_d<T, 3>(p, s); break;
        case 3: launch_adj_axis_d<T, 4>(p, s); break;
        case 4: launch_adj_axis_d<T, 5>(p, s); break;
        case 5: launch_adj_axis_d<T, 6>(p, s); break;
        default: launch_adj_axis_d<T, 0>(p, s); break;
    }
}

template <typename T, int D>
inline void launch_adj_axis0_t(const AxisPass &p, cudaStream_t s) {
    // QT columns x CT control points per CTA; few columns -> more control points
    const int QT = p.Q >= 32 ? 32 : (p.Q >= 16 ? 16 : (p.Q >= 8 ? 8 : (p.Q >= 4 ? 4 : (p.Q >= 2 ? 2 : 1))));
    const int CT = kAdj0Threads / QT;
    const int64_t gy = (p.Q + QT - 1) / QT;
    dim3 grid((unsigned)((p.n + CT - 1) / CT), gdim(gy, kMaxGridYZ));
    const size_t smem = (size_t)adj_axis0_smem_bytes<D, T>(QT);
    static bool attr_set = false;  // one instance per template instantiation
    if (!attr_set) {
        cudaFuncSetAttribute(k_adj_axis0<D, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)adj_axis0_smem_bytes<D, T>(32));
        attr_set = true;
    }
    launch(k_adj_axis0<D, T>, grid, kAdj0Threads, smem, s, p.idx, p.perm, p.lb, (const T *)p.B, p.ns, p.d,
           (const T *)p.X, p.n, p.Q, QT, (T *)p.Y);
}

// degrees <= 3: warp tasks of 32 columns x a chunk of control points (sg_warp.cuh); few
// columns get short chunks (at least 4 control points) so the tasks fill the GPU
template <typename T, int D>
inline void launch_adj0_warp(const AxisPass &p, cudaStream_t s) {
    const int64_t groups = (p.Q + 31) / 32;
    if (groups == 0 || p.n == 0) return;
    const int64_t want = (kAxis0Tasks + groups - 1) / groups;  // chunks wanted
    int64_t CC = (p.n + want - 1) / want;
    CC = CC < 4 ? 4 : CC;
    const int64_t tasks = groups * ((p.n + CC - 1) / CC);
    const int64_t blocks = (tasks + kWarpsPerBlock - 1) / kWarpsPerBlock;
    const int smem = kWarpsPerBlock * warp_adj0_smem<D, T>();
    static bool attr_set = false;  // one instance per template instantiation
    if (!attr_set) {
        cudaFuncSetAttribute(k_adj0_warp<D, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        attr_set = true;
    }
    launch(k_adj0_warp<D, T>, (unsigned)blocks, 32 * kWarpsPerBlock, smem, s, p.idx, p.perm, p.lb, (const T *)p.B,
           p.ns, p.d, (const T *)p.X, p.n, p.Q, CC, (T *)p.Y);
}

// The kernel of the adjoint pass over axis 0, degrees 0 to 5 (all give the same bits); the lines were
// drawn through the same measurements as adj_axis_kernel's.  A tile (32 columns x kA0Cp control
// points; kAdjLong) pays some 300 instructions a warp and a wait a segment, whatever it sums:
//  * Short sums (S < 18, Float64 9): one thread per output (4 samples, 1748157 columns, 2 control
//    points, degree 1: 29, tiles 149; 84462, 52, 14594: 16 and 22).  With very many outputs the
//    threads' loads are too scattered at degrees 2 and 3, and where a control point has hardly a
//    sample: warp tasks (12, 625777, 6, degree 3: 36 and 69; 13, 1477950, 16, degree 1: 122, 155).
//  * Fewer than 16 columns leave half of a tile's lanes idle: one thread per output, unless its sum
//    is long or there are few of them (Float64 182592, 3, 96247, degree 5: 16, tiles 65; 741545,
//    12, 16121, degree 3, S = 184: 188 and 62).
//  * Very many columns of few samples: warp tasks (20, 305766, 3, degree 2: 22, tiles 34).
//  * Unsorted samples: warp tasks, Float32 (67104, 300, 2615, degree 2: 157, tiles 454); the
//    CTA tiles of the runtime-degree path for degrees 4 and 5 (303904, 56, 56499, degree 4: 198, 450).
//  * The others: tiles (10168, 192, 137, degree 3: 18, threads 75).
template <typename T>
inline AdjKernel adj_axis0_kernel(const AxisPass &p) {
    constexpr bool f64 = sizeof(T) == 8;
    const double S = (double)p.ns * (p.d + 1) / (double)p.n;
    const int64_t O = p.n * p.Q;
    const bool warp = p.d <= 3;
    if (O > INT32_MAX || p.ns > INT32_MAX) return kAdjLong;  // k_adj_thread counts in 32 bits
    const int64_t V = p.ns * p.Q;
    if (p.perm && O >= 1 << 16 && V >= 1 << 19 && p.ns >= 12 && p.d >= 1) {
        if (warp && !f64) return kAdjWarp;
        if (!warp && V >= 1 << 22) return kAdjGeneric;
    }
    if constexpr (f64) {
        if (S < 9) return warp && p.Q >= 16 && O >= 150000 ? kAdjWarp : kAdjThread;
        if (p.Q < 16) return O >= 8192 && S < 4096 ? kAdjThread : kAdjLong;
        return warp && p.ns < 16 && O >= 80000 ? kAdjWarp : kAdjLong;
    } else {
        if (S < 18) {
            if (O < 12288 && S >= 8) return kAdjLong;
            const bool scattered = (p.d >= 2 && S >= 5) || 4 * p.ns < 5 * p.n;
            if (warp && scattered && O >= 1 << 20 && p.Q >= 32) return kAdjWarp;
            if (warp && p.d >= 2 && p.Q >= 1 << 16) return kAdjWarp;
            return kAdjThread;
        }
        if (warp && ((p.ns < 64 && p.Q >= 1 << 15) || (p.ns < 128 && p.Q >= 1 << 16))) return kAdjWarp;
        return p.Q < 16 && O >= 1 << 17 && S < 64 ? kAdjThread : kAdjLong;
    }
}

template <typename T, int D>
inline void launch_adj0(const AxisPass &p, cudaStream_t s) {
    const int64_t groups = (p.Q + 31) / 32, tiles = groups * ((p.n + kA0Cp - 1) / kA0Cp);
    if (tiles == 0) return;
    const AdjKernel k = adj_axis0_kernel<T>(p);
    if (k == kAdjThread) {
        launch_adj_thread<T, D>(p, s);
        return;
    }
    if constexpr (D <= 4) {
        if (k == kAdjWarp) {
            launch_adj0_warp<T, D>(p, s);
            return;
        }
    } else {
        if (k == kAdjGeneric) {
            launch_adj_axis0_t<T, 0>(p, s);
            return;
        }
    }
    if constexpr (sizeof(T) == 4) {
        if (!p.perm && p.ns % 4 == 0 && (uintptr_t)p.X % 16 == 0 && (uintptr_t)p.B % 16 == 0) {
            launch(k_adj0_tile<D, T, true>, (unsigned)tiles, 32 * kA0Warps, (a0_smem<D, T, true>()), s, p.perm, p.lb,
                   (const T *)p.B, p.ns, (const T *)p.X, p.n, p.Q, groups, (T *)p.Y);
            return;
        }
    }
    launch(k_adj0_tile<D, T, false>, (unsigned)tiles, 32 * kA0Warps, (a0_smem<D, T, false>()), s, p.perm, p.lb,
           (const T *)p.B, p.ns, (const T *)p.X, p.n, p.Q, groups, (T *)p.Y);
}

// Higher degrees (runtime-degree path) run as CTA tiles.
template <typename T>
inline void launch_adj_axis0(const AxisPass &p, cudaStream_t s) {
    switch (p.d) {
        case 0: launch_adj0<T, 1>(p, s); break;
        case 1: launch_adj0<T, 2>(p, s); break;
        case 2: launch_adj0<T, 3>(p, s); break;
        case 3: launch_adj0<T, 4>(p, s); break;
        case 4: launch_adj0<T, 5>(p, s); break;
        case 5: launch_adj0<T, 6>(p, s); break;
        default: launch_adj_axis0_t<T, 0>(p, s); break;
    }
}

// Nin = 1 with long supports: one cluster per (control point, column group)
template <typename T, int D, int QT>
inline int launch_adj_line_q(const AxisPass &p, cudaStream_t s) {
    const int64_t units = p.n * ((p.Q + QT - 1) / QT);
    int S = 1;  // more CTAs per control point while SMs are free and threads have several rounds
    while (S < 8 && units * S < kNumSMs * 4 && p.support > (int64_t)S * kLineThreads * 8) S *= 2;
    if (units * S > INT32_MAX) return set_error(SG_ERR_UNSUPPORTED, "adjoint: too many control points");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(units * S));
    cfg.blockDim = dim3(kLineThreads);
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)S;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch()
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cuda_check(cudaLaunchKernelEx(&cfg, k_adj_line<D, T, QT>, p.perm, p.lb, (const T *)p.B, p.ns,
                                         (const T *)p.X, p.n, p.Q, S, (T *)p.Y),
                      "adjoint launch");
}
template <typename T, int D>
inline int launch_adj_line_d(const AxisPass &p, cudaStream_t s) {
    return p.Q == 1 ? launch_adj_line_q<T, D, 1>(p, s) : p.Q == 2 ? launch_adj_line_q<T, D, 2>(p, s)
                                                                  : launch_adj_line_q<T, D, 4>(p, s);
}
template <typename T>
inline int launch_adj_line(const AxisPass &p, cudaStream_t s) {
    switch (p.d) {
        case 0: return launch_adj_line_d<T, 1>(p, s);
        case 1: return launch_adj_line_d<T, 2>(p, s);
        case 2: return launch_adj_line_d<T, 3>(p, s);
        case 3: return launch_adj_line_d<T, 4>(p, s);
        case 4: return launch_adj_line_d<T, 5>(p, s);
        default: return launch_adj_line_d<T, 6>(p, s);
    }
}

}  // namespace sg
