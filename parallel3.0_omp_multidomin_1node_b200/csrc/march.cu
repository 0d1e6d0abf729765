// Per-step kernels of the multi-domain TDBEM time march on B200.
//
//   rhs_kernel          history-convolution right-hand side for R load
//                       cases at once (one CTA per equation row): each 3x3
//                       history block is read from HBM once and applied to
//                       all R combined history vectors (block SpMM),
//                       DBEM1/multidomain.cpp:3843-3866; the head pass on
//                       the GMRES chain for two or more load cases and the
//                       one-step pass beside it
//   head_rows_kernel    the head pass of one load case over packed blocks
//   bulk_steps_kernel   the history steps k >= 2T + 1 of T time steps in
//                       one pass over the run layout (two or four load
//                       cases, or rows that share too little): each block
//                       read once for the T steps, each history vector of a
//                       run once, kept in registers
//   bulk_rows_kernel    the same for one load case over the step-major
//                       matrices
//   bulk_groups_kernel  the same for 8 or more load cases over groups of 8
//                       rows, on the FP64 tensor path
//   adj_history_kernel  the transposed history convolution of the adjoint
//                       march
//   gmres_cluster_kernel left-preconditioned GMRES(restart) for the R load
//                       cases in lockstep on one thread-block cluster
//                       (gmres.cuh): asynchronous remote stores completing
//                       on mbarriers, one SpMM of A' per Arnoldi step
//                       shared by all cases, DBEM1/pre_gmres.cpp:1369-1605;
//                       then the boundary write-back and history-state
//                       update, DBEM1/multidomain.cpp:3086-3225
//   rhs_models_kernel, gmres_models_kernel  the same for several models per
//                       launch
#include "march.cuh"

#include <algorithm>
#include <atomic>
#include <numeric>

#include "gmres.cuh"
#include "tdbem_common.cuh"

namespace tdbem {

namespace {

constexpr int kRhsThreads = 256;
constexpr int kHeadWarps = 4;          // warps per row of head_rows_kernel
constexpr int kMaxDevices = 64;        // launch attributes are kept per device

template <int R, int kCpt = (R >= 4 ? 4 : R)>
struct Lanes {
    static constexpr int CPT = kCpt;            // load cases per thread
    static constexpr int TPB = R / CPT;         // threads sharing one block
    static constexpr int BPW = 32 / TPB;        // blocks per warp iteration
};

// Device clock readings of the launches (MarchData::stamps)
__device__ __forceinline__ void stamp_start(const MarchData& d, int row, int which)
{
    if (d.stamps && blockIdx.x == 0 && threadIdx.x == 0) d.stamps[5 * (int64_t)row + which] = device_ns();
}
__device__ __forceinline__ void stamp_end(const MarchData& d, int row, int which)
{
    if (d.stamps && threadIdx.x == 0) atomicMax(d.stamps + 5 * (int64_t)row + which, device_ns());
}

// CPT consecutive values (16-byte aligned when CPT = 4 and R % 4 == 0)
template <int CPT>
__device__ __forceinline__ void load_cases(const float* p, float* v)
{
    if constexpr (CPT == 4) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else if constexpr (CPT == 2) {
        const float2 t = *reinterpret_cast<const float2*>(p);
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = *p;
    }
}

template <int CPT>
__device__ __forceinline__ void load_cases(const double* p, double* v)
{
    if constexpr (CPT == 4) {
        const double2 a = *reinterpret_cast<const double2*>(p);
        const double2 b = *reinterpret_cast<const double2*>(p + 2);
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    } else if constexpr (CPT == 2) {
        const double2 a = *reinterpret_cast<const double2*>(p);
        v[0] = a.x; v[1] = a.y;
    } else {
        v[0] = *p;
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// bd[0] conversion (BoundaryValue::Convert + AllLocToAbs,
// DBEM1/multidomain.cpp:3819-3821) and zeroed history rings.
__global__ void prepare_kernel(MarchData d)
{
    const int E = d.E;
    const long long n0 = (long long)d.R * E;
    const long long g0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, gs = gridDim.x * (long long)blockDim.x;
    for (long long t = g0; t < n0; t += gs) {
        const int r = (int)(t / E), i = (int)(t % E);
        const double* in = d.known_lu + ((long long)r * (d.nstep + 1) * E + i) * 3;
        double lu[3], lt[3];
        for (int c = 0; c < 3; ++c) {
            lu[c] = d.bcid[i] == 456 ? 0.0 : in[c];
            lt[c] = d.bcid[i] == 456 ? in[c] : 0.0;
        }
        const double* T = d.trans + 9 * i;
        double* ou = d.out_lu + ((long long)r * (d.nstep + 1) * E + i) * 3;
        double* ot = d.out_lt + ((long long)r * (d.nstep + 1) * E + i) * 3;
        for (int c = 0; c < 3; ++c) {
            ou[c] = T[c] * lu[0] + T[3 + c] * lu[1] + T[6 + c] * lu[2];
            ot[c] = T[c] * lt[0] + T[3 + c] * lt[1] + T[6 + c] * lt[2];
        }
    }
    const long long nx = 3LL * 2 * d.nh * 3 * d.R;
    for (long long t = g0; t < nx; t += gs) d.xring[t] = 0.0;
    const long long nw = (long long)d.SW * 2 * d.nh * 3 * d.R;
    for (long long t = g0; t < nw; t += gs) d.wring[t] = 0.0;
    for (long long t = g0; t < 8LL * 3 * d.E * d.R; t += gs) d.bulk[t] = 0.0;
    for (long long t = g0; t < 2LL * d.nstep; t += gs) d.audit[t] = 0.0;
    if (g0 < 4) d.status[g0] = 0;
}

// ---------------------------------------------------------------------------
// This warp's share of KnownM . known_step for equation row `row`
// (DBEM1/multidomain.cpp:3843-3846): known blocks j = first + w, first + w +
// NW, ... of the row; lane r < R takes load case r.  The warps' shares are
// summed with the history sums.
template <int R>
__device__ __forceinline__ void known_share(const MarchData& d, int row, int step, int w, int NW, int lane,
                                            double (&ka)[3])
{
    ka[0] = ka[1] = ka[2] = 0.0;
    if (lane >= R) return;
    const double* kv0 = d.known_lu + ((int64_t)lane * (d.nstep + 1) + step) * d.E * 3;
    const int je = d.k_rp[row + 1];
    for (int j = d.k_rp[row] + w; j < je; j += NW) {
        const double sg = d.k_sgn[j];
        const double* kv = kv0 + 3 * (int64_t)d.k_elem[j];
        const double x0 = sg * kv[0], x1 = sg * kv[1], x2 = sg * kv[2];
        const double* v = d.k_val + 9 * (int64_t)j;
        ka[0] += v[0] * x0 + v[1] * x1 + v[2] * x2;
        ka[1] += v[3] * x0 + v[4] * x1 + v[5] * x2;
        ka[2] += v[6] * x0 + v[7] * x1 + v[8] * x2;
    }
}

// ---------------------------------------------------------------------------
// Right-hand side of perm row p for steps k in [k_lo, k_hi]:
//   sum_k MGS_k . wT(s-k) - MTS_k . wU(s-k)     (MTS blocks stored negated)
// kBulk: write KnownM . known_s + sum to the bulk buffer of `step`.
// Otherwise write b = sum + the bulk buffer of `step` when add_bulk, else
// b = KnownM . known_s + sum.  Each block's 9 values are read once
// (streaming loads) and applied to the R load cases; a thread handles CPT
// cases.
template <int R, bool kMixed, bool kBulk, int kCpt>
__device__ __forceinline__ void rhs_row(const MarchData& d, const int p, const int step, const int add_bulk,
                                        const int k_lo, const int k_hi)
{
    // blocks in flight per lane group: measured best 6 (two CTAs per SM) for
    // 32 load cases, 4 (three CTAs per SM) for one
    constexpr int kUnroll = R >= 8 ? 6 : 4;
    using L = Lanes<R, kCpt>;
    constexpr int CPT = L::CPT, TPB = L::TPB, BPW = L::BPW;
    constexpr int NW = kRhsThreads / 32;
    // The head pass runs on the chain stream after the previous step's GMRES,
    // the only writer of the status word, so all its threads read one value.
    // The bulk pass runs beside a GMRES launch that may set the word at any
    // time: thread 0's reading is OR-ed across the CTA by the barrier itself,
    // so every thread takes the same branch.  (A form that broadcast the
    // reading through a shared variable made the 32-load mixed march 8%
    // slower, measured: the hot loop compiled differently.)
    if constexpr (!kBulk)
        if (*(volatile int*)d.status) return;
    extern __shared__ int slot_of_k[];
    __shared__ double red[NW][3][R];
    const int row = d.row_of[p];
    const int K = d.K, SW = d.SW;
    for (int k = threadIdx.x; k <= K; k += blockDim.x) slot_of_k[k] = (((step - k) % SW) + SW) % SW;
    if (__syncthreads_or(kBulk && threadIdx.x == 0 && *(volatile int*)d.status)) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int sub = lane / TPB, cgp = lane % TPB;
    double acc[3][CPT];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int q = 0; q < CPT; ++q) acc[c][q] = 0.0;
    if (k_hi >= k_lo) {
        const int64_t beg = d.h_kptr[(int64_t)row * (K + 1) + k_lo - 1];
        const int64_t end = d.h_kptr[(int64_t)row * (K + 1) + k_hi];
        const int64_t nnz = d.h_nnz;
        const int nh = d.nh;
#pragma unroll kUnroll
        for (int64_t i = beg + w * BPW + sub; i < end; i += NW * BPW) {
            const uint32_t cp = __ldcs(d.h_col + i);
            const int k = (int)(cp >> 21), type = (int)((cp >> 20) & 1u), col = (int)(cp & 0xFFFFFu);
            const int64_t wi = (((int64_t)slot_of_k[k] * 2 + type) * nh + col) * 3 * R + cgp * CPT;
            if constexpr (kMixed) {
                // FP32 block values (exact in FP64), FP64 history state and
                // products: rounding the state to FP32 instead costs ~10x the
                // displacement error of rounding the blocks
                const float* v = d.h_val32 + i;
                double m[9];
#pragma unroll
                for (int c = 0; c < 9; ++c) m[c] = (double)__ldcs(v + c * nnz);
                double w0[CPT], w1[CPT], w2[CPT];
                load_cases<CPT>(d.wring + wi, w0);
                load_cases<CPT>(d.wring + wi + R, w1);
                load_cases<CPT>(d.wring + wi + 2 * R, w2);
#pragma unroll
                for (int q = 0; q < CPT; ++q) {
                    acc[0][q] += m[0] * w0[q] + m[1] * w1[q] + m[2] * w2[q];
                    acc[1][q] += m[3] * w0[q] + m[4] * w1[q] + m[5] * w2[q];
                    acc[2][q] += m[6] * w0[q] + m[7] * w1[q] + m[8] * w2[q];
                }
            } else {
                const double* v = d.h_val + i;
                double m[9];
#pragma unroll
                for (int c = 0; c < 9; ++c) m[c] = __ldcs(v + c * nnz);
                double w0[CPT], w1[CPT], w2[CPT];
                load_cases<CPT>(d.wring + wi, w0);
                load_cases<CPT>(d.wring + wi + R, w1);
                load_cases<CPT>(d.wring + wi + 2 * R, w2);
#pragma unroll
                for (int q = 0; q < CPT; ++q) {
                    acc[0][q] += m[0] * w0[q] + m[1] * w1[q] + m[2] * w2[q];
                    acc[1][q] += m[3] * w0[q] + m[4] * w1[q] + m[5] * w2[q];
                    acc[2][q] += m[6] * w0[q] + m[7] * w1[q] + m[8] * w2[q];
                }
            }
        }
    }
    // sum the lanes that share a case group, then the warps
#pragma unroll
    for (int o = 16; o >= TPB && o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int q = 0; q < CPT; ++q) acc[c][q] += __shfl_xor_sync(0xffffffffu, acc[c][q], o);
    if (sub == 0)
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int q = 0; q < CPT; ++q) red[w][c][cgp * CPT + q] = acc[c][q];
    // the KnownM term goes with the pass that covers the step: the history
    // pass beside GMRES when there is one (the head then adds its buffer),
    // else the head
    if (kBulk || !add_bulk) {
        double ka[3];
        known_share<R>(d, row, step, w, NW, lane, ka);
        __syncwarp();
        if (lane < R)
#pragma unroll
            for (int c = 0; c < 3; ++c) red[w][c][lane] += ka[c];
    }
    __syncthreads();
    const int E = d.E;
    if (threadIdx.x < 3 * R) {
        const int c = threadIdx.x / R, r = threadIdx.x % R;
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < NW; ++q) s += red[q][c][r];
        const int64_t o = (int64_t)(3 * p + c) * R + r;
        double* bulk = d.bulk + (int64_t)(step & 7) * 3 * E * R;
        if constexpr (kBulk) {
            bulk[o] = s;
        } else {
            if (add_bulk) s += bulk[o];
            d.b[o] = s;
            if (d.rec_rhs && r == 0) d.rec_rhs[(int64_t)(step - 1) * 3 * E + 3 * row + c] = s;
        }
    }
}

template <int R, bool kMixed, bool kBulk, int kCpt>
__global__ void __launch_bounds__(kRhsThreads, R >= 8 ? 2 : 3) rhs_kernel(MarchData d, int step, int add_bulk)
{
    if constexpr (!kBulk) cudaTriggerProgrammaticLaunchCompletion();  // GMRES sets up beside it
    stamp_start(d, step, kBulk ? 3 : 0);
    rhs_row<R, kMixed, kBulk, kCpt>(d, blockIdx.x, step, add_bulk, d.k_lo, d.k_hi);
    if constexpr (kBulk) stamp_end(d, step, 4);
}

// The head pass of one load case over its packed blocks (MarchData hd_*): a row
// takes four warps.  What bounds it is latency: it runs on the
// chain, after a history pass that has swept the caches.  In the step-major
// matrices a row's few head blocks lie on ten pages (nine value planes and the
// columns) that no other row's head shares much of; packed, the part is 6% of the
// matrices in one piece.  Beside the half pass of bulk_rows_kernel, head of the
// 3,072-element bar: 47 us with rhs_kernel, 34 with warps over the step-major
// matrices, 27 packed (102 MB); of 1,728 elements: 24 -> 22 -> 18.  Four
// warps a row: with one, a step of the 120-element rod takes 69.7 us instead of
// 67.5 and of the 1,728-element bar 146 instead of 140; with eight, of 480 elements
// 69.6 instead of 67.1 and of the 3,072-element bar 205 instead of 200.  Loads that leave the blocks in L2
// make the head as fast and GMRES slower (168 -> 190), so they stream.
template <bool kMixed>
__global__ void __launch_bounds__(kRhsThreads, 3) head_rows_kernel(MarchData d, int step, int add_bulk)
{
    using V = typename std::conditional<kMixed, float, double>::type;
    constexpr int NW = kRhsThreads / 32, wpr = kHeadWarps, kUnroll = 4;
    constexpr size_t kTile = head_tile_bytes(kMixed);
    __shared__ double red[NW][3];
    cudaTriggerProgrammaticLaunchCompletion();  // GMRES sets up beside it
    if (*(volatile int*)d.status) return;       // set by GMRES before this launch only
    stamp_start(d, step, 0);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, part = w % wpr;
    const int p = blockIdx.x * (NW / wpr) + w / wpr;
    const bool on = p < d.E;
    double acc[3] = {0.0, 0.0, 0.0};
    if (on) {
        const int t0 = d.hd_ptr[p], t1 = d.hd_ptr[p + 1];
        const int64_t slot_len = 6LL * d.nh;
        const int SW = d.SW, s0 = step % SW, k_hi = d.k_hi;
#pragma unroll kUnroll
        for (int t = t0 + part; t < t1; t += wpr) {
            const unsigned char* tile = d.hd_tile + t * kTile;
            const uint32_t cp = __ldcs(reinterpret_cast<const unsigned*>(tile) + lane);
            const V* v = reinterpret_cast<const V*>(tile + 128) + lane;
            double m[9];
#pragma unroll
            for (int c = 0; c < 9; ++c) m[c] = (double)__ldcs(v + 32 * c);
            const int k = (int)(cp >> 21);
            int slot = s0 - k;
            if (slot < 0) slot += SW;
            const double* x = d.wring + slot * slot_len + ((int64_t)((cp >> 20) & 1u) * d.nh + (cp & 0xFFFFFu)) * 3;
            const bool in = k <= k_hi && cp;  // padding is 0
            const double x0 = in ? x[0] : 0.0, x1 = in ? x[1] : 0.0, x2 = in ? x[2] : 0.0;
#pragma unroll
            for (int c = 0; c < 3; ++c) acc[c] += m[3 * c] * x0 + m[3 * c + 1] * x1 + m[3 * c + 2] * x2;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    const int row = on ? d.row_of[p] : 0;
    if (lane == 0) {
        if (on && !add_bulk) {
            double ka[3];
            known_share<1>(d, row, step, part, wpr, lane, ka);
#pragma unroll
            for (int c = 0; c < 3; ++c) acc[c] += ka[c];
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) red[w][c] = acc[c];
    }
    __syncthreads();
    if (on && part == 0 && lane < 3) {
        double s = 0.0;
        for (int q = 0; q < wpr; ++q) s += red[w + q][lane];
        if (add_bulk) s += d.bulk[(int64_t)(step & 7) * 3 * d.E + 3 * p + lane];
        d.b[3 * p + lane] = s;
        if (d.rec_rhs) d.rec_rhs[(int64_t)(step - 1) * 3 * d.E + 3 * row + lane] = s;
    }
}

// Packs the blocks k <= head_k of each perm row into tiles of 32, zero-padded.
template <class V>
__global__ void pack_head_kernel(int E, int K, int head_k, const int32_t* row_of, const int64_t* kptr, const uint32_t* col,
                                 const V* val, int64_t nnz, const int32_t* ptr, unsigned char* tiles, int* infinite)
{
    const int p = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (p >= E) return;
    const int64_t b = kptr[(int64_t)row_of[p] * (K + 1)], e = kptr[(int64_t)row_of[p] * (K + 1) + head_k];
    for (int t = ptr[p]; t < ptr[p + 1]; ++t) {
        const int64_t i = b + (int64_t)(t - ptr[p]) * 32 + lane;
        unsigned char* tile = tiles + t * head_tile_bytes(sizeof(V) == 4);
        reinterpret_cast<uint32_t*>(tile)[lane] = i < e ? col[i] : 0u;
        V* v = reinterpret_cast<V*>(tile + 128) + lane;
        for (int c = 0; c < 9; ++c) {
            const V x = i < e ? val[c * nnz + i] : V(0);
            v[32 * c] = x;
            if (!isfinite(x)) *infinite = 1;
        }
    }
}

// ---------------------------------------------------------------------------
// History part k >= kr of the right-hand sides of the T steps t0 .. t0+T-1
// in one pass over the run layout (perm row blockIdx.x; the sums of
// DBEM1/multidomain.cpp:3843-3866 restricted to k >= kr, plus KnownM of each
// step).  Every block is read once for the T steps.  A lane group walks one
// run (one (type, column) pair, steps kf..kl) in increasing k keeping the
// window win[h] = W_{t0+h-k}, h < T, in registers: block k applies win[h] to
// step t0 + h, and moving to k + 1 shifts the window by one and loads only
// W_{t0-k-1}, so a run of n blocks loads n + T - 1 history vectors for T n
// products.  Needs the W slots up to t0 + T - 1 - kr, complete once the GMRES
// of step t0 + T - kr has run: kr = 2T + 1 leaves the T GMRES launches of
// steps t0 - T .. t0 - 1 to run beside.  Window entries of steps not yet
// reached (t0 + h - k < 0, only while t0 < K) are zero.
template <int R, bool kMixed, int kCpt, int T, int kUnroll = T>
__global__ void __launch_bounds__(kRhsThreads, 2) bulk_steps_kernel(MarchData d, int t0)
{
    using L = Lanes<R, kCpt>;
    constexpr int CPT = L::CPT, TPB = L::TPB, BPW = L::BPW;
    constexpr int NW = kRhsThreads / 32, NG = NW * BPW;
    __shared__ double red[NW][T][3][R];
    stamp_start(d, t0, 3);
    // runs beside GMRES launches that may set the status word: thread 0's
    // reading is OR-ed across the CTA by the barrier
    if (__syncthreads_or(threadIdx.x == 0 && *(volatile int*)d.status)) return;
    const int row = d.row_of[blockIdx.x];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int sub = lane / TPB, cgp = lane % TPB;
    const int K = d.K, SW = d.SW;
    const int klast = t0 + T - 1 < K ? t0 + T - 1 : K;  // last step of the last sum
    const int64_t nb = d.r_nb;
    const int64_t slot_len = 2LL * d.nh * 3 * R;
    double a[T][3][CPT];
#pragma unroll
    for (int h = 0; h < T; ++h)
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int q = 0; q < CPT; ++q) a[h][c][q] = 0.0;
    const int64_t rb = d.r_ptr[row], re = d.r_ptr[row + 1];
    for (int64_t r = rb + w * BPW + sub; r < re; r += NG) {
        const uint2 mt = __ldg(d.r_meta + r);
        const int kf = (int)(mt.y >> 16);
        const int kl = min(kf + (int)(mt.y & 0xFFFFu) - 1, klast);
        if (kl < kf) continue;
        const int64_t vb = __ldg(d.r_off + r) - kf;  // block of step k at vb + k
        const double* wc = d.wring + ((int64_t)(mt.x >> 20) * d.nh + (mt.x & 0xFFFFFu)) * 3 * R + cgp * CPT;
        double win[T][3][CPT];
        int slot = ((t0 - kf) % SW + SW) % SW;  // slot of W_{t0-k}, k = kf
#pragma unroll
        for (int h = 1; h < T; ++h) {
            if (t0 + h - kf >= 0) {
                const int sh = (slot + h) % SW;
#pragma unroll
                for (int c = 0; c < 3; ++c) load_cases<CPT>(wc + sh * slot_len + c * R, win[h][c]);
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int q = 0; q < CPT; ++q) win[h][c][q] = 0.0;
            }
        }
        // steps k <= t0: every window entry is a stored vector
        const int kb = kl < t0 ? kl : t0;
#pragma unroll kUnroll
        for (int k = kf; k <= kb; ++k) {
            double m[9];
            if constexpr (kMixed) {
#pragma unroll
                for (int c = 0; c < 9; ++c) m[c] = (double)__ldg(d.r_val32 + c * nb + vb + k);
            } else {
#pragma unroll
                for (int c = 0; c < 9; ++c) m[c] = __ldg(d.r_val + c * nb + vb + k);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) load_cases<CPT>(wc + slot * slot_len + c * R, win[0][c]);
            slot = slot == 0 ? SW - 1 : slot - 1;
#pragma unroll
            for (int h = 0; h < T; ++h)
#pragma unroll
                for (int q = 0; q < CPT; ++q)
#pragma unroll
                    for (int c = 0; c < 3; ++c)
                        a[h][c][q] += m[3 * c] * win[h][0][q] + m[3 * c + 1] * win[h][1][q] +
                                      m[3 * c + 2] * win[h][2][q];
#pragma unroll
            for (int h = T - 1; h > 0; --h)
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int q = 0; q < CPT; ++q) win[h][c][q] = win[h - 1][c][q];
        }
        // steps t0 < k <= t0 + T - 1 (only while t0 < K): W_{t0-k} does not
        // exist yet, the later steps' sums take the remaining entries
        for (int k = kb + 1 > kf ? kb + 1 : kf; k <= kl; ++k) {
            double m[9];
            if constexpr (kMixed) {
#pragma unroll
                for (int c = 0; c < 9; ++c) m[c] = (double)__ldg(d.r_val32 + c * nb + vb + k);
            } else {
#pragma unroll
                for (int c = 0; c < 9; ++c) m[c] = __ldg(d.r_val + c * nb + vb + k);
            }
#pragma unroll
            for (int h = 1; h < T; ++h)
#pragma unroll
                for (int q = 0; q < CPT; ++q)
#pragma unroll
                    for (int c = 0; c < 3; ++c)
                        a[h][c][q] += m[3 * c] * win[h][0][q] + m[3 * c + 1] * win[h][1][q] +
                                      m[3 * c + 2] * win[h][2][q];
#pragma unroll
            for (int h = T - 1; h > 1; --h)
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int q = 0; q < CPT; ++q) win[h][c][q] = win[h - 1][c][q];
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int q = 0; q < CPT; ++q) win[1][c][q] = 0.0;
        }
    }
    // sum the lanes that share a case group, then the warps
#pragma unroll
    for (int o = 16; o >= TPB && o > 0; o >>= 1)
#pragma unroll
        for (int h = 0; h < T; ++h)
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int q = 0; q < CPT; ++q) a[h][c][q] += __shfl_xor_sync(0xffffffffu, a[h][c][q], o);
    if (sub == 0)
#pragma unroll
        for (int h = 0; h < T; ++h)
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int q = 0; q < CPT; ++q) red[w][h][c][cgp * CPT + q] = a[h][c][q];
    // the KnownM terms of the T steps
    __syncwarp();
#pragma unroll 1
    for (int h = 0; h < T; ++h) {
        if (t0 + h > d.nstep) break;
        double ka[3];
        known_share<R>(d, row, t0 + h, w, NW, lane, ka);
        if (lane < R)
#pragma unroll
            for (int c = 0; c < 3; ++c) red[w][h][c][lane] += ka[c];
    }
    __syncthreads();
    const int64_t E3R = 3LL * d.E * R;
    for (int t = threadIdx.x; t < 3 * T * R; t += blockDim.x) {
        const int h = t / (3 * R), c = (t / R) % 3, r = t % R;
        if (t0 + h > d.nstep) continue;
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < NW; ++q) s += red[q][h][c][r];
        d.bulk[(int64_t)((t0 + h) & 7) * E3R + (int64_t)(3 * blockIdx.x + c) * R + r] = s;
    }
    stamp_end(d, t0, 4);
}

// The same part of the right-hand sides for one load case, over the step-major
// matrices of the one-step pass: each block is read once for the T steps (a run's
// blocks lie 8 bytes apart per lane in the run layout, too thin a read where a
// vector is one load case), with T vectors of 24 bytes from L2, in column order.
// What bounds it: HBM, 76 bytes a block (FP64).  On the 3,072-element bar, 1.68 GB
// of blocks, the one-step pass took 270 us a step, more than the GMRES it runs
// beside (223 us), and a step 339 us; with T = 2 a step takes 218 us (mixed
// precision: 201 -> 168).  T = 3 is slower (230), as the head then reads 14% of
// the blocks on the chain instead of 6%.  Of 128 to 1,024 threads with 1 to 8
// blocks in flight each, 256 with 4 (3 FP32) at two CTAs per SM was fastest: beside
// GMRES scheduled with the head, a step takes 169 us, 195 with 3. Each
// GMRES launch of the T has a T-th of the rows beside it (launched as one, a pass
// held up the next head and GMRES for an SM: 218 -> 206 us with the head above).
template <bool kMixed, int T>
__global__ void __launch_bounds__(kRhsThreads, 2) bulk_rows_kernel(MarchData d, int t0, int p0, int part)
{
    constexpr int NW = kRhsThreads / 32, kUnroll = T > 2 || kMixed ? 3 : 4;
    extern __shared__ int slot_of_k[];  // slot of W_{t0-k}
    __shared__ double red[NW][T][3];
    stamp_start(d, t0 + part, 3);
    const int p = p0 + blockIdx.x, row = d.row_of[p], K = d.K, SW = d.SW;
    for (int k = threadIdx.x; k <= K; k += blockDim.x) slot_of_k[k] = (((t0 - k) % SW) + SW) % SW;
    // runs beside GMRES launches that may set the status word: thread 0's
    // reading is OR-ed across the CTA by the barrier
    if (__syncthreads_or(threadIdx.x == 0 && *(volatile int*)d.status)) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t nnz = d.h_nnz, *kp = d.h_kptr + (int64_t)row * (K + 1);
    const int64_t slot_len = 6LL * d.nh;
    double a[T][3] = {};
    // apply(h0): blocks [beg, end) for the steps t0 + h, h >= h0
    auto apply = [&](auto first, int64_t beg, int64_t end) {
        constexpr int h0 = decltype(first)::value;
#pragma unroll kUnroll
        for (int64_t i = beg + threadIdx.x; i < end; i += kRhsThreads) {
            const uint32_t cp = __ldcs(d.h_col + i);
            int slot = slot_of_k[cp >> 21];
            const double* wc = d.wring + ((int64_t)((cp >> 20) & 1u) * d.nh + (cp & 0xFFFFFu)) * 3;
            double m[9];
#pragma unroll
            for (int c = 0; c < 9; ++c) {
                if constexpr (kMixed) m[c] = (double)__ldcs(d.h_val32 + c * nnz + i);
                else m[c] = __ldcs(d.h_val + c * nnz + i);
            }
#pragma unroll
            for (int h = 0; h < T; ++h) {
                if (h >= h0) {
                    const double* x = wc + slot * slot_len;
                    const double x0 = x[0], x1 = x[1], x2 = x[2];
#pragma unroll
                    for (int c = 0; c < 3; ++c) a[h][c] += m[3 * c] * x0 + m[3 * c + 1] * x1 + m[3 * c + 2] * x2;
                }
                slot = slot + 1 == SW ? 0 : slot + 1;
            }
        }
    };
    const int kb = t0 < K ? t0 : K;  // up to here every step has a stored vector
    if (kb >= d.kr) apply(std::integral_constant<int, 0>{}, kp[d.kr - 1], kp[kb]);
    // W_{t0+h-k} of t0 < k exists for the later steps only (while t0 < K)
    if (t0 < K && t0 + 1 >= d.kr) apply(std::integral_constant<int, 1>{}, kp[t0], kp[t0 + 1]);
    if constexpr (T > 2)
        if (t0 + 1 < K && t0 + 2 >= d.kr) apply(std::integral_constant<int, 2>{}, kp[t0 + 1], kp[t0 + 2]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int h = 0; h < T; ++h)
#pragma unroll
            for (int c = 0; c < 3; ++c) a[h][c] += __shfl_xor_sync(0xffffffffu, a[h][c], o);
#pragma unroll 1
    for (int h = 0; h < T; ++h) {
        double ka[3] = {0.0, 0.0, 0.0};
        if (t0 + h <= d.nstep) known_share<1>(d, row, t0 + h, w, NW, lane, ka);
        if (lane == 0)
#pragma unroll
            for (int c = 0; c < 3; ++c) red[w][h][c] = ka[c];
    }
    if (lane == 0)
#pragma unroll
        for (int h = 0; h < T; ++h)
#pragma unroll
            for (int c = 0; c < 3; ++c) red[w][h][c] += a[h][c];
    __syncthreads();
    if (threadIdx.x < 3 * T) {
        const int h = threadIdx.x / 3, c = threadIdx.x % 3;
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < NW; ++q) s += red[q][h][c];
        if (t0 + h <= d.nstep) d.bulk[(int64_t)((t0 + h) & 7) * 3 * d.E + 3 * p + c] = s;
    }
    stamp_end(d, t0 + part, 4);
}

// ---------------------------------------------------------------------------
// The same part of the right-hand sides over the group layout (8 or more load
// cases): a cluster of CTAs takes a group of 8 rows.  What bounds it: FP64
// multiply-adds (1.0 ms a launch at full rate on the 3,072-element bar with 32
// load cases).  bulk_steps_kernel spends 2.1 ms there: it reads a history
// vector of 768 bytes from L2 per block and two steps, 17.6 GB, and converts
// every FP32 block value in each lane that uses it, at a quarter of the
// multiply-add rate.  Here a segment is a product of matrices on the FP64
// tensor path (m8n8k4, as fast as scalar FP64 and one operand load per eight
// products): 24 equation components by 3 x steps, times 3 x steps by load
// cases, once per time step with the vectors shifted by a step.  A warp walks
// segments; the fragments and vectors come to its ring of stages by cp.async,
// kChunk steps each, and a vector read serves 8 rows and T steps, a value 8 T
// products.  The CTAs of a cluster split the segments (a CTA of some 0.2 ms
// does not hold up the GMRES clusters that wait for its SM) and sum in rank
// order.
__device__ __forceinline__ void copy16(uint32_t dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(__cvta_generic_to_global(src)) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// c += a b, 8 x 4 by 4 x 8: lane l holds a[l / 4][l % 4], b[l % 4][l / 4] and
// c[l / 4][2 (l % 4)], c[l / 4][2 (l % 4) + 1]
__device__ __forceinline__ void mma_f64(double& c0, double& c1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c0), "+d"(c1) : "d"(a), "d"(b));
}

template <int R, int T, class V>
struct GroupPass {
    // 8 cases make little of a step: longer chunks for them
    static constexpr int NW = 4, kThreads = 32 * NW, kChunk = R == 8 ? 8 : 4, kStages = 3, NT = R / 8;
    static constexpr int kSteps = kChunk / 4 * 3;                                 // contraction steps of a chunk
    static constexpr int kRowLen = R + 4;                                         // padded: no bank conflicts between fragment rows
    static constexpr int kVecs = (kChunk + T - 1) * 3 * kRowLen;                  // doubles of a stage's vectors
    static constexpr int kStage = kVecs * 8 + kSteps * 3 * 32 * (int)sizeof(V);  // bytes
    static constexpr int kSums = T * 24 * R;                            // doubles of a CTA's sums
    static constexpr size_t kRing = (size_t)NW * kStages * kStage, kRed = sizeof(double) * (size_t)(NW + 1) * kSums;
    static constexpr size_t kBytes = kRing > kRed ? kRing : kRed;
};

// One row's sum of one step by a warp, from the step-major matrices: only the
// products of stored blocks.  For histories with vectors that are not finite, which
// the group layout's zeros must not meet.
template <int R, class V>
__device__ __noinline__ void group_row_plain(const MarchData& d, int p, int step, int lane)
{
    constexpr int kLists = 32 / R;
    const int row = d.row_of[p], r = lane % R, K = d.K, SW = d.SW;
    const int64_t* kp = d.h_kptr + (int64_t)row * (K + 1);
    const int64_t slot_len = 2LL * d.nh * 3 * R, nnz = d.h_nnz;
    double acc[3];
    known_share<R>(d, row, step, 0, 1, lane, acc);
    const int64_t end = kp[step < K ? step : K];
#pragma unroll 1
    for (int64_t i = kp[d.kr - 1] + lane / R; i < end; i += kLists) {
        const uint32_t cp = d.h_col[i];
        const double* x = d.wring + ((step - (int)(cp >> 21)) % SW) * slot_len +
                          ((int64_t)((cp >> 20) & 1u) * d.nh + (cp & 0xFFFFFu)) * 3 * R + r;
        const V* v;
        if constexpr (sizeof(V) == 4) v = d.h_val32 + i;
        else v = d.h_val + i;
        const double x0 = x[0], x1 = x[R], x2 = x[2 * R];
#pragma unroll
        for (int c = 0; c < 3; ++c)
            acc[c] += (double)v[3 * c * nnz] * x0 + (double)v[(3 * c + 1) * nnz] * x1 + (double)v[(3 * c + 2) * nnz] * x2;
    }
#pragma unroll
    for (int o = 16; o >= R; o >>= 1)
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    if (lane < R)
#pragma unroll
        for (int c = 0; c < 3; ++c)
            d.bulk[(int64_t)(step & 7) * 3 * d.E * R + (int64_t)(3 * p + c) * R + lane] = acc[c];
}

template <int R, int T, class V>
__global__ void __launch_bounds__(GroupPass<R, T, V>::kThreads) bulk_groups_kernel(const __grid_constant__ MarchData d,
                                                                                   int t0, int split)
{
    using P = GroupPass<R, T, V>;
    constexpr int NT = P::NT, NW = P::NW;
    const int group = (int)blockIdx.x / split, rank = (int)blockIdx.x % split;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    stamp_start(d, t0, 3);
    // runs beside GMRES launches that may set the status words: the cluster
    // takes rank 0's reading.  A word that is set meanwhile for vectors that are
    // not finite is set for later ones than this pass reads.
    __shared__ int stop, stop_all;
    if (threadIdx.x == 0) stop = ((volatile int*)d.status)[0] ? 1 : ((volatile int*)d.status)[1] ? 2 : 0;
    unsigned char* const ring = reinterpret_cast<unsigned char*>(dsm) + w * P::kStages * P::kStage;
    for (int i = lane; i < P::kStages * P::kStage / 8; i += 32) reinterpret_cast<double*>(ring)[i] = 0.0;
    __syncthreads();
    if (split > 1) {
        cluster_barrier();
        if (threadIdx.x == 0) stop_all = *cg::this_cluster().map_shared_rank(&stop, 0);
        cluster_barrier();
    } else {
        if (threadIdx.x == 0) stop_all = stop;
        __syncthreads();
    }
    if (stop_all) {
        if (stop_all == 2)
            for (int i = rank * NW + w; i < 8 * T; i += NW * split) {
                const int p = __ldg(d.hg_rows + (int64_t)group * 8 + i % 8), step = t0 + i / 8;
                if (p >= 0 && step <= d.nstep) group_row_plain<R, V>(d, p, step, lane);
            }
        return;
    }
    const int SW = d.SW, klast = t0 + T - 1 < d.K ? t0 + T - 1 : d.K;  // last step of the last sum
    const int64_t slot_len = 2LL * d.nh * 3 * R;
    const int64_t seg_end = __ldg(d.hg_ptr + group + 1);
    const int seg_step = NW * split;
    // a position in the warp's sequence of chunks: its segments of the group
    // (longest first; the warps take them in turn, every other round in reverse,
    // so their totals are alike), kChunk steps at a time
    struct Pos {
        int64_t seg;
        int skip;            // to the warp's next segment
        const V* val;        // first fragment of the segment
        const double* vec;   // its (type, column) in slot 0 of the ring of vectors
        int k0, len, j;      // first step, steps within the last sum, next step
    };
    const int mine = rank * NW + w;
    auto next_seg = [&](Pos& p) {
        p.seg += p.skip;
        p.skip = 2 * seg_step - p.skip;
    };
    auto load_seg = [&](Pos& p) {
        // segments that start past the last sum's steps are skipped
        for (; p.seg < seg_end; next_seg(p)) {
            const uint2 mt = __ldg(d.hg_meta + p.seg);
            p.k0 = (int)(mt.y >> 16);
            p.len = min((int)(mt.y & 0xFFFFu), klast - p.k0 + 1);
            p.val = static_cast<const V*>(d.hg_val) + __ldg(d.hg_off + p.seg) * 96;
            p.vec = d.wring + ((int64_t)(mt.x >> 20) * d.nh + (mt.x & 0xFFFFFu)) * 3 * R;
            p.j = 0;
            if (p.len > 0) return;
        }
    };
    auto advance = [&](Pos& p) {
        p.j += P::kChunk;
        if (p.j >= p.len) {
            next_seg(p);
            load_seg(p);
        }
    };
    // One chunk into a stage: the vectors W_{t0+T-1-k0-j} and on, backwards in
    // time, one more than its steps need (its last fragment may reach into the
    // next step), then the fragments of its ceil(3 n / 4) contraction steps.
    // Vectors of steps not yet reached (only while t0 < K) are slots that are
    // still zero.
    auto issue = [&](const Pos& p, int stage) {
        const int n = min(P::kChunk, p.len - p.j), vecs = min(n + T, P::kChunk + T - 1), ks = (3 * n + 3) / 4;
        const uint32_t vdst = shared_addr(ring + stage * P::kStage), fdst = vdst + P::kVecs * 8;
        constexpr int kPieces = 3 * R / 2, kPer = 16 / sizeof(V);  // 16-byte pieces of a vector, values of a piece
        const int slot0 = ((t0 + T - 1 - p.k0 - p.j) % SW + SW) % SW;
        auto vector_piece = [&](int q, int slot, int i) {
            copy16(vdst + 8 * ((3 * q + i / (R / 2)) * P::kRowLen + 2 * (i % (R / 2))), p.vec + slot * slot_len + 2 * i);
        };
        if constexpr (kPieces < 16) {
            // a warp's copy takes pieces of several vectors
#pragma unroll 2
            for (int i = lane; i < vecs * kPieces; i += 32) {
                const int q = i / kPieces;
                vector_piece(q, slot0 >= q ? slot0 - q : slot0 - q + SW, i % kPieces);
            }
        } else {
            int slot = slot0;
#pragma unroll 1
            for (int q = 0; q < vecs; ++q) {
#pragma unroll
                for (int i0 = 0; i0 < kPieces; i0 += 32)
                    if (i0 + lane < kPieces) vector_piece(q, slot, i0 + lane);
                slot = slot == 0 ? SW - 1 : slot - 1;
            }
        }
        const V* f = p.val + (p.j / 4) * 288;
#pragma unroll 2
        for (int i = lane; i < ks * 96 / kPer; i += 32) copy16(fdst + 16 * i, f + kPer * i);
    };
    double acc[3][NT][T][2];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int q = 0; q < NT; ++q)
#pragma unroll
            for (int h = 0; h < T; ++h) acc[i][q][h][0] = acc[i][q][h][1] = 0.0;
    Pos cur{}, ahead{};
    cur.seg = __ldg(d.hg_ptr + group) + mine;
    cur.skip = 2 * (seg_step - mine) - 1;
    load_seg(cur);
    ahead = cur;
    for (int i = 0; i < P::kStages - 1; ++i) {
        if (ahead.seg < seg_end) {
            issue(ahead, i);
            advance(ahead);
        }
        copy_commit();
    }
    int stage = 0, fill = P::kStages - 1;
#pragma unroll 1
    while (cur.seg < seg_end) {
        copy_wait<P::kStages - 2>();
        __syncwarp();  // the stage's copies of all lanes; and the stage to fill is free
        if (ahead.seg < seg_end) {
            issue(ahead, fill);
            advance(ahead);
        }
        copy_commit();
        fill = fill + 1 == P::kStages ? 0 : fill + 1;
        const double* vs = reinterpret_cast<const double*>(ring + stage * P::kStage) + (lane & 3) * P::kRowLen + (lane >> 2);
        const V* fs = reinterpret_cast<const V*>(ring + stage * P::kStage + P::kVecs * 8) + lane;
        const int n = min(P::kChunk, cur.len - cur.j), ks = (3 * n + 3) / 4;
#pragma unroll
        for (int s = 0; s < P::kSteps; ++s) {
            if (s >= ks) break;
            double a[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) a[i] = (double)fs[(3 * s + i) * 32];
#pragma unroll
            for (int h = 0; h < T; ++h)
#pragma unroll
                for (int q = 0; q < NT; ++q) {
                    const double b = vs[(4 * s + 3 * (T - 1 - h)) * P::kRowLen + 8 * q];
#pragma unroll
                    for (int i = 0; i < 3; ++i) mma_f64(acc[i][q][h][0], acc[i][q][h][1], a[i], b);
                }
        }
        advance(cur);
        stage = stage + 1 == P::kStages ? 0 : stage + 1;
    }
    copy_wait<0>();
    __syncthreads();
    // the warps' sums; then, summed over them, with this CTA's share of the
    // KnownM terms of the T steps: [h][row component][case]
    double* const red = dsm;
    double* const sums = dsm + NW * P::kSums;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int q = 0; q < NT; ++q)
#pragma unroll
            for (int h = 0; h < T; ++h)
                *reinterpret_cast<double2*>(red + w * P::kSums + (h * 24 + 8 * i + (lane >> 2)) * R + 8 * q + 2 * (lane & 3)) =
                    make_double2(acc[i][q][h][0], acc[i][q][h][1]);
    __syncthreads();
    for (int t = threadIdx.x; t < P::kSums; t += P::kThreads) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < NW; ++q) s += red[q * P::kSums + t];
        sums[t] = s;
    }
    __syncthreads();
    const int32_t* rows = d.hg_rows + (int64_t)group * 8;
#pragma unroll 1
    for (int i = mine; i < 8 * T; i += seg_step) {
        const int p = __ldg(rows + i % 8), h = i / 8;
        if (p < 0 || t0 + h > d.nstep) continue;
        double ka[3];
        known_share<R>(d, d.row_of[p], t0 + h, 0, 1, lane, ka);
        if (lane < R)
#pragma unroll
            for (int c = 0; c < 3; ++c) sums[(h * 24 + 3 * (i % 8) + c) * R + lane] += ka[c];
    }
    if (split > 1) cluster_barrier();
    else __syncthreads();
    const int64_t E3R = 3LL * d.E * R;
    // each CTA adds up and writes its share of the group's sums
    for (int t = rank * P::kThreads + threadIdx.x; t < P::kSums; t += split * P::kThreads) {
        const int h = t / (24 * R), m = t / R % 24, r = t % R, p = __ldg(rows + m / 3);
        if (p < 0 || t0 + h > d.nstep) continue;
        double s = 0.0;
        for (int q = 0; q < split; ++q) {
            double v;
            peer_load1(peer_addr(shared_addr(sums + t), (uint32_t)q), v);
            s += v;
        }
        d.bulk[(int64_t)((t0 + h) & 7) * E3R + (int64_t)(3 * p + m % 3) * R + r] = s;
    }
    if (split > 1) cluster_barrier();  // peers still read this CTA's sums
    stamp_end(d, t0, 4);
}

// Copy one model's MarchData into shared memory (several models per launch).
__device__ __forceinline__ void load_model(const MarchData* ds, int m, MarchData& sd)
{
    const int* src = reinterpret_cast<const int*>(ds + m);
    int* dst = reinterpret_cast<int*>(&sd);
    for (int i = threadIdx.x; i < (int)(sizeof(MarchData) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
    __syncthreads();
}

// Several models' right-hand sides of one step in one launch: CTA b serves
// perm row b - row_off[m] of model m (row_off[m] <= b < row_off[m+1]); models
// whose march is shorter skip.  With kBulk the history steps 3..min(step, K_m)
// and KnownM go to the model's bulk buffer (computed one step ahead, beside
// GMRES); otherwise the head: k <= min(step, K_m, kmax_head) plus that bulk
// when k = 3.. applies (kmax_head = 2; KnownM itself before that), or KnownM
// and every history step (kmax_head = K_m).
template <int R, bool kMixed, bool kBulk, int kCpt>
__global__ void __launch_bounds__(kRhsThreads, R >= 8 ? 2 : 3) rhs_models_kernel(const MarchData* ds, const int* row_off,
                                                                                  int n_models, int step, int split)
{
    int lo = 0, hi = n_models - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((int)blockIdx.x >= row_off[mid]) lo = mid;
        else hi = mid - 1;
    }
    __shared__ MarchData sd;
    load_model(ds, lo, sd);
    if (step > sd.nstep) return;
    const int kcap = step > 1 ? (step < sd.K ? step : sd.K) : 0;
    const int p = (int)blockIdx.x - row_off[lo];
    if constexpr (kBulk) {
        if (kcap >= 3) rhs_row<R, kMixed, true, kCpt>(sd, p, step, 0, 3, kcap);
    } else if (split) {
        rhs_row<R, kMixed, false, kCpt>(sd, p, step, kcap >= 3 ? 1 : 0, 1, kcap < 2 ? kcap : 2);
    } else {
        rhs_row<R, kMixed, false, kCpt>(sd, p, step, 0, 1, kcap);
    }
}

// ---------------------------------------------------------------------------
// Transposed history convolution of the adjoint march at step n:
//   adj[type][c] = sum_k sum_r B(r, k, type, c)^T Omega_{n,k}[r]
//   Omega_{n,k} = lam_{n+k-1} (k >= 2) + 2 lam_{n+k} + lam_{n+k+1}, steps <= N,
// the transpose of the forward sum over k of B . (X_{s-k+1} + 2 X_{s-k} +
// X_{s-k-1}) (DBEM1/multidomain.cpp:3201-3225, 3843-3866) with B the stacked
// blocks (MTS negated).  Omega_{n,k} is row n + k of com, which adjoint_finish
// keeps so.  What bounds it: latency, then L2 bandwidth (76 bytes and one vector a
// block).  Four warps take a (type, column) pair's blocks of all k as one list; a
// warp that went through k by k, with three vectors a block, took 97 us a step of
// 480 elements (509,000 blocks) with cold caches, 15 now.
__global__ void __launch_bounds__(256, 3) adj_history_kernel(int N, int n, int K, int nh, int E, const int64_t* tptr,
                                                             const uint32_t* trow, const double* tval, const double* com,
                                                             double* adj)
{
    constexpr int kWarps = 4;  // per pair
    __shared__ double red[8][3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, part = w % kWarps;
    const int64_t seg = (int64_t)blockIdx.x * (8 / kWarps) + w / kWarps;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    if (seg < 2LL * nh) {
        const int kmax = K < N + 1 - n ? K : N + 1 - n;  // later rows of com are zero
        const int64_t b = tptr[seg * (K + 1)], e = tptr[seg * (K + 1) + kmax];
        const double* w0 = com + 3LL * n * E;
#pragma unroll 4
        for (int64_t j = b + part * 32 + lane; j < e; j += 32 * kWarps) {
            const uint32_t kr = __ldg(trow + j);  // k << 21 | row
            const double* x = w0 + 3 * ((int64_t)(kr >> 21) * E + (kr & 0x1FFFFFu));
            const double* B = tval + (j >> 5) * 288 + (j & 31);  // row-major B in planes; B^T x
            const double x0 = x[0], x1 = x[1], x2 = x[2];
            a0 += __ldg(B) * x0 + __ldg(B + 96) * x1 + __ldg(B + 192) * x2;
            a1 += __ldg(B + 32) * x0 + __ldg(B + 128) * x1 + __ldg(B + 224) * x2;
            a2 += __ldg(B + 64) * x0 + __ldg(B + 160) * x1 + __ldg(B + 256) * x2;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a0 += __shfl_xor_sync(0xffffffffu, a0, o);
        a1 += __shfl_xor_sync(0xffffffffu, a1, o);
        a2 += __shfl_xor_sync(0xffffffffu, a2, o);
    }
    if (lane == 0) {
        red[w][0] = a0;
        red[w][1] = a1;
        red[w][2] = a2;
    }
    __syncthreads();
    if (part == 0 && lane < 3 && seg < 2LL * nh) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < kWarps; ++q) s += red[w + q][lane];
        adj[3 * seg + lane] = s;
    }
}

cudaError_t adj_history(int N, int n, int K, int nh, int E, const int64_t* tptr, const uint32_t* trow,
                        const double* tval, const double* com, double* adj, cudaStream_t s)
{
    const int64_t segs = 2LL * nh;
    adj_history_kernel<<<(int)((segs + 1) / 2), 256, 0, s>>>(N, n, K, nh, E, tptr, trow, tval, com, adj);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
template <int R, bool kMixed, bool kLocal>
__global__ void __launch_bounds__(kGmresThreads, 1) gmres_cluster_kernel(const __grid_constant__ MarchData d, int step)
{
    gmres_body<R, kMixed, kLocal>(d, step, (int)(blockIdx.x / cg::this_cluster().num_blocks()));
    stamp_end(d, step, 2);
}

// Several models' GMRES of one step in one launch per form: cluster m solves
// model m (one group of R load cases each; every model laid out for the launch's
// cluster size); models of the other form and models whose march is shorter skip.
template <int R, bool kMixed, bool kLocal>
__global__ void __launch_bounds__(kGmresThreads, 1) gmres_models_kernel(const MarchData* ds, int step)
{
    __shared__ MarchData sd;
    load_model(ds, (int)(blockIdx.x / cg::this_cluster().num_blocks()), sd);
    if (step > sd.nstep || (sd.dsm_rows > 0) != kLocal) return;
    gmres_body<R, kMixed, kLocal>(sd, step, 0);
}

// ---------------------------------------------------------------------------
namespace {

// Dynamic shared memory of the GMRES kernel at most (of the 227 KB a CTA may
// have; the several-models form keeps its model there too).
constexpr size_t kGmresDsmMax = 224 * 1024;
// Basis vectors kept in shared memory at most: solves take 6 to 18 steps, and
// what shared memory leaves is L1.
constexpr int kVcapMax = 20, kVcapMin = 10;

// Threads of a GMRES CTA owning `rows` rows: a small range does not run its
// barriers over idle warps, but a warp per dot product pays.
int gmres_threads(int rows, int Rg)
{
    const int n = 3 * rows * Rg;
    return n <= 192 ? 256 : kGmresThreads;
}

// Caches leaf inverses and basis vectors in `room` bytes of shared memory and
// returns the bytes taken.  A step reads the inverses behind its product, whose
// stream of A' evicts them from L1 (one load case on the 3,072-element bar:
// 5,600 cycles per application against 2,200 cached); for one or two cases,
// whose vectors are short, only when kVcapMin vectors fit beside them.
size_t gmres_caches(MarchData& d, size_t room, int Rg, bool mixed)
{
    const size_t vec = sizeof(double) * 3 * (size_t)d.dsm_rows * Rg;
    const size_t leaf = 16 * (size_t)d.dsm_rows +
                        ((size_t)d.leaf_max * (mixed ? sizeof(float) : sizeof(double)) + 15) / 16 * 16;
    const size_t want = (size_t)std::min(d.restart + 1, kVcapMax);
    const size_t least = std::min<size_t>(want, Rg <= 2 ? kVcapMin : 0);
    size_t used = 0;
    d.leaf_cap = 0;
    if (leaf + least * vec <= room) {
        d.leaf_cap = d.leaf_max;
        used = leaf;
    }
    d.vcap = (int)std::min<size_t>((room - used) / vec, want);
    return used + vec * (size_t)d.vcap;
}

// Raises a kernel's dynamic shared memory to the most the device allows and,
// `clusters`, lets it run in clusters of 16, once per device: changing attributes between
// launches (models of different sizes marched side by side) would be a
// host-side attribute change per launch.  Returns that size in cap.
template <class K>
cudaError_t kernel_attributes(K kernel, std::atomic<int> (&dyn_max)[kMaxDevices], int& cap, bool clusters = true)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    cap = dyn_max[dev].load();
    if (cap != 0) return cudaSuccess;
    cudaFuncAttributes fa{};
    int optin = 0;
    if ((e = cudaFuncGetAttributes(&fa, kernel)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
    cap = optin - (int)fa.sharedSizeBytes;
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, cap)) != cudaSuccess) return e;
    if (clusters &&
        (e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess)
        return e;
    dyn_max[dev].store(cap);
    return cudaSuccess;
}

template <int R, bool kMixed, bool kLocal>
cudaError_t launch_gmres_form(const MarchData& d0, int step, cudaStream_t s)
{
    MarchData d = d0;
    static std::atomic<int> dyn_max[kMaxDevices];
    int cap = 0;
    cudaError_t e = kernel_attributes(gmres_cluster_kernel<R, kMixed, kLocal>, dyn_max, cap);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(d.cluster * d.groups);
    cfg.blockDim = dim3(gmres_threads(d.own_rows, R));
    cfg.dynamicSmemBytes = gmres_dsm_bytes(d.dsm_rows, d.halo_rows, R, kMixed);
    cfg.stream = s;
    if (cfg.dynamicSmemBytes > (size_t)cap) return cudaErrorInvalidValue;
    // the rest of the shared memory goes to leaf inverses and basis vectors
    if (kLocal) cfg.dynamicSmemBytes += gmres_caches(d, (size_t)cap - cfg.dynamicSmemBytes, R, kMixed);
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = d.cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = d.after_head ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, gmres_cluster_kernel<R, kMixed, kLocal>, d, step);
}

template <int R, bool kMixed>
cudaError_t launch_gmres(const MarchData& d, int step, cudaStream_t s)
{
    return d.dsm_rows > 0 ? launch_gmres_form<R, kMixed, true>(d, step, s)
                          : launch_gmres_form<R, kMixed, false>(d, step, s);
}

template <int R, bool kMixed>
int cluster_size_for(int device)
{
    (void)device;
    for (int c : {16, 8, 4, 2, 1}) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(c);
        cfg.blockDim = dim3(kGmresThreads);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = c;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (c > 8 && cudaFuncSetAttribute(gmres_cluster_kernel<R, kMixed, true>,
                                          cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, gmres_cluster_kernel<R, kMixed, true>, &cfg) == cudaSuccess && n >= 1)
            return c;
        cudaGetLastError();
    }
    return 1;
}

template <int R, bool kMixed, int kCpt>
cudaError_t launch_rhs_cpt(const MarchData& d, int step, bool bulk, int add_bulk, cudaStream_t s)
{
    const size_t smem = sizeof(int) * (size_t)(d.K + 1);
    if (bulk)
        rhs_kernel<R, kMixed, true, kCpt><<<d.E, kRhsThreads, smem, s>>>(d, step, 0);
    else
        rhs_kernel<R, kMixed, false, kCpt><<<d.E, kRhsThreads, smem, s>>>(d, step, add_bulk);
    return cudaGetLastError();
}

// d.rhs_cpt selects the load cases per thread (the R-tile; with it the blocks
// a warp takes per iteration, 32 / (R / cpt)): 4 or 2 for R >= 4, 2 or 1 for
// R = 2; 0 is the default, min(R, 4)
template <int R, bool kMixed>
cudaError_t launch_rhs(const MarchData& d, int step, bool bulk, int add_bulk, cudaStream_t s)
{
    if constexpr (R >= 4) {
        if (d.rhs_cpt == 2) return launch_rhs_cpt<R, kMixed, 2>(d, step, bulk, add_bulk, s);
        return launch_rhs_cpt<R, kMixed, 4>(d, step, bulk, add_bulk, s);
    } else if constexpr (R == 2) {
        if (d.rhs_cpt == 1) return launch_rhs_cpt<R, kMixed, 1>(d, step, bulk, add_bulk, s);
        return launch_rhs_cpt<R, kMixed, 2>(d, step, bulk, add_bulk, s);
    } else {
        if (bulk || !d.hd_ptr) return launch_rhs_cpt<R, kMixed, 1>(d, step, bulk, add_bulk, s);
        constexpr int rows = kRhsThreads / 32 / kHeadWarps;
        head_rows_kernel<kMixed><<<(d.E + rows - 1) / rows, kRhsThreads, 0, s>>>(d, step, add_bulk);
        return cudaGetLastError();
    }
}

// Group form of the T-step history pass: a cluster of hg_split CTAs per group.
template <int R, int T, class V>
cudaError_t launch_bulk_groups(const MarchData& d, int t0, cudaStream_t s)
{
    using P = GroupPass<R, T, V>;
    static std::atomic<int> dyn_max[kMaxDevices];
    int cap = 0;
    const cudaError_t e = kernel_attributes(bulk_groups_kernel<R, T, V>, dyn_max, cap, false);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(d.hg_n * d.hg_split);
    cfg.blockDim = dim3(P::kThreads);
    cfg.dynamicSmemBytes = P::kBytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = d.hg_split;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, bulk_groups_kernel<R, T, V>, d, t0, d.hg_split);
}

// T-step history pass (T = (kr - 1) / 2, 2 or 3): groups where there are any, the
// step-major matrices for one load case, else the run layout with two load cases
// per thread (the registers hold the T steps' sums and the window of T history
// vectors).  Measured against the run form and kept out of it: staging its history
// vectors and block values through shared memory with cp.async (72% more
// instructions, 1.5x slower; what pays for the staging in the group form is that
// eight rows use a vector) and L1 prefetches of the coming vectors (slower at every
// distance tried).
template <int R, bool kMixed>
cudaError_t launch_bulk_steps(const MarchData& d, int t0, int part, cudaStream_t s)
{
    if constexpr (R >= 8) {
        using V = typename std::conditional<kMixed, float, double>::type;
        if (d.hg_n > 0) return d.kr >= 7 ? launch_bulk_groups<R, 3, V>(d, t0, s) : launch_bulk_groups<R, 2, V>(d, t0, s);
    }
    if constexpr (R == 1) {
        const size_t slots = sizeof(int) * (d.K + 1);
        const int T = d.kr >= 7 ? 3 : 2, p0 = (int)((int64_t)d.E * part / T), p1 = (int)((int64_t)d.E * (part + 1) / T);
        if (p1 == p0) return cudaSuccess;
        if (T == 3) bulk_rows_kernel<kMixed, 3><<<p1 - p0, kRhsThreads, slots, s>>>(d, t0, p0, part);
        else bulk_rows_kernel<kMixed, 2><<<p1 - p0, kRhsThreads, slots, s>>>(d, t0, p0, part);
    } else {
        if (d.kr >= 7) bulk_steps_kernel<R, kMixed, 2, 3><<<d.E, kRhsThreads, 0, s>>>(d, t0);
        else bulk_steps_kernel<R, kMixed, 2, 2><<<d.E, kRhsThreads, 0, s>>>(d, t0);
    }
    return cudaGetLastError();
}

template <int R>
cudaError_t step_r(const MarchData& d0, int step, cudaStream_t s, cudaStream_t side, const StepEvents& ev, bool overlap)
{
    MarchData d = d0;
    const int kcap = step > 1 ? (step < d.K ? step : d.K) : 0;
    // T-step history passes: launched at steps 2, 2 + T, 2 + 2T, ..., the one
    // launched at step e covers steps e + T .. e + 2T - 1
    const int T = d.kr >= 5 ? (d.kr - 1) / 2 : 0;
    const bool pair = overlap && T >= 2;
    // one load case: part of the rows beside each of the T GMRES launches, so that
    // a part ends with its GMRES and the head finds the SMs free
    const int part = pair && step >= 2 ? (step - 2) % T : 0;
    const bool launches = pair && step >= 2 && (part == 0 || R == 1);
    cudaError_t e;
    // the first step a pass covers waits for it
    if (pair && step >= 2 + T && (step - 2) % T == 0 && ev.prev_pass) cudaStreamWaitEvent(s, ev.prev_pass, 0);
    if (!overlap) {
        d.k_lo = 1;
        d.k_hi = kcap;
        e = d.mixed ? launch_rhs<R, true>(d, step, false, 0, s) : launch_rhs<R, false>(d, step, false, 0, s);
    } else if (pair) {
        // head: k < kr, plus the part k >= kr and KnownM computed beside the
        // GMRES launches before this step (every step from 2 + T on)
        d.k_lo = 1;
        d.k_hi = kcap < d.kr - 1 ? kcap : d.kr - 1;
        const int add = step >= 2 + T ? 1 : 0;
        e = d.mixed ? launch_rhs<R, true>(d, step, false, add, s) : launch_rhs<R, false>(d, step, false, add, s);
    } else {
        // head: k in {1, 2}, plus the bulk (k >= 3 and KnownM) computed during
        // the previous step (every step from 3 on)
        d.k_lo = 1;
        d.k_hi = kcap < 2 ? kcap : 2;
        const int add = kcap >= 3 ? 1 : 0;
        e = d.mixed ? launch_rhs<R, true>(d, step, false, add, s) : launch_rhs<R, false>(d, step, false, add, s);
    }
    if (e != cudaSuccess) return e;
    // GMRES is scheduled while the head runs: without it a history pass takes the
    // SMs that the head leaves.  Steps of one load case: 120-element rod 57.2 ->
    // 55.0 us, 1,728-element bar 132 -> 117, 2,058 elements 179 -> 158.
    d.after_head = 1;
    switch (d.R / d.groups) {
    case 1: e = d.mixed ? launch_gmres<1, true>(d, step, s) : launch_gmres<1, false>(d, step, s); break;
    case 2: e = d.mixed ? launch_gmres<2, true>(d, step, s) : launch_gmres<2, false>(d, step, s); break;
    case 4: e = d.mixed ? launch_gmres<4, true>(d, step, s) : launch_gmres<4, false>(d, step, s); break;
    case 8: e = d.mixed ? launch_gmres<8, true>(d, step, s) : launch_gmres<8, false>(d, step, s); break;
    case 16: e = d.mixed ? launch_gmres<16, true>(d, step, s) : launch_gmres<16, false>(d, step, s); break;
    case 32: e = d.mixed ? launch_gmres<32, true>(d, step, s) : launch_gmres<32, false>(d, step, s); break;
    default: e = cudaErrorInvalidValue;
    }
    if (e != cudaSuccess) return e;
    cudaEventRecord(ev.gm, s);
    if (pair) {
        // part k >= kr of steps step+T .. step+2T-1 needs the states up to
        // step-1 only: it runs beside the GMRES of this step and the T - 1
        // after it
        if (ev.prev_gm) cudaStreamWaitEvent(side, ev.prev_gm, 0);
        const int t0 = step - part + T;
        if (launches && t0 <= d.nstep) {
            e = d.mixed ? launch_bulk_steps<R, true>(d0, t0, part, side) : launch_bulk_steps<R, false>(d0, t0, part, side);
            if (e != cudaSuccess) return e;
        }
        cudaEventRecord(ev.sync, side);
    } else if (overlap && step + 1 <= d.nstep) {
        // bulk of step+1 (k >= 3) needs the states up to step-1 only: run it on
        // the side stream while this step's GMRES runs; the next head waits.
        const int kc1 = step + 1 < d.K ? step + 1 : d.K;
        if (ev.prev_gm) cudaStreamWaitEvent(side, ev.prev_gm, 0);
        if (kc1 >= 3) {
            MarchData db = d0;
            db.k_lo = 3;
            db.k_hi = kc1;
            e = d.mixed ? launch_rhs<R, true>(db, step + 1, true, 0, side)
                        : launch_rhs<R, false>(db, step + 1, true, 0, side);
            if (e != cudaSuccess) return e;
        }
        cudaEventRecord(ev.sync, side);
        cudaStreamWaitEvent(s, ev.sync, 0);
    }
    return cudaSuccess;
}

}  // namespace

bool march_supported_loads(int R) { return R == 1 || R == 2 || R == 4 || R == 8 || R == 16 || R == 32; }

cudaError_t march_prepare(const MarchData& d, cudaStream_t s)
{
    prepare_kernel<<<296, 256, 0, s>>>(d);
    return cudaGetLastError();
}

cudaError_t march_step(const MarchData& d, int step, cudaStream_t s, cudaStream_t side, const StepEvents& ev,
                       bool overlap)
{
    switch (d.R) {
    case 1: return step_r<1>(d, step, s, side, ev, overlap);
    case 2: return step_r<2>(d, step, s, side, ev, overlap);
    case 4: return step_r<4>(d, step, s, side, ev, overlap);
    case 8: return step_r<8>(d, step, s, side, ev, overlap);
    case 16: return step_r<16>(d, step, s, side, ev, overlap);
    case 32: return step_r<32>(d, step, s, side, ev, overlap);
    }
    return cudaErrorInvalidValue;
}

cudaError_t gmres_solve_single(const MarchData& d, cudaStream_t s) { return launch_gmres<1, false>(d, 1, s); }

namespace {

size_t gmres_shared_bytes(int Rg)
{
    switch (Rg) {
    case 1: return (sizeof(GShared<1>) + 15) / 16 * 16;
    case 2: return (sizeof(GShared<2>) + 15) / 16 * 16;
    case 4: return (sizeof(GShared<4>) + 15) / 16 * 16;
    case 8: return (sizeof(GShared<8>) + 15) / 16 * 16;
    case 16: return (sizeof(GShared<16>) + 15) / 16 * 16;
    default: return (sizeof(GShared<32>) + 15) / 16 * 16;
    }
}

}  // namespace

size_t gmres_dsm_bytes(int rows, int halo, int Rg, bool mixed)
{
    const size_t row = 3 * (size_t)Rg, stride = Rg == 1 ? 4 : row, m = mixed ? sizeof(float) : sizeof(double);
    // shared state; product vector with its halo, work vector, product
    return gmres_shared_bytes(Rg) + (size_t)(rows + halo) * stride * sizeof(double) +
           (size_t)rows * (row * sizeof(double) + row * m);
}

bool gmres_dsm_fits(int rows, int halo, int Rg, bool mixed)
{
    return rows > 0 && gmres_dsm_bytes(rows, halo, Rg, mixed) <= kGmresDsmMax;
}

int gmres_row_capacity(int own_rows) { return (own_rows + 3) / 4 * 4; }  // 16-byte aligned vectors

void gmres_tile_index(const std::vector<int32_t>& cta_row, int own_cap, const std::vector<int32_t>& rp,
                      const std::vector<int32_t>& col, GmresTileIndex& out)
{
    const int C = (int)cta_row.size() - 1, E = cta_row[C];
    std::vector<int32_t> owner((size_t)E), slot((size_t)E, -1), mark((size_t)E, -1), remote, order;
    for (int c = 0; c < C; ++c)
        for (int p = cta_row[c]; p < cta_row[c + 1]; ++p) owner[p] = c;
    out = GmresTileIndex{};
    out.cs.assign((size_t)C + 1, 0);
    out.halo.assign((size_t)C, 0);
    std::vector<std::vector<int2>> send((size_t)C);
    for (int c = 0; c < C; ++c) {
        // rows of other CTAs that this CTA's rows use, in perm order
        remote.clear();
        for (int j = rp[cta_row[c]]; j < rp[cta_row[c + 1]]; ++j)
            if (owner[col[j]] != c && mark[col[j]] != c) {
                mark[col[j]] = c;
                remote.push_back(col[j]);
            }
        std::sort(remote.begin(), remote.end());
        for (size_t i = 0; i < remote.size(); ++i) {
            const int q = remote[i], o = owner[q];
            slot[q] = own_cap + (int)i;
            send[o].push_back(int2{(int)(((uint32_t)c << 24) | (uint32_t)(q - cta_row[o])), slot[q]});
        }
        out.halo[c] = (int32_t)remote.size();
        out.halo_max = std::max(out.halo_max, (int)remote.size());
        out.cs[c] = (int32_t)out.sp.size();
        // longest rows first: a slice's rows are of about one length (little
        // padding), and the warps' last slices are the short ones
        order.resize((size_t)(cta_row[c + 1] - cta_row[c]));
        std::iota(order.begin(), order.end(), cta_row[c]);
        std::stable_sort(order.begin(), order.end(),
                         [&](int a, int b) { return rp[a + 1] - rp[a] > rp[b + 1] - rp[b]; });
        for (size_t i0 = 0; i0 < order.size(); i0 += 4) {
            const size_t i1 = std::min(i0 + 4, order.size());
            const int most = rp[order[i0] + 1] - rp[order[i0]];
            out.sp.push_back(int2{(int)(out.col.size() / 32), most});
            for (size_t i = i0; i < i0 + 4; ++i) out.rows.push_back(i < i1 ? order[i] - cta_row[c] : -1);
            const size_t base = out.col.size(), tiles = (size_t)(most + 7) / 8;
            // padding: a zero block at the CTA's first row
            out.col.resize(base + 32 * tiles, 0);
            out.colg.resize(base + 32 * tiles, cta_row[c]);
            out.src.resize(base + 32 * tiles, -1);
            for (size_t i = i0; i < i1; ++i)
                for (int p = order[i], j = rp[p]; j < rp[p + 1]; ++j) {
                    const int b = j - rp[p], q = col[j];
                    const size_t at = base + 32 * (size_t)(b / 8) + 8 * (i - i0) + b % 8;
                    out.col[at] = owner[q] == c ? q - cta_row[c] : slot[q];
                    out.colg[at] = q;
                    out.src[at] = j;
                }
        }
    }
    out.cs[C] = (int32_t)out.sp.size();
    out.send_ptr.assign((size_t)C + 1, 0);
    for (int c = 0; c < C; ++c) {
        out.send.insert(out.send.end(), send[c].begin(), send[c].end());
        out.send_ptr[c + 1] = (int32_t)out.send.size();
    }
}

// Tile values from row-major 3x3 blocks; a block of the padding is zero.
__global__ void gather_tiles_kernel(int64_t n, const int32_t* src, const double* val9, double* out, float* out32)
{
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t tile = t / 288, c = (t - tile * 288) / 32, l = t & 31;
        const int32_t j = src[tile * 32 + l];
        const double v = j < 0 ? 0.0 : val9[9 * (int64_t)j + c];
        out[t] = v;
        if (out32) out32[t] = (float)v;
    }
}

cudaError_t pack_head(int E, int K, int head_k, const int32_t* row_of, const int64_t* kptr, const uint32_t* col,
                      const void* val, bool mixed, int64_t nnz, const int32_t* ptr, unsigned char* tiles, int* infinite,
                      cudaStream_t s)
{
    if (mixed)
        pack_head_kernel<<<(E + 7) / 8, 256, 0, s>>>(E, K, head_k, row_of, kptr, col, static_cast<const float*>(val), nnz,
                                                     ptr, tiles, infinite);
    else
        pack_head_kernel<<<(E + 7) / 8, 256, 0, s>>>(E, K, head_k, row_of, kptr, col, static_cast<const double*>(val), nnz,
                                                     ptr, tiles, infinite);
    return cudaGetLastError();
}

cudaError_t gather_tiles(int64_t tiles, const int32_t* src, const double* val9, double* out, float* out32,
                         cudaStream_t s)
{
    if (tiles <= 0) return cudaSuccess;
    const int64_t n = tiles * 288;
    gather_tiles_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 1184), 256, 0, s>>>(n, src, val9, out, out32);
    return cudaGetLastError();
}

namespace {

template <int R, bool kMixed, bool kLocal>
cudaError_t launch_gmres_models(const MarchData* ds, int n_models, int cluster, size_t gmres_dsm, int step,
                                cudaStream_t s)
{
    static std::atomic<int> dyn_max[kMaxDevices];
    int cap = 0;
    const cudaError_t e = kernel_attributes(gmres_models_kernel<R, kMixed, kLocal>, dyn_max, cap);
    if (e != cudaSuccess) return e;
    if (gmres_dsm > (size_t)cap) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cluster * n_models);
    cfg.blockDim = dim3(kGmresThreads);
    cfg.dynamicSmemBytes = gmres_dsm;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, gmres_models_kernel<R, kMixed, kLocal>, ds, step);
}

// One step of several models: the right-hand sides of every model in one launch,
// then one GMRES cluster of C CTAs per model, the models of the two forms side by
// side.
template <int R, bool kMixed>
cudaError_t models_step_r(const MarchData* ds, const int* row_off, int n_models, int total_rows, int cluster,
                          const ModelForms& forms, int max_K, int step, int phase, cudaStream_t s)
{
    constexpr int kC = R >= 4 ? 4 : R;
    const size_t smem = sizeof(int) * (size_t)(max_K + 1);
    if (phase == 2) {
        rhs_models_kernel<R, kMixed, true, kC><<<total_rows, kRhsThreads, smem, s>>>(ds, row_off, n_models, step, 1);
        return cudaGetLastError();
    }
    rhs_models_kernel<R, kMixed, false, kC><<<total_rows, kRhsThreads, smem, s>>>(ds, row_off, n_models, step, phase);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const bool both = forms.local && forms.global;
    cudaStream_t gs = both ? forms.other : s;
    if (both && ((e = cudaEventRecord(forms.fork, s)) != cudaSuccess ||
                 (e = cudaStreamWaitEvent(gs, forms.fork, 0)) != cudaSuccess))
        return e;
    if (forms.global)
        if ((e = launch_gmres_models<R, kMixed, false>(ds, n_models, cluster, gmres_dsm_bytes(0, 0, R, kMixed), step,
                                                       gs)) != cudaSuccess)
            return e;
    if (forms.local)
        if ((e = launch_gmres_models<R, kMixed, true>(ds, n_models, cluster, forms.dsm, step, s)) != cudaSuccess)
            return e;
    if (both && (e = cudaEventRecord(forms.join, gs)) == cudaSuccess) e = cudaStreamWaitEvent(s, forms.join, 0);
    return e;
}

}  // namespace

cudaError_t march_models_step(const MarchData* ds, const int* row_off, int n_models, int total_rows, int R,
                              bool mixed, int cluster, const ModelForms& forms, int max_K, int step, int phase,
                              cudaStream_t s)
{
#define TDBEM_MODELS_CASE(RR)                                                                                      \
    case RR:                                                                                                       \
        return mixed ? models_step_r<RR, true>(ds, row_off, n_models, total_rows, cluster, forms, max_K, step,     \
                                               phase, s)                                                           \
                     : models_step_r<RR, false>(ds, row_off, n_models, total_rows, cluster, forms, max_K, step,    \
                                                phase, s);
    switch (R) {
        TDBEM_MODELS_CASE(1)
        TDBEM_MODELS_CASE(2)
        TDBEM_MODELS_CASE(4)
        TDBEM_MODELS_CASE(8)
    }
#undef TDBEM_MODELS_CASE
    return cudaErrorInvalidValue;
}

int gmres_cluster_size(int device, int R, bool mixed)
{
    switch (R) {
    case 1: return mixed ? cluster_size_for<1, true>(device) : cluster_size_for<1, false>(device);
    case 2: return mixed ? cluster_size_for<2, true>(device) : cluster_size_for<2, false>(device);
    case 4: return mixed ? cluster_size_for<4, true>(device) : cluster_size_for<4, false>(device);
    case 8: return mixed ? cluster_size_for<8, true>(device) : cluster_size_for<8, false>(device);
    case 16: return mixed ? cluster_size_for<16, true>(device) : cluster_size_for<16, false>(device);
    case 32: return mixed ? cluster_size_for<32, true>(device) : cluster_size_for<32, false>(device);
    }
    return 1;
}

}  // namespace tdbem
