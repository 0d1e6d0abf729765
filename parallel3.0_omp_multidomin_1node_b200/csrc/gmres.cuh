// Left-preconditioned GMRES(restart) of one time step on one thread-block
// cluster, and the boundary write-back (included by march.cu).
//
// What bounds it: latency.  An Arnoldi step of one load case on the
// 3,072-element bar is 0.2 MFLOP of products over 0.4 MB of A' per CTA, so the
// time goes into the chain of phases, each waiting for the slowest thread and,
// three times, for the cluster.
// - A cluster barrier with release and acquire costs about 1,100 cycles here
//   (the fence), so inside the solve there is none: CTAs exchange data by
//   asynchronous remote stores that complete on the receiver's mbarrier (about
//   550 cycles), partial sums to every peer and basis vector values to the
//   CTAs whose rows use them, which then read only their own shared memory.
//   (Rows that do not fit shared memory: vectors in global memory, and a remote
//   arrival per peer instead of the values.)
// - A step runs straight through the code once, so its instructions have to
//   stay in the instruction cache: with every product, leaf application and
//   reduction inlined the kernel was 180 KB and each phase waited for its
//   instructions (a leaf application took 2,600 cycles, 900 when repeated at
//   once).  They are functions, and the two Gram-Schmidt passes one loop.
// Per time step, before (cluster barriers, W and A W carried along, everything
// inlined) and now, kernel alone: 3,072-element bar, one load case FP64 453 and
// 223 us (12.5 Arnoldi steps); 32 mixed 1,034 and 636 us; 120-element rod, one
// load case 99 and 55 us (5.9 steps).
#pragma once

#include "march.cuh"
#include "tdbem_common.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace tdbem {

__device__ __forceinline__ unsigned long long device_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
namespace {

constexpr int kGmresThreads = 512;  // at most (gmres_threads)
constexpr int kGmresWarps = kGmresThreads / 32;
static_assert(kGmresWarps == 16 && kGmresClusterMax == 16, "reductions use 16 lanes per value");
// cycles a CTA whose wait ran out stays after its peers have stopped, for their
// pushes still on the way to it (they take some 600)
constexpr long long kDrainCycles = 200000;

// basis vectors per cluster reduction, and Krylov columns whose small arrays
// (rotations, Hessenberg columns) are kept in shared memory: as many as the
// static shared memory holds for R cases
template <int R> constexpr int kDots = R == 1 ? 32 : R == 2 ? 16 : R == 4 ? 12 : R == 8 ? 8 : R == 16 ? 4 : 1;
template <int R> constexpr int kCols = R <= 4 ? 32 : R == 8 ? 24 : R == 16 ? 12 : 6;

// row stride of the product's source vector: a row of one case is padded to
// four values, so a block's three come as vector loads
template <int R> constexpr int kRowStride = R == 1 ? 4 : 3 * R;

template <int R>
__device__ __forceinline__ int mirror_index(int t)
{
    if constexpr (R == 1) return t + t / 3;
    else return t;
}

template <int R>
struct GShared {
    static constexpr int M = kDots<R> + 1;
    double wred[kGmresWarps][M * R + 1];            // per-warp partial sums
    double part[2][kGmresClusterMax][M * R];        // every CTA's partial sums, pushed by their owners
    double vals[M][R];                              // the cluster's sums
    double col[5][kCols<R>][R];                     // per column: cs, sn, h, c, f (SmallCol)
    double h1[R], phibar[R], n2b[R];
    int run[R], flag[R], inner[R], cycles[R], stag[R], check[R], jend[R];
    int any_run, any_cand, any_check;
    unsigned long long red_bar[2], vec_bar;         // mbarriers: partial sums of the two slots, vectors
    // the cluster and the vectors of this CTA
    int rank, C, nown, vcap, vs_off, vs_len, gl;    // basis vectors k < vcap at dsm + vs_off, vs_len apart
    int rl_off, pc_off;                             // cached leaf inverses: row table, values (doubles into dsm)
    double* vg;                                     // k >= vcap, vg_len apart
    double* G;                                      // small arrays in global memory, givens_stride per case
    int64_t vg_len, givens_stride;
};

enum { kCs = 0, kSn = 1, kH = 2, kC = 3, kF = 4 };

// ---- cluster primitives --------------------------------------------------
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_barrier()
{
    cluster_arrive();
    cluster_wait();
}
__device__ __forceinline__ uint32_t shared_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, uint32_t rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void peer_load1(uint32_t addr, double& v)
{
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
}
// asynchronous stores into a peer's shared memory, counted by its mbarrier
__device__ __forceinline__ void push8(uint32_t addr, unsigned long long v, uint32_t bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr), "l"(v), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void push16(uint32_t addr, unsigned long long v, unsigned long long w, uint32_t bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(addr), "l"(v),
                 "l"(w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void bar_init(unsigned long long* bar, uint32_t arrivals)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(shared_addr(bar)), "r"(arrivals) : "memory");
}
// one thread per CTA and phase: the phase ends when `bytes` have arrived
__device__ __forceinline__ void bar_expect(unsigned long long* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_addr(bar)), "r"(bytes) : "memory");
}
// State of a thread's exchanges: bit 0 slot of the next reduction, bits 1, 2 parity
// of the slots' current phases, bit 3 that of vec_bar, all the same in a CTA; bit 4
// a wait of this thread ran out, bit 5 its waits do so at once (a test's); from bit
// 8 on the limit of a wait, as a power of two in cycles.
constexpr uint32_t kDead = 16, kGiveUp = 32;
constexpr int kLimitShift = 8;

// Waits for a phase, at most about its limit.  When it runs out, this wait and the
// thread's later ones pass, and the thread arms no barrier and pushes nothing any
// more: a phase that did not end is never armed again, the waits of the CTA's other
// threads and of the peers that miss its share run out in turn, and every CTA comes
// to the barrier at the solve's end, where the step fails.
// kCluster: what other CTAs wrote to global memory is read next.  Otherwise the
// bytes counted lie in this CTA's shared memory and the wait acquires at CTA scope:
// a cluster-scope acquire also drops the SM's L1, and reading a 21-column leaf
// inverse after it took 3,700 cycles instead of 860 (measured).
template <bool kCluster = false>
__device__ __forceinline__ uint32_t bar_wait(unsigned long long* bar, uint32_t parity, uint32_t st)
{
    const uint32_t a = shared_addr(bar);
    long long start = 0;
    bool dead = (st & (kDead | kGiveUp)) != 0;
    while (!dead) {
        uint32_t done;
        if constexpr (kCluster)
            asm volatile("{.reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; "
                         "selp.u32 %0, 1, 0, p;}"
                         : "=r"(done) : "r"(a), "r"(parity) : "memory");
        else
            asm volatile("{.reg .pred p; mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2; "
                         "selp.u32 %0, 1, 0, p;}"
                         : "=r"(done) : "r"(a), "r"(parity) : "memory");
        if (done) return 0;
        const long long now = clock64();
        if (start == 0) start = now;
        else if ((now - start) >> (st >> kLimitShift) != 0) dead = true;
    }
    return kDead;
}

// the CPT cases of the three components of one row of a shared-memory vector
template <int R, int CPT>
__device__ __forceinline__ void vector_row(const double* a, double (&x)[3][CPT])
{
    if constexpr (R == 1) {
        const double2 t = *reinterpret_cast<const double2*>(a);
        x[0][0] = t.x;
        x[1][0] = t.y;
        x[2][0] = a[2];
    } else {
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int q = 0; q < CPT; q += 2) {
                const double2 t = *reinterpret_cast<const double2*>(a + c * R + q);
                x[c][q] = t.x;
                x[c][q + 1] = t.y;
            }
    }
}
template <int R, int CPT>
__device__ __forceinline__ void vector_row(const float* a, float (&x)[3][CPT])
{
    if constexpr (R == 1) {
        const float4 t = *reinterpret_cast<const float4*>(a);
        x[0][0] = t.x;
        x[1][0] = t.y;
        x[2][0] = t.z;
    } else if constexpr (CPT == 2) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 t = *reinterpret_cast<const float2*>(a + c * R);
            x[c][0] = t.x;
            x[c][1] = t.y;
        }
    } else {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float4 t = *reinterpret_cast<const float4*>(a + c * R);
            x[c][0] = t.x;
            x[c][1] = t.y;
            x[c][2] = t.z;
            x[c][3] = t.w;
        }
    }
}

// ---- cluster-wide sums ---------------------------------------------------
// This thread's contribution v to value q of its case.
template <int R>
__device__ __forceinline__ void red_put(GShared<R>& s, double v, int q)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o >= R && o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane < R) s.wred[w][q * R + lane] = v;
}

__device__ __forceinline__ double sum16(double v)
{
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

extern __shared__ __align__(16) double dsm[];

template <int R>
__device__ __forceinline__ GShared<R>& gshared()
{
    return *reinterpret_cast<GShared<R>*>(dsm);
}

// Sums of m values per case over the cluster, in dst[q * R + case] (shared
// memory) of every CTA.  Each CTA pushes its partial sums into every peer's
// shared memory, all reads are local and every CTA adds the same partials in
// the same order.  The two slots alternate: a peer pushes into a slot again
// only after it has received every CTA's partials of the reduction between,
// which a CTA pushes after its reads of the slot.
template <int R>
__device__ __noinline__ uint32_t red_finish(int m, int dst, uint32_t st)
{
    GShared<R>& s = gshared<R>();
    const int l = threadIdx.x & 15, g = threadIdx.x >> 4, per = blockDim.x >> 4, nw = blockDim.x >> 5;
    const int items = m * R, slot = st & 1u, C = s.C;
    const bool live = !(st & kDead);
    unsigned long long* bar = &s.red_bar[slot];
    __syncthreads();
    if (threadIdx.x == 0 && live) bar_expect(bar, (uint32_t)(sizeof(double) * items * C));
    const uint32_t peer = (uint32_t)(l < C ? l : s.rank);
    const uint32_t to = peer_addr(shared_addr(&s.part[slot][s.rank][0]), peer), to_bar = peer_addr(shared_addr(bar), peer);
#pragma unroll 1
    for (int i0 = 0; i0 < items; i0 += per) {
        const int i = i0 + g;
        const double v = sum16(i < items && l < nw ? s.wred[l][i] : 0.0);
        if (i < items && l < C && live) push8(to + 8 * i, (unsigned long long)__double_as_longlong(v), to_bar);
    }
    st |= bar_wait(bar, (st >> (1 + slot)) & 1u, st);
#pragma unroll 1
    for (int i0 = 0; i0 < items; i0 += per) {
        const int i = i0 + g;
        const double v = sum16(i < items && l < C ? s.part[slot][l][i] : 0.0);
        if (i < items && l == 0) dsm[dst + i] = v;
    }
    __syncthreads();
    return st ^ 1u ^ (2u << slot);
}

// Dot products of the work vector u (shared-memory offset, or a global pointer)
// with V_{q0} .. V_{q0+nq-1} and, `norm`, with itself, summed over the cluster
// into dst[value * R + case] of every CTA.  A warp takes a value: its lanes read
// consecutive elements, and for R <= 4 it pushes the CTA's sum straight to the
// peers (a value per thread and a second stage over the warps took twice the
// time for one load case).  For more cases, whose vectors are longer, several
// warps share a value.  Starts with a CTA barrier (u complete).
template <int R>
__device__ __noinline__ uint32_t gram_dots(int q0, int nq, bool norm, const double* u, int dst, uint32_t st)
{
    GShared<R>& s = gshared<R>();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5, C = s.C, slot = st & 1u;
    const int m = nq + norm, parts = R <= 4 || m >= nw ? 1 : nw / m, nown = s.nown;
    const int to_all = st & kDead ? 0 : C;  // peers to push to
    unsigned long long* bar = &s.red_bar[slot];
    const uint32_t to = shared_addr(&s.part[slot][s.rank][0]), to_bar = shared_addr(bar);
    __syncthreads();
    if (threadIdx.x == 0 && to_all) bar_expect(bar, (uint32_t)(sizeof(double) * m * R * C));
#pragma unroll 1
    for (int i = w; i < m * parts; i += nw) {
        const int k = i % m, part = i / m, kv = q0 + k, step = 32 * parts;
        const double* v = k >= nq ? u : kv < s.vcap ? dsm + s.vs_off + kv * s.vs_len : s.vg + kv * s.vg_len;
        double a0 = 0.0, a1 = 0.0;
#pragma unroll 1
        for (int t = lane + 32 * part; t < nown; t += 4 * step) {
            double x[4], y[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const bool on = t + q * step < nown;
                x[q] = on ? v[t + q * step] : 0.0;
                y[q] = on ? u[t + q * step] : 0.0;
            }
            a0 += x[0] * y[0];
            a1 += x[1] * y[1];
            a0 += x[2] * y[2];
            a1 += x[3] * y[3];
        }
        a0 += a1;
#pragma unroll
        for (int o = 16; o >= R && o > 0; o >>= 1) a0 += __shfl_xor_sync(0xffffffffu, a0, o);
        if constexpr (R <= 4) {
#pragma unroll
            for (int j = 0; j < (R + 1) / 2; ++j) {
                const int peer = lane / R + j * (32 / R);
                if (peer < to_all)
                    push8(peer_addr(to + 8 * (k * R + lane % R), (uint32_t)peer),
                          (unsigned long long)__double_as_longlong(a0), peer_addr(to_bar, (uint32_t)peer));
            }
        } else if (lane < R) {
            s.wred[part][k * R + lane] = a0;
        }
    }
    const int l = threadIdx.x & 15, g = threadIdx.x >> 4, per = blockDim.x >> 4, items = m * R;
    if constexpr (R > 4) {
        __syncthreads();
#pragma unroll 1
        for (int i0 = 0; i0 < items; i0 += per) {
            const int i = i0 + g;
            const double v = sum16(i < items && l < parts ? s.wred[l][i] : 0.0);
            if (i < items && l < to_all)
                push8(peer_addr(to + 8 * i, (uint32_t)l), (unsigned long long)__double_as_longlong(v),
                      peer_addr(to_bar, (uint32_t)l));
        }
    }
    st |= bar_wait(bar, (st >> (1 + slot)) & 1u, st);
#pragma unroll 1
    for (int i0 = 0; i0 < items; i0 += per) {
        const int i = i0 + g;
        const double v = sum16(i < items && l < C ? s.part[slot][l][i] : 0.0);
        if (i < items && l == 0) dsm[dst + i] = v;
    }
    __syncthreads();
    return st ^ 1u ^ (2u << slot);
}

// Publishes the owned rows of the product's source vector v (shared memory; row
// stride kRowStride<R>): pushes each row to the CTAs whose rows use it and waits
// for the `halo` rows this CTA uses.  The previous vector's rows are free: every
// peer has pushed its partial sums of a reduction after its product.
template <int R, class T>
__device__ __noinline__ uint32_t publish(const int2* __restrict__ send, int n_send, int halo, int v_off, uint32_t st)
{
    constexpr int kRowBytes = kRowStride<R> * (int)sizeof(T), kChunk = kRowBytes % 16 == 0 ? 16 : 8;
    constexpr int kChunks = kRowBytes / kChunk;
    GShared<R>& s = gshared<R>();
    const char* v = reinterpret_cast<const char*>(dsm + v_off);
    if (st & kDead) n_send = 0;
    __syncthreads();
    if (threadIdx.x == 0 && !(st & kDead)) bar_expect(&s.vec_bar, (uint32_t)(halo * kRowBytes));
    const uint32_t base = shared_addr(v), bar = shared_addr(&s.vec_bar);
#pragma unroll 1
    for (int i = threadIdx.x; i < n_send * kChunks; i += blockDim.x) {
        const int2 e = __ldg(send + i / kChunks);  // x = peer << 24 | row, y = row there
        const int o = (i % kChunks) * kChunk;
        const char* src = v + (e.x & 0xFFFFFF) * kRowBytes + o;
        const uint32_t peer = (uint32_t)e.x >> 24, to = peer_addr(base + (uint32_t)(e.y * kRowBytes + o), peer);
        if constexpr (kChunk == 16) {
            const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(src);
            push16(to, t.x, t.y, peer_addr(bar, peer));
        } else {
            push8(to, *reinterpret_cast<const unsigned long long*>(src), peer_addr(bar, peer));
        }
    }
    return (st | bar_wait(&s.vec_bar, (st >> 3) & 1u, st)) ^ 8u;
}

// The global-memory form's counterpart: this CTA's rows of a vector in global
// memory are complete, and every other CTA's are after it.  An arrival at each
// peer's vec_bar, with the limit of the other waits: the cluster barrier has none,
// and a CTA that gave up would have to keep count of its peers'.  A peer arrives
// for the next vector only after a reduction between, so after this CTA's wait.
template <int R>
__device__ __noinline__ uint32_t vectors_complete(uint32_t st)
{
    GShared<R>& s = gshared<R>();
    __syncthreads();
    if ((int)threadIdx.x < s.C && !(st & kDead))
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(
                         peer_addr(shared_addr(&s.vec_bar), threadIdx.x))
                     : "memory");
    return (st | bar_wait<true>(&s.vec_bar, (st >> 3) & 1u, st)) ^ 8u;
}

// ---- products ------------------------------------------------------------
// y = A' v on the owned rows.  A' comes as tiles of 4 rows x 8 blocks, values
// in 9 planes of 32, so a warp's load of one value index is one coalesced
// access (the row-major blocks it replaces, 72 bytes apart per lane, took
// eight times the memory wavefronts).  A warp takes a slice of 4 rows, 8 lanes
// per row; TPB lanes share a block (CPT cases each), BPR lane groups take the
// blocks of a row.  The source is this CTA's shared memory (kLocal: offset in dsm; its
// own rows and the halo it received) or a global vector, the columns
// accordingly.  Ends with a CTA barrier.
template <int R, bool kLocal, class AT, class ST, class Y>
__device__ __noinline__ void spmm_tiles(const int2* __restrict__ slices, const int32_t* __restrict__ srows,
                                        const int32_t* __restrict__ cols, const AT* __restrict__ tv, const ST* gsrc, int src_off, int rows,
                                        Y* y)
{
    constexpr int CPT = R >= 4 ? 4 : R, TPB = R / CPT;
    constexpr int BPR = TPB >= 8 ? 1 : 8 / TPB;
    constexpr bool kF = sizeof(AT) == 4, kAccF = kF && sizeof(ST) == 4;
    using Acc = typename std::conditional<kAccF, float, double>::type;
    const ST* src = reinterpret_cast<const ST*>(dsm + src_off);
    const int lane = threadIdx.x & 31;
    const int rsub = lane >> 3, bsub = (lane & 7) / TPB, cgp = lane % TPB;
#pragma unroll 1
    for (int sl = threadIdx.x >> 5; 4 * sl < rows; sl += (int)(blockDim.x >> 5)) {
        const int2 sp = __ldg(slices + sl);  // first tile, blocks of the longest row
        const int p = __ldg(srows + 4 * sl + rsub);
        const int tb = sp.x, its = (sp.y + BPR - 1) / BPR;
        Acc acc[3][CPT];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int q = 0; q < CPT; ++q) acc[c][q] = 0;
        // kU blocks per lane at once; those past the end load nothing
        constexpr int kU = R <= 2 ? 3 : 2;
#pragma unroll 1
        for (int i0 = 0; i0 < its; i0 += kU) {
            AT m[kU][9];
            int col[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int it = i0 + u, tile = tb + it * BPR / 8, at = rsub * 8 + (it * BPR) % 8 + bsub;
                const bool on = it < its;
                const AT* a = tv + (int64_t)tile * 288 + at;
                col[u] = on ? __ldg(cols + tile * 32 + at) : 0;
#pragma unroll
                for (int c = 0; c < 9; ++c) m[u][c] = on ? __ldg(a + 32 * c) : (AT)0;
            }
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                ST x[3][CPT];
                if constexpr (kLocal) {
                    vector_row<R, CPT>(src + col[u] * kRowStride<R> + cgp * CPT, x);
                } else {
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int q = 0; q < CPT; ++q)
                            x[c][q] = __ldcg(gsrc + (3 * (int64_t)col[u] + c) * R + cgp * CPT + q);
                }
#pragma unroll
                for (int q = 0; q < CPT; ++q)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        if constexpr (kF && !kAccF)
                            acc[c][q] += (double)(m[u][3 * c] * (float)x[0][q] + m[u][3 * c + 1] * (float)x[1][q] +
                                                  m[u][3 * c + 2] * (float)x[2][q]);
                        else
                            acc[c][q] += m[u][3 * c] * x[0][q] + m[u][3 * c + 1] * x[1][q] + m[u][3 * c + 2] * x[2][q];
                    }
            }
        }
#pragma unroll
        for (int o = TPB; o < 8; o <<= 1)
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int q = 0; q < CPT; ++q) acc[c][q] += __shfl_xor_sync(0xffffffffu, acc[c][q], o);
        if (p >= 0 && bsub == 0)
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int q = 0; q < CPT; ++q) y[(3 * p + c) * R + cgp * CPT + q] = (Y)acc[c][q];
    }
    __syncthreads();
}

// out = the block-diagonal product of `in` with the leaves' dense blocks m
// (GMRES_M_X, DBEM1/pre_gmres.cpp:837-895) at this thread's owned values (not
// stored when out is null); returns their sum of squares.  m is stored by columns, so the lanes of a
// leaf's rows read consecutive values.  FP64: one running sum over the leaf's
// columns, the reference's order.
template <int R, class MT, class ST>
__device__ __noinline__ double leaf_apply(const int4* __restrict__ row_leaf, const MT* __restrict__ m, const ST* in,
                                          int lo, double* out)
{
    const int nown = gshared<R>().nown;
    double p2 = 0.0;
#pragma unroll 1
    for (int t = threadIdx.x; t < nown; t += blockDim.x) {
        const int r = t % R, e = t / R, p = e / 3, c = e - 3 * p;
        const int4 lf = __ldg(row_leaf + lo + p);  // RowLeaf
        const int n3 = lf.w;
        const MT* a = m + (int64_t)(((uint64_t)(uint32_t)lf.y << 32) | (uint32_t)lf.x) + 3 * (lo + p - lf.z) + c;
        const ST* src = in + 3 * (lf.z - lo) * R + r;
        double v = 0.0;
        if constexpr (sizeof(MT) == 4 && sizeof(ST) == 4) {
            float s0 = 0.0f, s1 = 0.0f;
            int q = 0;
#pragma unroll 3
            for (; q + 1 < n3; q += 2) {
                s0 += __ldg(a) * src[q * R];
                s1 += __ldg(a + n3) * src[(q + 1) * R];
                a += 2 * n3;
            }
            if (q < n3) s0 += __ldg(a) * src[q * R];
            v = (double)(s0 + s1);
        } else {
            // n3 is a multiple of 3
#pragma unroll 2
            for (int q = 0; q < n3; q += 3) {
                MT w[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) w[i] = __ldg(a + i * n3);
                a += 3 * n3;
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    if constexpr (sizeof(MT) == 4) v += (double)(w[i] * (float)src[(q + i) * R]);
                    else v += w[i] * src[(q + i) * R];
                }
            }
        }
        if (out) out[t] = v;
        p2 += v * v;
    }
    return p2;
}

// leaf_apply for the inverses cached in shared memory (kLocal form): `in` an
// offset in dsm (in doubles) of ST values, out FP64.  Up to two cases: a thread
// per value; more: a thread per row and case, whose three components share the
// source values.  Ends without a barrier; the values' sum of squares is not
// taken (the caller's gram_dots does).
template <int R, class MT, class ST>
__device__ __noinline__ void leaf_apply_cached(int in_off, double* out)
{
    GShared<R>& s = gshared<R>();
    const MT* pc = reinterpret_cast<const MT*>(dsm + s.pc_off);
    const int4* rl = reinterpret_cast<const int4*>(dsm + s.rl_off);
    const ST* in = reinterpret_cast<const ST*>(dsm + in_off);
    const int nown = s.nown;
    if constexpr (R <= 2) {
#pragma unroll 1
        for (int t = threadIdx.x; t < nown; t += blockDim.x) {
            const int r = t % R, e = t / R, p = e / 3;
            const int4 lf = rl[p];  // offset of the row's first component, first source row * 3, -, n3
            const MT* a = pc + lf.x + (e - 3 * p);
            const ST* src = in + lf.y * R + r;
            const int n3 = lf.w;
            MT v0 = 0, v1 = 0;
#pragma unroll 2
            for (int q = 0; q < n3; q += 3) {
                const MT m0 = a[0], m1 = a[n3], m2 = a[2 * n3];
                const MT x0 = (MT)src[q * R], x1 = (MT)src[(q + 1) * R], x2 = (MT)src[(q + 2) * R];
                a += 3 * n3;
                if constexpr (sizeof(MT) == 4) {
                    if (q % 2 == 0) {
                        v0 += m0 * x0;
                        v1 += m1 * x1;
                        v0 += m2 * x2;
                    } else {
                        v1 += m0 * x0;
                        v0 += m1 * x1;
                        v1 += m2 * x2;
                    }
                } else {
                    v0 += m0 * x0;
                    v0 += m1 * x1;
                    v0 += m2 * x2;
                }
            }
            out[t] = (double)(v0 + v1);
        }
    } else {
        const int items = nown / 3;
#pragma unroll 1
        for (int i = threadIdx.x; i < items; i += blockDim.x) {
            const int r = i % R, p = i / R;
            const int4 lf = rl[p];
            const MT* a = pc + lf.x;
            const ST* src = in + lf.y * R + r;
            const int n3 = lf.w;
            MT v[2][3] = {};
#pragma unroll 2
            for (int q = 0; q < n3; q += 3)
#pragma unroll
                for (int h = 0; h < 3; ++h) {
                    const MT x = (MT)src[(q + h) * R];
#pragma unroll
                    for (int c = 0; c < 3; ++c) v[sizeof(MT) == 4 ? h & 1 : 0][c] += a[(q + h) * n3 + c] * x;
                }
#pragma unroll
            for (int c = 0; c < 3; ++c) out[(3 * p + c) * R + r] = (double)(v[0][c] + v[1][c]);
        }
    }
}

// A small array of one case: element k at p[k * stride].  Arrays of up to
// kCols<R> columns are read in shared memory; past that all columns are in
// global memory (the persistent ones, cs, sn and f, always too).
struct SmallCol {
    double* p;
    int stride;
    __device__ __forceinline__ double& operator[](int k) const { return p[k * stride]; }
};
template <int R>
__device__ __forceinline__ SmallCol small_col(GShared<R>& s, int which, int columns, int r)
{
    if (columns <= kCols<R>) return {&s.col[which][0][r], R};
    return {s.G + r * s.givens_stride + which * s.gl, 1};
}

// out = scale * (in + sign * sum_{k < nk} a_k V_k) at this thread's owned values
// (a: small array `which` of `columns` columns; in may be null), also to the
// product's source at dsm + src_off unless that is negative.
template <int R, class ST>
__device__ __noinline__ void combine(int which, int columns, int nk, const double* in, double sign, double scale,
                                     double* out, int src_off)
{
    GShared<R>& s = gshared<R>();
    const int nown = s.nown, vcap = s.vcap, len = s.vs_len, NT = (int)blockDim.x, r = threadIdx.x % R;
    ST* const pv = reinterpret_cast<ST*>(dsm + src_off);
    const double* vs = dsm + s.vs_off;
    if (R <= 2 && columns <= kCols<R> && nk <= vcap) {
        const double* a = &s.col[which][0][r];
#pragma unroll 1
        for (int t = threadIdx.x; t < nown; t += NT) {
            double v0 = 0.0, v1 = 0.0;
            const double x = in ? in[t] : 0.0;
#pragma unroll 1
            for (int k = 0; k < nk; k += 4) {
                double f[4], b[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    f[q] = k + q < nk ? a[(k + q) * R] : 0.0;
                    b[q] = k + q < nk ? vs[(k + q) * len + t] : 0.0;
                }
                v0 += f[0] * b[0];
                v1 += f[1] * b[1];
                v0 += f[2] * b[2];
                v1 += f[3] * b[3];
            }
            const double v = scale * (x + sign * (v0 + v1));
            out[t] = v;
            if (src_off >= 0) pv[mirror_index<R>(t)] = (ST)v;
        }
        return;
    }
    // kT values and two vectors at once
    constexpr int kT = R <= 2 ? 1 : 3;
    const SmallCol a = small_col<R>(s, which, columns, r);
    const double* vg = s.vg;
    const int64_t glen = s.vg_len;
#pragma unroll 1
    for (int t0 = threadIdx.x; t0 < nown; t0 += kT * NT) {
        double v[kT];
#pragma unroll
        for (int i = 0; i < kT; ++i) v[i] = 0.0;
#pragma unroll 1
        for (int k = 0; k < nk; k += 2) {
            const bool two = k + 1 < nk;
            const double f0 = a[k], f1 = two ? a[k + 1] : 0.0;
            const double* p0 = k < vcap ? vs + k * len : vg + k * glen;
            const double* p1 = k + 1 < vcap ? vs + (k + 1) * len : vg + (k + 1) * glen;
            double b0[kT], b1[kT];
#pragma unroll
            for (int i = 0; i < kT; ++i) {
                const bool on = t0 + i * NT < nown;
                b0[i] = on ? p0[t0 + i * NT] : 0.0;
                b1[i] = on && two ? p1[t0 + i * NT] : 0.0;
            }
#pragma unroll
            for (int i = 0; i < kT; ++i) v[i] += f0 * b0[i] + f1 * b1[i];
        }
#pragma unroll
        for (int i = 0; i < kT; ++i) {
            const int t = t0 + i * NT;
            if (t < nown) {
                const double x = scale * ((in ? in[t] : 0.0) + sign * v[i]);
                out[t] = x;
                if (src_off >= 0) pv[mirror_index<R>(t)] = (ST)x;
            }
        }
    }
}

// Boundary values of element i for load case r of the private solution x
// (ScatterUnknownToBoundary + AllLocToAbs, DBEM1/multidomain.cpp:3086-3200):
// displacement in g[0..2], traction in g[3..5], global frame.
template <int R>
__device__ __forceinline__ void boundary_values(const MarchData& d, const double* x, int i, int r, const double* in,
                                                double (&g)[6])
{
    const double* T = d.itf_trans + 9 * (int64_t)i;
    const double* F = d.trans + 9 * (int64_t)i;
#pragma unroll 1
    for (int type = 0; type < 2; ++type) {
        const double sg = __ldg((type ? d.tref_sign : d.uref_sign) + i);
        double l[3];
        if (__ldg((type ? d.tref_known : d.uref_known) + i)) {
#pragma unroll
            for (int c = 0; c < 3; ++c) l[c] = sg * __ldg(in + c);
        } else {
            const double* v = x + (int64_t)3 * __ldg(d.perm_of_unk + __ldg((type ? d.tref_block : d.uref_block) + i)) * R + r;
            const double v0 = __ldcg(v), v1 = __ldcg(v + R), v2 = __ldcg(v + 2 * R);
#pragma unroll
            for (int c = 0; c < 3; ++c)
                l[c] = sg * (__ldg(T + 3 * c) * v0 + __ldg(T + 3 * c + 1) * v1 + __ldg(T + 3 * c + 2) * v2);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double v = __ldg(F + c) * l[0] + __ldg(F + 3 + c) * l[1] + __ldg(F + 6 + c) * l[2];
            if (type) g[3 + c] = v;
            else g[c] = v;
        }
    }
}

// Write-back of a step for the load cases roff .. roff+R-1: boundary values,
// the history state X_s with the combined vectors W_{s-1} = (X_s + 2 X_{s-1}) +
// X_{s-2} and W_s = 2 X_s + X_{s-1} (BuildConvolutionVector's coefficients 1, 2,
// 1 and summation order; X_0 and unsolved states are zero,
// DBEM1/multidomain.cpp:3201-3225), and the interface audit
// (PrintInterfaceError, :3227-3257).  One pass without barriers: the thread
// of an element has X_s at hand for its W entries, and the thread of an
// interface's B side computes the A side's values again for the audit.
template <int R>
__device__ __noinline__ void write_back(const MarchData& d, int step, int roff, const double* x, int gtid, int gstride)
{
    const int E = d.E, RT = d.R, nh = d.nh;
    const int64_t per_type = (int64_t)nh * 3 * RT, per_slot = 2 * per_type;
    double* X = d.xring + (step % 3) * per_slot;
    const double* X1 = d.xring + ((step + 2) % 3) * per_slot;
    const double* X2 = d.xring + ((step + 1) % 3) * per_slot;
    double* Wa = d.wring + ((step - 1) % d.SW) * per_slot;
    double* Wb = d.wring + (step % d.SW) * per_slot;
    double worst[2] = {0.0, 0.0};  // displacement jump, traction balance
    double zero = 0.0;             // not any more once a combined vector is not finite (for the group pass)
#pragma unroll 1
    for (int t = gtid; t < E * R; t += gstride) {
        const int i = t / R, r = t % R, rg = roff + r;
        const int64_t base = ((int64_t)rg * (d.nstep + 1) + step) * E;
        double g[6], a[6];
        // the element, then the A side of its interface
        int e = i;
#pragma unroll 1
        for (int side = 0; side < 2; ++side) {
            boundary_values<R>(d, x, e, r, d.known_lu + (base + e) * 3, a);
            if (side) break;
#pragma unroll
            for (int c = 0; c < 6; ++c) g[c] = a[c];
            e = __ldg(d.itf_a + i);
            if (e < 0) break;
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            d.out_lu[(base + i) * 3 + c] = g[c];
            d.out_lt[(base + i) * 3 + c] = g[3 + c];
        }
        if (__ldg(d.hist_owner + i)) {
            const double su = __ldg(d.hu_sign + i), st = __ldg(d.ht_sign + i);
            const int64_t o = __ldg(d.hist_block + i) * 3 * RT + rg;
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                const double xs = (c < 3 ? su : st) * g[c];
                const int64_t p = o + (c < 3 ? 0 : per_type) + (c % 3) * RT;
                const double xm1 = X1[p], xm2 = X2[p];
                const double wa = (xs + 2.0 * xm1) + xm2, wb = 2.0 * xs + xm1;
                X[p] = xs;
                Wa[p] = wa;
                Wb[p] = wb;
                if (d.hg_n > 0) zero += 0.0 * wa + 0.0 * wb;
            }
        }
        if (e >= 0) {
            const double sg = __ldg(d.itf_asign + i);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                worst[0] = fmax(worst[0], fabs(a[c] - g[c]));
                worst[1] = fmax(worst[1], fabs(g[3 + c] - sg * a[3 + c]));
            }
        }
    }
    if (zero != 0.0) d.status[1] = 1;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) worst[k] = fmax(worst[k], __shfl_xor_sync(0xffffffffu, worst[k], o));
        // non-negative doubles order like their bit patterns
        if ((threadIdx.x & 31) == 0 && worst[k] > 0.0)
            atomicMax(reinterpret_cast<unsigned long long*>(d.audit + 2 * (step - 1) + k),
                      (unsigned long long)__double_as_longlong(worst[k]));
    }
    if (d.rec_x && roff == 0)
#pragma unroll 1
        for (int u = gtid; u < E; u += gstride)
            for (int c = 0; c < 3; ++c)
                d.rec_x[(int64_t)(step - 1) * 3 * E + 3 * u + c] = __ldcg(x + ((int64_t)3 * d.perm_of_unk[u] + c) * R);
}

}  // namespace

// GMRES for the R load cases of one step on one thread-block cluster, then
// the write-back.  Case r stops updating once converged; the cluster stops
// when every case has.  FP64 mode stops a case on its true residual b - A x
// (maxit = 1, as the reference).  Mixed mode runs the Arnoldi product and the
// preconditioner in FP32, keeps orthogonalisation and Givens in FP64, and
// restarts from the explicit FP64 residual until it meets the tolerance.
//
// The residual of each step comes without forming x: with z_j the
// preconditioned residual, z_j = V t with t built from the rotations, and
// r_j = M z_j with M the leaf blocks.  |r_j| >= |z_j| / |M^-1|, |z_j| =
// |phibar|, so steps whose phibar is above 1.01 |M^-1| tol |b| cannot have
// converged and skip it (the hundredth is for rounding).  x = x0 + V y is formed once, when the residual meets
// the tolerance.  (Carrying W_j = V_j R^-1 and A W_j through every step, as
// the reference's recurrence does, read and wrote 4 j + 6 vectors per step.)
template <int R, bool kMixed, bool kLocal>
__device__ __forceinline__ void gmres_body(const MarchData& d, const int step, const int grp)
{
    // element types of the Arnoldi product's source and result
    using MT = typename std::conditional<kMixed && kLocal, float, double>::type;
    using AT = typename std::conditional<kMixed, float, double>::type;
    constexpr int JC = kCols<R>, KD = kDots<R>;
    GShared<R>& s = gshared<R>();
    int rank, C;
    {
        cg::cluster_group cgc = cg::this_cluster();
        rank = (int)cgc.block_rank();
        C = (int)cgc.num_blocks();
    }
    // state of the exchanges; a limit of zero or less makes the last thread of the
    // last CTA give up its first wait
    uint32_t st = (uint32_t)abs(d.wait_log2) << kLimitShift;
    if (d.wait_log2 <= 0 && rank == C - 1 && threadIdx.x == blockDim.x - 1) st |= kGiveUp;
    const int NT = (int)blockDim.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int RT = d.R, roff = grp * R;  // total cases, first case of this group
    const int E = d.E, rs = d.restart;
    const int64_t n = 3LL * E * R;       // values of one private vector
    const int lo = __ldg(d.cta_row + rank), rows = __ldg(d.cta_row + rank + 1) - lo;
    const int64_t ob = 3LL * lo * R;
    const int nown = 3 * rows * R;
    static_assert(256 % R == 0, "a thread's values all belong to one case");
    const int tr = threadIdx.x % R;
    // Vectors of the owned rows.  kLocal, in shared memory: pv, the source of the
    // next product (V_j, or the solution in FP64) with its halo; us, work; aw,
    // the product; then the first vcap basis vectors.  Otherwise (the range is
    // too large) all in global memory, where products read other CTAs' values.
    constexpr int pv_off = (int)((sizeof(GShared<R>) + 15) / 16 * 2);
    double* const pv = kLocal ? dsm + pv_off : d.rv + (int64_t)grp * n + ob;
    MT* const pvm = reinterpret_cast<MT*>(pv);
    double* const us = kLocal ? dsm + pv_off + (d.dsm_rows + d.halo_rows) * kRowStride<R> : d.u + (int64_t)grp * n + ob;
    double* const aw64 = kLocal ? us + 3 * d.dsm_rows * R : d.aw + (int64_t)grp * n + ob;
    MT* const aw = reinterpret_cast<MT*>(aw64);
    // cached leaf inverses (row table, values) when the launch has room for them
    const int rl_off = kLocal ? (int)(aw64 - dsm) + 3 * d.dsm_rows * R * (int)sizeof(MT) / (int)sizeof(double) : 0;
    const int pc_off = rl_off + 2 * d.dsm_rows, leaf_vals = kLocal ? d.leaf_cap : 0;
    const int vs_off = leaf_vals ? pc_off + (leaf_vals * (int)sizeof(AT) + 15) / 16 * 2 : rl_off;
    double* const vs = dsm + vs_off;
    double* const vg = d.V + (int64_t)grp * (rs + 1) * n + ob;
    const int vcap = kLocal ? d.vcap : 0, vs_len = 3 * d.dsm_rows * R;
    if (threadIdx.x == 0) {
        bar_init(&s.red_bar[0], 1);
        bar_init(&s.red_bar[1], 1);
        bar_init(&s.vec_bar, kLocal ? 1 : C);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s.rank = rank;
        s.C = C;
        s.nown = nown;
        s.vcap = vcap;
        s.vs_off = vs_off;
        s.vs_len = vs_len;
        s.rl_off = rl_off;
        s.pc_off = pc_off;
        s.vg = vg;
        s.vg_len = n;
        s.gl = rs + 2;
        s.givens_stride = d.givens_stride;
        s.G = d.givens + ((int64_t)grp * C + rank) * R * d.givens_stride;
    }
    __syncthreads();
    cluster_arrive();  // waited for before the first push: every CTA of the cluster has its mbarriers set up
    // the rotated Hessenberg column j (upper triangle, diagonal as its reciprocal)
    auto tri = [&](int r, int j) {
        return s.G + r * d.givens_stride + kGivensArrays * (rs + 2) + (int64_t)j * (j + 1) / 2;
    };
    // element j of a persistent small array
    auto put_col = [&](int which, int j, int r, double v) {
        if (j < JC) s.col[which][j][r] = v;
        s.G[r * d.givens_stride + which * (rs + 2) + j] = v;
    };
    auto V = [&](int k) -> double* { return k < vcap ? vs + k * vs_len : vg + (int64_t)k * n; };
    auto pi = [&](int t) { return kLocal ? mirror_index<R>(t) : t; };
    auto rhs = [&](int t) { return __ldcg(d.b + (3LL * lo + t / R) * RT + roff + tr); };
    auto off = [&](const double* p) { return (int)(p - dsm); };
    const int2* const slices = d.g_sp + __ldg(d.g_cs + rank);
    const int32_t* const srows = d.g_rows + 4 * __ldg(d.g_cs + rank);
    const int4* const row_leaf = reinterpret_cast<const int4*>(d.row_leaf);
    const int e0 = __ldg(d.g_send_ptr + rank), n_send = __ldg(d.g_send_ptr + rank + 1) - e0, halo = __ldg(d.g_halo + rank);
    // y = A pv (FP64)
    auto product_x = [&](double* y) {
        if constexpr (kLocal) {
            st = publish<R, double>(d.g_send + e0, n_send, halo, pv_off, st);
            spmm_tiles<R, true, double, double, double>(slices, srows, d.g_col, d.g_val, nullptr, pv_off, rows, y);
        } else {
            st = vectors_complete<R>(st);
            spmm_tiles<R, false, double, double, double>(slices, srows, d.g_colg, d.g_val, pv - ob, 0, rows, y);
        }
    };
    const AT* pinv;
    if constexpr (kMixed) pinv = d.pinv32;
    else pinv = d.pinv;
    // in exact arithmetic 1 x |M^-1| bounds |z| / |r|; the rest is for rounding
    const double minv2 = 1.01 * __ldg(d.minv);
    // V_1's direction from the residual in us: z = M^-1 r (in V(0)), its sum of squares
    auto start_vector = [&]() { return leaf_apply<R, AT, double>(row_leaf, pinv, us, lo, V(0)); };
    if (leaf_vals) {
        const int4 f0 = __ldg(row_leaf + lo);
        const int64_t off0 = (int64_t)(((uint64_t)(uint32_t)f0.y << 32) | (uint32_t)f0.x);
        int4* rl = reinterpret_cast<int4*>(dsm + rl_off);
        AT* pc = reinterpret_cast<AT*>(dsm + pc_off);
        for (int p = threadIdx.x; p < rows; p += NT) {
            const int4 f = __ldg(row_leaf + lo + p);
            const int64_t o = (int64_t)(((uint64_t)(uint32_t)f.y << 32) | (uint32_t)f.x);
            rl[p] = make_int4((int)(o - off0) + 3 * (lo + p - f.z), 3 * (f.z - lo), 0, f.w);
        }
        const int4 fl = rows > 0 ? __ldg(row_leaf + lo + rows - 1) : f0;
        const int64_t end = (int64_t)(((uint64_t)(uint32_t)fl.y << 32) | (uint32_t)fl.x) + (int64_t)fl.w * fl.w;
        for (int i = threadIdx.x; rows > 0 && i < (int)(end - off0); i += NT) pc[i] = __ldg(pinv + off0 + i);
    }

    // all above read what setup laid out; the head pass, beside which this launch may
    // have started, is complete below
    cudaGridDependencySynchronize();
    if (d.stamps && blockIdx.x == 0 && threadIdx.x == 0) d.stamps[5 * (int64_t)step + 1] = device_ns();

    // start vector and residual (in us).  Mixed mode starts from the previous
    // steps' solutions extrapolated linearly (x_{s-1} at step 2); the FP64 path
    // starts from zero as the reference does (DBEM1/multidomain.cpp:3869-3870)
    double* const x = d.x + (int64_t)grp * n + ob;
    double* const xold = kMixed && d.xold ? d.xold + (int64_t)grp * n + ob : nullptr;
    const bool warm = xold != nullptr && step >= 2;
    double bb = 0.0, rr = 0.0;
    if (warm) {
        for (int t = threadIdx.x; t < nown; t += NT) {
            const double x1 = x[t], x2 = xold[t], x0 = step == 2 ? x1 : 2.0 * x1 - x2;
            xold[t] = x1;
            x[t] = x0;
            pv[pi(t)] = x0;
        }
        cluster_wait();
        product_x(us);
    }
    for (int t = threadIdx.x; t < nown; t += NT) {
        const double b = rhs(t);
        double res = b;
        if (warm) {
            res -= us[t];
        } else {
            x[t] = 0.0;
            if (xold) xold[t] = 0.0;
        }
        us[t] = res;
        bb += b * b;
        rr += res * res;
    }
    __syncthreads();
    const double zz = start_vector();
    if (!warm) cluster_wait();
    // |b|^2, |r|^2, |z|^2 in one reduction.  Another cluster of the launch
    // (another load-case group) may set the status word at any time: the last
    // value counts the CTAs that read it set, so the whole cluster takes the
    // same decision.
    const double stop = threadIdx.x < R && *(volatile int*)d.status ? 1.0 : 0.0;
    constexpr int kOnce = KD + 1 < 4 ? KD + 1 : 4;  // values per reduction
    bool aborted = false;
#pragma unroll
    for (int q0 = 0; q0 < 4; q0 += kOnce) {
#pragma unroll
        for (int q = q0; q < q0 + kOnce; ++q) red_put<R>(s, q == 0 ? bb : q == 1 ? rr : q == 2 ? zz : stop, q - q0);
        st = red_finish<R>(kOnce, off(&s.vals[0][0]), st);
        if (threadIdx.x < R) {
#pragma unroll
            for (int q = q0; q < q0 + kOnce; ++q) {
                const double v = s.vals[q - q0][tr];
                if (q == 0) s.n2b[tr] = sqrt(v);
                if (q == 1) s.phibar[tr] = sqrt(v);
                if (q == 2) s.h1[tr] = sqrt(v);
            }
        }
        if (q0 + kOnce == 4) aborted = s.vals[kOnce - 1][0] != 0.0;
        __syncthreads();
    }
    if (threadIdx.x < R) {
        s.flag[tr] = (s.n2b[tr] == 0.0 || s.phibar[tr] <= d.tol * s.n2b[tr]) ? 0 : 1;
        s.inner[tr] = 0;
        s.cycles[tr] = 0;
    }

    // R y = f by back substitution into the h column (jn columns), a warp per
    // case; columns from jend on get zero
    auto solve_columns = [&](int jn) {
#pragma unroll 1
        for (int r = w; r < R; r += NT >> 5) {
            const int je = s.jend[r];
            const SmallCol f = small_col<R>(s, kF, jn, r), y = small_col<R>(s, kH, jn, r);
#pragma unroll 1
            for (int k = lane; k < jn; k += 32) y[k] = k < je ? f[k] : 0.0;
            __syncwarp();
            // columns of R are fetched a step ahead of their use
            double next = je > 0 ? tri(r, je - 1)[min(lane, je - 1)] : 0.0, diag = je > 0 ? tri(r, je - 1)[je - 1] : 0.0;
#pragma unroll 1
            for (int l = je - 1; l >= 0; --l) {
                const double rc = next, yl = y[l] * diag;
                if (l > 0) {
                    next = tri(r, l - 1)[min(lane, l - 1)];
                    diag = tri(r, l - 1)[l - 1];
                }
                __syncwarp();
                if (lane < l) y[lane] -= rc * yl;
#pragma unroll 1
                for (int k = lane + 32; k < l; k += 32) y[k] -= tri(r, l)[k] * yl;
                if (lane == 0) y[l] = yl;
                __syncwarp();
            }
        }
        __syncthreads();
    };
    // V_k as the next product's source
    auto to_source = [&](int k) {
        if constexpr (kLocal) {
            const double* v = V(k);
            for (int t = threadIdx.x; t < nown; t += NT) pvm[mirror_index<R>(t)] = (MT)v[t];
        }
    };

    const int max_cycles = kMixed ? 8 : 1;
#pragma unroll 1
    for (int cycle = 0; cycle < max_cycles; ++cycle) {
        if (w == 0) {
            bool running = false;
            if (lane < R) {
                running = s.flag[lane] == 1 && !aborted;
                s.run[lane] = running;
                s.phibar[lane] = s.h1[lane];
                s.stag[lane] = 0;
                s.jend[lane] = 0;
                if (running) s.cycles[lane]++;
            }
            const unsigned any = __ballot_sync(0xffffffffu, running);
            if (lane == 0) s.any_run = any != 0;
        }
        __syncthreads();
        if (!s.any_run) break;
        // V_1 = z / |z|; zero for a case that does not run, whose z need not be finite
        combine<R, MT>(kH, 0, 0, R == 1 || s.run[tr] ? V(0) : nullptr, 0.0, s.run[tr] ? 1.0 / s.h1[tr] : 0.0, V(0),
                       kLocal ? pv_off : -1);
        int jn = 0;  // columns done
#pragma unroll 1
        for (int j = 0; j < rs; ++j) {
            // u = M^-1 A V_j (in us)
            if constexpr (kLocal) {
                st = publish<R, MT>(d.g_send + e0, n_send, halo, pv_off, st);
                if constexpr (kMixed)
                    spmm_tiles<R, true, float, float, float>(slices, srows, d.g_col, d.g_val32, nullptr, pv_off, rows, aw);
                else
                    spmm_tiles<R, true, double, double, double>(slices, srows, d.g_col, d.g_val, nullptr, pv_off, rows, aw);
            } else {
                st = vectors_complete<R>(st);
                if constexpr (kMixed)
                    spmm_tiles<R, false, float, double, double>(slices, srows, d.g_colg, d.g_val32, V(j) - ob, 0, rows, aw);
                else
                    spmm_tiles<R, false, double, double, double>(slices, srows, d.g_colg, d.g_val, V(j) - ob, 0, rows, aw);
            }
            if (leaf_vals) leaf_apply_cached<R, AT, MT>(off(aw64), us);
            else leaf_apply<R, AT, MT>(row_leaf, pinv, aw, lo, us);
            // Classical Gram-Schmidt applied twice (CGS2), one cluster
            // reduction per pass and KD basis vectors, instead of one per basis
            // vector as in MGS (DBEM1/pre_gmres.cpp:1462-1485).  The basis and
            // the Hessenberg column are MGS's up to rounding.  Pass 0: h_k =
            // V_k . u; pass 1: u' = u - sum_k h_k V_k (kept in us), c_k =
            // V_k . u' and, as one more value, |u'|^2.
            const int nb = j + 1;  // basis vectors
#pragma unroll 1
            for (int pass = 0; pass < 2; ++pass) {
                const int which = pass ? kC : kH, values = nb + pass;
                if (pass) {
                    combine<R, MT>(kH, nb + 1, nb, us, -1.0, 1.0, us, -1);
                }
#pragma unroll 1
                for (int q0 = 0; q0 < values; q0 += KD + 1) {
                    const int m = min(KD + 1, values - q0), nq = min(m, nb - q0);  // values, dot products among them
                    const bool small = nb + 1 <= JC;
                    st = gram_dots<R>(q0, nq, nq < m, us, off(small ? &s.col[which][q0][0] : &s.vals[0][0]), st);
                    if (!small) {
                        for (int i = threadIdx.x; i < m * R; i += NT)
                            small_col<R>(s, which, nb + 1, i % R)[q0 + i / R] = s.vals[i / R][i % R];
                        __syncthreads();
                    }
                }
            }
            // h(k, j) = h_k + c_k; |u''|^2 = |u'|^2 - sum c_k^2 unless that
            // cancels (near breakdown): then u'' and its norm explicitly
            double cc = 0.0, nn;
            {
                const SmallCol c = small_col<R>(s, kC, nb + 1, tr);
                nn = c[nb];
#pragma unroll 1
                for (int k0 = 0; k0 < nb; k0 += 4)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const double v = k0 + q < nb ? c[k0 + q] : 0.0;
                        cc += v * v;
                    }
            }
            const double est = nn - cc;
            const bool exact = !(est > 1.0e-4 * nn);
            double hn = exact ? 0.0 : sqrt(est);
            const bool any_exact = R == 1 ? exact : __syncthreads_or(exact) != 0;
            if (any_exact) {
                combine<R, MT>(kC, nb + 1, nb, us, -1.0, 1.0, us, -1);
                st = gram_dots<R>(0, 0, true, us, off(&s.vals[0][0]), st);
                hn = sqrt(s.vals[0][tr]);
            }
            jn = nb;
            // Givens by the last warp (the one with the fewest values), a lane
            // per case: column j of R, the new rotation, phibar, and which
            // cases may have converged; the other warps go on to V_{j+1}
            if (w == (NT >> 5) - 1) {
                bool cand = false, going = false;
                if (lane < R) {
                    const int r = lane;
                    double* rc = tri(r, j);
                    const SmallCol h = small_col<R>(s, kH, nb + 1, r), hc = small_col<R>(s, kC, nb + 1, r);
                    const SmallCol cs = small_col<R>(s, kCs, nb + 1, r), sn = small_col<R>(s, kSn, nb + 1, r);
                    double a = h[0] + hc[0];
#pragma unroll 1
                    for (int i = 0; i < j; i += 2) {
                        const bool two = i + 1 < j;
                        const double b1 = h[i + 1] + hc[i + 1], b2 = two ? h[i + 2] + hc[i + 2] : 0.0;
                        const double c1 = cs[i], s1 = sn[i], c2 = two ? cs[i + 1] : 1.0, s2 = two ? sn[i + 1] : 0.0;
                        rc[i] = c1 * a - s1 * b1;
                        a = s1 * a + c1 * b1;
                        if (two) {
                            rc[i + 1] = c2 * a - s2 * b2;
                            a = s2 * a + c2 * b2;
                        }
                    }
                    double c = 1.0, sv = 0.0;
                    const double inv = 1.0 / (hn != 0.0 ? sqrt(a * a + hn * hn) : a);
                    if (hn != 0.0) {
                        c = a * inv;
                        sv = -hn * inv;
                    }
                    rc[j] = inv;
                    put_col(kCs, j, r, c);
                    put_col(kSn, j, r, sv);
                    const double f = c * s.phibar[r], pb = sv * s.phibar[r];
                    put_col(kF, j, r, f);
                    s.phibar[r] = pb;
                    if (s.run[r]) {
                        s.inner[r]++;
                        s.jend[r] = nb;
                        if (f == 0.0) s.stag[r] = 1;
                        cand = s.stag[r] || fabs(pb) <= minv2 * (d.tol * s.n2b[r]);
                        if (kMixed && !cand && fabs(pb) <= 1.0e-5 * s.h1[r]) s.run[r] = 0;  // FP32 Krylov space exhausted: refine
                        going = s.run[r] != 0;
                    }
                }
                const unsigned any = __ballot_sync(0xffffffffu, cand), gg = __ballot_sync(0xffffffffu, going);
                if (lane == 0) {
                    s.any_cand = any != 0;
                    s.any_run = gg != 0;
                }
            }
            // V_{j+1} = (u' - sum_k c_k V_k) / h(j+1, j), zero when
            // h(j+1, j) <= 1e-12 (DBEM1/pre_gmres.cpp:1481-1485)
            combine<R, MT>(kC, nb + 1, any_exact ? 0 : nb, us, -1.0, hn <= 1.0e-12 ? 0.0 : 1.0 / hn, V(nb),
                           kLocal ? pv_off : -1);
            __syncthreads();
            if (!s.any_cand) {
                if (!s.any_run) break;
                continue;
            }
            // residual of the candidates: z_j = sum_k t_k V_k, t_{j+1} =
            // c_j phibar_j, t_k = c_{k-1} s_k ... s_j phibar_j; r_j = M z_j
            if (w == 0 && lane < R) {
                const SmallCol cs = small_col<R>(s, kCs, nb + 1, lane), sn = small_col<R>(s, kSn, nb + 1, lane);
                const SmallCol tz = small_col<R>(s, kC, nb + 1, lane);
                double p = s.phibar[lane];
                tz[nb] = cs[j] * p;
#pragma unroll 1
                for (int k = j; k >= 0; --k) {
                    const double c = k > 0 ? cs[k - 1] : 1.0;
                    p *= sn[k];
                    tz[k] = c * p;
                }
            }
            __syncthreads();
            combine<R, MT>(kC, nb + 1, nb + 1, nullptr, 1.0, 1.0, us, -1);
            __syncthreads();
            red_put<R>(s, leaf_apply<R, double, double>(row_leaf, d.pmat, us, lo, nullptr), 0);
            st = red_finish<R>(1, off(&s.vals[0][0]), st);
            if (w == 0) {
                bool check = false, going = false;
                if (lane < R) {
                    const int r = lane;
                    if (s.run[r]) {
                        if (sqrt(s.vals[0][r]) <= d.tol * s.n2b[r]) {
                            if (kMixed) s.run[r] = 0;  // decided on the FP64 residual after the cycle
                            else check = true;         // decided on the true residual now
                        } else if (s.stag[r]) {
                            s.run[r] = 0;
                            s.flag[r] = 3;
                        } else if (kMixed && fabs(s.phibar[r]) <= 1.0e-5 * s.h1[r]) {
                            s.run[r] = 0;
                        }
                    }
                    s.check[r] = check;
                    going = s.run[r] != 0;
                }
                const unsigned c = __ballot_sync(0xffffffffu, check), gg = __ballot_sync(0xffffffffu, going);
                if (lane == 0) {
                    s.any_check = c != 0;
                    s.any_run = gg != 0;
                }
            }
            __syncthreads();
            if constexpr (!kMixed) {
                if (s.any_check) {
                    // x = V y and the stopping test on b - A x (DBEM1/pre_gmres.cpp:1566-1578)
                    solve_columns(nb);
                    combine<R, MT>(kH, nb, nb, nullptr, 1.0, 1.0, us, -1);
                    for (int t = threadIdx.x; t < nown; t += NT) pv[pi(t)] = us[t];
                    product_x(aw64);
                    double p2 = 0.0;
                    for (int t = threadIdx.x; t < nown; t += NT) {
                        const double res = rhs(t) - aw64[t];
                        p2 += res * res;
                    }
                    red_put<R>(s, p2, 0);
                    st = red_finish<R>(1, off(&s.vals[0][0]), st);
                    if (s.check[tr] && sqrt(s.vals[0][tr]) <= d.tol * s.n2b[tr])
                        for (int t = threadIdx.x; t < nown; t += NT) x[t] = us[t];
                    if (w == 0) {
                        bool going = false;
                        if (lane < R) {
                            if (s.check[lane] && sqrt(s.vals[0][lane]) <= d.tol * s.n2b[lane]) {
                                s.run[lane] = 0;
                                s.flag[lane] = 0;
                            }
                            going = s.run[lane] != 0;
                        }
                        const unsigned gg = __ballot_sync(0xffffffffu, going);
                        if (lane == 0) s.any_run = gg != 0;
                    }
                    __syncthreads();
                    if (s.any_run) to_source(nb);
                }
            }
            if (!s.any_run) break;
        }
        if constexpr (!kMixed) {
            // cases that ended without converging: their last iterate
            int failed = 0;
            for (int r = 0; r < R; ++r) failed |= s.flag[r] != 0 && s.jend[r] > 0;
            if (failed) {
                solve_columns(jn);
                combine<R, MT>(kH, jn, jn, nullptr, 1.0, 1.0, us, -1);
                if (s.flag[tr] != 0)
                    for (int t = threadIdx.x; t < nown; t += NT) x[t] = us[t];
            }
        } else {
            // x += V y, its explicit FP64 residual, and the next cycle's start
            solve_columns(jn);
            combine<R, MT>(kH, jn, jn, x, 1.0, 1.0, x, -1);
            for (int t = threadIdx.x; t < nown; t += NT) pv[pi(t)] = x[t];
            product_x(us);
            double r2 = 0.0;
            for (int t = threadIdx.x; t < nown; t += NT) {
                const double res = rhs(t) - us[t];
                us[t] = res;
                r2 += res * res;
            }
            __syncthreads();
            red_put<R>(s, r2, 0);
            red_put<R>(s, start_vector(), 1);
            st = red_finish<R>(2, off(&s.vals[0][0]), st);
            if (threadIdx.x < R) {
                if (s.flag[tr] == 1 && sqrt(s.vals[0][tr]) <= d.tol * s.n2b[tr]) s.flag[tr] = 0;
                s.h1[tr] = sqrt(s.vals[1][tr]);
            }
            __syncthreads();
        }
    }
    const bool dead = __syncthreads_or(st & kDead) != 0;  // a wait ran out in this CTA: the step has failed
    int failed = dead;  // the flags are the same in every CTA otherwise
    for (int r = 0; r < R; ++r) failed |= s.flag[r] != 0;
    int* const fl = d.step_flags + ((int64_t)(step - 1) * RT + roff + tr) * 3;
    if (threadIdx.x < R && rank == 0 && !aborted) {
        fl[0] = s.flag[tr];
        fl[1] = s.cycles[tr];
        fl[2] = s.inner[tr];
        if (s.flag[tr] != 0) atomicExch(d.status, 1);
    }
    cluster_barrier();  // x complete; no peer is accessed below
    if (dead) {
        if (threadIdx.x < R) {
            fl[0] = 1;
            atomicExch(d.status, 1);
        }
        // all peers have stopped; what they had pushed may still be on its way here
        const long long t0 = clock64();
        while (clock64() - t0 < kDrainCycles) {}
    }
    if (failed || aborted || d.solve_only) return;
    write_back<R>(d, step, roff, d.x + (int64_t)grp * n, rank * NT + (int)threadIdx.x, C * NT);
}

}  // namespace tdbem
