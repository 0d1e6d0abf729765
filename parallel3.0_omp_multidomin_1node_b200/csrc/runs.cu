// Run layout of the stacked history blocks, read by the T-step history pass
// (bulk_steps_kernel in march.cu).
//
// The stacked layout keeps each equation row's blocks step-major (k = 1..K,
// then type and column), which suits a pass over one step.  The blocks of one
// (row, type, column) pair form an unbroken run of consecutive steps (the
// wave front passes a source-field pair during a window of steps), so the
// T-step pass walks runs instead: block k of a run meets the combined
// history vectors W_{s-k} .. W_{s+T-1-k} for steps s .. s + T - 1, and all but
// W_{s-k} are vectors its predecessor met, kept in registers.
//
// Built on the device from the stacked arrays: sort the blocks of steps
// k >= kr by (row, type, column, k), cut runs where the pair changes or k
// jumps, order each row's runs longest first (so the lane groups of one warp
// walk runs of similar length), and gather the block values into that order.
//
// The group layout (8 or more load cases) does the same for groups of
// neighbouring rows of one domain, whose waves arrive at about the same steps:
// a segment is one (type, column) pair over the steps in which any of the rows
// has a block, a matrix of the rows' blocks in the tensor path's fragments, so
// one history vector serves all the rows.
#include "assemble.cuh"
#include "march.cuh"

#include <climits>
#include <vector>

#include <cub/cub.cuh>

namespace tdbem {

namespace {

// one warp per row: sort keys row << 32 | type << 31 | column << 11 | k of the
// row's blocks of steps k >= kr, with their stacked index
__global__ void run_keys_kernel(int E, int K, int kr, const int64_t* __restrict__ kptr,
                                const int64_t* __restrict__ qoff, const uint32_t* __restrict__ col,
                                unsigned long long* __restrict__ key, uint32_t* __restrict__ idx)
{
    const int r = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (r >= E) return;
    const int64_t beg = kptr[(int64_t)r * (K + 1) + kr - 1], end = kptr[(int64_t)r * (K + 1) + K];
    const int64_t q0 = qoff[r] - beg;
    for (int64_t i = beg + lane; i < end; i += 32) {
        const uint32_t cp = col[i];
        const unsigned long long k = cp >> 21, type = (cp >> 20) & 1u, c = cp & 0xFFFFFu;
        key[q0 + i] = ((unsigned long long)r << 32) | (type << 31) | (c << 11) | k;
        idx[q0 + i] = (uint32_t)i;
    }
}

// 1 where sorted block q starts a run: a new (row, type, column) or a gap in k
__global__ void run_flags_kernel(int64_t nb, const unsigned long long* __restrict__ key, int* __restrict__ flag)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nb; q += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long a = key[q];
        int f = 1;
        if (q > 0) {
            const unsigned long long b = key[q - 1];
            f = (b >> 11) != (a >> 11) || (b & 0x7FFull) + 1 != (a & 0x7FFull);
        }
        flag[q] = f;
    }
}

// run j (inclusive scan of the flags minus one) starts at sorted block q
__global__ void run_starts_kernel(int64_t nb, const int* __restrict__ flag, const int* __restrict__ runid,
                                  int* __restrict__ start)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nb; q += (int64_t)gridDim.x * blockDim.x)
        if (flag[q]) start[runid[q] - 1] = (int)q;
}

// order key of run j: row << 16 | (0xFFFF - length), so a stable sort puts each
// row's runs longest first; counts the row's runs
__global__ void run_order_keys_kernel(int n_runs, int64_t nb, const int* __restrict__ start,
                                      const unsigned long long* __restrict__ key, unsigned long long* __restrict__ okey,
                                      int* __restrict__ oval, int* __restrict__ row_count)
{
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n_runs; j += gridDim.x * blockDim.x) {
        const int q = start[j];
        const int len = (j + 1 < n_runs ? start[j + 1] : (int)nb) - q;
        const unsigned long long row = key[q] >> 32;
        okey[j] = (row << 16) | (unsigned long long)(0xFFFF - len);
        oval[j] = j;
        atomicAdd(row_count + row, 1);
    }
}

__global__ void run_lengths_kernel(int n_runs, const unsigned long long* __restrict__ okey, int64_t* __restrict__ len)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_runs; i += gridDim.x * blockDim.x)
        len[i] = 0xFFFF - (int64_t)(okey[i] & 0xFFFFull);
}

// one warp per run (in final order): header, then the 9 values of each block
template <class T>
__global__ void run_gather_kernel(int n_runs, int64_t nb, int64_t nnz, const int* __restrict__ order,
                                  const int* __restrict__ start, const int64_t* __restrict__ len,
                                  const int64_t* __restrict__ off, const unsigned long long* __restrict__ key,
                                  const uint32_t* __restrict__ idx, const T* __restrict__ val, uint2* __restrict__ meta,
                                  int64_t* __restrict__ r_off, T* __restrict__ out)
{
    const int i = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (i >= n_runs) return;
    const int q = start[order[i]];
    const int n = (int)len[i];
    const int64_t o = off[i];
    if (lane == 0) {
        const unsigned long long a = key[q];
        const unsigned type = (unsigned)((a >> 31) & 1u), c = (unsigned)((a >> 11) & 0xFFFFFu),
                       kf = (unsigned)(a & 0x7FFu);
        meta[i] = make_uint2((type << 20) | c, (kf << 16) | (unsigned)n);
        r_off[i] = o;
    }
    for (int t = lane; t < n; t += 32) {
        const int64_t src = idx[q + t];
#pragma unroll
        for (int c = 0; c < 9; ++c) out[c * nb + o + t] = val[c * nnz + src];
    }
}

// As run_keys_kernel for groups of rows: key place / 8 << 35 | type << 34 |
// column << 14 | k << 3 | place % 8, so a group's blocks of one (type, column)
// come together, steps ascending.
__global__ void group_keys_kernel(int E, int K, int kr, const int32_t* __restrict__ place,
                                  const int64_t* __restrict__ kptr, const int64_t* __restrict__ qoff,
                                  const uint32_t* __restrict__ col, unsigned long long* __restrict__ key,
                                  uint32_t* __restrict__ idx)
{
    const int r = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (r >= E) return;
    const int64_t beg = kptr[(int64_t)r * (K + 1) + kr - 1], end = kptr[(int64_t)r * (K + 1) + K];
    const int64_t q0 = qoff[r] - beg;
    const unsigned long long g = (unsigned)(place[r] / kGroupRows), slot = (unsigned)(place[r] % kGroupRows);
    for (int64_t i = beg + lane; i < end; i += 32) {
        const uint32_t cp = col[i];
        const unsigned long long k = cp >> 21, type = (cp >> 20) & 1u, c = cp & 0xFFFFFu;
        key[q0 + i] = (g << 35) | (type << 34) | (c << 14) | (k << 3) | slot;
        idx[q0 + i] = (uint32_t)i;
    }
}

// 1 where sorted block q starts a segment: a new (group, type, column) or a
// step past the next one
__global__ void group_flags_kernel(int64_t nb, const unsigned long long* __restrict__ key, int* __restrict__ flag)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nb; q += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long a = key[q];
        int f = 1;
        if (q > 0) {
            const unsigned long long b = key[q - 1];
            f = (b >> 14) != (a >> 14) || ((a >> 3) & 0x7FFull) > ((b >> 3) & 0x7FFull) + 1;
        }
        flag[q] = f;
    }
}

// order key of segment j: group << 16 | (0xFFFF - length in steps); counts the
// group's segments
__global__ void group_order_keys_kernel(int n_segs, int64_t nb, const int* __restrict__ start,
                                        const unsigned long long* __restrict__ key,
                                        unsigned long long* __restrict__ okey, int* __restrict__ oval,
                                        int* __restrict__ group_count)
{
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n_segs; j += gridDim.x * blockDim.x) {
        const int q = start[j], e = (j + 1 < n_segs ? start[j + 1] : (int)nb) - 1;
        const int len = (int)((key[e] >> 3) & 0x7FFull) - (int)((key[q] >> 3) & 0x7FFull) + 1;
        const unsigned long long g = key[q] >> 35;
        okey[j] = (g << 16) | (unsigned long long)(0xFFFF - len);
        oval[j] = j;
        atomicAdd(group_count + g, 1);
    }
}

// contraction steps of n history steps
__global__ void group_steps_kernel(int n_segs, const unsigned long long* __restrict__ okey, int64_t* __restrict__ steps)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_segs; i += gridDim.x * blockDim.x)
        steps[i] = (3 * (0xFFFF - (int64_t)(okey[i] & 0xFFFFull)) + 3) / 4;
}

// one warp per segment (in final order): header, then its blocks to their
// places in the fragments (which start at zero): entry (3 slot + i, 3 (k - k0) +
// j) of the segment's matrix.  *infinite is set when a value is not finite.
template <class V>
__global__ void group_scatter_kernel(int n_segs, int64_t nb, int64_t nnz, const int* __restrict__ order,
                                     const int* __restrict__ start, const unsigned long long* __restrict__ okey,
                                     const int64_t* __restrict__ off, const unsigned long long* __restrict__ key,
                                     const uint32_t* __restrict__ idx, const V* __restrict__ val,
                                     uint2* __restrict__ meta, int64_t* __restrict__ s_off, V* __restrict__ out,
                                     int* __restrict__ infinite)
{
    const int i = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (i >= n_segs) return;
    const int j = order[i], q = start[j], e = j + 1 < n_segs ? start[j + 1] : (int)nb;
    const int64_t o = off[i];
    const unsigned long long a = key[q];
    const int k0 = (int)((a >> 3) & 0x7FFull);
    if (lane == 0) {
        meta[i] = make_uint2((unsigned)((a >> 34) & 1u) << 20 | (unsigned)((a >> 14) & 0xFFFFFu),
                             ((unsigned)k0 << 16) | (unsigned)(0xFFFF - (okey[i] & 0xFFFFull)));
        s_off[i] = o;
    }
    for (int t = q + lane; t < e; t += 32) {
        const unsigned long long b = key[t];
        const int step = (int)((b >> 3) & 0x7FFull) - k0, slot = (int)(b & 7u);
        const int64_t src = idx[t];
#pragma unroll
        for (int c = 0; c < 9; ++c) {
            const int m = 3 * slot + c / 3, kk = 3 * step + c % 3;
            const V v = val[c * nnz + src];
            out[((o + kk / 4) * 3 + m / 8) * 32 + (m % 8) * 4 + kk % 4] = v;
            if (!isfinite(v)) *infinite = 1;
        }
    }
}

struct Tmp {
    void* p = nullptr;
    Tmp() = default;
    Tmp(const Tmp&) = delete;
    Tmp& operator=(const Tmp&) = delete;
    ~Tmp() { release(); }
    void release()
    {
        if (p) cudaFree(p);
        p = nullptr;
    }
    cudaError_t alloc(size_t n)
    {
        release();
        return cudaMalloc(&p, n ? n : 1);
    }
    template <class T>
    T* as() const { return static_cast<T*>(p); }
};

int bits_for(unsigned long long v)
{
    int b = 0;
    while (b < 64 && (v >> b) != 0) ++b;
    return b;
}

}  // namespace

#define RUN_TRY(x)                          \
    do {                                    \
        cudaError_t e_ = (x);               \
        if (e_ != cudaSuccess) return e_;   \
    } while (0)

size_t history_runs_bytes(int64_t nb, bool mixed)
{
    // per block: sort keys and indices (double-buffered), flags, run ids and
    // the radix sort's scratch; per run (about nine blocks on the models
    // measured; counted as four): start, order keys and values
    // (double-buffered), length, offset and header; the output values.  An
    // estimate: the caller falls back to the one-step pass when an
    // allocation fails all the same.
    const size_t per_block = 2 * 8 + 2 * 4 + 4 + 4 + 16;
    const size_t per_run = 4 + 2 * 8 + 2 * 4 + 8 + 8 + 8 + 8;
    return (size_t)nb * (per_block + 9 * (mixed ? sizeof(float) : sizeof(double))) + (size_t)nb / 4 * per_run;
}

cudaError_t build_history_runs(int E, int K, int kr, const std::vector<int64_t>& kptr, const int64_t* d_kptr,
                               const uint32_t* d_col, const void* d_val, int64_t nnz, bool mixed, HistoryRuns& out,
                               cudaStream_t s)
{
    out = HistoryRuns{};
    if (kr < 1 || kr > K) return cudaSuccess;
    std::vector<int64_t> qoff(E + 1, 0);
    for (int r = 0; r < E; ++r)
        qoff[r + 1] = qoff[r] + kptr[(size_t)r * (K + 1) + K] - kptr[(size_t)r * (K + 1) + kr - 1];
    const int64_t nb = qoff[E];
    if (nb <= 0 || nb > INT_MAX || nnz >= (int64_t)UINT_MAX) return cudaSuccess;
    const int n = (int)nb;
    Tmp d_qoff, k1, k2, i1, i2, flag, runid;
    RUN_TRY(d_qoff.alloc(sizeof(int64_t) * (E + 1)));
    RUN_TRY(cudaMemcpyAsync(d_qoff.p, qoff.data(), sizeof(int64_t) * (E + 1), cudaMemcpyHostToDevice, s));
    RUN_TRY(k1.alloc(8 * (size_t)nb));
    RUN_TRY(k2.alloc(8 * (size_t)nb));
    RUN_TRY(i1.alloc(4 * (size_t)nb));
    RUN_TRY(i2.alloc(4 * (size_t)nb));
    run_keys_kernel<<<(E + 7) / 8, 256, 0, s>>>(E, K, kr, d_kptr, d_qoff.as<int64_t>(), d_col,
                                               k1.as<unsigned long long>(), i1.as<uint32_t>());
    RUN_TRY(cudaGetLastError());
    const int end_bit = 32 + bits_for((unsigned long long)E);
    size_t sort_bytes = 0;
    RUN_TRY(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, k1.as<unsigned long long>(),
                                            k2.as<unsigned long long>(), i1.as<uint32_t>(), i2.as<uint32_t>(), n, 0,
                                            end_bit, s));
    {
        Tmp temp;
        RUN_TRY(temp.alloc(sort_bytes));
        RUN_TRY(cub::DeviceRadixSort::SortPairs(temp.p, sort_bytes, k1.as<unsigned long long>(),
                                                k2.as<unsigned long long>(), i1.as<uint32_t>(), i2.as<uint32_t>(), n,
                                                0, end_bit, s));
    }
    // k2 / i2: blocks in (row, type, column, k) order
    RUN_TRY(flag.alloc(4 * (size_t)nb));
    RUN_TRY(runid.alloc(4 * (size_t)nb));
    run_flags_kernel<<<1184, 256, 0, s>>>(nb, k2.as<unsigned long long>(), flag.as<int>());
    RUN_TRY(cudaGetLastError());
    size_t scan_bytes = 0;
    RUN_TRY(cub::DeviceScan::InclusiveSum(nullptr, scan_bytes, flag.as<int>(), runid.as<int>(), n, s));
    {
        Tmp temp;
        RUN_TRY(temp.alloc(scan_bytes));
        RUN_TRY(cub::DeviceScan::InclusiveSum(temp.p, scan_bytes, flag.as<int>(), runid.as<int>(), n, s));
    }
    int n_runs = 0;
    RUN_TRY(cudaMemcpyAsync(&n_runs, runid.as<int>() + (nb - 1), sizeof(int), cudaMemcpyDeviceToHost, s));
    RUN_TRY(cudaStreamSynchronize(s));
    k1.release();  // not needed past the sort
    i1.release();
    Tmp start, okey1, okey2, ov1, ov2, lens, offs;
    RUN_TRY(start.alloc(4 * (size_t)n_runs));
    run_starts_kernel<<<1184, 256, 0, s>>>(nb, flag.as<int>(), runid.as<int>(), start.as<int>());
    RUN_TRY(cudaGetLastError());
    RUN_TRY(okey1.alloc(8 * (size_t)n_runs));
    RUN_TRY(okey2.alloc(8 * (size_t)n_runs));
    RUN_TRY(ov1.alloc(4 * (size_t)n_runs));
    RUN_TRY(ov2.alloc(4 * (size_t)n_runs));
    // runs per row (E + 1 entries, the last one stays zero)
    Tmp rcnt32;
    RUN_TRY(rcnt32.alloc(sizeof(int) * (E + 1)));
    RUN_TRY(cudaMemsetAsync(rcnt32.p, 0, sizeof(int) * (E + 1), s));
    run_order_keys_kernel<<<1184, 256, 0, s>>>(n_runs, nb, start.as<int>(), k2.as<unsigned long long>(),
                                               okey1.as<unsigned long long>(), ov1.as<int>(), rcnt32.as<int>());
    RUN_TRY(cudaGetLastError());
    const int end2 = 16 + bits_for((unsigned long long)E);
    RUN_TRY(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, okey1.as<unsigned long long>(),
                                            okey2.as<unsigned long long>(), ov1.as<int>(), ov2.as<int>(), n_runs, 0,
                                            end2, s));
    {
        Tmp temp;
        RUN_TRY(temp.alloc(sort_bytes));
        RUN_TRY(cub::DeviceRadixSort::SortPairs(temp.p, sort_bytes, okey1.as<unsigned long long>(),
                                                okey2.as<unsigned long long>(), ov1.as<int>(), ov2.as<int>(), n_runs,
                                                0, end2, s));
    }
    RUN_TRY(lens.alloc(8 * (size_t)n_runs));
    RUN_TRY(offs.alloc(8 * (size_t)n_runs));
    run_lengths_kernel<<<1184, 256, 0, s>>>(n_runs, okey2.as<unsigned long long>(), lens.as<int64_t>());
    RUN_TRY(cudaGetLastError());
    RUN_TRY(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, lens.as<int64_t>(), offs.as<int64_t>(), n_runs, s));
    {
        Tmp temp;
        RUN_TRY(temp.alloc(scan_bytes));
        RUN_TRY(cub::DeviceScan::ExclusiveSum(temp.p, scan_bytes, lens.as<int64_t>(), offs.as<int64_t>(), n_runs,
                                              s));
    }
    // row pointers: exclusive sum of the per-row run counts (E + 1 entries,
    // the last count is zero)
    Tmp ptr32;
    RUN_TRY(ptr32.alloc(sizeof(int) * (E + 1)));
    RUN_TRY(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, rcnt32.as<int>(), ptr32.as<int>(), E + 1, s));
    {
        Tmp temp;
        RUN_TRY(temp.alloc(scan_bytes));
        RUN_TRY(cub::DeviceScan::ExclusiveSum(temp.p, scan_bytes, rcnt32.as<int>(), ptr32.as<int>(), E + 1, s));
    }
    std::vector<int> hp(E + 1);
    RUN_TRY(cudaMemcpyAsync(hp.data(), ptr32.p, sizeof(int) * (E + 1), cudaMemcpyDeviceToHost, s));
    RUN_TRY(cudaStreamSynchronize(s));
    std::vector<int64_t> hp64(hp.begin(), hp.end());
    const size_t vs = mixed ? sizeof(float) : sizeof(double);
    RUN_TRY(cudaMalloc(reinterpret_cast<void**>(&out.ptr), sizeof(int64_t) * (E + 1)));
    RUN_TRY(cudaMemcpyAsync(out.ptr, hp64.data(), sizeof(int64_t) * (E + 1), cudaMemcpyHostToDevice, s));
    RUN_TRY(cudaMalloc(reinterpret_cast<void**>(&out.meta), sizeof(uint2) * (size_t)n_runs));
    RUN_TRY(cudaMalloc(reinterpret_cast<void**>(&out.off), sizeof(int64_t) * (size_t)n_runs));
    RUN_TRY(cudaMalloc(&out.val, vs * 9 * (size_t)nb));
    const int gb = (int)(((int64_t)n_runs * 32 + 255) / 256);
    if (mixed)
        run_gather_kernel<float><<<gb, 256, 0, s>>>(n_runs, nb, nnz, ov2.as<int>(), start.as<int>(),
                                                    lens.as<int64_t>(), offs.as<int64_t>(),
                                                    k2.as<unsigned long long>(), i2.as<uint32_t>(),
                                                    static_cast<const float*>(d_val), out.meta, out.off,
                                                    static_cast<float*>(out.val));
    else
        run_gather_kernel<double><<<gb, 256, 0, s>>>(n_runs, nb, nnz, ov2.as<int>(), start.as<int>(),
                                                     lens.as<int64_t>(), offs.as<int64_t>(),
                                                     k2.as<unsigned long long>(), i2.as<uint32_t>(),
                                                     static_cast<const double*>(d_val), out.meta, out.off,
                                                     static_cast<double*>(out.val));
    RUN_TRY(cudaGetLastError());
    RUN_TRY(cudaStreamSynchronize(s));
    out.nb = nb;
    out.runs = n_runs;
    out.kr = kr;
    return cudaSuccess;
}

cudaError_t exclusive_sum(const int64_t* in, int64_t* out, int64_t n, cudaStream_t s)
{
    size_t bytes = 0;
    RUN_TRY(cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, n, s));
    Tmp temp;
    RUN_TRY(temp.alloc(bytes));
    return cub::DeviceScan::ExclusiveSum(temp.p, bytes, in, out, n, s);
}

size_t history_groups_bytes(int64_t nb, bool mixed)
{
    // per block: sort keys and indices (double-buffered), flags, segment ids and
    // the radix sort's scratch; per segment (about 70 blocks; counted as 16)
    // start, order keys and values (double-buffered), length, offset, header;
    // the matrices at the least fill accepted
    const size_t per_block = 2 * 8 + 2 * 4 + 4 + 4 + 16, per_seg = 4 + 2 * 8 + 2 * 4 + 8 + 8 + 8 + 8;
    return (size_t)nb * per_block + (size_t)((double)nb * 9.0 * (mixed ? sizeof(float) : sizeof(double)) / kGroupFillMin) +
           (size_t)nb / 16 * per_seg;
}

cudaError_t build_history_groups(int E, int K, int kr, const std::vector<int32_t>& place, int groups,
                                 const std::vector<int64_t>& kptr, const int64_t* d_kptr, const uint32_t* d_col,
                                 const void* d_val, int64_t nnz, bool mixed, HistoryGroups& out, cudaStream_t s)
{
    out = HistoryGroups{};
    if (kr < 1 || kr > K) return cudaSuccess;
    std::vector<int64_t> qoff(E + 1, 0);
    for (int r = 0; r < E; ++r)
        qoff[r + 1] = qoff[r] + kptr[(size_t)r * (K + 1) + K] - kptr[(size_t)r * (K + 1) + kr - 1];
    const int64_t nb = qoff[E];
    if (nb <= 0 || nb > INT_MAX || nnz >= (int64_t)UINT_MAX) return cudaSuccess;
    const int n = (int)nb;
    Tmp d_qoff, d_place, k1, k2, i1, i2, flag, segid;
    RUN_TRY(d_qoff.alloc(sizeof(int64_t) * (E + 1)));
    RUN_TRY(cudaMemcpyAsync(d_qoff.p, qoff.data(), sizeof(int64_t) * (E + 1), cudaMemcpyHostToDevice, s));
    RUN_TRY(d_place.alloc(sizeof(int32_t) * E));
    RUN_TRY(cudaMemcpyAsync(d_place.p, place.data(), sizeof(int32_t) * E, cudaMemcpyHostToDevice, s));
    RUN_TRY(k1.alloc(8 * (size_t)nb));
    RUN_TRY(k2.alloc(8 * (size_t)nb));
    RUN_TRY(i1.alloc(4 * (size_t)nb));
    RUN_TRY(i2.alloc(4 * (size_t)nb));
    group_keys_kernel<<<(E + 7) / 8, 256, 0, s>>>(E, K, kr, d_place.as<int32_t>(), d_kptr, d_qoff.as<int64_t>(),
                                                 d_col, k1.as<unsigned long long>(), i1.as<uint32_t>());
    RUN_TRY(cudaGetLastError());
    const int end_bit = 35 + bits_for((unsigned long long)groups);
    size_t bytes = 0;
    RUN_TRY(cub::DeviceRadixSort::SortPairs(nullptr, bytes, k1.as<unsigned long long>(), k2.as<unsigned long long>(),
                                            i1.as<uint32_t>(), i2.as<uint32_t>(), n, 0, end_bit, s));
    {
        Tmp temp;
        RUN_TRY(temp.alloc(bytes));
        RUN_TRY(cub::DeviceRadixSort::SortPairs(temp.p, bytes, k1.as<unsigned long long>(),
                                                k2.as<unsigned long long>(), i1.as<uint32_t>(), i2.as<uint32_t>(), n,
                                                0, end_bit, s));
    }
    RUN_TRY(flag.alloc(4 * (size_t)nb));
    RUN_TRY(segid.alloc(4 * (size_t)nb));
    group_flags_kernel<<<1184, 256, 0, s>>>(nb, k2.as<unsigned long long>(), flag.as<int>());
    RUN_TRY(cudaGetLastError());
    RUN_TRY(cub::DeviceScan::InclusiveSum(nullptr, bytes, flag.as<int>(), segid.as<int>(), n, s));
    {
        Tmp temp;
        RUN_TRY(temp.alloc(bytes));
        RUN_TRY(cub::DeviceScan::InclusiveSum(temp.p, bytes, flag.as<int>(), segid.as<int>(), n, s));
    }
    int n_segs = 0;
    RUN_TRY(cudaMemcpyAsync(&n_segs, segid.as<int>() + (nb - 1), sizeof(int), cudaMemcpyDeviceToHost, s));
    RUN_TRY(cudaStreamSynchronize(s));
    k1.release();  // not needed past the sort
    i1.release();
    Tmp start, okey1, okey2, ov1, ov2, lens, offs, gcnt, gptr;
    RUN_TRY(start.alloc(4 * (size_t)n_segs));
    run_starts_kernel<<<1184, 256, 0, s>>>(nb, flag.as<int>(), segid.as<int>(), start.as<int>());
    RUN_TRY(cudaGetLastError());
    RUN_TRY(okey1.alloc(8 * (size_t)n_segs));
    RUN_TRY(okey2.alloc(8 * (size_t)n_segs));
    RUN_TRY(ov1.alloc(4 * (size_t)n_segs));
    RUN_TRY(ov2.alloc(4 * (size_t)n_segs));
    RUN_TRY(gcnt.alloc(sizeof(int) * (groups + 1)));
    RUN_TRY(gptr.alloc(sizeof(int) * (groups + 1)));
    RUN_TRY(cudaMemsetAsync(gcnt.p, 0, sizeof(int) * (groups + 1), s));
    group_order_keys_kernel<<<1184, 256, 0, s>>>(n_segs, nb, start.as<int>(), k2.as<unsigned long long>(),
                                                 okey1.as<unsigned long long>(), ov1.as<int>(), gcnt.as<int>());
    RUN_TRY(cudaGetLastError());
    const int end2 = 16 + bits_for((unsigned long long)groups);
    RUN_TRY(cub::DeviceRadixSort::SortPairs(nullptr, bytes, okey1.as<unsigned long long>(),
                                            okey2.as<unsigned long long>(), ov1.as<int>(), ov2.as<int>(), n_segs, 0,
                                            end2, s));
    {
        Tmp temp;
        RUN_TRY(temp.alloc(bytes));
        RUN_TRY(cub::DeviceRadixSort::SortPairs(temp.p, bytes, okey1.as<unsigned long long>(),
                                                okey2.as<unsigned long long>(), ov1.as<int>(), ov2.as<int>(), n_segs,
                                                0, end2, s));
    }
    RUN_TRY(lens.alloc(8 * (size_t)(n_segs + 1)));
    RUN_TRY(offs.alloc(8 * (size_t)(n_segs + 1)));
    RUN_TRY(cudaMemsetAsync(lens.p, 0, 8 * (size_t)(n_segs + 1), s));
    group_steps_kernel<<<1184, 256, 0, s>>>(n_segs, okey2.as<unsigned long long>(), lens.as<int64_t>());
    RUN_TRY(cudaGetLastError());
    RUN_TRY(cub::DeviceScan::ExclusiveSum(nullptr, bytes, lens.as<int64_t>(), offs.as<int64_t>(), n_segs + 1, s));
    {
        Tmp temp;
        RUN_TRY(temp.alloc(bytes));
        RUN_TRY(cub::DeviceScan::ExclusiveSum(temp.p, bytes, lens.as<int64_t>(), offs.as<int64_t>(), n_segs + 1, s));
    }
    RUN_TRY(cub::DeviceScan::ExclusiveSum(nullptr, bytes, gcnt.as<int>(), gptr.as<int>(), groups + 1, s));
    {
        Tmp temp;
        RUN_TRY(temp.alloc(bytes));
        RUN_TRY(cub::DeviceScan::ExclusiveSum(temp.p, bytes, gcnt.as<int>(), gptr.as<int>(), groups + 1, s));
    }
    std::vector<int> hp(groups + 1);
    int64_t steps = 0;
    RUN_TRY(cudaMemcpyAsync(hp.data(), gptr.p, sizeof(int) * (groups + 1), cudaMemcpyDeviceToHost, s));
    RUN_TRY(cudaMemcpyAsync(&steps, offs.as<int64_t>() + n_segs, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    RUN_TRY(cudaStreamSynchronize(s));
    if ((double)nb * 9.0 < kGroupFillMin * 96.0 * (double)steps) return cudaSuccess;
    std::vector<int64_t> hp64(hp.begin(), hp.end());
    RUN_TRY(cudaMalloc(reinterpret_cast<void**>(&out.ptr), sizeof(int64_t) * (groups + 1)));
    RUN_TRY(cudaMemcpyAsync(out.ptr, hp64.data(), sizeof(int64_t) * (groups + 1), cudaMemcpyHostToDevice, s));
    RUN_TRY(cudaMalloc(reinterpret_cast<void**>(&out.meta), sizeof(uint2) * (size_t)n_segs));
    RUN_TRY(cudaMalloc(reinterpret_cast<void**>(&out.off), sizeof(int64_t) * (size_t)n_segs));
    const size_t val_bytes = (mixed ? sizeof(float) : sizeof(double)) * 96 * (size_t)steps;
    RUN_TRY(cudaMalloc(&out.val, val_bytes));
    RUN_TRY(cudaMemsetAsync(out.val, 0, val_bytes, s));
    const int gb = (int)(((int64_t)n_segs * 32 + 255) / 256);
    int infinite = 0;
    int* d_infinite = gcnt.as<int>();  // free again
    RUN_TRY(cudaMemsetAsync(d_infinite, 0, sizeof(int), s));
    if (mixed)
        group_scatter_kernel<float><<<gb, 256, 0, s>>>(n_segs, nb, nnz, ov2.as<int>(), start.as<int>(),
                                                       okey2.as<unsigned long long>(), offs.as<int64_t>(),
                                                       k2.as<unsigned long long>(), i2.as<uint32_t>(),
                                                       static_cast<const float*>(d_val), out.meta, out.off,
                                                       static_cast<float*>(out.val), d_infinite);
    else
        group_scatter_kernel<double><<<gb, 256, 0, s>>>(n_segs, nb, nnz, ov2.as<int>(), start.as<int>(),
                                                        okey2.as<unsigned long long>(), offs.as<int64_t>(),
                                                        k2.as<unsigned long long>(), i2.as<uint32_t>(),
                                                        static_cast<const double*>(d_val), out.meta, out.off,
                                                        static_cast<double*>(out.val), d_infinite);
    RUN_TRY(cudaGetLastError());
    RUN_TRY(cudaMemcpyAsync(&infinite, d_infinite, sizeof(int), cudaMemcpyDeviceToHost, s));
    RUN_TRY(cudaStreamSynchronize(s));
    if (infinite) return cudaSuccess;
    out.steps = steps;
    out.segments = n_segs;
    out.kr = kr;
    return cudaSuccess;
}

}  // namespace tdbem
