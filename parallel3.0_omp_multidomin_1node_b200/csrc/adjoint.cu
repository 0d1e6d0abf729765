// Device-side set-up of the adjoint march: the stacked history blocks
// regrouped by (type, column) and step for the transposed convolution
// (adj_history_kernel), by a stable radix sort so that each group keeps the
// ascending-row order of the stacked matrix.
#include <cub/cub.cuh>

#include "march.cuh"
#include "tdbem_common.cuh"

namespace tdbem {

namespace {

// One warp per equation row: group key of every block of the row,
// group = (type * nh + column) * (K + 1) + k, its row, and the group sizes.
__global__ void hist_keys_kernel(int E, int K, int nh, const int64_t* kptr, const uint32_t* hcol, uint32_t* key,
                                 uint32_t* idx, int32_t* rowof, unsigned long long* counts)
{
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= E) return;
    const int64_t b = kptr[(int64_t)row * (K + 1)], e = kptr[(int64_t)row * (K + 1) + K];
    for (int64_t j = b + lane; j < e; j += 32) {
        const uint32_t c = hcol[j];
        const uint32_t seg = ((c >> 20) & 1u) * (uint32_t)nh + (c & 0xFFFFFu);
        const uint32_t g = seg * (uint32_t)(K + 1) + (c >> 21);
        key[j] = g;
        idx[j] = (uint32_t)j;
        rowof[j] = row;
        atomicAdd(counts + g, 1ull);
    }
}

// Gather rows and values in group order: k << 21 | row, and tiles of 32 blocks in
// 9 planes.
__global__ void hist_gather_kernel(int64_t nnz, int K, const uint32_t* key, const uint32_t* order, const int32_t* rowof,
                                   const double* hval, uint32_t* trow, double* tval)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = order[i];
        trow[i] = (key[i] % (uint32_t)(K + 1)) << 21 | (uint32_t)rowof[j];
#pragma unroll
        for (int q = 0; q < 9; ++q) tval[(i >> 5) * 288 + 32 * q + (i & 31)] = hval[(int64_t)q * nnz + j];
    }
}

struct Scratch {
    void* p = nullptr;
    ~Scratch()
    {
        if (p) cudaFree(p);
    }
    cudaError_t alloc(size_t bytes) { return cudaMalloc(&p, bytes ? bytes : 1); }
};

#define ADJ_TRY(x)                                 \
    do {                                           \
        const cudaError_t e_ = (x);                \
        if (e_ != cudaSuccess) return e_;          \
    } while (0)

}  // namespace

cudaError_t adjoint_history_groups(int E, int K, int nh, int64_t nnz, const int64_t* kptr, const uint32_t* hcol,
                                   const double* hval, int64_t* tptr, uint32_t* trow, double* tval, cudaStream_t s)
{
    const int64_t groups = 2LL * nh * (K + 1);
    if (nnz >= (1LL << 31) || groups >= (1LL << 31) || E > (1 << 21)) return cudaErrorInvalidValue;
    int end_bit = 1;
    while (end_bit < 32 && (1LL << end_bit) < groups) ++end_bit;
    const size_t n = (size_t)std::max<int64_t>(nnz, 1);
    Scratch keys, keys2, idx, idx2, rowof, counts;
    ADJ_TRY(keys.alloc(4 * n));
    ADJ_TRY(keys2.alloc(4 * n));
    ADJ_TRY(idx.alloc(4 * n));
    ADJ_TRY(idx2.alloc(4 * n));
    ADJ_TRY(rowof.alloc(4 * n));
    ADJ_TRY(counts.alloc(8 * (size_t)groups));
    auto* k1 = static_cast<uint32_t*>(keys.p);
    auto* k2 = static_cast<uint32_t*>(keys2.p);
    auto* i1 = static_cast<uint32_t*>(idx.p);
    auto* i2 = static_cast<uint32_t*>(idx2.p);
    auto* cnt = static_cast<unsigned long long*>(counts.p);
    ADJ_TRY(cudaMemsetAsync(cnt, 0, 8 * (size_t)groups, s));
    hist_keys_kernel<<<ceil_div(E, 8), 256, 0, s>>>(E, K, nh, kptr, hcol, k1, i1, static_cast<int32_t*>(rowof.p), cnt);
    ADJ_TRY(cudaGetLastError());
    // group ends (the layout adj_history_kernel reads)
    size_t scan_bytes = 0, sort_bytes = 0;
    ADJ_TRY(cub::DeviceScan::InclusiveSum(nullptr, scan_bytes, cnt, reinterpret_cast<unsigned long long*>(tptr),
                                          (int)groups, s));
    ADJ_TRY(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, k1, k2, i1, i2, (int)nnz, 0, end_bit, s));
    Scratch temp;
    ADJ_TRY(temp.alloc(std::max(scan_bytes, sort_bytes)));
    ADJ_TRY(cub::DeviceScan::InclusiveSum(temp.p, scan_bytes, cnt, reinterpret_cast<unsigned long long*>(tptr),
                                          (int)groups, s));
    if (nnz > 0) {
        ADJ_TRY(cub::DeviceRadixSort::SortPairs(temp.p, sort_bytes, k1, k2, i1, i2, (int)nnz, 0, end_bit, s));
        const int grid = (int)std::min<int64_t>(ceil_div(nnz, 256), 8 * 148);
        hist_gather_kernel<<<grid, 256, 0, s>>>(nnz, K, k2, i2, static_cast<int32_t*>(rowof.p), hval, trow, tval);
        ADJ_TRY(cudaGetLastError());
    }
    // the scratch is released when this returns: wait for its last use
    return cudaStreamSynchronize(s);
}

}  // namespace tdbem

namespace tdbem {

namespace {

// Cotangent of element i's displacement (which = 0) or traction (1) reference at
// step n in its local frame: that of the global-frame output plus the history
// adjoint, back through LocToAbs.
__device__ __forceinline__ void reference_cotangent(const AdjWriteBack& a, int n, int64_t i, int which, double (&cl)[3])
{
    const int64_t o = ((int64_t)n * a.E + i) * 3;
    const double* cot = which ? a.cot_lt : a.cot_lu;
    double cg[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) cg[c] = cot ? cot[o + c] : 0.0;
    if (a.adj && a.hist_owner[i]) {
        const double* adj = a.adj + 3 * ((which ? (int64_t)a.nh : 0) + a.hist_block[i]);
        const double sg = which ? a.ht_sign[i] : a.hu_sign[i];
#pragma unroll
        for (int c = 0; c < 3; ++c) cg[c] += sg * adj[c];
    }
    const double* F = a.trans + 9 * i;  // gu = F^T l  ->  dl = F dgu
#pragma unroll
    for (int j = 0; j < 3; ++j) cl[j] = F[3 * j] * cg[0] + F[3 * j + 1] * cg[1] + F[3 * j + 2] * cg[2];
}

// Transposed write-back of reverse step n, a thread per element and perm (A'
// column) row t: prescribed references of element t add to gk, and the unknown of
// row t sums its (at most two) references in element order into the right-hand
// side of the transposed solve.  The solve's status word is cleared here, and the
// solve sets up beside this launch.
__global__ void adj_writeback_kernel(AdjWriteBack a, int n, const int32_t* unk_src, const int32_t* unk_of, double* gp,
                                     int* status)
{
    cudaTriggerProgrammaticLaunchCompletion();
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) *status = 0;
    if (t >= a.E) return;
    for (int which = 0; which < 2; ++which) {
        if (!(which ? a.tref_known[t] : a.uref_known[t])) continue;
        double cl[3];
        reference_cotangent(a, n, t, which, cl);
        const double sg = which ? a.tref_sign[t] : a.uref_sign[t];
        double* g = a.gk + ((int64_t)n * a.E + t) * 3;
        for (int c = 0; c < 3; ++c) g[c] += sg * cl[c];
    }
    const int64_t u = unk_of[t];
    double g[3] = {0.0, 0.0, 0.0};
    for (int k = 0; k < 2; ++k) {
        const int src = unk_src[2 * u + k];
        if (src < 0) continue;
        const int64_t i = src >> 1;
        const int which = src & 1;
        double cl[3];
        reference_cotangent(a, n, i, which, cl);
        const double sg = which ? a.tref_sign[i] : a.uref_sign[i];
        const double* T = a.itf_trans + 9 * i;
        for (int j = 0; j < 3; ++j) g[j] += sg * (T[j] * cl[0] + T[3 + j] * cl[1] + T[6 + j] * cl[2]);
    }
    for (int c = 0; c < 3; ++c) gp[3 * t + c] = g[c];
}

// After the solve of step n: lam_n (equation rows) from x (perm rows), the sums
// com_m = lam_{m-1} + 2 lam_m + lam_{m+1} of what is known by now, and KnownM^T
// lam_n into the prescribed-value gradient, a warp per known block.
__global__ void __launch_bounds__(256) adj_finish_kernel(AdjFinish a, int n, int rows_ctas)
{
    const int64_t per = 3LL * a.E;
    if ((int)blockIdx.x < rows_ctas) {
        const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
        if (t >= per) return;
        const double l = a.x[3LL * a.perm_of_row[t / 3] + t % 3];
        a.lam[n * per + t] = l;
        a.com[n * per + t] = 2.0 * l + a.lam[(n + 1) * per + t];
        a.com[(n + 1) * per + t] += l;
        return;
    }
    const int kb = ((int)blockIdx.x - rows_ctas) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (kb >= a.n_known) return;
    double acc[3] = {0.0, 0.0, 0.0};
    for (int j = a.kt_ptr[kb] + lane; j < a.kt_ptr[kb + 1]; j += 32) {
        const double* B = a.k_val + 9 * (int64_t)a.kt_blk[j];
        const double* l = a.x + 3LL * a.perm_of_row[a.kt_row[j]];
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] += B[c] * l[0] + B[3 + c] * l[1] + B[6 + c] * l[2];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    if (lane == 0) {
        double* g = a.gk + ((int64_t)n * a.E + a.known_elem[kb]) * 3;
        for (int c = 0; c < 3; ++c) g[c] += a.known_sign[kb] * acc[c];
    }
}

// Step 0 of the gradient: bd[0] is the prescribed value converted to the
// global frame (lu for BCID 123, lt for 456), so its cotangent goes back
// through the frame: gk[0][i] = F_i^T-applied cotangent.
__global__ void adj_step0_kernel(int E, const double* trans, const int32_t* bcid, const double* cot_lu,
                                 const double* cot_lt, double* gk)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= E) return;
    const double* c = bcid[i] == 456 ? cot_lt : cot_lu;
    if (!c) return;
    const double* F = trans + 9 * i;
    for (int j = 0; j < 3; ++j)
        gk[3 * i + j] += F[3 * j] * c[3 * i] + F[3 * j + 1] * c[3 * i + 1] + F[3 * j + 2] * c[3 * i + 2];
}

}  // namespace

cudaError_t adjoint_step0(int E, const double* trans, const int32_t* bcid, const double* cot_lu, const double* cot_lt,
                          double* gk, cudaStream_t s)
{
    adj_step0_kernel<<<ceil_div(E, 128), 128, 0, s>>>(E, trans, bcid, cot_lu, cot_lt, gk);
    return cudaGetLastError();
}

cudaError_t adjoint_writeback(const AdjWriteBack& a, int n, const int32_t* unk_src, const int32_t* unk_of, double* gp,
                              int* status, cudaStream_t s)
{
    adj_writeback_kernel<<<ceil_div(a.E, 64), 64, 0, s>>>(a, n, unk_src, unk_of, gp, status);
    return cudaGetLastError();
}

cudaError_t adjoint_finish(const AdjFinish& a, int n, cudaStream_t s)
{
    const int rows = ceil_div(3LL * a.E, 256);
    adj_finish_kernel<<<rows + ceil_div(a.n_known, 8), 256, 0, s>>>(a, n, rows);
    return cudaGetLastError();
}

}  // namespace tdbem
