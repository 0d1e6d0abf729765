// Time-march kernels: history right-hand side (batched over load cases),
// cluster-resident GMRES and the boundary write-back (host-side launch
// wrappers).
#pragma once

#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

namespace tdbem {

// Everything the per-step kernels read or write, all device pointers.
// Index spaces: "perm" = leaf order of the mapped-leaf preconditioner
// (row p is equation row row_of[p]; unknown p is unknown block
// unk_of[p] = preferred unknown of row_of[p]), so the preconditioner is
// block diagonal and every GMRES CTA owns one contiguous perm range.
// Vectors over the 3E unknowns are stored [3E][R], load case fastest.
struct RowLeaf {
    int64_t off;    // of the leaf's dense block
    int32_t begin;  // its first perm row
    int32_t n3;     // 3 x its rows
};

struct MarchData {
    int E;            // elements = equation rows = unknown blocks
    int n_known;      // known blocks
    int nh;           // history blocks
    int K;            // history steps
    int R;            // load cases
    int nstep;
    int SW;           // W-ring slots (K + 1)
    int mixed;        // FP32 history + mixed-precision GMRES
    int k_lo, k_hi;   // right-hand side split: k in [k_lo, k_hi] (see march_step)
    // stacked history matrix: per equation row, blocks of k = 1..K, each k
    // with MGS_k (type 1, traction history) then MTS_k (type 0, negated)
    const int64_t* h_kptr;  // [E][K+1]: entry k = first block with step > k; entry 0 = row start
    const uint32_t* h_col;  // packed (k << 21) | (type << 20) | history column
    const double* h_val;    // SoA [9][nnz]
    const float* h_val32;   // SoA [9][nnz] (mixed)
    int64_t h_nnz;
    // head pass of one load case: the blocks of the first steps (below kr, or 1 and
    // 2) of each perm row again, in tiles of 32 columns and 9 planes of 32 values
    // (head_tile_bytes), zero-padded; null: none
    const int32_t* hd_ptr;  // [E+1] first tile of each perm row
    const unsigned char* hd_tile;
    // run layout of the blocks of steps k >= kr = 2T + 1, for the T-step
    // history pass: per equation row, runs of one (type, column) pair over
    // consecutive steps, longest first; kr = 0 when there is none
    const int64_t* r_ptr;   // [E+1] first run of each equation row
    const uint2* r_meta;    // x = (type << 20) | column, y = (first step << 16) | length
    const int64_t* r_off;   // block of the run's first step in r_val / r_val32
    const double* r_val;    // SoA [9][r_nb] (FP64 mode)
    const float* r_val32;   // SoA [9][r_nb] (mixed)
    int64_t r_nb;
    int kr;
    // group layout of the same blocks, instead of the run layout when there are
    // groups (8 or more load cases): per group of 8 rows, segments of one (type,
    // column) pair over consecutive steps, longest first; a segment of n steps is
    // a 24 x 3n matrix (zero where a row has no block) in fragments of 8 x 4:
    // [ceil(3n / 4)][3][lane]
    int hg_n, hg_split;     // groups, CTAs per group
    const int64_t* hg_ptr;  // [hg_n+1] first segment of each group
    const uint2* hg_meta;   // x = (type << 20) | column, y = (first step << 16) | length
    const int64_t* hg_off;  // first of each segment's ceil(3n / 4) contraction steps
    const void* hg_val;     // [contraction step][3][32], FP32 (mixed) or FP64
    const int32_t* hg_rows; // [hg_n][8] perm rows, -1 past the end
    // KnownM (natural rows), known blocks map to (element, sign)
    const int32_t* k_rp;
    const int32_t* k_col;
    const double* k_val;    // [nnz][9]
    const int32_t* known_elem;
    const double* known_sign;
    const int32_t* k_elem;  // per KnownM block: known_elem of its column
    const double* k_sgn;    // per KnownM block: known_sign of its column
    // permuted system matrix A' and preconditioner, laid out for the GMRES
    // cluster (GmresTiles): CTA c owns the perm rows cta_row[c] .. cta_row[c+1]
    // and the slices (4 rows each) g_cs[c] .. g_cs[c+1]; slice s starts at tile
    // g_sp[s].x of 4 rows x 8 blocks, g_sp[s].y blocks in its longest row, its
    // rows (within the range, -1 past the end) at g_rows[4 s]; a tile holds 32 columns and 9 planes of 32 values, padded with zero blocks.
    // Columns are rows of the CTA's product vector (g_col): its own rows, then
    // from dsm_rows on the g_halo[c] rows of other CTAs that its rows use, which
    // their owners send (g_send_ptr[c] .. of g_send: x = peer << 24 | own row,
    // y = row there); or perm rows (g_colg)
    const int32_t* cta_row;
    const int32_t* g_cs;
    const int2* g_sp;
    const int32_t* g_rows;
    const int32_t* g_halo;
    const int32_t* g_send_ptr;
    const int2* g_send;
    const int32_t* g_col;
    const int32_t* g_colg;
    const double* g_val;
    const float* g_val32;
    const int32_t* row_of;  // perm -> equation row
    const int32_t* perm_of_unk; // unknown block -> perm
    const RowLeaf* row_leaf;  // leaf of each perm row
    const double* pinv;       // dense (3L x 3L) leaf inverses, column-major
    const float* pinv32;
    const double* pmat;       // the leaves' dense blocks, column-major
    const double* minv;       // largest Frobenius norm of a leaf inverse
    int own_rows;             // rows of the largest owned range
    int dsm_rows;             // row capacity of the shared-memory vectors; 0 = vectors in global memory
    int halo_rows;            // largest g_halo
    int leaf_max;             // values of the largest CTA's leaf inverses
    int leaf_cap;             // room for cached leaf inverses, in values (0: not cached), and
    int vcap;                 // basis vectors kept in shared memory; both set at launch
    // per-element write-back data
    const int64_t* uref_block; const double* uref_sign; const int32_t* uref_known;
    const int64_t* tref_block; const double* tref_sign; const int32_t* tref_known;
    const int64_t* hist_block; const double* hu_sign; const double* ht_sign;
    const int32_t* hist_owner;  // 1 when the element feeds the history state (not an interface B side)
    const double* itf_trans;    // [E][9] local transform of interface B sides (identity elsewhere)
    const double* trans;        // [E][9] element frames
    const int32_t* bcid;
    const int32_t* itf_a;       // [E] A-side element of an interface's B-side element, else -1
    const double* itf_asign;    // [E] its normal sign
    // state
    double* xring;    // [3][2][nh][3][R] physical history states X_s (type 0 = U, 1 = T)
    double* wring;    // [SW][2][nh][3][R] combined history vectors
    double* bulk;     // [8][3E][R] part of the right-hand side of step s at s % 8 computed
                      // ahead beside GMRES: history k >= 3 (k >= kr with the run layout), KnownM
    double* b;        // [3E][R] perm right-hand side
    // GMRES: `groups` clusters, cluster g solves load cases [g*Rg, (g+1)*Rg)
    // with private Krylov storage ([3E][Rg] per vector) at offset g
    int groups;
    double* x;        // [groups][3E][Rg] perm solution
    double* xold;     // [groups][3E][Rg] solution of the step before (mixed-mode start vector), or null
    double* V;        // [groups][restart+1][3E][Rg] basis vectors beyond vcap
    // vectors of the global-memory form (dsm_rows = 0): solution, product, work
    double* rv;       // [groups][3E][Rg]
    double* aw;       // [groups][3E][Rg]
    double* u;        // [groups][3E][Rg]
    double* givens;   // [groups][C][Rg] small arrays of gmres_givens_doubles(restart) each
    int* status;      // [0] abort, [1] a combined history vector is not finite (with groups)
    // [nstep+4][5] device clock (ns): start of the step's head pass, start and end of
    // its GMRES, start and end of the history pass launch kept under it; or null
    unsigned long long* stamps;
    int* step_flags;  // [nstep][R][3] flag, refinements, inner iterations
    double* audit;    // [nstep][2] max interface jump, balance
    const double* known_lu; // [R][nstep+1][E][3] device input
    double* out_lu;          // [R][nstep+1][E][3]
    double* out_lt;
    double* rec_rhs;         // optional [nstep][E*3] (load 0, natural row order)
    double* rec_x;           // optional [nstep][E*3] (load 0, natural unknown order)
    int restart;
    double tol;
    int cluster;             // CTAs in the GMRES cluster
    int rhs_cpt;             // history pass: load cases per thread (0 = default: min(R, 4))
    int64_t givens_stride;   // doubles per (CTA, case) in givens
    int wait_log2;           // limit of the GMRES clusters' waits for one another, 2^wait_log2 cycles
    int after_head;          // 1: the GMRES launch follows the step's head pass in its stream and may
                             // start beside it (its caches of leaf inverses fill meanwhile)
    int solve_only;          // 1: GMRES alone, no write-back, history update or audit (bare solve)
};

// Small arrays per (GMRES CTA, load case) in MarchData::givens: restart+2
// doubles each of rotation cosines and sines, the Hessenberg column, the second
// Gram-Schmidt pass's coefficients and the rotated right-hand side (the columns
// that do not fit in shared memory), then the rotated Hessenberg columns.
constexpr int kGivensArrays = 5;
constexpr int64_t gmres_givens_doubles(int restart)
{
    return (int64_t)kGivensArrays * (restart + 2) + (int64_t)(restart + 1) * (restart + 2) / 2;
}
constexpr int kGmresClusterMax = 16;
// 2^32 cycles (about two seconds) after which a wait of a GMRES cluster gives up and
// the step fails; a wait takes microseconds.
constexpr int kGmresWaitLog2 = 32;

// A' in the tile form of MarchData::g_*, built on the host as block indices and
// gathered on the device (gather_tiles): src[tile][32] is the block of the
// row-major array, or -1.  own_cap: row capacity of the owned part of a CTA's
// product vector.
struct GmresTileIndex {
    std::vector<int32_t> cs, rows, halo, send_ptr, col, colg, src;
    std::vector<int2> sp, send;
    int halo_max = 0;
};
int gmres_row_capacity(int own_rows);
void gmres_tile_index(const std::vector<int32_t>& cta_row, int own_cap, const std::vector<int32_t>& rp,
                      const std::vector<int32_t>& col, GmresTileIndex& out);
cudaError_t gather_tiles(int64_t tiles, const int32_t* src, const double* val9, double* out, float* out32,
                         cudaStream_t s);

// Run layout of the stacked history blocks of steps k >= kr (MarchData r_*),
// built on the device from the stacked arrays (kptr on the host and the
// device, packed columns, values FP32 when mixed, else FP64).  The arrays are
// the caller's (cudaFree each); kr = 0 on return when there is nothing to
// lay out or the sizes exceed the 32-bit sort indices.
struct HistoryRuns {
    int64_t* ptr = nullptr;   // [E+1]
    uint2* meta = nullptr;    // [runs]
    int64_t* off = nullptr;   // [runs]
    void* val = nullptr;      // SoA [9][nb]
    int64_t nb = 0, runs = 0;
    int kr = 0;
};
cudaError_t build_history_runs(int E, int K, int kr, const std::vector<int64_t>& kptr, const int64_t* d_kptr,
                               const uint32_t* d_col, const void* d_val, int64_t nnz, bool mixed, HistoryRuns& out,
                               cudaStream_t s);
// Device memory the build takes at most for nb blocks (outputs included).
size_t history_runs_bytes(int64_t nb, bool mixed);

// Group layout of the same blocks (MarchData hg_*): place[row] = group * 8 + slot
// of every equation row.  Left out (kr = 0) when the sizes exceed the sort's
// indices, the blocks fill less than kGroupFillMin of the matrices, or a value is
// not finite (a fragment also meets the zero vectors of steps not yet reached).
struct HistoryGroups {
    int64_t* ptr = nullptr;   // [groups+1]
    uint2* meta = nullptr;    // [segments]
    int64_t* off = nullptr;   // [segments]
    void* val = nullptr;      // [steps][3][32]
    int64_t steps = 0, segments = 0;  // contraction steps
    int kr = 0;
};
constexpr double kGroupFillMin = 0.4;
constexpr int kGroupRows = 8;
cudaError_t build_history_groups(int E, int K, int kr, const std::vector<int32_t>& place, int groups,
                                 const std::vector<int64_t>& kptr, const int64_t* d_kptr, const uint32_t* d_col,
                                 const void* d_val, int64_t nnz, bool mixed, HistoryGroups& out, cudaStream_t s);
size_t history_groups_bytes(int64_t nb, bool mixed);

// Blocks of steps 1 .. head_k of each perm row to tiles (MarchData hd_*); sets
// *infinite when a value is not finite (the head multiplies blocks of steps not yet
// reached by zero).
constexpr size_t head_tile_bytes(bool mixed) { return 128 + 9 * 32 * (mixed ? 4 : 8); }
cudaError_t pack_head(int E, int K, int head_k, const int32_t* row_of, const int64_t* kptr, const uint32_t* col,
                      const void* val, bool mixed, int64_t nnz, const int32_t* ptr, unsigned char* tiles, int* infinite,
                      cudaStream_t s);

// Sizes of the R template instantiations.
bool march_supported_loads(int R);
cudaError_t march_prepare(const MarchData& d, cudaStream_t s);
// One time step.  With `overlap`, the history part k >= 3 of step+1 is
// launched on `side` concurrently with this step's GMRES (it only needs
// states up to step-1), and this step's right-hand side adds the part
// computed during the previous step.  With the run layout (d.kr = 2T + 1,
// T = 2 or 3) steps 2, 2 + T, 2 + 2T, ... instead launch the part k >= kr of
// the T steps step+T .. step+2T-1 in one pass (it needs states up to step-1
// as well and has the GMRES of step .. step+T-1 to run beside), and the head
// covers k < kr.
// Events of one step: gm after its GMRES (the side stream waits on prev_gm, that of
// the step before), sync after its launch on the side stream; prev_pass is sync of
// the launch that ends the pass before: of step-T, of step-1 with one load case
// (the first step a T-step pass covers waits on it).  The phases' times come from
// MarchData::stamps: with seven timed events a step and their reading back, and two
// buffers allocated anew, a step of the 120-element rod took 76.9 us, without 57.7.
struct StepEvents {
    cudaEvent_t gm, sync, prev_gm, prev_pass;
};
cudaError_t march_step(const MarchData& d, int step, cudaStream_t s, cudaStream_t side, const StepEvents& ev,
                       bool overlap);
int gmres_cluster_size(int device, int R, bool mixed);
// The forms of GMRES that several models take: vectors in shared memory
// (MarchData::dsm_rows > 0; dsm: the largest dynamic shared memory one needs) or in
// global memory.  With both, the second form's launch goes to `other` between the
// events.
struct ModelForms {
    bool local, global;
    size_t dsm;
    cudaStream_t other;
    cudaEvent_t fork, join;
};
// Launches of one time step of several models of R load cases each (R in 1,
// 2, 4, 8).  phase 0: every model's right-hand side over all history steps,
// then one GMRES cluster of `cluster` CTAs per model (a launch per form); phase 1: the same with
// the head right-hand side (KnownM, k <= 2, plus the bulk computed ahead);
// phase 2: only the bulk (history steps k >= 3) of `step` into the models'
// bulk buffers.  ds: device array of the models' MarchData (each laid out for
// `cluster`); row_off: [n_models + 1] prefix sums of their element counts;
// forms: which forms of GMRES the models take; max_K: the largest history length.
cudaError_t march_models_step(const MarchData* ds, const int* row_off, int n_models, int total_rows, int R,
                              bool mixed, int cluster, const ModelForms& forms, int max_K, int step, int phase,
                              cudaStream_t s);
// The FP64 single-load GMRES step kernel on caller-supplied storage: d.R = 1,
// d.groups = 1, d.nstep = 1, step 1.  Every pointer it writes (b, x, rv,
// aw, u, V, givens, status, step_flags, and unless d.solve_only the write-back
// targets out_lu, out_lt, xring, wring, audit) must be sized for that shape.
cudaError_t gmres_solve_single(const MarchData& d, cudaStream_t s);
// Adjoint march, step n: adj[type][col][3] (type 0 = U, 1 = T) = the
// transposed history convolution of the adjoint right-hand sides
// lam[0..N+1][E][3]; tptr [2 nh][K+1] gives each (type, column)'s blocks of
// step k, trow their equation rows, tval their 9 stacked values.
// One recorded step's right-hand side split into its parts (diagnostics):
// out [4][3E] = KnownM k_n, sum MGS_k W1, -sum MTS_k W0 and A x_n, rows in
// equation order.  xh: [N+1][2][nh][3] history states (X_0 = 0); known:
// [N+1][E][3]; a_*: A in equation-row order with 9 doubles per block; x: x_n
// in unknown order.
struct RhsSplitArgs {
    int E, K, nh, n;
    const int64_t* h_kptr;
    const uint32_t* h_col;
    const double* h_val;
    int64_t h_nnz;
    const double* xh;
    const int32_t* k_rp;
    const int32_t* k_col;
    const double* k_val;
    const int32_t* known_elem;
    const double* known_sign;
    const int32_t* k_elem;  // per KnownM block: known_elem of its column
    const double* k_sgn;    // per KnownM block: known_sign of its column
    const double* known;
    const int32_t* a_rp;
    const int32_t* a_col;
    const double* a_val;
    const double* x;
    double* out;
};
cudaError_t rhs_split(const RhsSplitArgs& a, cudaStream_t s);

// The stacked history blocks regrouped for adj_history: tptr [2 nh (K+1)]
// group ends, group (type * nh + column) * (K + 1) + k in ascending row order;
// trow [nnz] k << 21 | row, tval tiles of 32 blocks in 9 planes.  Synchronises the
// stream.
cudaError_t adjoint_history_groups(int E, int K, int nh, int64_t nnz, const int64_t* kptr, const uint32_t* hcol,
                                   const double* hval, int64_t* tptr, uint32_t* trow, double* tval, cudaStream_t s);
// Transposed write-back of one reverse step (adjoint march), device arrays.
struct AdjWriteBack {
    int E, nh;
    const double* cot_lu;      // [N+1][E][3] or null
    const double* cot_lt;      // [N+1][E][3] or null
    const double* adj;         // [2][nh][3] history adjoint of this step, or null
    const int32_t* hist_owner;
    const int64_t* hist_block;
    const double* hu_sign;
    const double* ht_sign;
    const double* trans;       // [E][9] local frames
    const double* itf_trans;   // [E][9] interface transforms
    const double* uref_sign;
    const double* tref_sign;
    const int32_t* uref_known;
    const int32_t* tref_known;
    double* gk;                // [N+1][E][3] prescribed-value gradient (added to)
};
// Write-back of step n to the transposed solve's right-hand side gp in perm order
// (unk_src: [E][2] (element * 2 + U/T) sources of each unknown, -1 for none;
// unk_of: unknown of each perm row); clears *status.
cudaError_t adjoint_writeback(const AdjWriteBack& a, int n, const int32_t* unk_src, const int32_t* unk_of, double* gp,
                              int* status, cudaStream_t s);
// What follows the transposed solve of a reverse step, device arrays.
struct AdjFinish {
    int E, n_known;
    const double* x;             // [E][3] solution, perm rows
    const int32_t* perm_of_row;
    double* lam;                 // [N+2][E][3] by equation rows; rows past the last step zero
    double* com;                 // [N+2][E][3] lam_{m-1} + 2 lam_m + lam_{m+1}, so far
    const int32_t* kt_ptr;       // [n_known+1] KnownM by columns, in row order: kt_row, kt_blk (block
    const int32_t* kt_row;       // of k_val, 9 doubles row-major)
    const int32_t* kt_blk;
    const double* k_val;
    const int32_t* known_elem;
    const double* known_sign;
    double* gk;                  // [N+1][E][3] prescribed-value gradient (added to)
};
cudaError_t adjoint_finish(const AdjFinish& a, int n, cudaStream_t s);
// gk (step 0) += the cotangent of bd[0] through the local frame (lu for BCID
// 123, lt for 456); cot_* are the device cotangents of step 0 (or null).
cudaError_t adjoint_step0(int E, const double* trans, const int32_t* bcid, const double* cot_lu, const double* cot_lt,
                          double* gk, cudaStream_t s);
cudaError_t adj_history(int N, int n, int K, int nh, int E, const int64_t* tptr, const uint32_t* trow,
                        const double* tval, const double* com, double* adj, cudaStream_t s);
// Shared memory of the GMRES kernel for Rg load cases per cluster, a row
// capacity of `rows` (0: the global-memory form) and `halo` rows from other
// CTAs, without cached leaf inverses and basis vectors; and whether that fits
// (else the global-memory form runs).
size_t gmres_dsm_bytes(int rows, int halo, int Rg, bool mixed);
bool gmres_dsm_fits(int rows, int halo, int Rg, bool mixed);

}  // namespace tdbem
