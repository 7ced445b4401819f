// Host-callable launchers of the kernels in cfs_kernels.cuh and cfs_march.cuh.
// Each policy's kernels live in the translation unit whose compile flags they
// need: kernels_exact.cu (-fmad=false), kernels_fast.cu and march_inst.cu (FMA
// on; the latter once per form and feature set).
#pragma once
#include <cuda_runtime.h>

#include <cmath>

#include "cfs_layout.h"

namespace cfs {

enum Prec : int { kF64 = 0, kF32Mixed = 1, kF64Exact = 2 };

// Tile of the stage kernel: TI rows (x) by TJ columns (y, contiguous).
constexpr int kTileI = 8;
constexpr int kTileJ = 32;

cudaError_t launch_stage(Prec p, const StageArgs& a, cudaStream_t s);
cudaError_t launch_ib_fill(int elem_bytes, const IbArgs& a, cudaStream_t s);
// Before a stage of the throughput forms: the immersed-ghost fill (ib; null:
// none) and the fluxes through the Dirichlet boundary faces (a; null: none).
cudaError_t launch_pre_stage(Prec p, const IbArgs* ib, const StageArgs* a, cudaStream_t s);
cudaError_t launch_wmax(int elem_bytes, const void* U, const Layout& L, const uint8_t* types, double g, double dx,
                        double dy, unsigned long long* out, cudaStream_t s);
// CFL maxima of every case of a batch: args[c].in into args[c].P->wmax[0].
cudaError_t launch_batch_wmax(int elem_bytes, const StageArgs* args, int ncases, cudaStream_t s);
// Sums of the four planes of a device FP64 state [4][n], deterministic; the 4
// sums land at scratch[plane_sums_scratch_doubles() - 4 ..].
int plane_sums_scratch_doubles();
cudaError_t launch_plane_sums(const double* U, long long n, double* scratch, double* out4, cudaStream_t s);
// The parameters of an advance to the device (P), and results to the host's
// pinned memory (null sources are left out): one-thread kernels in the place of
// copies of a few bytes, each of which took the copy engine and two to three
// microseconds more.  wmax is set back to 0 behind the read.
cudaError_t launch_set_params(DevParams* P, const DevParams& v, cudaStream_t s);
cudaError_t launch_results(HostResults* out, const DevParams* P, unsigned long long* wmax, const unsigned int* err,
                           cudaStream_t s);
// Sums of the four planes over fluid cells, deterministic (fixed order);
// scratch holds plane_sums_scratch_doubles() doubles, the 4 sums go to out.
cudaError_t launch_totals(int elem_bytes, const void* U, const Layout& L, const uint8_t* types, double* scratch,
                          double* out, cudaStream_t s);
cudaError_t launch_pack(int elem_bytes, const double* src, void* dst, const Layout& L, cudaStream_t s);
cudaError_t launch_unpack(int elem_bytes, const void* src, double* dst, const Layout& L, cudaStream_t s);
// Ghost layers of the three state buffers, in one launch.
cudaError_t launch_ghost_fill(int elem_bytes, void* const U[3], const Layout& L, const BcSides& sides, cudaStream_t s);
cudaError_t launch_viscous(Prec p, const ViscArgs& a, cudaStream_t s);
cudaError_t launch_weno_faces(Prec p, int n, const double* st, double* left, double* right, double g, double eps,
                              cudaStream_t s);
cudaError_t launch_hll_faces(Prec p, int n, int dir, const double* L, const double* R, double* F, double g,
                             int variant, cudaStream_t s);

// TMA load schedule: one tensor map (CUtensorMap, 128 bytes, 64-byte
// aligned) per state buffer, box of 4 variables x kTmaBoxCells cells x 1 row
// (tma_maps.cpp; the row march's ring rows are that wide).
constexpr int kTmaBoxCells = 36;
constexpr int kTensorMapBytes = 128;
cudaError_t encode_state_map(const void* base, const Layout& L, void* map);

// Stage-kernel variants of the throughput forms (march_kernel template shapes).
struct MarchVariant {
    int rows, warps, min_blocks;
    int load;  // load schedule of the row march: 0 at use, 1 early in the iteration, 2 rows ahead,
               // 3 rows staged in shared memory by cp.async, 4 rows staged by TMA
};
constexpr int kNumVariants = 13;
constexpr MarchVariant kVariants[kNumVariants] = {
    {64, 4, 1, 0}, {32, 4, 5, 0}, {64, 8, 2, 0}, {32, 4, 4, 1}, {64, 8, 2, 1},
    {32, 4, 5, 2}, {32, 4, 5, 3}, {32, 4, 4, 3}, {64, 4, 4, 3}, {32, 4, 6, 3},
    {32, 4, 5, 4}, {32, 4, 4, 4}, {64, 4, 4, 4},
};
// 1-based defaults, from the committed tuning table
// (2d_compressible_flow_solver_b200/tuning.json): FP32 stages its ring rows by
// per-lane 16-byte cp.async (variant 7: 13,997 Mcell-steps/s at 4096^2 against
// 12,717 for the same shape staged by TMA, whose lane-0 issue and mbarrier
// waits cost more instructions than the copies they replace once cells are
// interleaved), FP64 too (variant 8: 4096^2 7,302 against 6,984; 1024^2 5,550
// against 5,302).  The defaults also run with the launch's scheme compiled in
// (launch_march_default); 5 blocks of 96 registers hold the FP32 loop with edge
// code as well.
constexpr int kDefaultVariantF32 = 7;
constexpr int kDefaultVariantF64 = 8;
// FP64 ring blocks per SM (4 warps at 128 registers; 37 KB dynamic + 4.6 KB
// static shared memory), and the register-window variant the FP64 default
// falls back to when the ring's last wave would run nearly empty
// (launch_stage_f64).
constexpr int kRingBlocksPerSmF64 = 4;
constexpr int kWindowVariantF64 = 4;

// Row chunk of a launch whose warps (nseg per chunk of rows, w per block) run
// on `slots` resident blocks.  An item costs its R rows plus about 2 more (the x-work of
// the row above and below the chunk), and the launch ends with a partly
// filled stretch of about half an item, so the launch lasts about
// (R + 2) (blocks / slots + 1/2): short chunks pay the per-item rows, long
// ones the tail -- and, on a grid of few items, the chain of one warp's rows
// (1.2 us a row in FP32, 2.0 in FP64), which is all that such a launch waits
// for.  The minimum lies near R = 2 sqrt(nseg nrows / (w slots)): 28 rows
// at 4096^2, 14 at 2048^2, 7 at 1024^2 (FP32, 740 slots), 2 at 256^2, 1 at
// 64 x 48.  Fitted to a sweep of fixed chunks of 8 .. 196 rows at 512^2 ..
// 4096^2, FP32 and FP64 (a whole-wave model that ignored the tail picked 196
// rows at 4096^2 and lost 12 % against 32), and followed by a sweep of 1 .. 24
// rows below: periodic SSP3 steps with chunks of at least 6 rows (the search's
// end before) against the chosen ones, 64 x 48 FP64 49.2 -> 20.4 us, 256^2
// FP32 37.0 -> 25.2, 512^2 FP32 51.2 -> 47.0.  Searched over 1 .. 128 rows
// (the whole range when it is shorter), ties to the longer chunk.
inline int choose_rows(int nseg, int w, int nrows, long long slots) {
    int best_r = 32;
    long long best_cost = -1;
    const int r_max = nrows < 128 ? nrows : 128;
    for (int r = 1; r <= r_max; ++r) {
        const long long blocks = (static_cast<long long>(nseg) * ((nrows + r - 1) / r) + w - 1) / w;
        const long long cost = static_cast<long long>(r + 2) * (2 * blocks + slots);
        if (best_cost < 0 || cost <= best_cost) {
            best_cost = cost;
            best_r = r;
        }
    }
    return best_r;
}

// Row chunks of a launch in two lengths: long ones first, one to each of the
// `w slots` resident warps (two where a warp's share is 50 rows or more) and
// about 84 % of the rows together, then short ones that fill what the warps'
// different ends leave open.  Against equal chunks (choose_rows) fewer rows are
// repeated at chunk ends and the last stretch is shorter: SSP3 steps at 4096^2
// FP32 1,252 -> 1,203 us, 1024^2 112 -> 105, 2048^2 FP64 631 -> 614, 2048 x 1024
// cylinder FP32 250 -> 228, 1021 x 1537 FP32 155 -> 145 (one long chunk per warp
// instead of two: 4096^2 1,304, 3100^2 759 against 715; two instead of one: 1800^2
// FP64 491 against 477).  The short chunks' length balances the rows they
// repeat (2 each) against the half chunk the launch ends with.  Grids of fewer
// than 4 rows per warp keep equal chunks (605 x 301 FP64 lost 9 to 16 % with a
// long chunk of 2 rows).
struct RowChunks {
    int rows, long_chunks, rows_short;
};
inline RowChunks choose_chunks(int nseg, int w, int nrows, long long slots) {
    const double per_warp = static_cast<double>(nseg) * nrows / (static_cast<double>(slots) * w);
    const int waves = per_warp < 50 ? 1 : 2;
    const long long n = waves * slots * w / nseg;  // long chunks per segment
    if (per_warp >= 4 && n >= 1) {
        const int rows = static_cast<int>(0.84 * nrows / n + 0.5);
        const double left = 1.0 - static_cast<double>(rows) * n / nrows;
        if (left > 0.08) {
            const int s = static_cast<int>(2 * std::sqrt(left * per_warp) + 0.5);
            return {rows, static_cast<int>(n), s < 2 ? 2 : s};
        }
    }
    const int rows = choose_rows(nseg, w, nrows, slots);
    return {rows, (nrows + rows - 1) / rows, rows};
}

// Batched forms (cfs_batch_*): one launch covers every case of a batch.
constexpr int kBatchWarps = 4;
// 4 blocks of 4 warps per SM (128 registers): the uneven 512-case batch ran
// 6,074 / 7,241 / 6,629 Mcell-steps/s at 5 / 4 / 3 blocks per SM.
constexpr int kBatchMinBlocksF32 = 4;
constexpr int kBatchLoadF32 = 3;  // FP32 batches stage rows in the shared ring
constexpr int kBatchMinBlocksF64 = 4;
// FP64 batches stage rows in the ring too (dynamic shared memory, 4 blocks per
// SM): the uneven 512-case batch 3,230 against 2,938 Mcell-steps/s without it
// (the earlier ring that also held U^0 rows allowed 3 blocks and lost, 2,775).
constexpr int kBatchLoadF64 = 3;
// Longest batch work unit the library cuts by itself (append_units): longer
// ones gain nothing (128 uneven cases to 768 cells at 128 / 96 / 64 rows, FP32
// 2,131 / 2,066 / 2,069 us a step).
constexpr int kBatchMaxRows = 96;
// Work-unit counters of a batch, [parity][stage][feature group]: the group
// launches of a stage count their own up from 0 and put every counter of the
// other stages back to 0 (nothing else of the batch runs then), so no stage
// needs a clearing launch.
constexpr int kBatchMaxGroups = 4;  // the feature sets a batch launches: 0, Pos, Edge, Edge | Pos
constexpr int kBatchCounters = 2 * 3 * kBatchMaxGroups;
cudaError_t launch_batch_stage(Prec p, const StageArgs* args, const BatchUnit* units, int total, unsigned int* counters,
                               int slot, int grid, int feat, int scheme,
                               cudaStream_t s);  // feat: kFeatPos | kFeatEdge bits; scheme: known_scheme
// The same for a batch: the immersed-ghost cells of every case (total; may be
// 0) and the Dirichlet faces of every case (ncases; 0: none).
cudaError_t launch_batch_pre_stage(Prec p, const IbArgs* ibs, const int* cases, const int* local, int total,
                                   const StageArgs* args, int ncases, int max_edge, cudaStream_t s);
int batch_blocks_per_sm(Prec p);

// Per-policy entry points behind the dispatchers above.
cudaError_t launch_stage_exact(const StageArgs& a, cudaStream_t s);
cudaError_t launch_stage_f64(const StageArgs& a, cudaStream_t s);
cudaError_t launch_stage_f32(const StageArgs& a, cudaStream_t s);
// Row march of one form and feature set (march_inst.cu, kFeat* bits), variant v (1-based).
cudaError_t launch_march_f64_0(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f64_1(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f64_2(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f64_3(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f64_4(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f64_5(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f64_6(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f64_7(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f32_0(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f32_1(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f32_2(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f32_3(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f32_4(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f32_5(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f32_6(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_march_f32_7(const StageArgs& a, int v, cudaStream_t s);
cudaError_t launch_viscous_f64(const ViscArgs& a, cudaStream_t s);
cudaError_t launch_viscous_f32(const ViscArgs& a, cudaStream_t s);
cudaError_t launch_weno_faces_exact(int n, const double* st, double* l, double* r, double g, double eps, cudaStream_t s);
cudaError_t launch_weno_faces_f64(int n, const double* st, double* l, double* r, double g, double eps, cudaStream_t s);
cudaError_t launch_weno_faces_f32(int n, const double* st, double* l, double* r, double g, double eps, cudaStream_t s);
cudaError_t launch_hll_faces_exact(int n, int dir, const double* L, const double* R, double* F, double g, int v, cudaStream_t s);
cudaError_t launch_hll_faces_f64(int n, int dir, const double* L, const double* R, double* F, double g, int v, cudaStream_t s);
cudaError_t launch_hll_faces_f32(int n, int dir, const double* L, const double* R, double* F, double g, int v, cudaStream_t s);

}  // namespace cfs
