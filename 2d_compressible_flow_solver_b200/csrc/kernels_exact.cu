// Kernels whose FP64 rounding must follow the reference's operation order:
// built with -fmad=false so no multiply-add is contracted, IEEE division and
// square root (nvcc defaults).  Holds the CFS_FP64_EXACT stage, the immersed-
// ghost fill, the CFL reduction and the layout helpers for both storage types.
#include "cfs_kernels.cuh"
#include "cfs_launch.h"
#include "cfs_march.cuh"
#include "cfs_resident.h"

namespace cfs {

namespace {
inline dim3 stage_grid(const Layout& L) {
    return dim3((L.ny + kTileJ - 1) / kTileJ, (L.nx + kTileI - 1) / kTileI);
}
inline int flat_blocks(long long work, int nt) {
    long long b = (work + nt - 1) / nt;
    if (b < 1) b = 1;
    if (b > 148 * 16) b = 148 * 16;
    return static_cast<int>(b);
}
}  // namespace

// Two blocks per SM at 96 registers; a grid of more than two rounds of those runs
// three at 72: TVD2 600 x 500 235 -> 214 us a step, 1024^2 TVD3 1,059 -> 937, but
// 256^2 62 -> 80.
cudaError_t launch_stage_exact(const StageArgs& a, cudaStream_t s) {
    constexpr int nt = (kTileI + 1) * kTileJ;
    static ResidentCache cache;
    const dim3 grid = stage_grid(a.L);
    const bool many = static_cast<long long>(grid.x) * grid.y > 2 * resident_blocks(cache, stage_kernel<PolExact, kTileI, kTileJ, 2>, nt, 0);
    return launch_after(many ? stage_kernel<PolExact, kTileI, kTileJ, 3> : stage_kernel<PolExact, kTileI, kTileJ, 2>, grid, nt, 0, s, a);
}

cudaError_t launch_ib_fill(int elem_bytes, const IbArgs& a, cudaStream_t s) {
    if (a.n <= 0) return cudaSuccess;
    const int nt = 128, nb = (a.n + nt - 1) / nt;
    return launch_after(elem_bytes == 8 ? ib_fill_kernel<double> : ib_fill_kernel<float>, nb, nt, 0, s, a);
}

// What a stage of the throughput forms needs before its march, in one launch:
// the immersed-ghost fill (blocks below ib_blocks; n cells) and the fluxes
// through the Dirichlet boundary faces (face_blocks blocks of 128 faces per
// side).  Both are chains of a few microseconds on a few blocks; in two launches
// they cost the 605 x 301 FP64 cylinder 10 of a stage's 27 us (step 79.9 -> 73.1
// us; 2048 x 1024 FP32 258 -> 251, the uneven batch 901 -> 889).  A face flux reads the
// cells next to its side, so a body whose ghosts lie there fills first, in a
// launch of its own.
constexpr int kPreThreads = 128;
template <class Pol>
__global__ void __launch_bounds__(kPreThreads) pre_stage_kernel(const IbArgs ib, const __grid_constant__ StageArgs a,
                                                                int ib_blocks, int face_blocks) {
    const int b = static_cast<int>(blockIdx.x), t = static_cast<int>(threadIdx.x);
    let_next_in();
    after_previous();
    if (b < ib_blocks) {
        if (b * kPreThreads + t < ib.n) ib_fill_one<typename Pol::T>(ib, b * kPreThreads + t);
    } else {
        maybe_boundary_flux<Pol>(a, (b - ib_blocks) / face_blocks, (b - ib_blocks) % face_blocks * kPreThreads + t);
    }
}

cudaError_t launch_pre_stage(Prec p, const IbArgs* ib, const StageArgs* a, cudaStream_t s) {
    static const StageArgs no_faces{};
    const int ib_blocks = ib ? (ib->n + kPreThreads - 1) / kPreThreads : 0;
    const int n = !a ? 0 : a->L.nx > a->L.ny ? a->L.nx : a->L.ny;
    const int face_blocks = (n + kPreThreads - 1) / kPreThreads;
    const int blocks = ib_blocks + 4 * face_blocks;
    if (blocks == 0) return cudaSuccess;
    if (a && !a->bflux) return cudaErrorInvalidValue;
    return launch_after(p == kF32Mixed ? pre_stage_kernel<PolF32> : pre_stage_kernel<PolF64>, blocks, kPreThreads, 0, s,
                        ib ? *ib : IbArgs{}, a ? *a : no_faces, ib_blocks, face_blocks);
}

// Batched form: immersed-ghost cell g of the batch is cell local[g] of case
// cases[g] (ibs[c]: case c's fill description); the faces of every case with a
// Dirichlet side (args[c].bflux; face_blocks covers the largest edge).
template <class Pol>
__global__ void __launch_bounds__(kPreThreads) batch_pre_stage_kernel(const IbArgs* __restrict__ ibs, const int* __restrict__ cases,
                                                                      const int* __restrict__ local, int total, int ib_blocks,
                                                                      const StageArgs* __restrict__ args, int face_blocks) {
    const int b = static_cast<int>(blockIdx.x), t = static_cast<int>(threadIdx.x);
    let_next_in();
    after_previous();
    if (b < ib_blocks) {
        const int g = b * kPreThreads + t;
        if (g >= total) return;
        const IbArgs ib = ibs[cases[g]];
        ib_fill_one<typename Pol::T>(ib, local[g]);
    } else {
        const int f = b - ib_blocks, side = f / face_blocks;
        const StageArgs& a = args[side / 4];
        if (a.bflux) maybe_boundary_flux<Pol>(a, side % 4, f % face_blocks * kPreThreads + t);
    }
}

cudaError_t launch_batch_pre_stage(Prec p, const IbArgs* ibs, const int* cases, const int* local, int total,
                                   const StageArgs* args, int ncases, int max_edge, cudaStream_t s) {
    const int ib_blocks = (total + kPreThreads - 1) / kPreThreads;
    const int face_blocks = ncases > 0 ? (max_edge + kPreThreads - 1) / kPreThreads : 0;
    const long long blocks = ib_blocks + 4LL * face_blocks * ncases;
    if (blocks == 0) return cudaSuccess;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    return launch_after(p == kF32Mixed ? batch_pre_stage_kernel<PolF32> : batch_pre_stage_kernel<PolF64>,
                        static_cast<unsigned>(blocks), kPreThreads, 0, s, ibs, cases, local, total, ib_blocks, args, face_blocks);
}

cudaError_t launch_wmax(int elem_bytes, const void* U, const Layout& L, const uint8_t* types, double g, double dx,
                        double dy, unsigned long long* out, cudaStream_t s) {
    constexpr int nt = 256;
    const int nb = flat_blocks(static_cast<long long>(L.nx) * L.ny, nt);
    if (elem_bytes == 8) wmax_kernel<double, nt><<<nb, nt, 0, s>>>(static_cast<const double*>(U), L, types, g, dx, dy, out);
    else wmax_kernel<float, nt><<<nb, nt, 0, s>>>(static_cast<const float*>(U), L, types, g, dx, dy, out);
    return cudaGetLastError();
}

cudaError_t launch_batch_wmax(int elem_bytes, const StageArgs* args, int ncases, cudaStream_t s) {
    constexpr int nt = 256, per_case = 64;
    for (int c0 = 0; c0 < ncases; c0 += 65535) {  // gridDim.y limit
        const int nc = ncases - c0 < 65535 ? ncases - c0 : 65535;
        if (elem_bytes == 8) batch_wmax_kernel<double, nt><<<dim3(per_case, nc), nt, 0, s>>>(args + c0);
        else batch_wmax_kernel<float, nt><<<dim3(per_case, nc), nt, 0, s>>>(args + c0);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Sums of the four planes of a host-order FP64 state [4][n], in a fixed order
// (the same bits on every run): kSumBlocks strided partial sums per plane,
// each reduced as a tree in its block, then the partials added in index order.
constexpr int kSumBlocks = 256, kSumThreads = 256;

__global__ void __launch_bounds__(kSumThreads) plane_partial_sums_kernel(const double* U, long long n, double* partial) {
    __shared__ double red[kSumThreads];
    const int v = blockIdx.y;
    double s = 0.0;
    for (long long k = static_cast<long long>(blockIdx.x) * kSumThreads + threadIdx.x; k < n;
         k += static_cast<long long>(kSumBlocks) * kSumThreads)
        s += U[v * n + k];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kSumThreads / 2; w > 0; w >>= 1) {
        if (static_cast<int>(threadIdx.x) < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[v * kSumBlocks + blockIdx.x] = red[0];
}

__global__ void plane_final_sums_kernel(const double* partial, double* out4) {
    const int v = threadIdx.x;
    if (v >= kVars) return;
    double s = 0.0;
    for (int b = 0; b < kSumBlocks; ++b) s += partial[v * kSumBlocks + b];
    out4[v] = s;
}

int plane_sums_scratch_doubles() { return kVars * kSumBlocks + kVars; }

cudaError_t launch_plane_sums(const double* U, long long n, double* scratch, double* out4, cudaStream_t s) {
    plane_partial_sums_kernel<<<dim3(kSumBlocks, kVars), kSumThreads, 0, s>>>(U, n, scratch);
    plane_final_sums_kernel<<<1, 32, 0, s>>>(scratch, out4);
    return cudaGetLastError();
}

cudaError_t launch_totals(int elem_bytes, const void* U, const Layout& L, const uint8_t* types, double* scratch,
                          double* out, cudaStream_t s) {
    const dim3 grid(kSumBlocks, kVars);
    if (elem_bytes == 8)
        totals_partial_kernel<double, kSumThreads, kSumBlocks><<<grid, kSumThreads, 0, s>>>(static_cast<const double*>(U), L, types, scratch);
    else
        totals_partial_kernel<float, kSumThreads, kSumBlocks><<<grid, kSumThreads, 0, s>>>(static_cast<const float*>(U), L, types, scratch);
    plane_final_sums_kernel<<<1, 32, 0, s>>>(scratch, out);
    return cudaGetLastError();
}

cudaError_t launch_pack(int elem_bytes, const double* src, void* dst, const Layout& L, cudaStream_t s) {
    const int nt = 256, nb = flat_blocks(4LL * L.nx * L.ny, nt);
    if (elem_bytes == 8) pack_kernel<double><<<nb, nt, 0, s>>>(src, static_cast<double*>(dst), L);
    else pack_kernel<float><<<nb, nt, 0, s>>>(src, static_cast<float*>(dst), L);
    return cudaGetLastError();
}

cudaError_t launch_unpack(int elem_bytes, const void* src, double* dst, const Layout& L, cudaStream_t s) {
    const int nt = 256, nb = flat_blocks(4LL * L.nx * L.ny, nt);
    if (elem_bytes == 8) unpack_kernel<double><<<nb, nt, 0, s>>>(static_cast<const double*>(src), dst, L);
    else unpack_kernel<float><<<nb, nt, 0, s>>>(static_cast<const float*>(src), dst, L);
    return cudaGetLastError();
}

__global__ void set_params_kernel(DevParams* P, const DevParams v) { *P = v; }

__global__ void results_kernel(HostResults* out, const DevParams* P, unsigned long long* wmax, const unsigned int* err) {
    after_previous();
    if (P) out->params = *P;
    if (wmax) {
        out->wmax = *wmax;
        *wmax = 0ull;
    }
    if (err) out->err = *err;
}

cudaError_t launch_set_params(DevParams* P, const DevParams& v, cudaStream_t s) {
    set_params_kernel<<<1, 1, 0, s>>>(P, v);
    return cudaGetLastError();
}

cudaError_t launch_results(HostResults* out, const DevParams* P, unsigned long long* wmax, const unsigned int* err,
                           cudaStream_t s) {
    return launch_after(results_kernel, 1, 1, 0, s, out, P, wmax, err);
}

cudaError_t launch_ghost_fill(int elem_bytes, void* const U[3], const Layout& L, const BcSides& sides, cudaStream_t s) {
    const int per = L.nx > L.ny ? L.nx : L.ny;
    const int nt = 256, nb = flat_blocks(4LL * kGhost * per * kVars + 4LL * kGhost * kGhost * kVars, nt);
    const dim3 grid(nb, 3);
    if (elem_bytes == 8) ghost_fill_kernel<<<grid, nt, 0, s>>>(static_cast<double*>(U[0]), static_cast<double*>(U[1]), static_cast<double*>(U[2]), L, sides);
    else ghost_fill_kernel<<<grid, nt, 0, s>>>(static_cast<float*>(U[0]), static_cast<float*>(U[1]), static_cast<float*>(U[2]), L, sides);
    return cudaGetLastError();
}

cudaError_t launch_weno_faces_exact(int n, const double* st, double* l, double* r, double g, double eps, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    weno_faces_kernel<PolExact><<<(n + 127) / 128, 128, 0, s>>>(n, st, l, r, g, eps);
    return cudaGetLastError();
}

cudaError_t launch_hll_faces_exact(int n, int dir, const double* L, const double* R, double* F, double g, int v,
                                   cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    hll_faces_kernel<PolExact><<<(n + 127) / 128, 128, 0, s>>>(n, dir, L, R, F, g, v);
    return cudaGetLastError();
}

}  // namespace cfs
