// Kernels of the throughput forms: FP64 with FMA contraction and the
// FP32-mixed form.  Built with FMA contraction on (nvcc default).
#include <atomic>

#include "cfs_kernels.cuh"
#include "cfs_launch.h"
#include "cfs_march.cuh"
#include "cfs_resident.h"
#include "cfs_viscous.cuh"

namespace cfs {

constexpr int kMaxDev = ResidentCache::kMaxDev;

// SM count of the current device (cached per device).
int sm_count() {
    static std::atomic<int> count[kMaxDev] = {};  // every writer stores the same value
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return 148;
    int c = count[dev].load(std::memory_order_relaxed);
    if (c == 0) {
        int n = 0;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        c = n > 0 ? n : 148;
        count[dev].store(c, std::memory_order_relaxed);
    }
    return c;
}

// The FP64 default variant stages rows in a shared ring, kRingBlocksPerSmF64
// blocks per SM.  When its grid fills more than one but fewer than three such
// waves and the last one is under half full, the register-window variant
// finishes first (measured with the earlier 3-block ring on the Mach-3
// cylinder, 2048 x 1024: 2,105 against 1,832 Mcell-steps/s; the 4-block ring
// now fills that grid in one wave and runs it at 2,376).
int default_variant_f64(const Layout& L, int rows) {
    const MarchVariant& d = kVariants[kDefaultVariantF64 - 1];
    const long long nseg = (L.ny + kSeg - 1) / kSeg;
    const long long blocks = (nseg * ((L.nx + rows - 1) / rows) + d.warps - 1) / d.warps;
    const double waves = static_cast<double>(blocks) / (static_cast<double>(sm_count()) * kRingBlocksPerSmF64);
    if (waves > 1.0 && waves < 3.0 && waves - static_cast<double>(static_cast<long long>(waves)) < 0.5)
        return kWindowVariantF64;
    return kDefaultVariantF64;
}

cudaError_t launch_stage_f64(const StageArgs& a, cudaStream_t s) {
    // (with the row chunk chosen per launch to fill whole waves, the ring
    // variant stays; the fallback serves fixed chunks)
    const int v = a.variant > 0 ? a.variant : a.rows > 0 ? default_variant_f64(a.L, a.rows) : kDefaultVariantF64;
    switch (march_features(a)) {
        case 0: return launch_march_f64_0(a, v, s);
        case 1: return launch_march_f64_1(a, v, s);
        case 2: return launch_march_f64_2(a, v, s);
        case 3: return launch_march_f64_3(a, v, s);
        case 4: return launch_march_f64_4(a, v, s);
        case 5: return launch_march_f64_5(a, v, s);
        case 6: return launch_march_f64_6(a, v, s);
        default: return launch_march_f64_7(a, v, s);
    }
}

cudaError_t launch_stage_f32(const StageArgs& a, cudaStream_t s) {
    const int v = a.variant > 0 ? a.variant : kDefaultVariantF32;
    switch (march_features(a)) {
        case 0: return launch_march_f32_0(a, v, s);
        case 1: return launch_march_f32_1(a, v, s);
        case 2: return launch_march_f32_2(a, v, s);
        case 3: return launch_march_f32_3(a, v, s);
        case 4: return launch_march_f32_4(a, v, s);
        case 5: return launch_march_f32_5(a, v, s);
        case 6: return launch_march_f32_6(a, v, s);
        default: return launch_march_f32_7(a, v, s);
    }
}

// The batch's feature set is common to its cases: positivity, and the edge
// code when some case has a physical side or cell types (batches keep no RHS
// and have no viscous terms).
// Dynamic shared memory of a batched march (the FP64 ring), 0 for the others.
template <class Pol, int kLoad>
constexpr size_t batch_dyn_bytes() {
    return (kLoad == 3 && sizeof(typename Pol::T) == 8) ? static_cast<size_t>(kBatchWarps) * ring_words<double, kLoad>() * 8 : 0;
}

template <class Kernel>
cudaError_t allow_dyn(Kernel k, size_t bytes) {
    if (bytes == 0) return cudaSuccess;
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}

template <class Pol, int kMinBlocks, int kLoad, int kFeat>
cudaError_t launch_batch_kernel(const StageArgs* args, const BatchUnit* units, int total, unsigned int* counters, int slot, int grid,
                                cudaStream_t s) {
    constexpr size_t dyn = batch_dyn_bytes<Pol, kLoad>();
    const cudaError_t e = allow_dyn(batch_march_kernel<Pol, kBatchWarps, kMinBlocks, kLoad, kFeat>, dyn);
    if (e != cudaSuccess) return e;
    return launch_after(batch_march_kernel<Pol, kBatchWarps, kMinBlocks, kLoad, kFeat>, grid, 32 * kBatchWarps, dyn, s, args,
                        units, total, counters, slot);
}

template <class Pol, int kMinBlocks, int kLoad, int kScheme, class... Args>
cudaError_t launch_batch_feat(int feat, Args... args) {
    switch (feat) {
        case 0: return launch_batch_kernel<Pol, kMinBlocks, kLoad, kScheme>(args...);
        case kFeatPos: return launch_batch_kernel<Pol, kMinBlocks, kLoad, kFeatPos | kScheme>(args...);
        case kFeatEdge: return launch_batch_kernel<Pol, kMinBlocks, kLoad, kFeatEdge | kScheme>(args...);
        case kFeatEdge | kFeatPos:
            return launch_batch_kernel<Pol, kMinBlocks, kLoad, kFeatEdge | kFeatPos | kScheme>(args...);
        default: return cudaErrorInvalidValue;
    }
}

template <class Pol, int kMinBlocks, int kLoad, class... Args>
cudaError_t launch_batch_scheme(int scheme, int feat, Args... args) {
    switch (scheme) {
        case kScheme0: return launch_batch_feat<Pol, kMinBlocks, kLoad, kScheme0>(feat, args...);
        case kScheme1: return launch_batch_feat<Pol, kMinBlocks, kLoad, kScheme1>(feat, args...);
        case kScheme2: return launch_batch_feat<Pol, kMinBlocks, kLoad, kScheme2>(feat, args...);
        default: return launch_batch_feat<Pol, kMinBlocks, kLoad, 0>(feat, args...);
    }
}

cudaError_t launch_batch_stage(Prec p, const StageArgs* args, const BatchUnit* units, int total, unsigned int* counters,
                               int slot, int grid, int feat, int scheme, cudaStream_t s) {
    if (total <= 0) return cudaSuccess;
    if (p == kF32Mixed)
        return launch_batch_scheme<PolF32, kBatchMinBlocksF32, kBatchLoadF32>(
            scheme, feat, args, units, total, counters, slot, grid, s);
    return launch_batch_scheme<PolF64, kBatchMinBlocksF64, kBatchLoadF64>(
        scheme, feat, args, units, total, counters, slot, grid, s);
}

int batch_blocks_per_sm(Prec p) {
    int n = 0;
    if (p == kF32Mixed)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &n, batch_march_kernel<PolF32, kBatchWarps, kBatchMinBlocksF32, kBatchLoadF32, kFeatEdge | kFeatPos>,
            32 * kBatchWarps, 0);
    else
    {
        constexpr size_t dyn = batch_dyn_bytes<PolF64, kBatchLoadF64>();
        auto k = batch_march_kernel<PolF64, kBatchWarps, kBatchMinBlocksF64, kBatchLoadF64, kFeatEdge | kFeatPos>;
        if (allow_dyn(k, dyn) == cudaSuccess) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, 32 * kBatchWarps, dyn);
    }
    return n > 0 ? n : 1;
}

// Rows of a viscous work item by the row march's rule: an item of R rows
// costs about R + 2.5 (five more rows are loaded and converted, one more
// x-face formed).
template <class Pol, int kMinBlocks>
cudaError_t launch_viscous_form(const ViscArgs& a_in, cudaStream_t s) {
    static ResidentCache cache;
    const long long slots = resident_blocks(cache, viscous_kernel<Pol, kMinBlocks>, 32 * kViscWarps, 0);
    ViscArgs a = a_in;
    const int nseg = (a.L.ny + kViscSeg - 1) / kViscSeg;
    a.rows = slots > 0 ? choose_rows(nseg, kViscWarps, a.L.nx, slots) : 32;
    const long long items = static_cast<long long>(nseg) * ((a.L.nx + a.rows - 1) / a.rows);
    const long long blocks = (items + kViscWarps - 1) / kViscWarps;
    return launch_after(viscous_kernel<Pol, kMinBlocks>, static_cast<unsigned>(blocks), 32 * kViscWarps, 0, s, a);
}

cudaError_t launch_viscous_f64(const ViscArgs& a, cudaStream_t s) { return launch_viscous_form<PolF64, 3>(a, s); }
cudaError_t launch_viscous_f32(const ViscArgs& a, cudaStream_t s) { return launch_viscous_form<PolF32, 5>(a, s); }

cudaError_t launch_weno_faces_f64(int n, const double* st, double* l, double* r, double g, double eps, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    weno_faces_kernel<PolF64><<<(n + 127) / 128, 128, 0, s>>>(n, st, l, r, g, eps);
    return cudaGetLastError();
}

cudaError_t launch_weno_faces_f32(int n, const double* st, double* l, double* r, double g, double eps, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    weno_faces_kernel<PolF32><<<(n + 127) / 128, 128, 0, s>>>(n, st, l, r, g, eps);
    return cudaGetLastError();
}

cudaError_t launch_hll_faces_f64(int n, int dir, const double* L, const double* R, double* F, double g, int v,
                                 cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    hll_faces_kernel<PolF64><<<(n + 127) / 128, 128, 0, s>>>(n, dir, L, R, F, g, v);
    return cudaGetLastError();
}

cudaError_t launch_hll_faces_f32(int n, int dir, const double* L, const double* R, double* F, double g, int v,
                                 cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    hll_faces_kernel<PolF32><<<(n + 127) / 128, 128, 0, s>>>(n, dir, L, R, F, g, v);
    return cudaGetLastError();
}

}  // namespace cfs
