// Row-march launchers of one (form, feature set): compiled once per pair, with
//   -DCFS_MARCH_POL=PolF32|PolF64  -DCFS_MARCH_FEAT=0..7  -DCFS_MARCH_FN=<launcher name>
// (the build gives each pair its own object, so the kernels compile in
// parallel).  The launcher runs the variant `v` of kVariants (1-based).
#include <mutex>

#include "cfs_kernels.cuh"
#include "cfs_launch.h"
#include "cfs_march.cuh"
#include "cfs_resident.h"
#include "cfs_tile.cuh"

#if !defined(CFS_MARCH_POL) || !defined(CFS_MARCH_FEAT) || !defined(CFS_MARCH_FN)
#error "march_inst.cu needs CFS_MARCH_POL, CFS_MARCH_FEAT and CFS_MARCH_FN"
#endif

namespace cfs {
namespace {

constexpr int kMaxDev = ResidentCache::kMaxDev;

template <class Pol, int R, int W, int B, int Ld, int F>
cudaError_t launch_march(const StageArgs& a_in, cudaStream_t s) {
    const int nseg = (a_in.L.ny + kSeg - 1) / kSeg;
    const int nrows = stage_row_hi(a_in) - stage_row_lo(a_in);
    if (nrows <= 0) return cudaSuccess;
    size_t dyn = 0;
    const StageArgs& a = a_in;
    if constexpr (Ld == 4) {
        if (!a.has_tmaps || !a.err) return cudaErrorInvalidValue;
    }
    if constexpr (Ld >= 3 && sizeof(typename Pol::T) == 8) {
        // the FP64 ring lives in dynamic shared memory; allow it once per
        // device (std::call_once: host threads may make their first launches
        // on one device at the same time)
        static std::once_flag once[kMaxDev];
        static cudaError_t allow_err[kMaxDev];
        dyn = static_cast<size_t>(W) * ring_words<double, Ld>() * sizeof(double);
        auto allow = [dyn] {
            return cudaFuncSetAttribute(march_kernel<Pol, R, W, B, Ld, F>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(dyn));
        };
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        if (dev < 0 || dev >= kMaxDev) {
            e = allow();
        } else {
            std::call_once(once[dev], [&] { allow_err[dev] = allow(); });
            e = allow_err[dev];
        }
        if (e != cudaSuccess) return e;
    }
    static ResidentCache cache;
    const long long slots = resident_blocks(cache, march_kernel<Pol, R, W, B, Ld, F>, 32 * W, dyn);
    StageArgs b = a;
    if (a.rows > 0 || slots <= 0) {  // fixed rows (also where the query of the slots failed)
        b.rows = b.rows_short = a.rows > 0 ? a.rows : R;
        b.long_chunks = (nrows + b.rows - 1) / b.rows;
    } else {
        const RowChunks c = choose_chunks(nseg, W, nrows, slots);
        b.rows = c.rows;
        b.long_chunks = c.long_chunks;
        b.rows_short = c.rows_short;
    }
    const int covered = b.long_chunks * b.rows;
    const int chunks = b.long_chunks + (covered < nrows ? (nrows - covered + b.rows_short - 1) / b.rows_short : 0);
    // one warp per (segment, row chunk), segments fastest
    const long long items = static_cast<long long>(nseg) * chunks;
    const dim3 grid(static_cast<unsigned>((items + W - 1) / W));
    // A launch of more blocks than fit at once starts before the one ahead of it
    // ends (launch_after).  A smaller one waits for it: its blocks would go to
    // whichever SMs have room, two and three to some, and the stage lasts as long
    // as those (SSP3 steps with and without: 256^2 FP32 22.9 / 21.4 us, 384^2
    // Navier-Stokes 52 / 43, but 768^2 70.6 / 72.5).
    if (static_cast<long long>(grid.x) > slots) return launch_after(march_kernel<Pol, R, W, B, Ld, F>, grid, 32 * W, dyn, s, b);
    march_kernel<Pol, R, W, B, Ld, F><<<grid, 32 * W, dyn, s>>>(b);
    return cudaGetLastError();
}

template <class Pol, int K, int F>
cudaError_t launch_march_k(const StageArgs& a, cudaStream_t s) {
    constexpr MarchVariant v = kVariants[K];
    return launch_march<Pol, v.rows, v.warps, v.min_blocks, v.load, F>(a, s);
}

// The tile form with W warps per block, when its blocks fit `rounds` times on
// the device; false: not launched.
template <class Pol, int W, int F>
bool launch_tile(const StageArgs& a, int rounds, cudaStream_t s, cudaError_t& e) {
    auto kernel = tile_kernel<Pol, W, tile_min_blocks<typename Pol::T>(W), F>;
    static ResidentCache cache;
    const long long slots = resident_blocks(cache, kernel, 32 * W, 0);
    const int nseg = (a.L.ny + kSeg - 1) / kSeg;
    const int nrows = stage_row_hi(a) - stage_row_lo(a);
    const long long blocks = static_cast<long long>(nseg) * ((nrows + W - 3) / (W - 2));
    if (blocks > rounds * slots) return false;
    e = nrows <= 0 ? cudaSuccess : launch_after(kernel, dim3(static_cast<unsigned>(blocks)), 32 * W, 0, s, a);
    return true;
}

// A grid too small to fill the GPU runs in the tile form: the smaller tile
// while all its blocks are resident at once, the larger one up to two rounds
// of it; others march.  SSP3 steps (us) with the march / 4 warps / 10 (FP32)
// or 8 (FP64) warps: FP32 periodic 64^2 14.3 / 11.3 / 12.5, 160^2 17.4 / 15.1 /
// 15.0, 256^2 21.4 / 22.7 / 16.3, 352^2 29.7 / 33.7 / 26.9, 384^2 30.7 / 39.8 /
// 33.4; FP64 64^2 18.4 / 13.4 / 15.4, 192^2 29.7 / 27.0 / 22.4, 352^2 46.0 /
// 53.8 / 43.8, 384^2 46.1 / 60.1 / 50.4; cylinder 400 x 200 FP32 43.2 / 46.0 /
// 39.3, FP64 59.3 / 60.1 / 54.5.  A caller that fixes the march's rows or
// variant gets the march (the same bits).
template <class Pol, int K, int F>
cudaError_t launch_default_scheme(const StageArgs& a, cudaStream_t s) {
    if (a.rows == 0 && a.variant == 0) {
        cudaError_t e = cudaSuccess;
        if (launch_tile<Pol, 4, F>(a, 1, s, e) || launch_tile<Pol, Pol::kMixed ? 10 : 8, F>(a, 2, s, e)) return e;
    }
    return launch_march_k<Pol, K, F>(a, s);
}

// The variant that runs by default, with the launch's scheme compiled in.
template <class Pol, int K, int F>
cudaError_t launch_march_default(const StageArgs& a, cudaStream_t s) {
    const bool last_of_step = a.stage == (a.rk == kRkTvd2 ? 1 : 2);
    const bool sr = !Pol::kMixed || stage_rounds_stochastically(a.rounding, last_of_step);
    switch (known_scheme(a.hll == kHllDavis, a.rk == kRkTvd3Ref, a.stage, sr)) {
        case kScheme0: return launch_default_scheme<Pol, K, F | kScheme0>(a, s);
        case kScheme1: return launch_default_scheme<Pol, K, F | kScheme1>(a, s);
        case kScheme2: return launch_default_scheme<Pol, K, F | kScheme2>(a, s);
        default: return launch_default_scheme<Pol, K, F>(a, s);
    }
}

}  // namespace

cudaError_t CFS_MARCH_FN(const StageArgs& a, int v, cudaStream_t s) {
    using P = CFS_MARCH_POL;
    constexpr int F = CFS_MARCH_FEAT;
    static_assert(kNumVariants == 13, "variant table and dispatch disagree");
    constexpr int kDefault = P::kMixed ? kDefaultVariantF32 : kDefaultVariantF64;
    if (v == kDefault) return launch_march_default<P, kDefault - 1, F>(a, s);
    switch (v) {
        case 1: return launch_march_k<P, 0, F>(a, s);
        case 2: return launch_march_k<P, 1, F>(a, s);
        case 3: return launch_march_k<P, 2, F>(a, s);
        case 4: return launch_march_k<P, 3, F>(a, s);
        case 5: return launch_march_k<P, 4, F>(a, s);
        case 6: return launch_march_k<P, 5, F>(a, s);
        case 7: return launch_march_k<P, 6, F>(a, s);
        case 8: return launch_march_k<P, 7, F>(a, s);
        case 9: return launch_march_k<P, 8, F>(a, s);
        case 10: return launch_march_k<P, 9, F>(a, s);
        case 11: return launch_march_k<P, 10, F>(a, s);
        case 12: return launch_march_k<P, 11, F>(a, s);
        case 13: return launch_march_k<P, 12, F>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace cfs
