// Tile form of the stage for small grids: the row march's arithmetic (the same
// device functions, so the same bits) with a warp per row instead of a warp
// per chunk of rows.
//
// On a grid that does not fill the GPU a stage lasts as long as one warp's
// chain of rows, and a row march of R rows is R + 2 row bodies long (two x
// reconstructions are repeated at its ends).  Here a block takes kTileRows
// rows of a 30-column segment with kTileRows + 2 warps: every warp reconstructs
// its own row in x (the outer two only that) and forms the y part of its row's
// RHS; left states pass to the row above through shared memory, each x-flux is
// formed once, passed down the same way, and the rows are updated.  So a stage
// is one row body long, and the repeated reconstructions are 2 in kTileRows.
// Step times of both forms, and where the line between them lies: launch_default_scheme
// (march_inst.cu).  Beyond it the march is faster: its 20 warps per SM never wait
// for each other, where a tile's wait twice a row body.
// No ring and no window: the stencils are read straight from the state (from
// L1 and L2 at these sizes), all loads issued before the first use.
#pragma once
#include "cfs_march.cuh"

namespace cfs {

// left x-states (7 values) and x-fluxes of the block's rows, by lane
template <class C, int kWarps>
struct TileSmem {
    C L[kWarps][7][32];
    C F[kWarps][kVars][32];
};

// Blocks per SM asked of the compiler: 16 warps (128 registers); the FP32
// 10-warp tile 2 blocks (102).
template <class T>
constexpr int tile_min_blocks(int warps) { return sizeof(T) == 4 && warps == 10 ? 2 : 16 / warps; }

template <class Pol, int kWarps, int kMinBlocks, int kFeat>
__global__ void __launch_bounds__(32 * kWarps, kMinBlocks) tile_kernel(const __grid_constant__ StageArgs a) {
    using T = typename Pol::T;
    using C = typename Pol::C;
    constexpr int kTileRows = kWarps - 2;
    constexpr bool kPos = (kFeat & kFeatPos) != 0;
    constexpr bool kExtra = (kFeat & kFeatExtra) != 0;
    constexpr bool kEdge = (kFeat & kFeatEdge) != 0;
    const int hll = (kFeat & kSchemeDavis) ? kHllDavis : (kFeat & kSchemeHllRef) ? kHllReference : a.hll;
    __shared__ TileSmem<C, kWarps> sm;
    const Layout& L = a.L;
    const int lane = threadIdx.x & 31;
    const int wid = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // (uniform to the compiler)
    const int nseg = (L.ny + kSeg - 1) / kSeg;
    const int j0 = static_cast<int>(blockIdx.x % nseg) * kSeg;
    const int i0 = stage_row_lo(a) + static_cast<int>(blockIdx.x / nseg) * kTileRows;
    const int i1 = min(i0 + kTileRows, stage_row_hi(a));
    const int r = i0 - 1 + wid;                  // this warp's row
    const int j = j0 - 1 + lane;                 // this lane's column
    const bool active = r <= i1;                 // row i0 - 1 and row i1 in x only
    const bool inner = r >= i0 && r < i1;
    const bool owner = inner && lane >= 1 && lane <= kSeg && j < L.ny;  // updates its cell
    const T* in = static_cast<const T*>(a.in);
    const C eps = C(a.eps);
    const double g = a.gamma;
    let_next_in();
    after_previous();
    const UpdateCoefs uc = update_coefs<Pol, kFeat>(a);
    if (a.P && a.first_stage && blockIdx.x == 0 && threadIdx.x == 0) begin_step(a, uc.dt);

    auto full = [&](const C w[kVars], C out[kVars]) {
#pragma unroll
        for (int v = 0; v < kVars; ++v) out[v] = Pol::kMixed ? w[v] + C(L.off[v]) : w[v];
    };
    // stored values: the 5 rows of this lane's column, the 5 columns of this
    // row (columns past the padded row repeat its last one: their lanes feed no owner)
    const int jmax = L.ny + kGhost - 1;
    C win[5][kVars], st[5][kVars];
    T u0c[kVars] = {T(0), T(0), T(0), T(0)}, u1c[kVars] = {T(0), T(0), T(0), T(0)};
    T rvc[kRvWords] = {T(0), T(0), T(0)};
    unsigned int f_r = 0u;
    if (active) {
#pragma unroll
        for (int k = 0; k < 5; ++k) ld_cell<T>(in, L.offset(r - 2 + k, min(j, jmax)), win[k]);
        if (kEdge && a.cflags && j <= L.ny) f_r = a.cflags[static_cast<long long>(r + 1) * (L.ny + 2) + (j + 1)];
    }
    if (inner) {
#pragma unroll
        for (int k = 0; k < 5; ++k)
            if (k != 2) ld_cell<T>(in, L.offset(r, min(j - 2 + k, jmax)), st[k]);
    }
    if (owner) {
        if (a.stage >= 1) ld_cell<T>(static_cast<const T*>(a.u0), L.offset(r, j), u0c);
        if (uc.x1_u1) ld_cell<T>(static_cast<const T*>(a.u1), L.offset(r, j), u1c);
        if (kExtra && a.rv) ld_rv<T>(static_cast<const T*>(a.rv), static_cast<long long>(r) * L.ny + j, rvc);
    }
    // ---- x reconstruction of row r; its left state to the row above
    Face5<C> Lr{}, Rr{};
    C RY[kVars] = {C(0), C(0), C(0), C(0)};
    if (active) {
        cell_states<Pol>(win, eps, g, Lr, Rr, Pol::kMixed ? L.off : nullptr);
        if constexpr (kPos) {
            C cc[kVars];
            full(win[2], cc);
            fix_states<Pol>(f_r & kCellLowXhi, f_r & kCellLowXlo, cc, g, Lr, Rr);
        }
        C(*s)[32] = sm.L[wid];
        s[0][lane] = Lr.r;
        s[1][lane] = Lr.mx;
        s[2][lane] = Lr.my;
        s[3][lane] = Lr.E;
        s[4][lane] = Lr.p;
        s[5][lane] = Lr.a;
        s[6][lane] = Lr.ri;
    }
    // ---- y part of row r
    if (inner) {
#pragma unroll
        for (int v = 0; v < kVars; ++v) st[2][v] = win[2][v];
        const bool lo_y = kEdge && physical_side(a, 2), hi_y = kEdge && physical_side(a, 3);
        const bool ybnd = (j == -1 && lo_y) || (j == L.ny - 1 && hi_y);
        const bool warp_ybnd = __any_sync(0xffffffffu, ybnd);
        const C* const bfl = static_cast<const C*>(a.bflux);
        const C* const bfy = ybnd && (j == -1 ? a.bc[2] == kDirichlet : a.bc[3] == kDirichlet)
                                 ? bfl + (j == -1 ? bflux_side_offset(L, 2) : bflux_side_offset(L, 3)) : nullptr;
        y_part<Pol, kFeat, Pol::kMixed>(a, uc, r, j, hll, st, eps, f_r, warp_ybnd, ybnd, bfy, RY);
    }
    __syncthreads();
    // ---- x-flux through the face below row r
    C FX[kVars];
    if (active && wid >= 1) {
        Face5<C> Lx;
        const C(*s)[32] = sm.L[wid - 1];
        Lx.r = s[0][lane];
        Lx.mx = s[1][lane];
        Lx.my = s[2][lane];
        Lx.E = s[3][lane];
        Lx.p = s[4][lane];
        Lx.a = s[5][lane];
        Lx.ri = s[6][lane];
        hll_flux<Pol>(Lx, Rr, 0, hll, g, FX);
        if (kEdge && ((r == 0 && physical_side(a, 0)) || (r == L.nx && physical_side(a, 1)))) {
            C c[kVars];
            if (r == 0) full(win[2], c);
            else full(win[1], c);
            boundary_x_flux<Pol>(a, r, j, c, FX);
        }
#pragma unroll
        for (int v = 0; v < kVars; ++v) sm.F[wid][v][lane] = FX[v];
    }
    __syncthreads();
    // ---- update of row r
    double wloc = 0.0;
    if (owner) {
        C FXu[kVars];
#pragma unroll
        for (int v = 0; v < kVars; ++v) FXu[v] = sm.F[wid + 1][v][lane];
        const bool fluid = !kEdge || !(f_r & kCellSolid);
        T cur[kVars];
#pragma unroll
        for (int v = 0; v < kVars; ++v) cur[v] = T(win[2][v]);
        update_cell<Pol, kFeat>(a, uc, r, j, FXu, FX, RY, rvc, cur, a.stage >= 1 ? u0c : cur, u1c, fluid, wloc);
    }
    if (uc.do_cfl && inner) raise_wmax(a, wloc);
}

}  // namespace cfs
