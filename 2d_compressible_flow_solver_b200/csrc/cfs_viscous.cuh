// Viscous (Navier-Stokes) terms of one state as a row march.
//
// No reference counterpart is live: the reference computes a viscous flux but
// never adds it (Cell.cpp:128-133, Run.cpp:177,188).  Here: u, v and
// T = gamma Ma^2 p / rho; cell-centred 4th-order derivatives with the
// reference's table theta_c (FourthOrderCS.h:34-36); at each face the normal
// derivative from theta_r[1] over 6 cells (FourthOrderCS.h:28-32), the cross
// derivative and u, v interpolated with zeta_r[1] (FourthOrderCS.h:38-42);
// stresses sigma_11 = mu (4/3 u_x - 2/3 v_y), sigma_12 = mu (u_y + v_x), heat
// flux kT T_x with kT = mu / ((gamma-1) Ma^2 Pr).  The tables are
// antisymmetric (derivatives) or symmetric (interpolation), so a stencil
// takes one difference or sum per pair of cells and one multiply-add each.
//
// A warp's 32 lanes hold columns j0-3 .. j0+28 of a 26-column segment and
// march down x.  Everything along x comes from registers: (u, v) and T of the
// last six rows and (u_y, v_y) of the last four (the row loop is unrolled by
// six, so a row's place in the window is known at compile time and no values
// are moved).  What a lane needs of its neighbours in y -- the row's values,
// and (u_x, v_x) for the cross derivatives -- goes through per-warp rows in
// shared memory, ordered by __syncwarp: no block barriers, no halo tile.  Row q
// is converted (its load issued three rows earlier) and its y-derivatives
// taken; then the x-face between rows q-3 and q-2 and the y-faces of row q-3
// have all their values, and row q-3 is finished.  u and v of a lane share
// packed FP32 instructions.
//
// Bound by instruction issue (202 instructions per cell in FP32, 0.61 issued a
// cycle) and, cold, by its loads.  The kernel before worked on 16 x 32 tiles
// (FP64 8 x 32) with a 3-cell halo, five phases through shared memory with
// block barriers between them: 526 instructions per cell.  2048^2 FP32: 87 ->
// 45 us a launch (ncu, cold); whole Navier-Stokes SSP3 steps 1024^2 FP32 177
// -> 155 us, 2048^2 FP64 1,091 (an earlier form of this kernel) -> 928.  Three
// words a cell stored, in scalar stores: 1024^2 145.5 us with a fourth, unused
// word in one 16-byte store, 144.2 without.
// 26 columns a warp rather than 28 with a second pass for two halo columns:
// the pass would cost more than the two lanes.  5 blocks of 4 warps per SM in
// FP32 (89 registers) and 3 in FP64 (158): 4 blocks of either ran 2048^2 3 to
// 4 % slower, FP64 with spills.
#pragma once
#include "cfs_kernels.cuh"

namespace cfs {

constexpr int kViscSeg = 26;   // columns a warp finishes
constexpr int kViscWin = 6;    // rows of the window, and of the shared value ring
constexpr int kViscWarps = 4;

// (u, v) pairs: packed FP32 instructions, two FP64 ones.
template <class C> struct Pair;
template <> struct Pair<float> { using type = float2; };
template <> struct Pair<double> { using type = double2; };
__device__ __forceinline__ double2 add2(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 sub2(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 mul2(double2 a, double2 b) { return make_double2(mul(a.x, b.x), mul(a.y, b.y)); }
__device__ __forceinline__ double2 fma2(double2 a, double2 b, double2 c) {
    return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
__device__ __forceinline__ double2 p2(double a) { return make_double2(a, a); }

__device__ __forceinline__ float2 make_pair_of(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 make_pair_of(double a, double b) { return make_double2(a, b); }

// A warp's shared rows: pairs and temperatures apart, so that consecutive
// lanes read consecutive words.
template <class C>
struct ViscSmem {
    typename Pair<C>::type uv[kViscWin][32 + 6];  // column of lane l at l + 3 (neighbours of the outer lanes unused)
    C T[kViscWin][32 + 6];
    typename Pair<C>::type gx[2][32 + 4];         // (u_x, v_x) of lane l at l + 1, of even and odd rows
};

// Constants of one direction's faces: the normal derivative's table over h
// (t), and mu and kT over h as well, so that differences of fluxes need no
// scaling; pairs for the packed operations.
template <class C, class V>
struct ViscDir {
    V t0, t1, t2;
    C mu43, mu23, mu, kT;
    __device__ __forceinline__ ViscDir(C inv_h, C m, C k)
        : t0(p2(C(75.0 / 64) * inv_h)), t1(p2(C(-25.0 / 384) * inv_h)), t2(p2(C(3.0 / 640) * inv_h)),
          mu43(C(4.0 / 3.0) * m * inv_h), mu23(C(2.0 / 3.0) * m * inv_h), mu(m * inv_h), kT(k * inv_h) {}
};

// Stress and heat fluxes (over h) through the face between the cells 2 and 3
// of a normal's six: (u, v) pairs w and temperatures T of the six, cross
// derivatives cr at the face; nrm picks the normal velocity (0 u, 1 v).  F: u-
// and v-momentum and energy.
template <class C, class V>
__device__ __forceinline__ void visc_flux(int nrm, const ViscDir<C, V>& k, V w0, V w1, V w2, V w3, V w4, V w5, C T0, C T1,
                                          C T2, C T3, C T4, C T5, V cr, V n16, V m16, C F[3]) {
    const V dn = fma2(k.t0, sub2(w3, w2), fma2(k.t1, sub2(w4, w1), mul2(k.t2, sub2(w5, w0))));
    const C dT = fma(k.t0.x, T3 - T2, fma(k.t1.x, T4 - T1, mul(k.t2.x, T5 - T0)));
    const V f = fma2(n16, add2(w2, w3), mul2(m16, add2(w1, w4)));
    const C snn = nrm == 0 ? fma(k.mu43, dn.x, -mul(k.mu23, cr.y)) : fma(k.mu43, dn.y, -mul(k.mu23, cr.x));
    const C snt = nrm == 0 ? mul(k.mu, cr.x + dn.y) : mul(k.mu, dn.x + cr.y);
    F[0] = nrm == 0 ? snn : snt;
    F[1] = nrm == 0 ? snt : snn;
    F[2] = fma(f.x, F[0], fma(f.y, F[1], mul(k.kT, dT)));
}

// Cell-centred derivatives, scaled for the interpolation that reads them:
// cross_of(g..) = (9 (g1 + g2) - (g0 + g3))/16 of derivatives g is -9 (g1 + g2) + (g0 + g3)
// of derivatives held times -1/16 (the factor s = -1/(12 16 h)).
template <class V> __device__ __forceinline__ V centred(V m2, V m1, V p1, V pp2, V eight_s, V s) {
    return fma2(eight_s, sub2(p1, m1), mul2(s, sub2(m2, pp2)));
}
template <class V> __device__ __forceinline__ V cross_of(V g0, V g1, V g2, V g3, V minus9) {
    return fma2(minus9, add2(g1, g2), add2(g0, g3));
}

template <class Pol, int kMinBlocks>
__global__ void __launch_bounds__(32 * kViscWarps, kMinBlocks) viscous_kernel(const ViscArgs a) {
    using T = typename Pol::T;
    using C = typename Pol::C;
    using V = typename Pair<C>::type;
    __shared__ ViscSmem<C> smem[kViscWarps];
    const Layout& L = a.L;
    const int lane = threadIdx.x & 31;
    const int wid = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // (uniform to the compiler)
    ViscSmem<C>& sm = smem[wid];
    const int nseg = (L.ny + kViscSeg - 1) / kViscSeg;
    const long long gw = static_cast<long long>(blockIdx.x) * kViscWarps + wid;
    const int i0 = static_cast<int>(gw / nseg) * a.rows;
    let_next_in();
    after_previous();
    if (i0 >= L.nx) return;  // (a warp past the last item; nothing below is block-wide)
    const int i1 = min(i0 + a.rows, L.nx);
    const int j = static_cast<int>(gw % nseg) * kViscSeg - 3 + lane;  // this lane's column
    const bool stores = lane >= 3 && lane < 3 + kViscSeg && j < L.ny;

    constexpr bool kF = sizeof(C) == 4;  // FP32 form: constants rounded on the host
    const C idx = kF ? C(a.inv_dx_f) : C(a.inv_dx), idy = kF ? C(a.inv_dy_f) : C(a.inv_dy);
    const C mu = kF ? C(a.mu_f) : C(a.mu), kT = kF ? C(a.kT_f) : C(a.kT);
    const C cTg = (kF ? C(a.cT_f) : C(a.gamma * a.mach2)) * (kF ? C(a.gm1_f) : C(a.gamma - 1));
    const ViscDir<C, V> X(idx, mu, kT), Y(idy, mu, kT);
    const V sx = p2(C(-1.0 / 192) * idx), sx8 = p2(C(-8.0 / 192) * idx), sy = p2(C(-1.0 / 192) * idy), sy8 = p2(C(-8.0 / 192) * idy);
    const V minus9 = p2(C(-9)), n16 = p2(C(9.0 / 16)), m16 = p2(C(-1.0 / 16));

    const T* src = static_cast<const T*>(a.in) + Layout::at(L.offset(i0 - 3, min(j, L.ny + kGhost - 1)), 0);
    const long long row_step = static_cast<long long>(L.pitch) * kVars;
    T raw[3][kVars];
#pragma unroll
    for (int k = 0; k < 3; ++k, src += row_step) ld_cell<T>(src, 0, raw[k]);

    constexpr int W = kViscWin;
    V uv[W], gy[W];
    C tt[W], FXp[3];
    // row q into slot k (a compile-time constant): u, v, T; the load slot takes row q + 3
    auto convert = [&](int k, int q) {
        C c[kVars];
#pragma unroll
        for (int v = 0; v < kVars; ++v) c[v] = decc<T, C>(raw[k % 3][v], L, v);
        if (q + 3 <= i1 + 2) ld_cell<T>(src, 0, raw[k % 3]);
        src += row_step;
        const C ri = rcp_pos(c[0]);
        uv[k] = mul2(make_pair_of(c[1], c[2]), p2(ri));
        tt[k] = mul(mul(cTg, fma(C(-0.5), fma(c[1], uv[k].x, mul(c[2], uv[k].y)), c[3])), ri);
        sm.uv[k][lane + 3] = uv[k];
        sm.T[k][lane + 3] = tt[k];
    };
    auto y_derivative = [&](int k) {
        gy[k] = centred(sm.uv[k][lane + 1], sm.uv[k][lane + 2], sm.uv[k][lane + 4], sm.uv[k][lane + 5], sy8, sy);
    };
    // x-face between rows q-3 and q-2, row q in slot k (row q-5+m of the window is slot (k+1+m) % 6)
    auto x_face = [&](int k, C F[3]) {
        visc_flux<C, V>(0, X, uv[(k + 1) % W], uv[(k + 2) % W], uv[(k + 3) % W], uv[(k + 4) % W], uv[(k + 5) % W], uv[k],
                        tt[(k + 1) % W], tt[(k + 2) % W], tt[(k + 3) % W], tt[(k + 4) % W], tt[(k + 5) % W], tt[k],
                        cross_of(gy[(k + 2) % W], gy[(k + 3) % W], gy[(k + 4) % W], gy[(k + 5) % W], minus9), n16, m16, F);
    };
    // rows i0-3 .. i0+2 fill the window; the item's first x-face
#pragma unroll
    for (int k = 0; k < W; ++k) {
        convert(k, i0 - 3 + k);
        __syncwarp();
        if (k >= 1) y_derivative(k);  // (row i0-3's is not read)
    }
    x_face(W - 1, FXp);
    T* out = static_cast<T*>(a.rv) + (static_cast<long long>(i0) * L.ny + j) * kRvWords;
    for (int pb = i0; pb < i1; pb += W) {
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const int p = pb + k;  // the row finished here; row q = p + 3 enters slot k
            if (p >= i1) break;
            // ---- values of row q and x-derivatives of row p to the lanes
            V* const gx = sm.gx[k & 1];
            gx[lane + 1] = centred(uv[(k + 1) % W], uv[(k + 2) % W], uv[(k + 4) % W], uv[(k + 5) % W], sx8, sx);
            convert(k, p + 3);
            __syncwarp();
            y_derivative(k);
            C FX[3], GY[3];
            x_face(k, FX);
            // ---- the y-face above this lane's cell of row p: columns j-2 .. j+3
            const V* w = &sm.uv[(k + 3) % W][lane + 1];
            const C* t = &sm.T[(k + 3) % W][lane + 1];
            visc_flux<C, V>(1, Y, w[0], w[1], w[2], w[3], w[4], w[5], t[0], t[1], t[2], t[3], t[4], t[5],
                            cross_of(gx[lane], gx[lane + 1], gx[lane + 2], gx[lane + 3], minus9), n16, m16, GY);
#pragma unroll
            for (int v = 0; v < kRvWords; ++v) {
                const C below = __shfl_up_sync(0xffffffffu, GY[v], 1);
                const T o = T((FX[v] - FXp[v]) + (GY[v] - below));
                if (stores) out[v] = o;
                FXp[v] = FX[v];
            }
            out += static_cast<long long>(L.ny) * kRvWords;
        }
    }
}

}  // namespace cfs
