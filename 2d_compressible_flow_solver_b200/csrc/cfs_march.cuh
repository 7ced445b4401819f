// Row-marching stage kernel of the throughput forms (CFS_FP64, CFS_FP32_MIXED).
//
// Work decomposition: a warp owns a segment of kSeg = 30 consecutive y-cells
// (columns j0 .. j0+29); its 32 lanes hold columns j0-1 .. j0+30, so every
// interior cell has both y-neighbours' reconstructions inside the warp.  The
// warp marches down x (rows) from i0-1 to i1:
//  * the x-stencil of a lane is a 5-row register window of its column, one new
//    row loaded per step (no shared memory, no block barrier);
//  * the y-stencil comes from a per-warp row buffer in shared memory (the 32
//    lane values plus 2 halo columns each side), synchronised with __syncwarp;
//  * each cell reconstructs its own left- and right-biased WENO5 states per
//    direction and variable from ONE set of smoothness indicators (the
//    indicators of the two states are the same three numbers in mirrored
//    order), then each face's HLL flux takes the left state of the cell below
//    it and the right state of the cell above (a shuffle in y, the previous
//    march step in x);
//  * the RK update of row r-1 happens at step r, when its upper x-face exists.
// Physical boundary faces use the reference's stencil (CellInterface.cpp:
// 172-178: both walkers stop, so interior slots repeat the first interior cell).
#pragma once
#include "cfs_kernels.cuh"
#include "cfs_launch.h"

namespace cfs {

constexpr int kSeg = 30;

// Left- and right-biased WENO5 states of the middle cell of v0..v4
// (Weno5th.cpp:4-28 applied to v0..v4 and to v4..v0), rewritten on the
// differences D1..D4 (Dk = v_k - v_{k-1}) so that both states share one set of
// smoothness indicators and weight products and are formed as v2 plus a small
// correction (fewer operations, and in FP32 a rounding error relative to the
// correction instead of to the value):
//   indicators: 13/12 d^2 + 1/4 e^2 with (d, e) = (D2-D1, 3 D2-D1),
//     (D3-D2, D2+D3), (D4-D3, D4-3 D3), multiplied out and scaled by 3/4 (with
//     eps alike, which leaves the normalised weights unchanged) so that every
//     coefficient is a short binary fraction and eps enters a fused
//     multiply-add:
//       D1 (D1 - 11/4 D2) + 5/2 D2^2,  D2 (D2 - 5/4 D3) + D3^2,
//       D4 (D4 - 11/4 D3) + 5/2 D3^2;
//     the forms are positive definite (at least 0.24 D1^2, 0.61 D2^2, ...), so
//     multiplying out costs a relative rounding of at most about 13 units in an
//     indicator and no sign;
//   weights d_k / q_k with q_k = (eps + beta_k)^2 as products of the other two
//     q: X = q1 q2, Y = q0 q2, Z = q0 q1 times (1, 6, 3) on the left, (3, 6, 1)
//     on the right (the linear weights 0.1, 0.6, 0.3 times 10);
//   candidates v2 + c_k: c = (5/6 A0, A1/3, 2/3 A2) with A0 = D2 - 2/5 D1,
//     A1 = D3 + 1/2 D2, A2 = D3 - 1/4 D4, one fused multiply-add each, and
//     mirrored with a sign on the right (D1 <-> D4, D2 <-> D3);
//   left  = v2 + (5/12 X A0 + Y A1 + Z A2) / (X/2 + 3 Y + 3/2 Z),
//   right = v2 - (5/12 Z B0 + Y B1 + X B2) / (Z/2 + 3 Y + 3/2 X), the sums as
//     3/2 (X + Z + 2 Y) - X and - Z.
// 41 operations and two reciprocals per variable (52 before, with d, e and the
// candidates formed separately): the row march is bound by issue (FP32) and
// by the FP64 pipe, and this is more than half of its arithmetic.  Measured with
// the HLL flux written from the left flux (hll_flux): SSP3 step of 4096^2
// FP32-mixed 1,536 -> 1,412 us, of 2048^2 FP64 759 -> 690 us.
template <class C>
__device__ __forceinline__ void weno5_pair_diff(C v0, C v1, C v2, C v3, C v4, C eps, C& left, C& right) {
    const C D1 = v1 - v0, D2 = v2 - v1, D3 = v3 - v2, D4 = v4 - v3;
    const C P2 = mul(D2, D2), P3 = mul(D3, D3);
    C q0 = fma(D1, fma(C(-2.75), D2, D1), fma(C(2.5), P2, eps));  // eps: the WENO eps times 3/4
    C q1 = fma(D2, fma(C(-1.25), D3, D2), P3 + eps);
    C q2 = fma(D4, fma(C(-2.75), D3, D4), fma(C(2.5), P3, eps));
    q0 *= q0;
    q1 *= q1;
    q2 *= q2;
    const C X = mul(q1, q2), Y = mul(q0, q2), Z = mul(q0, q1);
    const C X5 = mul(C(5.0 / 12.0), X), Z5 = mul(C(5.0 / 12.0), Z);
    const C h = fma(C(2), Y, X + Z);
    const C A0 = fma(C(-0.4), D1, D2), A1 = fma(C(0.5), D2, D3), A2 = fma(C(-0.25), D4, D3);
    const C B0 = fma(C(-0.4), D4, D3), B1 = fma(C(0.5), D3, D2), B2 = fma(C(-0.25), D1, D2);
    // (the weight sums are >= 5 eps^4 > 0: rcp_pos)
    left = fma(fma(X5, A0, fma(Y, A1, mul(Z, A2))), rcp_pos(fma(C(1.5), h, -X)), v2);
    right = fma(fma(Z5, B0, fma(Y, B1, mul(X, B2))), -rcp_pos(fma(C(1.5), h, -Z)), v2);
}

template <class C>
__device__ __forceinline__ void weno5_pair(C v0, C v1, C v2, C v3, C v4, C eps, C& left, C& right) {
    weno5_pair_diff(v0, v1, v2, v3, v4, mul(C(0.75), eps), left, right);
}

// The same pair for two variables at once in packed FP32 (sm_100 FFMA2 /
// FADD2 / FMUL2: two independent FP32 operations per instruction, each rounded
// as its scalar form), for the FP32-mixed form, whose row loop is bound by
// instruction issue.  The weights are taken relative to the middle one: X =
// (q1 / q0)^2, Y = 1, Z = (q1 / q2)^2, from two scalar reciprocals (the sums take
// two more).  q0 and q2 hold 1e-12 of the square beyond them as well: X and Z
// stay below 1e25 at any jump, and a weight is moved only where it is 1e9 times
// the others and more.  So the states are finite, and the weights what they are
// in more bits, on jumps and ramps of up to 1e18 a cell and for any eps in the FP32
// range.  (With X = (q1 q2)^2, Y = (q0 q2)^2, Z = (q0 q1)^2 the indicators had to be
// capped at 1e9, which made the weights of larger jumps the linear ones, and the sums
// still overflowed on a ramp of 2e4 a cell; this form has the reciprocals on their own
// pipe in the place of six scalar caps: 4096^2 step 1,219 -> 1,196 us, 48 batched
// cases 825 -> 804.)
__device__ __forceinline__ float2 rcp2(float2 q) { return make_float2(rcp_fast(q.x), rcp_fast(q.y)); }

__device__ __forceinline__ void weno5_pair_x2(float2 v0, float2 v1, float2 v2, float2 v3, float2 v4, float eps,
                                              float2& left, float2& right) {
    const float2 D1 = sub2(v1, v0), D2 = sub2(v2, v1), D3 = sub2(v3, v2), D4 = sub2(v4, v3);
    const float2 P2 = mul2(D2, D2), P3 = mul2(D3, D3);
    const float2 es = p2(0.75f * eps), tiny = p2(kWenoTiny);
    const float2 q1 = fma2(D2, fma2(p2(-1.25f), D3, D2), add2(P3, es));
    const float2 q0 = fma2(D1, fma2(p2(-2.75f), D2, D1), fma2(p2(2.5f), P2, fma2(tiny, P3, es)));
    const float2 q2 = fma2(D4, fma2(p2(-2.75f), D3, D4), fma2(p2(2.5f), P3, fma2(tiny, P2, es)));
    const float2 r0 = mul2(q1, rcp2(q0)), r2 = mul2(q1, rcp2(q2));
    const float2 X = mul2(r0, r0), Z = mul2(r2, r2);
    const float2 X5 = mul2(p2(float(5.0 / 12.0)), X), Z5 = mul2(p2(float(5.0 / 12.0)), Z);
    const float2 h = add2(add2(X, Z), p2(2.0f));
    const float2 A0 = fma2(p2(-0.4f), D1, D2), A1 = fma2(p2(0.5f), D2, D3), A2 = fma2(p2(-0.25f), D4, D3);
    const float2 B0 = fma2(p2(-0.4f), D4, D3), B1 = fma2(p2(0.5f), D3, D2), B2 = fma2(p2(-0.25f), D1, D2);
    // (both sums negated, one packed operation each; the left reciprocals' sign is taken back in their argument)
    const float2 sL = fma2(p2(-1.5f), h, X), sR = fma2(p2(-1.5f), h, Z);
    const float2 iL = make_float2(rcp_fast(-sL.x), rcp_fast(-sL.y)), iR = rcp2(sR);
    left = fma2(fma2(X5, A0, fma2(Z, A2, A1)), iL, v2);
    right = fma2(fma2(Z5, B0, fma2(X, B2, B1)), iR, v2);
}

// finish_state of a cell's two states at once (FP32-mixed: a state whose
// kinetic energy exceeds 90 % of E takes the FP64 path of finish_state).
// Scalar: the packed form did the same operations in half the instructions
// but moved eight values into register pairs first, and a packed operation
// keeps the FMA pipe busy as long as two scalar ones (4096^2 step 1,308 ->
// 1,278 us).  With ke = m^2 / rho / 2
// and t = E - ke: p = (g - 1) t, a = sqrt(g (g - 1) t / rho).
template <class Pol>
__device__ __forceinline__ void finish_pair(Face5<typename Pol::C>& L, Face5<typename Pol::C>& R, double g) {
    if constexpr (Pol::kMixed) {
        const float gm1 = float(g - 1), gg = float(g) * float(g - 1);
        const float riL = rcp_fast(L.r), riR = rcp_fast(R.r);
        const float tL = fmaf(-0.5f, mul(fmaf(L.mx, L.mx, mul(L.my, L.my)), riL), L.E);
        const float tR = fmaf(-0.5f, mul(fmaf(R.mx, R.mx, mul(R.my, R.my)), riR), R.E);
        if (tL < 0.1f * L.E || tR < 0.1f * R.E) {
            finish_state<Pol>(L, g);
            finish_state<Pol>(R, g);
            return;
        }
        L.ri = riL;
        R.ri = riR;
        L.p = mul(gm1, tL);
        R.p = mul(gm1, tR);
        L.a = sqrt_fast(mul(mul(gg, tL), riL));
        R.a = sqrt_fast(mul(mul(gg, tR), riR));
    } else {
        finish_state<Pol>(L, g);
        finish_state<Pol>(R, g);
    }
}

// Both states of one cell from a 5-cell stencil st[k][v] (k = 0..4).  The
// FP32-mixed form pairs (rho, rho u) and (rho v, E) in packed instructions.
// With `off` the stencil holds stored deviations (value - off[v]): WENO5 is
// translation invariant (the difference form sees only differences), so the
// states are reconstructed from the deviations and the offsets added once.
template <class Pol>
__device__ __forceinline__ void cell_states(const typename Pol::C st[5][kVars], typename Pol::C eps, double g,
                                            Face5<typename Pol::C>& L, Face5<typename Pol::C>& R,
                                            const float* off = nullptr) {
    if constexpr (Pol::kMixed) {
        float2 l, r;
        weno5_pair_x2(make_float2(st[0][0], st[0][1]), make_float2(st[1][0], st[1][1]), make_float2(st[2][0], st[2][1]),
                      make_float2(st[3][0], st[3][1]), make_float2(st[4][0], st[4][1]), eps, l, r);
        if (off) {
            const float2 o = make_float2(off[0], off[1]);
            l = add2(l, o);
            r = add2(r, o);
        }
        L.r = l.x;
        L.mx = l.y;
        R.r = r.x;
        R.mx = r.y;
        weno5_pair_x2(make_float2(st[0][2], st[0][3]), make_float2(st[1][2], st[1][3]), make_float2(st[2][2], st[2][3]),
                      make_float2(st[3][2], st[3][3]), make_float2(st[4][2], st[4][3]), eps, l, r);
        if (off) {
            const float2 o = make_float2(off[2], off[3]);
            l = add2(l, o);
            r = add2(r, o);
        }
        L.my = l.x;
        L.E = l.y;
        R.my = r.x;
        R.E = r.y;
    } else {
        weno5_pair(st[0][0], st[1][0], st[2][0], st[3][0], st[4][0], eps, L.r, R.r);
        weno5_pair(st[0][1], st[1][1], st[2][1], st[3][1], st[4][1], eps, L.mx, R.mx);
        weno5_pair(st[0][2], st[1][2], st[2][2], st[3][2], st[4][2], eps, L.my, R.my);
        weno5_pair(st[0][3], st[1][3], st[2][3], st[3][3], st[4][3], eps, L.E, R.E);
    }
    finish_pair<Pol>(L, R, g);
}

// Reference boundary face between an interior cell value c and a ghost value g
// (lo = true: ghost below, stencil [g g g | c c c]; lo = false: [c c c | g g g]).
template <class Pol>
__device__ __forceinline__ void boundary_face_states(const typename Pol::C c[kVars], const typename Pol::C gh[kVars],
                                                     bool lo, typename Pol::C eps, double g,
                                                     Face5<typename Pol::C>& L, Face5<typename Pol::C>& R) {
    using C = typename Pol::C;
    C* lp[4] = {&L.r, &L.mx, &L.my, &L.E};
    C* rp[4] = {&R.r, &R.mx, &R.my, &R.E};
#pragma unroll
    for (int v = 0; v < kVars; ++v) {
        const C a = lo ? gh[v] : c[v], b = lo ? c[v] : gh[v];
        // stencil s = (a, a, a, b, b, b): left from s0..s4, right from s5..s1
        *lp[v] = weno5<Pol>(a, a, a, b, b, eps);
        *rp[v] = weno5<Pol>(b, b, b, a, a, eps);
    }
    finish_state<Pol>(L, g);
    finish_state<Pol>(R, g);
}

// Asynchronous global -> shared copies (cp.async, sm_80+): 16 bytes each,
// bypassing L1, zero filled without reading when `valid` is false (gmem must
// still be a valid address); completion per thread in commit groups.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n) : "memory");
}
// one cell of the stored state (all four variables), zero filled when not valid
template <class T>
__device__ __forceinline__ void cp_async_cell(T* smem, const T* gmem, bool valid) {
    cp_async16(smem, gmem, valid);
    if constexpr (sizeof(T) == 8) cp_async16(smem + 2, gmem + 2, valid);
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Ring of staged rows of the row march (load schedules 3 and 4), per warp:
// kRingRows rows of its 36 columns (the segment and 2 halo columns each side,
// whole cells), stored values, and (FP32 storage) the rows of U^0.  The FP64
// ring leaves U^0 out (each lane loads it early in the row's iteration): its
// rows of doubles would otherwise cost a fourth block per SM.
//
// cp.async (schedule 3): rows packed (576 / 1,152 bytes), U^0 rows of the 32
// lanes' own columns.  (Keeping the first four slots once more behind the
// last, so that an x-stencil's five rows are immediate offsets from one
// address, takes 27 instructions per cell-stage less but lost: 1,329 against
// 1,317 us for the 4096^2 step, FP64 677 against 647 at 2048^2; the ring then
// takes all of the SM's shared memory.)
//
// TMA (schedule 4): one box per row; a row starts 128-byte
// aligned, as a TMA copy's shared-memory destination must (its stride rounded
// up to 128 bytes: FP32 640, FP64 1,152), U^0 rows alike.
constexpr int kRingRows = 8, kRingDist = 2;
constexpr int kRingCols = 36;
template <class T>
__host__ __device__ constexpr int ring_row_words() {
    return ((kRingCols * kVars * static_cast<int>(sizeof(T)) + 127) / 128) * 128 / static_cast<int>(sizeof(T));
}
template <class T, int kLoad>
__host__ __device__ constexpr int ring_words() {
    if (kLoad == 3) return kRingRows * (kRingCols + (sizeof(T) == 4 ? 32 : 0)) * kVars;
    return (sizeof(T) == 4 ? 2 : 1) * kRingRows * ring_row_words<T>();
}
static_assert(ring_row_words<float>() * 4 % 128 == 0 && ring_row_words<double>() * 8 % 128 == 0,
              "TMA ring rows start 128-byte aligned");
static_assert(ring_words<float, 4>() * 4 % 128 == 0 && ring_words<double, 4>() * 8 % 128 == 0 &&
                  ring_words<float, 3>() * 4 % 128 == 0 && ring_words<double, 3>() * 8 % 128 == 0,
              "each warp's ring starts 128-byte aligned");

// ---- TMA staging (load schedule 4).  One elected lane of a warp copies a
// whole ring row -- the 4 variables of 36 cells, one box of the state
// buffer's 3-D tensor map (variables, columns, rows) -- with one bulk tensor
// copy that signals an mbarrier of the row's ring slot; the lanes wait on
// that barrier instead of issuing per-lane copies.  The tensor maps travel in
// the kernel's __grid_constant__ argument block (StageArgs::tmap_in,
// tmap_u0) and cover this GPU's own state buffers only; no copy is
// multicast.  Every wait is bounded: a copy that never lands sets
// *StageArgs::err and ends the work item.
__device__ __forceinline__ unsigned smem_addr(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0u;
}
// try_wait suspends the thread for a system-dependent time per attempt; this
// many attempts is far beyond any copy's latency (a row lands within a few
// microseconds); the drain after a failure tries less
constexpr int kMbarMaxTries = 1 << 20;
constexpr int kMbarDrainTries = 1 << 14;
__device__ __forceinline__ bool mbar_wait_bounded(unsigned bar, unsigned parity, int tries = kMbarMaxTries) {
    for (int k = 0; k < tries; ++k)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// generic-proxy accesses of this thread (and, after a __syncwarp, of its warp)
// before later async-proxy (TMA) writes to shared memory
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void tma_load_row(unsigned dst, const void* tmap, int col, int row, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n"
        ::"r"(dst), "l"(tmap), "r"(0), "r"(col), "r"(row), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_prefetch_map(const void* tmap) {
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(tmap) : "memory");
}

// One column's 4 variables to / from the shared row buffer in vector accesses.
template <class C>
__device__ __forceinline__ void put_slot(C (&slot)[kVars], const C v[kVars]) {
    if constexpr (sizeof(C) == 4) {
        *reinterpret_cast<float4*>(slot) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
        reinterpret_cast<double2*>(slot)[0] = make_double2(v[0], v[1]);
        reinterpret_cast<double2*>(slot)[1] = make_double2(v[2], v[3]);
    }
}

template <class C>
__device__ __forceinline__ void get_slot(const C (&slot)[kVars], C v[kVars]) {
    if constexpr (sizeof(C) == 4) {
        const float4 t = *reinterpret_cast<const float4*>(slot);
        v[0] = t.x;
        v[1] = t.y;
        v[2] = t.z;
        v[3] = t.w;
    } else {
        const double2 a = reinterpret_cast<const double2*>(slot)[0], b = reinterpret_cast<const double2*>(slot)[1];
        v[0] = a.x;
        v[1] = a.y;
        v[2] = b.x;
        v[3] = b.y;
    }
}

// Positivity fallback of one cell's two reconstructed states in one direction
// (no reference counterpart).  A state is admissible when rho > 0 and p > 0
// (NaN fails); a state that is not, or that lies on a face flagged low order
// (a non-fluid cell in the face's stencil), becomes the cell's own value (first
// order).  `c` is the cell's value; the replacement is finished only when a
// state needs it.
template <class Pol>
__device__ __forceinline__ bool admissible(const Face5<typename Pol::C>& s) {
    return s.r > typename Pol::C(0) && s.p > typename Pol::C(0);
}

template <class Pol>
__device__ __forceinline__ void fix_states(bool lowL, bool lowR, const typename Pol::C c[kVars], double g,
                                           Face5<typename Pol::C>& L, Face5<typename Pol::C>& R) {
    const bool bl = lowL || !admissible<Pol>(L), br = lowR || !admissible<Pol>(R);
    if (bl || br) {
        Face5<typename Pol::C> s;
        s.r = c[0];
        s.mx = c[1];
        s.my = c[2];
        s.E = c[3];
        finish_state<Pol>(s, g);
        if (bl) L = s;
        if (br) R = s;
    }
}

// The same for the 32 lanes of a warp together (all of them call): flags f, of
// which lowL and lowR mark the low-order faces.  One test over both states and
// a branch that the warp takes as one (tested and branched per lane, with the
// flags' address and range test formed in every row, the kernel of a cylinder
// grid ran 830 instructions per cell-stage in FP32, 787 with it; 48 batched cases
// 846 -> 818 us a step).
template <class Pol>
__device__ __forceinline__ void fix_states_warp(unsigned int f, unsigned int lowL, unsigned int lowR,
                                                const typename Pol::C c[kVars], double g, Face5<typename Pol::C>& L,
                                                Face5<typename Pol::C>& R) {
    using C = typename Pol::C;
    const bool ok = (L.r > C(0)) & (L.p > C(0)) & (R.r > C(0)) & (R.p > C(0)) & !(f & (lowL | lowR));
    if (!__all_sync(0xffffffffu, ok)) fix_states<Pol>(f & lowL, f & lowR, c, g, L, R);
}

// The same fallback on the two states of a physical boundary face, each taking
// the value of the cell on its side (cl left of the face, cr right of it).
template <class Pol>
__device__ __forceinline__ void fix_face(bool low, const typename Pol::C cl[kVars], const typename Pol::C cr[kVars],
                                         double g, Face5<typename Pol::C>& L, Face5<typename Pol::C>& R) {
    Face5<typename Pol::C> dummy = R;
    fix_states<Pol>(low, false, cl, g, L, dummy);
    dummy = L;
    fix_states<Pol>(false, low, cr, g, dummy, R);
}

// Flux through a transmissive face whose cell value is c: the ghosts repeat c
// (NeummanBoundary.cpp:31-45), so the face's whole stencil [c c c | c c c]
// reconstructs c on both sides (a positivity fallback gives c again) and the
// HLL flux of two equal states is the physical flux; a negative pressure or
// density (a NaN sound speed) still gives a NaN flux.
template <class Pol>
__device__ __forceinline__ void wall_flux(const typename Pol::C c[kVars], int dir, double g, typename Pol::C F[kVars]) {
    using C = typename Pol::C;
    Face5<C> s;
    s.r = c[0];
    s.mx = c[1];
    s.my = c[2];
    s.E = c[3];
    finish_state<Pol>(s, g);
    phys_flux<Pol>(s, dir, F);
    const C nan_or_0 = s.a - s.a;
#pragma unroll
    for (int v = 0; v < kVars; ++v) F[v] += nan_or_0;
}

// Fluxes through the Dirichlet boundary faces of one stage (the reference's
// boundary stencil [g g g | c c c], CellInterface.cpp:172-178, then the
// positivity fallback and HLL), computed by pre_stage_kernel before the
// row march, which reads them (StageArgs::bflux) instead of reconstructing
// there.  (Transmissive faces need no stencil: the march forms them itself,
// wall_flux, which saves their grids this launch -- 3.8 us a stage at
// 64 x 48.)
template <class Pol>
__device__ __forceinline__ void boundary_face_flux(const StageArgs& a, int s, int k) {
    using T = typename Pol::T;
    using C = typename Pol::C;
    const Layout& L = a.L;
    const T* in = static_cast<const T*>(a.in);
    // interior cell (ii, jj) and ghost cell (gi, gj) of face k of side s
    int ii, jj, gi, gj;
    if (s < 2) {
        jj = gj = k;
        ii = s == 0 ? 0 : L.nx - 1;
        gi = s == 0 ? -1 : L.nx;
    } else {
        ii = gi = k;
        jj = s == 2 ? 0 : L.ny - 1;
        gj = s == 2 ? -1 : L.ny;
    }
    C c[kVars], gh[kVars];
    T cs[kVars], gs[kVars];
    ld_cell<T>(in, L.offset(ii, jj), cs);
    ld_cell<T>(in, L.offset(gi, gj), gs);
#pragma unroll
    for (int v = 0; v < kVars; ++v) {
        c[v] = decc<T, C>(cs[v], L, v);
        gh[v] = decc<T, C>(gs[v], L, v);
    }
    const bool lo = s == 0 || s == 2;
    Face5<C> Lf, Rf;
    boundary_face_states<Pol>(c, gh, lo, C(a.eps), a.gamma, Lf, Rf);
    if (a.positivity) {
        // face flags [nx+1][ny+1]: bit 0 x-face (i-1/2, j), bit 1 y-face (i, j-1/2)
        bool low = false;
        if (a.lowo) {
            const long long f = s == 0 ? jj : s == 1 ? static_cast<long long>(L.nx) * (L.ny + 1) + jj
                              : s == 2 ? static_cast<long long>(ii) * (L.ny + 1) : static_cast<long long>(ii) * (L.ny + 1) + L.ny;
            low = a.lowo[f] & (s < 2 ? 1 : 2);
        }
        fix_face<Pol>(low, lo ? gh : c, lo ? c : gh, a.gamma, Lf, Rf);
    }
    C F[kVars];
    hll_flux<Pol>(Lf, Rf, s < 2 ? 0 : 1, a.hll, a.gamma, F);
    C* out = static_cast<C*>(a.bflux) + bflux_side_offset(L, s);
    const int n = s < 2 ? L.ny : L.nx;
#pragma unroll
    for (int v = 0; v < kVars; ++v) out[static_cast<long long>(v) * n + k] = F[v];
}

// Face k of side s when that is a Dirichlet side's.
template <class Pol>
__device__ __forceinline__ void maybe_boundary_flux(const StageArgs& a, int s, int k) {
    if (a.bc[s] == kDirichlet && k < (s < 2 ? a.L.ny : a.L.nx)) boundary_face_flux<Pol>(a, s, k);
}

// What the update of a stage's cells shares.
struct UpdateCoefs {
    double dt, inv_dx, inv_dy;
    float inv_dxf, inv_dyf;
    // FP32: new = cA x0 + cB x1 + (c dt) R with x0 = U^0 (or the current state
    // at stage 0), x1 = U^1 (TVD3 as written, stage 2) or the current state
    // (TVD2rdRK.h:16-19, TVD3rdRK.h:14-18).  cA + cB must be exactly 1 in FP32,
    // else the deviation form scales the stored deviations by (cA + cB) every
    // step: cB = fl(2/3), cA = 1 - cB (an exact FP32 subtraction).
    float cA, cB, cdt;
    bool x1_u1, sr;
    unsigned int step_seed;
    bool do_cfl;
};

template <class Pol, int kFeat>
__device__ __forceinline__ UpdateCoefs update_coefs(const StageArgs& a) {
    UpdateCoefs k;
    const double dt = stage_dt(a);
    k.dt = dt;
    k.inv_dx = 1.0 / a.dx;
    k.inv_dy = 1.0 / a.dy;
    k.inv_dxf = float(k.inv_dx);
    k.inv_dyf = float(k.inv_dy);
    k.cA = 1.0f;
    k.cB = 0.0f;
    double cdtd = dt;  // dt coefficient of the stage, FP64
    k.x1_u1 = false;
    if (a.stage == 1) {
        if (a.rk == kRkTvd2) { k.cA = 0.5f; k.cB = 0.5f; cdtd = 0.5 * dt; }
        else { k.cA = 0.75f; k.cB = 0.25f; cdtd = 0.25 * dt; }
    } else if (a.stage == 2) {
        k.cB = float(2.0 / 3.0);
        k.cA = 1.0f - k.cB;
        cdtd = (2.0 / 3.0) * dt;
        k.x1_u1 = a.rk == kRkTvd3Ref;
    }
    if (kFeat & kSchemeU1) k.x1_u1 = true;
    if (kFeat & kSchemeNoU1) k.x1_u1 = false;
    k.cdt = float(cdtd);
    // Stochastic rounding of the state that ends each step (the last stage), or
    // of every stage (CFS_ROUND_STOCHASTIC_ALL); otherwise round to nearest.
    // Rounding an intermediate stage to nearest leaves a small mass bias: its
    // increments are dt times differences of FP32 fluxes, a coarse lattice on
    // the stored grid, so the rounding errors do not average out.
    const bool last_of_step = a.rk == kRkTvd2 ? a.stage == 1 : a.stage == 2;
    k.sr = Pol::kMixed && ((kFeat & kSchemeSr) || stage_rounds_stochastically(a.rounding, last_of_step));
    k.step_seed = (a.P ? a.P->seed[a.parity] : a.seed) * 4u + static_cast<unsigned int>(a.stage);
    k.do_cfl = a.P && a.last_stage && a.P->use_cfl;  // read once: stores to `out` may alias P for the compiler
    return k;
}

// Start of a step in graph mode: the next step's CFL slot, the time, the seed
// (one thread of the grid's first item).
__device__ __forceinline__ void begin_step(const StageArgs& a, double dt) {
    a.P->wmax[1 - a.parity] = 0ull;
    a.P->t += dt;
    a.P->dt_last = dt;
    a.P->seed[1 - a.parity] = a.P->seed[a.parity] + 1u;
}

// Update of cell (i, j) from its x-fluxes FX (upper) and FXp (lower), the y
// part RY of its RHS and, with kFeatExtra, its viscous RHS rvc; cur, u0, u1:
// stored values of the current state, U^0 and U^1 (as the stage reads them).
// Stores the new state and its ghost copies and raises wloc to the cell's
// CFL term.
template <class Pol, int kFeat>
__device__ __forceinline__ void update_cell(const StageArgs& a, const UpdateCoefs& k, int i, int j,
                                            const typename Pol::C FX[kVars], const typename Pol::C FXp[kVars],
                                            const typename Pol::C RY[kVars], const typename Pol::T rvc[kRvWords],
                                            const typename Pol::T cur[kVars], const typename Pol::T u0[kVars],
                                            const typename Pol::T u1[kVars], bool fluid, double& wloc) {
    using T = typename Pol::T;
    using C = typename Pol::C;
    constexpr bool kPos = (kFeat & kFeatPos) != 0;
    constexpr bool kExtra = (kFeat & kFeatExtra) != 0;
    const Layout& L = a.L;
    const double g = a.gamma;
    double* const rhs_out = kExtra ? a.rhs : nullptr;
    const bool has_rv = kExtra && a.rv;
    C nv[kVars];  // new state in the form's arithmetic type, for the CFL maximum
    T sv[kVars];
    if constexpr (Pol::kMixed) {
        // FP32 update of the stored deviations (value - off): the RK
        // coefficients of a stage sum to 1, so the offsets cancel and
        // the rounding step is that of the deviation.
        // (formed for every cell and selected: a non-fluid cell keeps its state)
        float rvf[kVars], x1[kVars], ndv[kVars];
#pragma unroll
        for (int v = 0; v < kVars; ++v) {
            rvf[v] = fmaf(-(FX[v] - FXp[v]), k.inv_dxf, RY[v]);
            if (has_rv && v >= 1) rvf[v] += rvc[v - 1];
            // (stage 0: cB = 0 and x1 - x0 = 0, so x1 adds nothing)
            x1[v] = k.x1_u1 ? u1[v] : cur[v];
        }
        if (k.sr) {
            // Stochastic rounding of x0 + cB (x1 - x0) + cdt R (cA = 1 - cB
            // exactly): the increment is formed first, at its own
            // spacing (roundings near 1e-12 of the state, far below the
            // stored spacing), gets a dither uniform over one stored
            // spacing of the result's binade, and is added to x0 with
            // one rounding; two variables per packed instruction.
            const unsigned int h = cell_hash(i, j, k.step_seed);
            const float u[kVars] = {dither_bits<0>(h), dither_bits<1>(h), dither_bits<2>(h), dither_bits<3>(h)};
#pragma unroll
            for (int v = 0; v < kVars; v += 2) {
                const float2 a0 = make_float2(u0[v], u0[v + 1]);
                const float2 inc = fma2(p2(k.cB), sub2(make_float2(x1[v], x1[v + 1]), a0),
                                        mul2(p2(k.cdt), make_float2(rvf[v], rvf[v + 1])));
                const float2 f = add2(a0, inc);
                const float2 t = add2(make_float2(u[v], u[v + 1]), p2(-kDitherCentre));
                const float2 r = add2(a0, fma2(make_float2(binade(f.x), binade(f.y)), t, inc));
                ndv[v] = r.x;
                ndv[v + 1] = r.y;
            }
        } else {
#pragma unroll
            for (int v = 0; v < kVars; ++v) ndv[v] = fmaf(k.cdt, rvf[v], fmaf(k.cA, u0[v], mul(k.cB, x1[v])));
        }
#pragma unroll
        for (int v = 0; v < kVars; ++v) {
            const float nd = fluid ? ndv[v] : cur[v];
            sv[v] = nd;
            nv[v] = nd + L.off[v];
            if (kExtra && rhs_out)
                rhs_out[static_cast<long long>(v) * L.nx * L.ny + static_cast<long long>(i) * L.ny + j] = fluid ? double(rvf[v]) : 0.0;
        }
    } else {
#pragma unroll
        for (int v = 0; v < kVars; ++v) {
            double rv = fma(-(FX[v] - FXp[v]), k.inv_dx, RY[v]);
            if (has_rv && v >= 1) rv += rvc[v - 1];
            const double val = fluid ? rk_update_fast(a.rk, a.stage, k.dt, u0[v], k.x1_u1 ? u1[v] : cur[v], rv) : cur[v];
            sv[v] = val;
            nv[v] = val;
            if (kExtra && rhs_out)
                rhs_out[static_cast<long long>(v) * L.nx * L.ny + static_cast<long long>(i) * L.ny + j] = fluid ? rv : 0.0;
        }
    }
    if (kPos && a.positivity >= kPosFloor && fluid) {
        // p > floor, multiplied by rho > 0: (g-1)(rho E - |m|^2/2) > floor rho
        const C q = fma(nv[3], nv[0], C(-0.5) * fma(nv[1], nv[1], mul(nv[2], nv[2])));
        if (!(nv[0] > C(kRhoFloor)) || !(C(g - 1.0) * q > C(kPFloor) * nv[0])) {
            double s[kVars];
#pragma unroll
            for (int v = 0; v < kVars; ++v)
                s[v] = Pol::kMixed ? double(sv[v]) + double(L.off[v]) : double(nv[v]);
            floor_state(s, g);
#pragma unroll
            for (int v = 0; v < kVars; ++v) {
                sv[v] = Pol::kMixed ? T(s[v] - double(L.off[v])) : T(s[v]);
                nv[v] = C(s[v]);
            }
        }
    }
    store_cell4<T>(static_cast<T*>(a.out), L, a.bc, i, j, sv);
    if (k.do_cfl) {
        const double w = cfl_term(double(wave_sum_fast<C>(nv[0], nv[1], nv[2], nv[3], C(g), C(k.inv_dx), C(k.inv_dy))));
        if (fluid && w > wloc) wloc = w;
    }
}

// The CFL maximum of a warp's cells: one atomic per warp (no block barrier, so
// the warps of a block never wait for each other).
__device__ __forceinline__ void raise_wmax(const StageArgs& a, double wloc) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wloc = fmax(wloc, __shfl_xor_sync(0xffffffffu, wloc, o));
    if ((threadIdx.x & 31) == 0 && wloc > 0.0)
        atomicMax(&a.P->wmax[1 - a.parity], static_cast<unsigned long long>(__double_as_longlong(wloc)));
}

// Flux through the x-face below row r in the column j where that face is a
// physical one (r = 0 or nx): the cell's own (transmissive; c: the interior
// cell's values) or the precomputed one (Dirichlet).
template <class Pol>
__device__ __forceinline__ void boundary_x_flux(const StageArgs& a, int r, int j, const typename Pol::C c[kVars],
                                                typename Pol::C FX[kVars]) {
    const Layout& L = a.L;
    // (no side index computed at run time: it would put the batch's argument block into local memory)
    if (r == 0 ? a.bc[0] == kNeumann : a.bc[1] == kNeumann) {
        wall_flux<Pol>(c, 0, a.gamma, FX);
    } else if (j >= 0 && j < L.ny) {
        const typename Pol::C* b = static_cast<const typename Pol::C*>(a.bflux) + bflux_side_offset(L, r == 0 ? 0 : 1);
#pragma unroll
        for (int v = 0; v < kVars; ++v) FX[v] = b[static_cast<long long>(v) * L.ny + j];
    }
}

// The y part of row r's RHS, RY, for the lanes of a warp on consecutive
// columns j (the warp's first lane on the segment's first column less one): WENO
// states of the 5-cell stencils st, the flux above each lane's cell, the
// difference of the two.  The outer lanes' RY are not those of their cells.
template <class Pol, int kFeat, bool kDeviations>
__device__ __forceinline__ void y_part(const StageArgs& a, const UpdateCoefs& k, int r, int j, int hll,
                                       const typename Pol::C st[5][kVars], typename Pol::C eps, unsigned int f_r,
                                       bool warp_ybnd, bool ybnd, const typename Pol::C* bfy, typename Pol::C RY[kVars]) {
    using C = typename Pol::C;
    const Layout& L = a.L;
    const double g = a.gamma;
    auto full = [&](const C w[kVars], C out[kVars]) {
#pragma unroll
        for (int v = 0; v < kVars; ++v) out[v] = kDeviations ? w[v] + C(L.off[v]) : w[v];
    };
    Face5<C> Ly, Ry;
    cell_states<Pol>(st, eps, g, Ly, Ry, kDeviations ? L.off : nullptr);
    if constexpr ((kFeat & kFeatPos) != 0) {
        C cc[kVars];
        full(st[2], cc);
        fix_states_warp<Pol>(f_r, kCellLowYhi, kCellLowYlo, cc, g, Ly, Ry);
    }
    // right state of the cell above (lane + 1)
    Face5<C> Rn;
    Rn.r = __shfl_down_sync(0xffffffffu, Ry.r, 1);
    Rn.mx = __shfl_down_sync(0xffffffffu, Ry.mx, 1);
    Rn.my = __shfl_down_sync(0xffffffffu, Ry.my, 1);
    Rn.E = __shfl_down_sync(0xffffffffu, Ry.E, 1);
    Rn.p = __shfl_down_sync(0xffffffffu, Ry.p, 1);
    Rn.a = __shfl_down_sync(0xffffffffu, Ry.a, 1);
    Rn.ri = __shfl_down_sync(0xffffffffu, Ry.ri, 1);
    // face between column j and j+1 (face index j+1)
    C FY[kVars];
    hll_flux<Pol>(Ly, Rn, 1, hll, g, FY);
    if (warp_ybnd && ybnd) {
        if (bfy) {
#pragma unroll
            for (int v = 0; v < kVars; ++v) FY[v] = bfy[static_cast<long long>(v) * L.nx + r];
        } else {  // the interior cell: column 0 for the lane below it, this lane's at the top
            C c[kVars];
#pragma unroll
            for (int v = 0; v < kVars; ++v) c[v] = j == -1 ? st[3][v] : st[2][v];
            full(c, c);
            wall_flux<Pol>(c, 1, g, FY);
        }
    }
#pragma unroll
    for (int v = 0; v < kVars; ++v) {
        const C below = __shfl_up_sync(0xffffffffu, FY[v], 1);
        RY[v] = mul(below - FY[v], Pol::kMixed ? C(k.inv_dyf) : C(k.inv_dy));
    }
}

// One work item: rows [by*rows, by*rows + rows) of segment `seg` (columns
// seg*30 .. seg*30+29), one warp.  The warps of a block share nothing but their
// slices of the row buffer and their rings.  kLoad, where global loads
// are issued (the trade is latency hidden against registers held):
//   0 at their use;
//   1 early in the iteration: the next row, the y halo columns and the RK
//     operands right after the row's x reconstruction, ahead of the update and
//     the y work that precede their use;
//   2 ahead: the next row two iterations ahead, the halo columns one row ahead,
//     the RK operands before the x reconstruction;
//   3 staged: every row of the segment (with its halo columns) and, in the
//     FP32 form, of U^0 is copied asynchronously (cp.async) into a per-warp
//     shared ring `ring` kRingDist rows ahead of its use; the x and y stencils,
//     the stored value and (FP32) U^0 of the update are read from the ring, so
//     no row window is held in registers and load latency overlaps rows of
//     arithmetic (the FP64 form loads U^0 early in the row's iteration and
//     keeps its ring in dynamic shared memory).
//
// The row loop holds no rarely taken code of any size: a transmissive face's
// flux is the cell's own (wall_flux), a Dirichlet one is read from
// pre_stage_kernel, and cell types and low-order faces
// come from one flag byte per cell (StageArgs::cflags), both compiled in only
// with kFeatEdge; the positivity fallback is a select of the cell's own state
// (kFeatPos); the RHS copy and viscous RHS come with kFeatExtra.  A loop body that outgrows the
// instruction cache stalls every warp on instruction fetch, whatever the share
// of the rare code actually executed.
template <class Pol, int kWarps, int kLoad, int kFeat>
__device__ __forceinline__ bool march_item(const StageArgs& a, int seg, int i0, int i1, bool first,
                                           typename Pol::C (&rbuf)[kWarps][36][kVars],
                                           typename Pol::T* ring, int wid, unsigned long long* bars = nullptr,
                                           unsigned* phase = nullptr) {
    using T = typename Pol::T;
    using C = typename Pol::C;
    constexpr bool kTma = kLoad == 4;
    constexpr bool kRing = kLoad >= 3;
    constexpr int kL = kLoad;
    constexpr bool kPos = (kFeat & kFeatPos) != 0;
    constexpr bool kExtra = (kFeat & kFeatExtra) != 0;
    constexpr bool kEdge = (kFeat & kFeatEdge) != 0;
    const int hll = (kFeat & kSchemeDavis) ? kHllDavis : (kFeat & kSchemeHllRef) ? kHllReference : a.hll;
    const Layout& L = a.L;
    const int lane = threadIdx.x & 31;
    const int j0 = seg * kSeg;
    const int j = j0 - 1 + lane;                 // this lane's column
    const bool col_ok = j <= L.ny + kGhost - 1;  // inside the padded row
    const bool owner = lane >= 1 && lane <= kSeg && j < L.ny;  // updates cells of this column
    const T* in = static_cast<const T*>(a.in);
    const C eps = C(a.eps);
    const double g = a.gamma;
    const UpdateCoefs uc = update_coefs<Pol, kFeat>(a);
    // physical boundary faces: the cell's own flux (transmissive) or a precomputed one (Dirichlet)
    // rows below which a physical x-face lies (-2: none)
    const int wall_lo = kEdge && physical_side(a, 0) ? 0 : -2, wall_hi = kEdge && physical_side(a, 1) ? L.nx : -2;
    const bool lo_y = kEdge && physical_side(a, 2), hi_y = kEdge && physical_side(a, 3);
    const C* const bfl = static_cast<const C*>(a.bflux);
    const uint8_t* const flags = kEdge ? a.cflags : nullptr;
    const T* const rv_in = kExtra ? static_cast<const T*>(a.rv) : nullptr;
    if (a.P && a.first_stage && first && lane == 0) begin_step(a, uc.dt);
    const bool active_warp = j0 < L.ny;  // uniform per warp

    auto load_row = [&](int r, C out[kVars]) {
        if (col_ok) {
            T cv[kVars];
            ld_cell<T>(in, L.offset(r, j), cv);
#pragma unroll
            for (int v = 0; v < kVars; ++v) out[v] = decc<T, C>(cv[v], L, v);
        } else {
#pragma unroll
            for (int v = 0; v < kVars; ++v) out[v] = C(0);
        }
    };

    auto load_halo = [&](int r, C h[kVars]) {
        if (lane < 2 || lane >= 30) {  // halo columns j0-3, j0-2 and j0+31, j0+32
            const int hc = lane < 2 ? j0 - 3 + lane : j0 + 1 + lane;
            if (hc <= L.ny + kGhost - 1) {
                T cv[kVars];
                ld_cell<T>(in, L.offset(r, hc), cv);
#pragma unroll
                for (int v = 0; v < kVars; ++v) h[v] = decc<T, C>(cv[v], L, v);
            } else {
#pragma unroll
                for (int v = 0; v < kVars; ++v) h[v] = C(0);
            }
        }
    };
    // Flag byte of cell (r, j) (kCell* bits), from a pointer that steps one row
    // per call; columns past ny (no face of an owned cell reads them) repeat
    // column ny's.  Called for rows i0 - 1 .. i1 in turn, all of them within the
    // flags' -1 .. nx.
    const uint8_t* fp = flags ? flags + static_cast<long long>(i0) * (L.ny + 2) + (min(j, L.ny) + 1) : nullptr;
    auto load_flags = [&]() -> unsigned int {
        unsigned int f = 0u;
        if (flags) {  // uniform per warp
            f = *fp;
            fp += L.ny + 2;
        }
        return f;
    };
    // this lane's upper y-face is a physical one; warp-uniform screen for the rare lanes
    const bool ybnd = (j == -1 && lo_y) || (j == L.ny - 1 && hi_y);
    const bool warp_ybnd = __any_sync(0xffffffffu, ybnd);
    const C* const bfy = ybnd && (j == -1 ? a.bc[2] == kDirichlet : a.bc[3] == kDirichlet)
                             ? bfl + (j == -1 ? bflux_side_offset(L, 2) : bflux_side_offset(L, 3)) : nullptr;
    // RK operands of cell (i, j): the stored value (FP32 form), U^0.
    // (U^1, read by the reference's TVD3 stage 2 only, is loaded at its use.)
    T pf_cur[kVars], pf_u0[kVars];
    auto load_update = [&](int i) {
        const long long off = L.offset(i, j);
        if (Pol::kMixed) ld_cell<T>(in, off, pf_cur);
        if (a.stage >= 1) ld_cell<T>(static_cast<const T*>(a.u0), off, pf_u0);
    };

    // Load schedules 3, 4: this warp's ring (rows, and U^0 rows in FP32; ring_words).
    constexpr bool kU0Ring = kRing && sizeof(T) == 4;
    constexpr int kRowWords = kTma ? ring_row_words<T>() : kRingCols * kVars;
    constexpr int kU0Words = kTma ? ring_row_words<T>() : 32 * kVars;
    T* const rw = kRing ? ring + wid * ring_words<T, kLoad>() : nullptr;
    T* const ru0 = kU0Ring ? rw + kRingRows * kRowWords + (kTma ? 2 * kVars : 0) : nullptr;
    auto ring_row = [&](int q) -> T* { return rw + (q & (kRingRows - 1)) * kRowWords; };
    auto ring_u0 = [&](int q) -> T* { return ru0 + (q & (kRingRows - 1)) * kU0Words; };
    // cp.async: ring column c is cell j0 - 3 + c; a lane copies columns lane
    // and (lanes 0..3) 32 + lane, and its own column of U^0, from pointers that
    // step one row per issued row; a column past the padded row is zero filled
    // from column 0's address.  (Addresses formed from row and column for each
    // copy, with the halo columns on lanes 0, 1, 30 and 31, took 30 more
    // instructions per cell-stage: SSP3 step of 4096^2 FP32-mixed 1,356 ->
    // 1,308 us, 2048^2 FP64 666 -> 647.)
    const bool src_ok = j0 - 3 + lane <= L.ny + kGhost - 1, src2_ok = j0 + 29 + lane <= L.ny + kGhost - 1;
    const T* src = nullptr;
    const T* src2 = nullptr;
    const T* src_u0 = nullptr;
    const long long row_step = static_cast<long long>(L.pitch) * kVars;
    const int u0_rows = a.stage >= 1 ? i1 - i0 : 0;  // rows whose U^0 is staged, from i0
    if constexpr (kLoad == 3) {
        src = in + Layout::at(L.offset(i0 - 3, src_ok ? j0 - 3 + lane : 0), 0);
        src2 = in + Layout::at(L.offset(i0 - 3, src2_ok ? j0 + 29 + lane : 0), 0);
        if (kU0Ring) src_u0 = static_cast<const T*>(a.u0) + Layout::at(L.offset(i0 - 3, col_ok ? j : 0), 0);
    }
    // Issue the copies of row q and, for an updated row, of its U^0; one commit
    // group per row (empty past the last row needed, so group counts stay
    // uniform).
    // TMA: lane 0 copies the row's 36 cells (and U^0's) as one box each,
    // completing on the slot's mbarrier.
    constexpr unsigned kRowBytes = kRingCols * kVars * sizeof(T);
    const int tcol = L.joff + j0 - 3;  // buffer column of ring column 0 (j0 - 3)
    int issued = i0 - 4;               // TMA: rows <= issued have been issued
    auto issue_row = [&](int q) {
        if constexpr (kTma) {
            if (q > i1 + 2) return;
            issued = q;
            if (lane == 0) {
                const bool u0row = kU0Ring && a.stage >= 1 && q >= i0 && q < i1;
                const unsigned bar = smem_addr(bars + (q & (kRingRows - 1)));
                const unsigned dst = smem_addr(ring_row(q)), dst0 = u0row ? smem_addr(ring_u0(q) - 2 * kVars) : 0u;
                if (((dst | dst0) & 127u) != 0u) {
                    // self-check: never issue a copy to a misaligned row;
                    // complete the slot's phase without data and flag it
                    atomicOr(a.err, kErrTmaAlign);
                    mbar_arrive(bar);
                } else {
                    fence_proxy_async_smem();
                    mbar_expect_tx(bar, u0row ? 2u * kRowBytes : kRowBytes);
                    tma_load_row(dst, a.tmap_in, tcol, q + kGhost, bar);
                    if (u0row) tma_load_row(dst0, a.tmap_u0, tcol, q + kGhost, bar);
                }
            }
        } else if constexpr (kRing) {
            if (q <= i1 + 2) {
                T* const dst = ring_row(q) + lane * kVars;
                cp_async_cell<T>(dst, src, src_ok);
                if (lane < 4) cp_async_cell<T>(dst + 32 * kVars, src2, src2_ok);
                if (kU0Ring && static_cast<unsigned>(q - i0) < static_cast<unsigned>(u0_rows))
                    cp_async_cell<T>(ring_u0(q) + lane * kVars, src_u0, col_ok);
            }
            src += row_step;
            src2 += row_step;
            if (kU0Ring) src_u0 += row_step;
            cp_async_commit();
        }
    };
    // TMA: wait until row q has landed in its slot (each row is waited on
    // exactly once, in order, so one phase bit per slot tracks its fills)
    bool tma_ok = true;
    int waited = i0 - 4;  // rows <= waited have been waited on
    auto wait_row = [&](int q) {
        if constexpr (kTma) {
            if (q > i1 + 2 || !tma_ok) return;
            const int sl = q & (kRingRows - 1);
            // warp-uniform outcome: every lane continues or every lane stops
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(smem_addr(bars + sl), (*phase >> sl) & 1u))) {
                tma_ok = false;
                return;
            }
            *phase ^= 1u << sl;
            waited = q;
        }
    };
    // full value of a stencil cell (the ring holds stored deviations)
    auto full = [&](const C w[kVars], C out[kVars]) {
#pragma unroll
        for (int v = 0; v < kVars; ++v) out[v] = (kRing && Pol::kMixed) ? w[v] + C(L.off[v]) : w[v];
    };

    C win[5][kVars];
    C nxt[kVars];   // kLoad 1, 2: the row after win[4]
    C hal[kVars];   // kLoad 1, 2: halo columns of the next y row
    Face5<C> Lx{};                             // left x-state of the previous row
    C FXp[kVars] = {C(0), C(0), C(0), C(0)};   // x-flux through the lower face of the previous row
    C RY[kVars] = {C(0), C(0), C(0), C(0)};    // y part of the previous row's RHS
    unsigned int f_prev = 0u, f_next = 0u;     // flags of rows r-1 and r+1
    T rv_cur[kRvWords] = {T(0), T(0), T(0)}, rv_pf[kRvWords] = {T(0), T(0), T(0)};  // kExtra: viscous RHS of rows r-1, r
    double wloc = 0.0;
    if (active_warp && kRing) {
        if constexpr (kTma) __syncwarp();  // a previous item's reads of the ring end before lane 0's copies
        for (int q = i0 - 3; q <= i0 + 1 + kRingDist; ++q) issue_row(q);
        if constexpr (kTma) {
            for (int q = i0 - 3; q <= i0; ++q) wait_row(q);  // the first iteration waits for row i0 + 1
        }
    } else if (active_warp) {
#pragma unroll
        for (int k = 0; k < 5; ++k) load_row(i0 - 3 + k, win[k]);
        if constexpr (kL == 2) {
            load_row(i0 + 2, nxt);
            load_halo(i0, hal);
        }
    }
    if (active_warp) f_next = load_flags();
    for (int r = i0 - 1; active_warp && r <= i1; ++r) {
        const unsigned int f_r = f_next;
        if (r == i1) let_next_in();
        else f_next = load_flags();
        if constexpr (kRing && !kU0Ring) {  // FP64 ring: U^0 of row r-1, ahead of the x reconstruction
            if (a.stage >= 1 && owner && r - 1 >= i0) ld_cell<T>(static_cast<const T*>(a.u0), L.offset(r - 1, j), pf_u0);
        }
        if constexpr (kExtra) {  // viscous RHS of row r, a whole iteration ahead of its update
#pragma unroll
            for (int q = 0; q < kRvWords; ++q) rv_cur[q] = rv_pf[q];
            if (rv_in && owner && r >= i0 && r < i1) ld_rv<T>(rv_in, static_cast<long long>(r) * L.ny + j, rv_pf);
        }
        if constexpr (kRing) {
            // every lane is done with the previous iteration's slots; the slot
            // now refilled held row r+3+kRingDist-kRingRows, last read at r-1
            __syncwarp();
            issue_row(r + 3 + kRingDist);
            if constexpr (kTma) {
                wait_row(r + 2);  // rows <= r+2 have landed
                if (!tma_ok) break;
            } else {
                cp_async_wait<kRingDist + 1>();  // this lane's copies of rows <= r+2 have landed
                __syncwarp();                    // ... and every lane's
            }
#pragma unroll
            for (int k = 0; k < 5; ++k) {  // stored deviations; offsets added after the reconstruction
                ld_cell<T>(ring_row(r - 2 + k), lane + 2, win[k]);
            }
        }
        if constexpr (kL == 2) {
            if (r - 1 >= i0 && owner) load_update(r - 1);
        }
        // ---- x reconstruction of row r
        Face5<C> Lr, Rr;
        cell_states<Pol>(win, eps, g, Lr, Rr, (kRing && Pol::kMixed) ? L.off : nullptr);
        if constexpr (kPos) {
            C cc[kVars];
            full(win[2], cc);
            fix_states_warp<Pol>(f_r, kCellLowXhi, kCellLowXlo, cc, g, Lr, Rr);
        }
        if constexpr (kL == 1) {
            if (r < i1) load_row(r + 3, nxt);
            if (r - 1 >= i0 && owner) load_update(r - 1);
            if (r >= i0 && r < i1) load_halo(r, hal);
        }
        C FX[kVars] = {C(0), C(0), C(0), C(0)};
        if (r >= i0) {
            // (computed on a boundary row too and replaced there: a flux in a
            // branch of its own would not overlap the surrounding work)
            hll_flux<Pol>(Lx, Rr, 0, hll, g, FX);
            if (kEdge && (r == wall_lo || r == wall_hi)) {  // uniform per warp
                C c[kVars];
                if (r == 0) full(win[2], c);
                else full(win[1], c);
                boundary_x_flux<Pol>(a, r, j, c, FX);
            }
            // ---- update of row r-1 (its upper x-face is r - 1/2)
            const int i = r - 1;
            if (i >= i0 && owner) {
                if constexpr (kRing) {
                    const T* cs = ring_row(i) + (lane + 2) * kVars;
                    ld_cell<T>(cs, 0, pf_cur);
                    if constexpr (kU0Ring) {
                        // U^0 (stage 0: the current state, the update's x0 then)
                        const T* us = a.stage >= 1 ? ring_u0(i) + lane * kVars : cs;
                        ld_cell<T>(us, 0, pf_u0);
                    }
                } else if constexpr (kL == 0) {
                    load_update(i);
                }
                const bool fluid = !kEdge || !(f_prev & kCellSolid);
                T u1c[kVars] = {T(0), T(0), T(0), T(0)};  // U^1 (TVD3 as written, stage 2 only)
                if (uc.x1_u1) ld_cell<T>(static_cast<const T*>(a.u1), L.offset(i, j), u1c);
                if constexpr (!Pol::kMixed && !kRing) {
#pragma unroll
                    for (int v = 0; v < kVars; ++v) pf_cur[v] = T(win[1][v]);
                }
                update_cell<Pol, kFeat>(a, uc, i, j, FX, FXp, RY, rv_cur, pf_cur,
                                        (kU0Ring || a.stage >= 1) ? pf_u0 : pf_cur, u1c, fluid, wloc);
            }
        }
        // ---- y work of row r
        if (r >= i0 && r < i1) {
            // slot-major row buffer: the 4 variables of a column are one
            // 16-byte (FP32) or two 16-byte (FP64) shared accesses
            C st[5][kVars];
            if constexpr (kRing) {
                const T* row = ring_row(r);
#pragma unroll
                for (int k = 0; k < 5; ++k) ld_cell<T>(row, lane + k, st[k]);  // deviations
            } else {
                C(*rb)[kVars] = rbuf[wid];
                put_slot<C>(rb[lane + 2], win[2]);
                if constexpr (kL == 0) load_halo(r, hal);
                if (lane < 2 || lane >= 30) put_slot<C>(rb[lane < 2 ? lane : lane + 4], hal);
                __syncwarp();
#pragma unroll
                for (int k = 0; k < 5; ++k) get_slot<C>(rb[lane + k], st[k]);
            }
            y_part<Pol, kFeat, kRing && Pol::kMixed>(a, uc, r, j, hll, st, eps, f_r, warp_ybnd, ybnd, bfy, RY);
            __syncwarp();
        }
        // ---- carry to the next row
#pragma unroll
        for (int v = 0; v < kVars; ++v) FXp[v] = FX[v];
        Lx = Lr;
        f_prev = f_r;
        if (!kRing && r < i1) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int v = 0; v < kVars; ++v) win[k][v] = win[k + 1][v];
            if constexpr (kL == 2) {
#pragma unroll
                for (int v = 0; v < kVars; ++v) win[4][v] = nxt[v];
                if (r + 4 <= i1 + 2) load_row(r + 4, nxt);
                if (r + 1 < i1) load_halo(r + 1, hal);
            } else if constexpr (kL == 1) {
#pragma unroll
                for (int v = 0; v < kVars; ++v) win[4][v] = nxt[v];
            } else {
                load_row(r + 3, win[4]);
            }
        }
    }
    if constexpr (kTma) {
        if (!tma_ok) {
            // a copy never landed: report it, and wait (bounded) for the
            // copies still in flight so that none outlives the item
            if (lane == 0) atomicOr(a.err, kErrTmaTimeout);
            for (int q = waited + 1; q <= issued; ++q) {
                const int sl = q & (kRingRows - 1);
                if (__all_sync(0xffffffffu, mbar_wait_bounded(smem_addr(bars + sl), (*phase >> sl) & 1u, kMbarDrainTries)))
                    *phase ^= 1u << sl;
            }
            return false;
        }
    } else if constexpr (kRing) {
        cp_async_wait_all();  // no copy into the ring outlives the item
    }
    if (uc.do_cfl) raise_wmax(a, wloc);
    return true;
}

// Per-warp mbarriers of the TMA ring: initialised once per launch by lane 0,
// made visible to the async proxy before the first copy.
template <int kWarps>
__device__ __forceinline__ void init_ring_bars(unsigned long long (&bars)[kWarps][kRingRows], int wid) {
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int k = 0; k < kRingRows; ++k) mbar_init(smem_addr(&bars[wid][k]), 1u);
        mbar_init_fence();
    }
    __syncwarp();
}

template <class Pol, int kRows, int kWarps, int kMinBlocks, int kLoad, int kFeat>
__global__ void __launch_bounds__(32 * kWarps, kMinBlocks) march_kernel(const __grid_constant__ StageArgs a) {
    // warps numbered over (segment, row chunk), segments fastest, so no block
    // carries idle warps when the segments of a row are not a multiple of its
    // warps; a warp past the last item runs an empty one.  The long chunks come
    // first, the short ones behind them fill the launch's end.
    // (the warp index taken from lane 0, so that the compiler knows the item's
    // rows and columns to be the same in all lanes: the row tests' branches need
    // no convergence code.  685 -> 670 instructions per cell-stage in FP32, the
    // 4096^2 step 1,384 -> 1,356 us, 2048^2 FP64 689 -> 666)
    const int nseg = (a.L.ny + kSeg - 1) / kSeg;
    const int wid = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const long long gw = static_cast<long long>(blockIdx.x) * kWarps + wid;
    const int chunk = static_cast<int>(gw / nseg), lo = stage_row_lo(a), hi = stage_row_hi(a);
    const bool is_long = chunk < a.long_chunks;
    const long long at = is_long ? static_cast<long long>(chunk) * a.rows
                                 : static_cast<long long>(a.long_chunks) * a.rows +
                                       static_cast<long long>(chunk - a.long_chunks) * a.rows_short;
    const bool item = at < hi - lo;
    const int seg = item ? static_cast<int>(gw % nseg) : nseg;
    const int i0 = item ? lo + static_cast<int>(at) : lo;
    const int i1 = min(i0 + (is_long ? a.rows : a.rows_short), hi);
    const bool first = gw == 0;
    after_previous();
    // (the ring forms use no row buffer)
    __shared__ __align__(16) typename Pol::C rbuf[kLoad >= 3 ? 1 : kWarps][36][kVars];
    using RB = typename Pol::C(&)[kWarps][36][kVars];
    if constexpr (kLoad == 4) {
        __shared__ __align__(8) unsigned long long bars[kWarps][kRingRows];
        init_ring_bars<kWarps>(bars, wid);
        if ((threadIdx.x & 31) == 0) {
            tma_prefetch_map(a.tmap_in);
            if (a.stage >= 1 && sizeof(typename Pol::T) == 4) tma_prefetch_map(a.tmap_u0);
        }
        unsigned phase = 0u;
        if constexpr (sizeof(typename Pol::T) == 4) {
            __shared__ __align__(128) typename Pol::T ring[kWarps * ring_words<typename Pol::T, kLoad>()];
            march_item<Pol, kWarps, kLoad, kFeat>(a, seg, i0, i1, first, reinterpret_cast<RB>(rbuf), ring, wid,
                                                  bars[wid], &phase);
        } else {
            // FP64 ring: dynamic shared memory, sized at launch
            extern __shared__ __align__(128) unsigned char march_dyn_smem[];
            march_item<Pol, kWarps, kLoad, kFeat>(a, seg, i0, i1, first, reinterpret_cast<RB>(rbuf),
                                                  reinterpret_cast<typename Pol::T*>(march_dyn_smem), wid, bars[wid],
                                                  &phase);
        }
    } else if constexpr (kLoad == 3 && sizeof(typename Pol::T) == 4) {
        __shared__ __align__(128) typename Pol::T ring[kWarps * ring_words<typename Pol::T, kLoad>()];
        march_item<Pol, kWarps, kLoad, kFeat>(a, seg, i0, i1, first, reinterpret_cast<RB>(rbuf), ring, wid);
    } else if constexpr (kLoad == 3) {
        // FP64 ring: kWarps * ring_words<double, 3>() doubles (36.9 KB for 4
        // warps); dynamic shared memory, sized at launch
        extern __shared__ __align__(128) unsigned char march_dyn_smem[];
        march_item<Pol, kWarps, kLoad, kFeat>(a, seg, i0, i1, first, reinterpret_cast<RB>(rbuf),
                                              reinterpret_cast<typename Pol::T*>(march_dyn_smem), wid);
    } else {
        march_item<Pol, kWarps, kLoad, kFeat>(a, seg, i0, i1, first, rbuf, nullptr, wid);
    }
}

// Persistent batched form: one launch runs one stage of every case of a batch.
// Each warp pulls work units (case, segment, row chunk) from a global counter,
// largest cases first, until none are left; warps share nothing, so a case
// whose segment count is not a multiple of the block's warps leaves no warp
// idle.  args[c] holds case c's stage arguments (its own layout, boundaries,
// buffers, dt slot); a unit is one 16-byte record (cut by append_units, cfs_batch.cpp).
template <class Pol, int kWarps, int kMinBlocks, int kLoad, int kFeat>
__global__ void __launch_bounds__(32 * kWarps, kMinBlocks)
    batch_march_kernel(const StageArgs* __restrict__ args, const BatchUnit* __restrict__ units, int total,
                       unsigned int* counters, int slot) {
    using C = typename Pol::C;
    constexpr bool kRing = kLoad == 3;
    __shared__ __align__(16) C rbuf[kRing ? 1 : kWarps][36][kVars];  // (the ring forms use no row buffer)
    constexpr bool kDynRing = kRing && sizeof(typename Pol::T) == 8;  // FP64: ring in dynamic shared memory
    __shared__ __align__(128) typename Pol::T ring_static[kRing && !kDynRing ? kWarps * ring_words<typename Pol::T, kLoad>() : 1];
    extern __shared__ __align__(128) unsigned char batch_dyn_smem[];
    typename Pol::T* const ring = kDynRing ? reinterpret_cast<typename Pol::T*>(batch_dyn_smem) : ring_static;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned int* const counter = counters + slot;
    let_next_in();
    after_previous();
    if (blockIdx.x == 0 && threadIdx.x < kBatchCounters && threadIdx.x / kBatchMaxGroups != slot / kBatchMaxGroups)
        counters[threadIdx.x] = 0u;  // the other stages' (see kBatchCounters)
    C(&wbuf)[1][36][kVars] = *reinterpret_cast<C(*)[1][36][kVars]>(&rbuf[kRing ? 0 : wid]);
    for (;;) {
        unsigned int w = 0u;
        if (lane == 0) w = atomicAdd(counter, 1u);
        w = __shfl_sync(0xffffffffu, w, 0);
        if (w >= static_cast<unsigned int>(total)) break;
        const int4 u = __ldg(reinterpret_cast<const int4*>(units) + w);  // a BatchUnit
        const StageArgs a = args[u.x];
        march_item<Pol, 1, kLoad, kFeat>(a, u.y, u.z, u.w, u.y == 0 && u.z == 0, wbuf, kRing ? ring + wid * ring_words<typename Pol::T, kLoad>() : nullptr, 0);
    }
}

}  // namespace cfs
