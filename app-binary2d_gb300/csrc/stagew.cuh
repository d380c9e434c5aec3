// stagew.cuh — the FP32 RK-stage kernel: every warp marches down a strip of
// its own.
//
// One launch performs one call of try_advance_rk (src/scheme.rs:88-173) for
// every run of a context, on the FP64 state or on the compensated FP32 state:
// cons→prim (scheme.rs:185-199), PLM slopes and HLLE + viscous fluxes
// (scheme.rs:216-268), flux divergence + sources + RK average
// (scheme.rs:290-305, state.rs:183-199), the per-block source ledger's pieces
// (scheme.rs:288-313) and, on the last stage of an advance, the max signal
// speed of the next dt (state.rs:121-133).
//
//  * A warp is on its own: it is a CTA, so that its loop and addresses are
//    uniform.  It owns 60 columns of a row chunk, two adjacent columns a lane
//    (lanes 0 and 31 are the two guard pairs on either side), and goes down its
//    rows without a barrier: neighbouring columns come by shuffle, the rows
//    above from registers, and the guard columns are computed again by the
//    next strip's warp (2 of 32 lanes).  The twelve warps of an SM drift apart
//    and fill each other's stalls.
//  * Packed arithmetic.  Every per-column quantity is a float2 and the
//    arithmetic runs as Blackwell's packed FADD2 / FMUL2 / FFMA2; min / max,
//    compares, selects and the special-function unit stay per column.
//  * Row staging.  Asynchronous copies bring the rows ahead into a ring in
//    shared memory, one group per row: the stage input a row ahead of its use,
//    and what the update reads besides (low words, background, RK base).  Where
//    four columns are an aligned 16 bytes (an FP32 state whose sides are
//    multiples of 4; any pair of an FP64 state) the copies go past the L1: with
//    8-byte copies through it every row in flight holds three lines per plane,
//    more than the L1 has beside the rings (Euler 4096^2 474 us a stage with
//    28 KB of L1 left, 392 with 60 KB, 375 past it).  Other sides copy pairs or
//    single words.  (Bulk copies (TMA) cost more here: a warp's row is 15 planes
//    of 240 bytes, each an instruction of its own with uniform addresses, 180 of
//    970 instructions a row.)
//  * Constants that packed instructions take are kept twice, as a pair, in
//    shared memory: one load instead of two moves per use.  All shared memory is
//    one block behind one address.
//  * Pipeline.  Iteration n converts row n, forms slopes and stresses of row
//    g = n - 1, its upper x faces and its y faces, and updates row g - 1.
//  * Ledger.  The items that are live everywhere are summed per column in
//    registers; a block's part is reduced over the warp at the last row of
//    each block row and at the chunk's end, one piece per strip and chunk.  The
//    pieces of all stages are folded, in order, after the last of them: a fence,
//    a counter and a fold in the stage's tail cost it about 5 us.
//
// What bounds it: instruction issue (620 warp instructions per row of 60
// columns and isothermal first stage, guard rows and set-up included, 290 of
// them packed or special-function arithmetic and min / max; a warp in flight
// waits 4.5 cycles per instruction and a scheduler has three), not memory (4.0
// of 6.7 TB/s).  Measured per stage of queued advances, with the kernels that it
// took the place of, as this file began, and now:
//   isothermal 2048^2          127 -> 109 -> 71 us (10 warps a CTA in step over 512 columns)
//   isothermal 384^2            33 -> 22 -> 11.6 us
//   the sweep of 64 runs      1050 -> 690 -> 520 us
//   Euler 4096^2               650 -> 550 -> 365 us
//   Euler 768^2                 48 -> 42 -> 26.0 us
//   blocks of 50^2, RK3, alpha 163 -> 25 -> 10.3 us (a thread per column of a block)
//   FP64 state 1024^2          106 -> 94 -> 38 us
// Of this, forming FP32 pairs of FP64 words and widening increments with integer
// instructions gave the FP64 state 47 us where the FP64 pipe's conversions take 50
// to 70, and letting a stage begin in the last row of the one before 12.5 -> 12.1
// us at 384^2 and 12.6 -> 11.9 on blocks of 50^2.
//
// Tried and slower: the row loop unrolled twice (104 against 98 us at 2048^2:
// spills); the same later without spills (76 to 78 against 73 us: 5 % fewer
// instructions, but waits for instructions nearly double); the run's descriptor as
// a kernel argument (99 against 92); letting the next stage in from the start
// (768^2: 47 against 40 us); 16 warps per SM with 128 registers (85 against 78 us:
// more instructions, and four warps share what three nearly fill); pairs carried
// from row to row as 64-bit values (76 against 73 us: more moves); the first rows
// converted before the loop, or requested four at once (75 to 76).
#pragma once

#include "split.cuh"
#include "stage.cuh"

namespace b2d {

constexpr int SW_SLOTS = 4;              // stencil ring: rows n - 2 (for its update) to n + 1
constexpr int SW_USLOTS = 2;             // update rows: one in use, one ahead

// Constants as pairs, with what can be folded into them: the limiter works on
// slopes over theta, the stress on (slope / dx) times c, the sound speed on
// masses over Mach^2, the buffer on powers of two.
enum {
    C_ITHETA2,               // 1 / (2 theta), and 0 for theta = 0
    C_EDGE, C_NEDGE,         // theta / 2: half a slope
    C_NHALF, C_HALF, C_ONE,
    C_TN, C_TT, C_VISC,      // 4/3 + lambda, -2/3 + lambda; theta c / dx of the cell's stress
    C_CM1, C_CM2,            // m / Mach^2
    C_M1, C_M2, C_NM1DT, C_NM2DT, C_SOFT2,
    C_BUF_SLOPE, C_RADIUS, C_BUF_RATE, C_NDT_DX, C_GAMMA, C_GM1, C_INV_GM1, C_COOL, C_ALPHA, C_COUNT
};

// How a warp copies its rows: a word, a pair of columns or four columns at a
// time, by what divides the mesh's side (four columns of FP32 words, two of FP64).
enum { COPY_WORDS, COPY_PAIRS, COPY_QUADS };

// Shared memory of one warp.
template <int NF, int STORE, int COPY> struct SWShape {
    using E = typename std::conditional<STORE == 1, float, double>::type;
    static constexpr int NU = (STORE == 1 ? 4 : 2) * NF;  // update planes: (lo,) bg, base hi (, base lo)
    static constexpr int ITEMS = NF == 3 ? 16 : 19;       // ledger items: live everywhere, sinks, fake mass
    static constexpr int SINKS_AT = NF == 3 ? 7 : 11, FAKE_AT = 13;
    // a staged plane's row: columns -2 to 61 of the strip (quads: -4 to 63), and of the
    // update's planes too (quads: 0 to 59)
    static constexpr int S_PITCH = COPY == COPY_QUADS ? 68 : 64, S_FIRST = COPY == COPY_QUADS ? 2 : 0;
    static constexpr int U_PITCH = COPY == COPY_QUADS ? 60 : 64, U_FIRST = COPY == COPY_QUADS ? -2 : 0;
    static constexpr int PARTIALS = NF == 3 ? 4 : 1;
    // The warp's tables.  They lie with the rings in one block, whose address is held in a register:
    // the compiler forms the address of every shared array of its own anew wherever it is used.
    struct Tables {
        float2 K[C_COUNT];
        float2 dyc1[32], dyc2[32], dyv1[32], dyv2[32], yc[32];   // of the pair's centres and left faces
        float2 rows[5][32];                                 // dx1, dx2 and x^2 of zone rows, dx1, dx2 of the faces above
        float2 part[PARTIALS][32];                          // dy^2 + s^2 of faces and centres to either body (isothermal)
        Binary<float> B;
        float B_lo[10];
        DevParamsF P;                                       // a batched launch's parameters
    };
    static constexpr int TABLES = ((int)sizeof(Tables) + 127) / 128 * 128;
    static constexpr int STENCIL = NF * S_PITCH;          // elements of a staged row
    static constexpr int UPDATE = NU * U_PITCH;
    static constexpr int BYTES = TABLES + (SW_SLOTS * STENCIL + SW_USLOTS * UPDATE + (COPY == COPY_QUADS ? 4 : 0)) * (int)sizeof(E);
    static constexpr int CTAS = 12;   // per SM
    // A lane's items' sums (words 2 lane, 2 lane + 1 of rows of 64 FP32 words) cover only words that it alone
    // copies and reads: not where the planes' words are FP64, or lie at another pitch.
    static constexpr bool SUMS_OVER_OWN = STORE == 1 && COPY != COPY_QUADS;
    static_assert(SINKS_AT * 64 * 4 <= UPDATE * (int)sizeof(E), "a consumed update row takes the items' sums");
};

// ---------------------------------------------------------------------------
// Packed FP32x2 arithmetic (sm_100+ FADD2 / FMUL2 / FFMA2, round to nearest).
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
// (no intrinsic for it; as b * (-1) + a it takes the constant's two registers)
__device__ __forceinline__ float2 sub2(float2 a, float2 b)
{
    union U { float2 f; unsigned long long u; } x, y, d;
    x.f = a;
    y.f = b;
    asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d.u) : "l"(x.u), "l"(y.u));
    return d.f;
}
// 1 / a: __fdividef(1, a) gives the same values and tests for |a| > 2^126 besides
__device__ __forceinline__ float rcp(float a)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a));
    return y;
}
__device__ __forceinline__ float2 rcp2(float2 a) { return make_float2(rcp(a.x), rcp(a.y)); }
__device__ __forceinline__ float2 sqrt2(float2 a) { return make_float2(sqrtf(a.x), sqrtf(a.y)); }
__device__ __forceinline__ float2 rsqrt2(float2 a) { return make_float2(rsqrtf(a.x), rsqrtf(a.y)); }

// Knuth TwoSum / Dekker Fast2Sum on pairs (the compensated state update).
struct df2 { float2 hi, lo; };

__device__ __forceinline__ df2 fast_two_sum2(float2 a, float2 b)
{
    const float2 s = add2(a, b);
    return {s, sub2(b, sub2(s, a))};
}

__device__ __forceinline__ df2 two_sum2(float2 a, float2 b)
{
    const float2 s = add2(a, b);
    const float2 bb = sub2(s, a);
    return {s, add2(sub2(a, sub2(s, bb)), sub2(b, bb))};
}

__device__ __forceinline__ df2 df_add2(df2 a, df2 b)
{
    const df2 s = two_sum2(a.hi, b.hi);
    return fast_two_sum2(s.hi, add2(s.lo, add2(a.lo, b.lo)));
}

__device__ __forceinline__ df2 df_mul2(df2 a, df32 b)
{
    const float2 bh = f2(b.hi), bl = f2(b.lo);
    const float2 p = mul2(a.hi, bh);
    float2 e = fma2(a.hi, bh, mul2(p, f2(-1.0f)));
    e = fma2(a.hi, bl, fma2(a.lo, bh, e));
    return fast_two_sum2(p, e);
}

// Three-input FP32 minimum and maximum (PTX min/max with three sources, sm_100+).
__device__ __forceinline__ float min3f(float a, float b, float c)
{
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float max3f(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// The generalised minmod of differences a and b and of y = (a + b) / (2 theta)
// (godunov-core's plm_gradient, restated; over theta): the median of min(a, y, b),
// max(a, y, b) and 0 — the minimum when all three are positive, the maximum when
// all are negative, else 0: min(max(lo, 0), hi) for lo <= hi.
__device__ __forceinline__ float minmod3(float a, float y, float b)
{
    return fminf(fmaxf(min3f(a, y, b), 0.0f), max3f(a, y, b));
}

__device__ __forceinline__ float exp2_fast(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float log2_fast(float x)
{
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// e^x - 1 of two small arguments (|x| <= 0.35): the Taylor series
// x (1 + x/2 + x^2/6 + ... + x^7/8!) in Horner form; the first omitted term,
// x^9/9!, is below 6e-10 |x| there.
__device__ __forceinline__ float2 expm1_small2(float2 x)
{
    float2 p = f2(1.0f / 40320.0f);
    p = fma2(p, x, f2(1.0f / 5040.0f));
    p = fma2(p, x, f2(1.0f / 720.0f));
    p = fma2(p, x, f2(1.0f / 120.0f));
    p = fma2(p, x, f2(1.0f / 24.0f));
    p = fma2(p, x, f2(1.0f / 6.0f));
    p = fma2(p, x, f2(0.5f));
    p = fma2(p, x, f2(1.0f));
    return mul2(p, x);
}

// ---------------------------------------------------------------------------
// Scalar FP32 pieces, written with explicit roundings (fmaf, __fmul_rn,
// __fadd_rn: no contraction left to the compiler), so that every instantiation
// of the kernel rounds them alike and the states depend neither on the tiling
// nor on the batch.

// cons -> prim without floors (hydro-iso2d / hydro-euler; physics.rs:696).
template <int NF> __device__ __forceinline__ void prim_exact(const DevParamsF& P, const float* u, float* p)
{
    const float ir = __fdividef(1.0f, u[0]);
    p[0] = u[0];
    p[1] = __fmul_rn(u[1], ir);
    p[2] = __fmul_rn(u[2], ir);
    if constexpr (NF == 4) {
        const float v2 = fmaf(p[1], p[1], __fmul_rn(p[2], p[2]));
        p[3] = __fmul_rn(fmaf(__fmul_rn(-0.5f, u[0]), v2, u[3]), P.gm1);
    }
}

// Physics::sink_kernel (physics.rs:388-397): rate (1 - r^2 / s^2)^2 inside the sink radius s.
__device__ __forceinline__ float sink_rate_exact(const DevParamsF& P, float dx, float dy)
{
    const float r2 = fmaf(dx, dx, __fmul_rn(dy, dy));
    if (r2 < P.sink_r2) {
        const float t = fmaf(-r2, P.inv_sink_r2, 1.0f);
        return __fmul_rn(P.sink_rate, __fmul_rn(t, t));
    }
    return 0.0f;
}

// The torque-free sink velocity: the gas velocity relative to the body,
// projected on the radial direction, plus the body's velocity (physics.rs:743-756).
__device__ __forceinline__ void torque_free_exact(const DevParamsF& P, const PointMass<float>& b, float ddx, float ddy,
                                                  float vx, float vy, float& vxc, float& vyc)
{
    const float vxb = P.one_body ? 0.0f : b.vx, vyb = P.one_body ? 0.0f : b.vy;
    const float r = sqrtf(fmaf(ddx, ddx, __fmul_rn(ddy, ddy)));
    const float rx = __fdividef(ddx, r), ry = __fdividef(ddy, r);
    const float dvdotr = fmaf(vx - vxb, rx, __fmul_rn(vy - vyb, ry));
    vxc = fmaf(dvdotr, rx, vxb);
    vyc = fmaf(dvdotr, ry, vyb);
}

// The sink items of one zone (the sink part of source_terms, physics.rs:
// 528-582, 683-774): -rate u dt (impartial sinks) or -rate dt times the
// torque-free state, at (dx1, dy1) from body 1 and (dx2, dy2) from body 2.
template <int NF>
__device__ __noinline__ void sink_items_exact(const DevParamsF& P, const Binary<float>& B, const float* u, float dx1,
                                              float dy1, float dx2, float dy2, float dt, float* s1, float* s2)
{
    const float sr1 = __fmul_rn(sink_rate_exact(P, dx1, dy1), -dt);
    const float sr2 = __fmul_rn(sink_rate_exact(P, dx2, dy2), -dt);
    if (P.sink_model == 0) {
#pragma unroll
        for (int k = 0; k < NF; ++k) {
            s1[k] = __fmul_rn(u[k], sr1);
            s2[k] = __fmul_rn(u[k], sr2);
        }
        return;
    }
    float p[NF];
    prim_exact<NF>(P, u, p);
    float v1x, v1y, v2x, v2y;
    torque_free_exact(P, B.p1, dx1, dy1, p[1], p[2], v1x, v1y);
    torque_free_exact(P, B.p2, dx2, dy2, p[1], p[2], v2x, v2y);
    const float sd = p[0];
    float a1[NF], a2[NF];
    a1[0] = a2[0] = sd;
    a1[1] = __fmul_rn(sd, v1x); a1[2] = __fmul_rn(sd, v1y);
    a2[1] = __fmul_rn(sd, v2x); a2[2] = __fmul_rn(sd, v2y);
    if constexpr (NF == 4) {
        const float e0 = __fmul_rn(__fdividef(p[3], p[0]), P.inv_gm1), hs = __fmul_rn(0.5f, sd);
        a1[3] = fmaf(sd, e0, __fmul_rn(hs, fmaf(v1x, v1x, __fmul_rn(v1y, v1y))));
        a2[3] = fmaf(sd, e0, __fmul_rn(hs, fmaf(v2x, v2x, __fmul_rn(v2y, v2y))));
    }
#pragma unroll
    for (int k = 0; k < NF; ++k) {
        s1[k] = __fmul_rn(a1[k], sr1);
        s2[k] = __fmul_rn(a2[k], sr2);
    }
}

// ---------------------------------------------------------------------------
// Faces.
//
// Viscous stress, factored.  The face stress of stress_field (physics.rs:
// 322-349) with the `nu` closure of scheme.rs:230-247 is
//   tau_nn = (rho_l nu_l (s_nn,l + lambda bulk_l) + rho_r nu_r (s_nn,r + lambda bulk_r)) / 2
// (and tau_t alike with s_xy and no bulk term).  nu_l = nu_r = nu for a
// constant viscosity; for the alpha model nu_side = K(face) * cs2 with
// K = alpha / Omega_2(face) / sqrt(gamma - 1), cs2 taken at the face from the
// potential (isothermal, so nu_l = nu_r again) or from the cell's own
// pressure (Euler).  Each cell therefore carries T_nn = c rho (s_nn + lambda
// bulk) and T_xy = c rho s_xy with c = nu (constant), 1 (isothermal alpha) or
// gamma p / rho (Euler alpha), and a face needs tau = K (T_l + T_r) / 2 with
// K = 1 for the constant model.

// -0.5 K of the alpha model at two faces at these distances from the bodies, an
// isothermal face's cs2 left out.  1 / a^3 is taken as rsqrt(a^2)^3: the reference's
// a = |d| + 1e-12 dx (scheme.rs:244) differs from |d| below FP32 resolution
// unless |d| is under about 1e-7 dx, and at |d| = 0 both give K = 0.
__device__ __forceinline__ float2 alpha_nhalf_k2(const float2* K, float2 dx1, float2 dx2, float2 dy1, float2 dy2)
{
    const float2 q1 = rsqrt2(fma2(dy1, dy1, mul2(dx1, dx1))), q2 = rsqrt2(fma2(dy2, dy2, mul2(dx2, dx2)));
    const float2 w2 = fma2(K[C_M1], mul2(q1, mul2(q1, q1)), mul2(K[C_M2], mul2(q2, mul2(q2, q2))));
    return mul2(K[C_ALPHA], rsqrt2(w2));
}

// Two faces normal to AXIS (intercell_flux, physics.rs:584-607, 776-803, with
// hydro-iso2d's and hydro-euler's HLLE) from the states reconstructed on
// either side.  cs2: the isothermal face sound speed; k: minus half the alpha
// model's factor (-1/2 for a constant viscosity); tn, tt: the sums of the two
// cells' factored stresses; vxs, vys: the sums of their velocities (Euler).
//
// With wl = a+ / (a+ + b), wr = b / (a+ + b) and b = -a- the HLLE flux is
//   F = fl wl + fr wr - (ur - ul) b wl,
// and f = u v + pressure terms, so that the states enter through two products,
//   F = ul A + ur B + pressure terms, A = wl (vl + b), B = wr (vr - a+):
// 16 packed operations of an isothermal face pair where forming the conserved
// states and the fluxes on either side takes 22.
//
// Where the flow is supersonic the downwind state's weight is a product with a
// zero, so that it drops out exactly, whichever way the flow goes: as 1 - wl it
// is 1e-7 of that state, which beside a light zone is no small part of the flux.
// What the two rounded weights miss to 1 is then shared out over them (a weight
// of 0 stays 0, that of a state on its own becomes 1): without that the flux is
// off by the reciprocal's rounding, and over 40 disks of 256^2 and 512^2 the
// state's error against 64 bits 3 to 14 % larger (2048^2 without it 29.9 ms a
// pass, with it 30.3).
template <int NF, int AXIS>
__device__ __forceinline__ void faces2(const float2* K, const float2* pl, const float2* pr, float2 cs2, float2 k,
                                       float2 tn, float2 tt, float2 vxs, float2 vys, float2* F)
{
    constexpr int VN = 1 + AXIS, VT = 2 - AXIS;
    const float2 vl = pl[VN], vr = pr[VN];
    float2 csl, csr;
    if constexpr (NF == 3) csl = csr = sqrt2(cs2);
    else {
        csl = sqrt2(mul2(mul2(K[C_GAMMA], pl[3]), rcp2(pl[0])));
        csr = sqrt2(mul2(mul2(K[C_GAMMA], pr[3]), rcp2(pr[0])));
    }
    // outer wave speeds: a+ and -a-
    const float2 alp = add2(vl, csl), arp = add2(vr, csr), blm = sub2(csl, vl), brm = sub2(csr, vr);
    const float2 ap = make_float2(max3f(alp.x, arp.x, 0.0f), max3f(alp.y, arp.y, 0.0f));
    const float2 bm = make_float2(max3f(blm.x, brm.x, 0.0f), max3f(blm.y, brm.y, 0.0f));
    const float2 r = rcp2(add2(ap, bm)), wl1 = mul2(ap, r), wr1 = mul2(bm, r);
    const float2 miss = sub2(K[C_ONE], add2(wl1, wr1)), wl = fma2(wl1, miss, wl1), wr = fma2(wr1, miss, wr1);
    const float2 A = mul2(wl, add2(vl, bm)), B = mul2(wr, sub2(vr, ap));
    const float2 ml = mul2(pl[0], A), mr = mul2(pr[0], B);
    F[0] = add2(ml, mr);
    F[VT] = fma2(ml, pl[VT], mul2(mr, pr[VT]));
    F[VN] = fma2(ml, vl, mul2(mr, vr));
    if constexpr (NF == 3) {
        F[VN] = fma2(cs2, fma2(pl[0], wl, mul2(pr[0], wr)), F[VN]);
        F[VN] = fma2(k, tn, F[VN]);
        F[VT] = fma2(k, tt, F[VT]);
    } else {
        F[VN] = fma2(pl[3], wl, fma2(pr[3], wr, F[VN]));
        // energy: E = rho v^2 / 2 + p / (gamma - 1)
        const float2 el = mul2(K[C_HALF], fma2(pl[1], pl[1], mul2(pl[2], pl[2])));
        const float2 er = mul2(K[C_HALF], fma2(pr[1], pr[1], mul2(pr[2], pr[2])));
        F[3] = fma2(pl[3], fma2(A, K[C_INV_GM1], mul2(vl, wl)), mul2(ml, el));
        F[3] = fma2(pr[3], fma2(B, K[C_INV_GM1], mul2(vr, wr)), fma2(mr, er, F[3]));
        const float2 sn = mul2(k, tn), st = mul2(k, tt);
        F[VN] = add2(F[VN], sn);
        F[VT] = add2(F[VT], st);
        F[3] = fma2(K[C_HALF], fma2(sn, AXIS == 0 ? vxs : vys, mul2(st, AXIS == 0 ? vys : vxs)), F[3]);
    }
}

// Sum K values (a power of two, K <= 32) over the 32 lanes of a warp by
// recursive halving: after the call lane l holds the warp total of value
// item_of_lane(l, K); 2K - 1 shuffles in all.
template <int K> __device__ __forceinline__ float warp_sum_items(float (&v)[K], int lane)
{
#pragma unroll
    for (int half = K / 2, off = 16; half >= 1; half >>= 1, off >>= 1) {
        const bool upper = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float send = upper ? v[i] : v[i + half];
            const float keep = upper ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
    float s = v[0];
    for (int off = 16 / K; off >= 1; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    return s;
}

// Which value of warp_sum_items lane l ends up holding.
template <int K> __device__ __forceinline__ int item_of_lane(int lane)
{
    int item = 0;
    for (int half = K / 2, off = 16; half >= 1; half >>= 1, off >>= 1)
        if (lane & off) item += half;
    return item;
}

// The ledger word (item * NF + field) of a strip's ledger row m.
template <int NF> __device__ __forceinline__ int ledger_word(int m)
{
    if constexpr (NF == 3) {
        if (m < 4) return (GRAV1 + m / 2) * 3 + 1 + m % 2;
        if (m < 7) return BUFFER * 3 + m - 4;
        if (m < 13) return SINK1 * 3 + m - 7;
        return FAKE_MASS * 3 + m - 13;
    } else {
        if (m < 6) return (GRAV1 + m / 3) * 4 + 1 + m % 3;
        if (m < 10) return BUFFER * 4 + m - 6;
        if (m == 10) return COOLING * 4 + 3;
        return SINK1 * 4 + m - 11;
    }
}

// A strip's ledger pieces of block row `brow`, by its warp: for every block
// under the strip the sums over the columns inside it, in the piece's slot of
// the block's.  Out of line, so that it does not weigh on the row loop's
// register allocation.
template <int NF, int STORE, int COPY>
__device__ __noinline__ void flush_strip(const RunDev& rd, int stage, int strip, int ti, int brow, const float* sums,
                                         const float2* led, bool sinks, bool fake)
{
    using T = SWShape<NF, STORE, COPY>;
    constexpr int NL = NITEMS * NF, K = NF == 3 ? 16 : 32;
    const int lane = threadIdx.x & 31;
    const int N = rd.N, bs = rd.bs;
    const int j0 = strip * STRIP_COLS, w = min(STRIP_COLS, N - j0), c0 = 2 * lane - 2;
    const int nc = chunks_in_block_row(brow, bs, N, rd.chunks), first_chunk = chunk_of_row(brow * bs, N, rd.chunks);
    for (int b = j0 / bs; b <= (j0 + w - 1) / bs; ++b) {
        const int lo = max(b * bs - j0, 0), hi = min(b * bs + bs - j0, w);
        const bool inx = c0 >= lo && c0 < hi, iny = c0 + 1 >= lo && c0 + 1 < hi;
        float v[K];
#pragma unroll
        for (int m = 0; m < K; ++m) {
            const bool on = m < T::SINKS_AT || (m < (NF == 3 ? T::FAKE_AT : T::ITEMS) ? sinks : m < T::ITEMS && fake);
            v[m] = 0.0f;
            if (on) {
                const float2 q = m < T::SINKS_AT ? *(const float2*)(sums + m * 64 + 2 * lane) : led[m - T::SINKS_AT];
                v[m] = (inx ? q.x : 0.0f) + (iny ? q.y : 0.0f);
            }
        }
        const float s = warp_sum_items<K>(v, lane);
        const int m = item_of_lane<K>(lane);
        const int piece = strip_piece(strip, ti, b, bs, nc, first_chunk);
        if ((lane & (32 / K - 1)) == 0 && m < T::ITEMS)
            stage_pieces(rd, stage, brow * rd.nb + b, NL)[(size_t)piece * NL + ledger_word<NF>(m)] = (double)s;
    }
}

template <bool SINGLE>
__device__ __forceinline__ const DevParamsF& params_for(const StageArgs& a, const DevParamsF& shared_copy)
{
    // a single-run launch reads its parameters from the kernel arguments
    // (constant-bank operands), a batched one from shared memory
    if constexpr (SINGLE) return a.pf1;
    else return shared_copy;
}

// Programmatic dependent launch: once every CTA of a stage has let the next
// start (or is gone), the next stage's CTAs may take the places of those that
// finish; they wait for the whole stage, and for its writes, before they touch
// anything that a stage writes.
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Asynchronous copy of BYTES bytes (4, 8 or 16, aligned to it) from global to shared memory.
template <int BYTES> __device__ __forceinline__ void copy_async(void* dst, const void* src)
{
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst)), "l"(src), "n"(BYTES) : "memory");
}
// row + 16 place bytes, in one instruction
__device__ __forceinline__ const void* chunk_at(const void* row, unsigned place)
{
    unsigned long long p;
    asm("mad.wide.u32 %0, %1, 16, %2;" : "=l"(p) : "r"(place), "l"(row));
    return (const void*)p;
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING> __device__ __forceinline__ void copy_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// A staged pair, and the pairs of all fields at the stencil's precision (an
// FP64 state's by integer operations: the FP64 pipe converts two lanes a clock).
__device__ __forceinline__ float2 pair_of(const float* p) { return *(const float2*)p; }
template <int NF, int PITCH> __device__ __forceinline__ void pairs_of(const float* p, float2* u)
{
#pragma unroll
    for (int f = 0; f < NF; ++f) u[f] = pair_of(p + f * PITCH);
}
template <int NF, int PITCH> __device__ __forceinline__ void pairs_of(const double* p, float2* u)
{
    double2 v[NF];
    bool ok = true;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        v[f] = *(const double2*)(p + f * PITCH);
        ok = ok && split_range(v[f].x) && split_range(v[f].y);
    }
    if (ok) {
#pragma unroll
        for (int f = 0; f < NF; ++f) u[f] = make_float2(narrow_bits(v[f].x), narrow_bits(v[f].y));
    } else {
#pragma unroll
        for (int f = 0; f < NF; ++f) u[f] = make_float2(narrow(v[f].x), narrow(v[f].y));
    }
}

// ---------------------------------------------------------------------------
template <int NF, int STORE, bool SINGLE, int COPY>
__global__ void __launch_bounds__(32, SWShape<NF, STORE, COPY>::CTAS) stagew_kernel(const __grid_constant__ StageArgs a)
{
    using T = SWShape<NF, STORE, COPY>;
    constexpr bool EVEN = COPY != COPY_WORDS;               // a pair of columns is one aligned word
    using E = typename T::E;
    const int lane = threadIdx.x;

    const int g = blockIdx.x;
    const int ri = SINGLE ? 0 : find_run(a, g);
    const RunDev& rd = a.runs[ri];

    extern __shared__ __align__(128) unsigned char smem_raw[];   // one declaration for every stage kernel
    poison_dynamic_smem(smem_raw);
    unsigned smem_base = smem_addr(smem_raw);
    asm volatile("" : "+r"(smem_base));
    unsigned char* smem = (unsigned char*)__cvta_shared_to_generic(smem_base);
    __builtin_assume(__isShared(smem));
    typename T::Tables& S = *(typename T::Tables*)smem;
    const DevParamsF& P = params_for<SINGLE>(a, S.P);
    const Binary<float>& B = S.B;
    const float2* K = S.K;
    const float* B_lo = S.B_lo;
    const int N = rd.N, bs = rd.bs;
    const size_t nn = (size_t)N * N;
    // rows [i0, i0 + TH) of the strip from column j0: row chunk ti of C (chunk_start, runtime.cuh)
    const int lt = g - rd.tile_base;
    const int strip = lt % rd.tiles_j, ti = rd.chunk0 + lt / rd.tiles_j;
    const int i0 = chunk_start(ti, N, rd.chunks), TH = chunk_start(ti + 1, N, rd.chunks) - i0;
    const int j0 = strip * STRIP_COLS, w = min(STRIP_COLS, N - j0);
    const int c0 = 2 * lane - 2;                            // this lane's columns c0, c0 + 1
    const bool inx = c0 >= 0 && c0 < w, iny = EVEN ? inx : c0 >= 0 && c0 + 1 < w;
    const bool has_base = a.base_slot >= 0;

    const E* uin = (const E*)rd.slot[a.in_slot];
    const E* ubase = has_base ? (const E*)rd.slot[a.base_slot] : nullptr;
    const E* ubg = (const E*)rd.bg;

    E* stencil = (E*)(smem + T::TABLES);                              // [SW_SLOTS][NF][64]: this lane's pair at 2 lane
    E* update = stencil + SW_SLOTS * T::STENCIL;            // [SW_USLOTS][NU][64]
    float2 led[T::ITEMS - T::SINKS_AT];                     // the items that few warps have: local memory
    E* my_stencil = stencil + T::S_FIRST + 2 * lane;        // this lane's pair
    E* my_update = update + T::U_FIRST + 2 * lane;

    // ---- row staging -------------------------------------------------------------
    constexpr int PARTS = STORE == 1 ? 2 : 1;               // planes per field: hi and lo words
    const int colx = ((j0 + c0) % N + N) % N, coly = colx + 1 == N ? 0 : colx + 1;   // this lane's columns in the mesh
    const unsigned bx = colx * (unsigned)sizeof(E), by = coly * (unsigned)sizeof(E);
    auto copy_pair = [&](E* dst, const E* row) {
        if constexpr (EVEN) copy_async<2 * sizeof(E)>(dst, (const char*)row + bx);
        else {
            copy_async<sizeof(E)>(dst, (const char*)row + bx);
            copy_async<sizeof(E)>(dst + 1, (const char*)row + by);
        }
    };
    // Quads: lane l copies the chunks of four columns l, l + 32, ... of a row's planes of one kind,
    // 17 a plane of the stencil, 15 of the update; their places from the row's start, in chunks.
    constexpr int CHUNKS_S = 17 * NF, CHUNKS_U = 15 * NF;
    unsigned quad_s[(CHUNKS_S + 31) / 32], quad_u[(CHUNKS_U + 31) / 32];
    if constexpr (COPY == COPY_QUADS) {
#pragma unroll
        for (int k = 0; 32 * k < CHUNKS_S; ++k) {
            const int c = min(lane + 32 * k, CHUNKS_S - 1), col = ((j0 - 4 + 4 * (c % 17)) % N + N) % N;
            quad_s[k] = (unsigned)((PARTS * (c / 17) * nn + col) / 4);
        }
#pragma unroll
        for (int k = 0; 32 * k < CHUNKS_U; ++k) {
            const int c = min(lane + 32 * k, CHUNKS_U - 1), col = min(j0 + 4 * (c % 15), N - 4);
            quad_u[k] = (unsigned)((PARTS * (c / 15) * nn + col) / 4);
        }
    }
    // (the last lanes repeat the last chunk: a branch costs more)
    const int last_s = 4 * (min(lane + CHUNKS_S / 32 * 32, CHUNKS_S - 1)), last_u = 4 * (min(lane + CHUNKS_U / 32 * 32, CHUNKS_U - 1));
    auto copy_quads_s = [&](E* dst, const E* row) {
#pragma unroll
        for (int k = 0; 32 * k < CHUNKS_S; ++k)
            copy_async<16>(dst + (32 * k + 32 <= CHUNKS_S ? 4 * lane + 128 * k : last_s), chunk_at(row, quad_s[k]));
    };
    auto copy_quads_u = [&](E* dst, const E* row) {
#pragma unroll
        for (int k = 0; 32 * k < CHUNKS_U; ++k)
            copy_async<16>(dst + (32 * k + 32 <= CHUNKS_U ? 4 * lane + 128 * k : last_u), chunk_at(row, quad_u[k]));
    };
    // row rs of the stencil and row ru of the update, as one group
    int gi = wrap(wrap(i0 - 2, N), N);                      // mesh row of rs (a mesh may be one zone wide)
    const E *row_s = uin + (size_t)gi * N, *row_lo = uin + nn + (size_t)i0 * N, *row_bg = ubg + (size_t)i0 * N;
    const E *row_b = has_base ? ubase + (size_t)i0 * N : nullptr;
    auto issue = [&](int rs, int ru) {
        if (rs <= TH + 1) {
            const E* row = row_s;
            row_s += N;
            if (++gi == N) { gi = 0; row_s = uin; }
            const int at = ((rs + 2) & (SW_SLOTS - 1)) * T::STENCIL;
            if constexpr (COPY == COPY_QUADS) copy_quads_s(stencil + at, row);
            else {
#pragma unroll
                for (int f = 0; f < NF; ++f) copy_pair(my_stencil + at + f * T::S_PITCH, row + (size_t)(PARTS * f) * nn);
            }
        }
        if (ru >= 0 && ru < TH) {
            const int at = (ru & 1) * T::UPDATE;
            constexpr int KIND = NF * T::U_PITCH;           // elements of the planes of one kind
            if constexpr (COPY == COPY_QUADS) {
                copy_quads_u(update + at, row_lo);
                copy_quads_u(update + at + KIND, row_bg);
                if (has_base) {
                    copy_quads_u(update + at + 2 * KIND, row_b);
                    copy_quads_u(update + at + 3 * KIND, row_b + nn);
                }
            } else {
#pragma unroll
                for (int f = 0; f < NF; ++f) {
                    E* d = my_update + at + f * T::U_PITCH;
                    if constexpr (STORE == 1) copy_pair(d, row_lo + (size_t)(2 * f) * nn);
                    copy_pair(d + (STORE == 1 ? KIND : 0), row_bg + (size_t)(PARTS * f) * nn);
                    if (has_base) {
                        copy_pair(d + PARTS * KIND, row_b + (size_t)(PARTS * f) * nn);
                        if constexpr (STORE == 1) copy_pair(d + 3 * KIND, row_b + (size_t)(2 * f + 1) * nn);
                    }
                }
            }
            row_lo += N;
            row_bg += N;
            if (has_base) row_b += N;
        }
        copy_commit();
    };
    // What else comes from memory is asked for before any of it is used: on a small mesh a stage
    // is little more than these latencies.  None of this is written by a stage, so it does not
    // wait for the previous one, of which the last rows may still be running.
    auto at = [](int k, int n) { return min(max(k, 0), n); };
    const float2 ya = rd.xcf[at(j0 + c0, N - 1)], yb = rd.xcf[at(j0 + c0 + 1, N - 1)];
    const float2 va = rd.xvf[at(j0 + c0, N)], vb = rd.xvf[at(j0 + c0 + 1, N)];
    const float2 row_x = rd.xcf[at(i0 - 1 + lane, N - 1)], row_f = rd.xvf[at(i0 - 1 + lane, N)];
    const double orbit_word = lane < 10 ? rd.orbit[a.stage * 10 + lane] : 0.0;
    wait_for_previous();
    issue(-2, -1);
    if (!SINGLE)
        for (int k = lane; k < (int)(sizeof(DevParamsF) / 4); k += 32) ((unsigned*)&S.P)[k] = ((const unsigned*)&rd.pf)[k];
    if (lane < 10) {
        const float hi = (float)orbit_word;
        ((float*)&S.B)[lane] = hi;
        S.B_lo[lane] = (float)(orbit_word - (double)hi);
    }
    if (left_out(a.failure, a.stage)) {
        copy_wait<0>();
        return;
    }
    __syncwarp();
    const float dt = (float)*rd.dt;
    const float time = (float)rd.stage_time[a.stage];
    const float itheta2 = P.plm != 0.0f ? __fdividef(0.5f, P.plm) : 0.0f;
    if (lane == 0) {
        float2* K = S.K;
        const float visc = P.visc == 0 ? P.nu : (NF == 3 ? 1.0f : P.gamma), log2e = 1.4426950408889634f;
        K[C_ITHETA2] = f2(itheta2);
        K[C_EDGE] = f2(0.5f * P.plm);
        K[C_NEDGE] = f2(-0.5f * P.plm);
        K[C_NHALF] = f2(-0.5f);
        K[C_HALF] = f2(0.5f);
        K[C_ONE] = f2(1.0f);
        K[C_TN] = f2(4.0f / 3.0f + P.lambda);
        K[C_TT] = f2(-2.0f / 3.0f + P.lambda);
        K[C_VISC] = f2(__fmul_rn(__fmul_rn(P.plm, visc), P.inv_dx));
        K[C_CM1] = f2(__fmul_rn(B.p1.m, P.inv_mach2));
        K[C_CM2] = f2(__fmul_rn(B.p2.m, P.inv_mach2));
        K[C_M1] = f2(B.p1.m);
        K[C_M2] = f2(B.p2.m);
        K[C_NM1DT] = f2(__fmul_rn(-B.p1.m, dt));
        K[C_NM2DT] = f2(__fmul_rn(-B.p2.m, dt));
        K[C_SOFT2] = f2(P.soft2);
        K[C_BUF_SLOPE] = f2(__fmul_rn(-2.0f * P.inv_buffer_scale, log2e));
        K[C_RADIUS] = f2(P.domain_radius);
        K[C_BUF_RATE] = f2(__fmul_rn(-2.0f * dt, P.half_rate_omega));
        K[C_NDT_DX] = f2(__fmul_rn(-P.inv_dx, dt));
        K[C_GAMMA] = f2(P.gamma);
        K[C_GM1] = f2(P.gm1);
        K[C_INV_GM1] = f2(P.inv_gm1);
        K[C_COOL] = f2(__fmul_rn(-dt, P.inv_cool_beta));
        K[C_ALPHA] = f2(__fmul_rn(__fmul_rn(-0.5f, P.nu), P.inv_sqrt_gm));
    }
    __syncwarp();

    const float pdt = P.pdt;
    const df32 w1{a.w1f.hi, a.w1f.lo}, wb{a.bff.hi, a.bff.lo};
    const bool half_avg = a.half_avg != 0;
    const bool want_amax = a.amax_flag != 0, fake_on = NF == 3 && P.fake_rate != 0.0f;
    // the T^4 law's slow-start factor exp(-2 pi / (t + dt)) of this stage (physics.rs:683-774)
    const float slow = NF == 4 && P.cooling_slow_start ? __expf(-6.283185307f / (time + dt)) : 1.0f;
    // Distances to the bodies, from positions as double-floats (close to a body the difference of
    // FP32 positions is off by 1e-6), as tables: per lane along y, in shared memory since registers
    // are scarce, and per row along x, 31 rows at a time (loads in the row loop would be waited for
    // in every row).
    auto from = [](float2 x, float hi, float lo) { return __fadd_rn(__fadd_rn(x.x, -hi), __fadd_rn(x.y, -lo)); };
    S.yc[lane] = make_float2(ya.x, yb.x);
    S.dyc1[lane] = make_float2(from(ya, B.p1.y, B_lo[2]), from(yb, B.p1.y, B_lo[2]));
    S.dyc2[lane] = make_float2(from(ya, B.p2.y, B_lo[7]), from(yb, B.p2.y, B_lo[7]));
    S.dyv1[lane] = make_float2(from(va, B.p1.y, B_lo[2]), from(vb, B.p1.y, B_lo[2]));
    S.dyv2[lane] = make_float2(from(va, B.p2.y, B_lo[7]), from(vb, B.p2.y, B_lo[7]));
    enum { R_C1, R_C2, R_XX, R_F1, R_F2 };
    auto fill_rows = [&](float2 xa, float2 fa) {            // centres of 32 rows and faces below them, one each
        __syncwarp();
        S.rows[R_C1][lane] = f2(from(xa, B.p1.x, B_lo[1]));
        S.rows[R_C2][lane] = f2(from(xa, B.p2.x, B_lo[6]));
        S.rows[R_XX][lane] = f2(__fmul_rn(xa.x, xa.x));
        S.rows[R_F1][lane] = f2(from(fa, B.p1.x, B_lo[1]));
        S.rows[R_F2][lane] = f2(from(fa, B.p2.x, B_lo[6]));
        __syncwarp();
    };
    fill_rows(row_x, row_f);
    const float near2 = (P.sink_r2 + P.soft2) * 1.0001f;    // the sinks' vote: softened distance, with a margin
    constexpr int NPART = T::PARTIALS;
    if constexpr (NF == 3) {
        auto col_part = [&](float2 d) { return fma2(d, d, K[C_SOFT2]); };
        S.part[0][lane] = col_part(S.dyv1[lane]);
        S.part[1][lane] = col_part(S.dyv2[lane]);
        S.part[2][lane] = col_part(S.dyc1[lane]);
        S.part[3][lane] = col_part(S.dyc2[lane]);
    }
    // cs2 = -phi / M^2 (physics.rs:584-607) with the Plummer potential, of two faces dx1, dx2 from the bodies along x
    auto sound2 = [&](float2 dx1, float2 dx2, int which) {
        const float2 r1 = rsqrt2(fma2(dx1, dx1, S.part[which % NPART][lane]));
        const float2 r2 = rsqrt2(fma2(dx2, dx2, S.part[(which + 1) % NPART][lane]));
        return fma2(K[C_CM1], r1, mul2(K[C_CM2], r2));
    };

    float2 dP[NF], P0[NF];            // primitives of row g, and less those of row g - 1
    int trigger = 0;                  // rows whose densities are below the trigger: two bits for g - 1, for g and for g + 1
    float2 xl[NF], xtn, xtt;          // row g - 1: state at its lower x faces, stresses
    float2 div[NF];                   // row g - 1's y fluxes' difference less the flux through its upper x faces
    constexpr int NACC = T::SINKS_AT;
    float2 acc[NACC];                 // ledger items that are live everywhere, summed over rows
#pragma unroll
    for (int m = 0; m < NACC; ++m) acc[m] = f2(0.0f);
#pragma unroll
    for (int f = 0; f < NF; ++f) dP[f] = P0[f] = xl[f] = div[f] = f2(0.0f);
    xtn = xtt = f2(0.0f);
    bool sinks_seen = false, fake_seen = false;
    float amax = 0.0f;
    int brow = i0 / bs, next_flush = bs - i0 % bs;          // row count at which block row `brow` ends
    E* out = (E*)rd.slot[a.out_slot];
    __builtin_assume(__isGlobal(out));
    out += (size_t)i0 * N + j0 + c0;                        // this pair of row g - 1

    int next_fill = 31;
    for (int n = -2; n <= TH + 1; ++n) {
        if constexpr (COPY == COPY_QUADS) __syncwarp();     // a slot is read by other lanes than those that fill it
        issue(n + 1, n - 1);
        // (in the Euler kernel after the loop: here it costs its schedule 4 %)
        if (NF == 3 && n == TH + 1) let_next_start();
        const int gr = n - 1;
        if (gr == next_fill) {   // the table holds rows gr - 1 to gr + 30
            fill_rows(rd.xcf[at(i0 + gr - 1 + lane, N - 1)], rd.xvf[at(i0 + gr - 1 + lane, N)]);
            next_fill += 31;
        }
        const int rt = gr - (next_fill - 32);               // row g's place in it

        // ---- row n -> primitives (try_block_primitive, scheme.rs:185-199) ------------
        float2 pn[NF];
        {
            copy_wait<1>();   // the row's group, and that of the update below
            if constexpr (COPY == COPY_QUADS) __syncwarp();
            const E* sb = my_stencil + ((n + 2) & (SW_SLOTS - 1)) * T::STENCIL;
            float2 u[NF];
            pairs_of<NF, T::S_PITCH>(sb, u);
            int ea = 0, eb = 0;
            if constexpr (NF == 3) {
                if (P.has_density_floor) {
                    if (u[0].x < P.density_floor) { u[0].x = P.density_floor; u[1].x = u[2].x = 0.0f; }
                    if (u[0].y < P.density_floor) { u[0].y = P.density_floor; u[1].y = u[2].y = 0.0f; }
                }
                const float2 ir = rcp2(u[0]);
                pn[0] = u[0];
                pn[1] = mul2(u[1], ir);
                pn[2] = mul2(u[2], ir);
                ea = u[0].x < 0.0f;
                eb = u[0].y < 0.0f;
            } else {
                const float2 ir = rcp2(u[0]);
                pn[0] = u[0];
                pn[1] = mul2(u[1], ir);
                pn[2] = mul2(u[2], ir);
                pn[3] = mul2(sub2(u[3], mul2(mul2(K[C_HALF], u[0]), fma2(pn[1], pn[1], mul2(pn[2], pn[2])))), K[C_GM1]);
                // the floors and checks of Euler::try_to_primitive (physics.rs:631-660)
                if (P.has_density_floor) {
                    if (pn[0].x < P.density_floor) {
                        pn[0].x = P.density_floor;
                        pn[1].x = pn[2].x = 0.0f;
                        pn[3].x = P.density_floor_pow_gamma;
                    }
                    if (pn[0].y < P.density_floor) {
                        pn[0].y = P.density_floor;
                        pn[1].y = pn[2].y = 0.0f;
                        pn[3].y = P.density_floor_pow_gamma;
                    }
                }
                if (P.has_pressure_floor) {
                    if (pn[3].x < P.pressure_floor && !(pn[0].x < 0.0f)) pn[3].x = P.pressure_floor;
                    if (pn[3].y < P.pressure_floor && !(pn[0].y < 0.0f)) pn[3].y = P.pressure_floor;
                }
                ea = pn[0].x < 0.0f ? 1 : (pn[3].x <= 0.0f ? 2 : 0);
                eb = pn[0].y < 0.0f ? 1 : (pn[3].y <= 0.0f ? 2 : 0);
            }
            if (__any_sync(0xffffffffu, ea || eb) && n >= 0 && n < TH) {
                if (ea && inx) atomicMin(&a.failure->key, error_key(a.stage, ri, rd, i0 + n, j0 + c0, ea));
                if (eb && iny) atomicMin(&a.failure->key, error_key(a.stage, ri, rd, i0 + n, j0 + c0 + 1, eb));
            }
        }

        float2 dn[NF];                                      // rows n less n - 1
#pragma unroll
        for (int f = 0; f < NF; ++f) dn[f] = sub2(pn[f], P0[f]);
        if (pdt > 0.0f) trigger = trigger >> 2 | (pn[0].x < pdt ? 16 : 0) | (pn[0].y < pdt ? 32 : 0);

        if (gr >= -1) {
            // ---- slopes and stresses of row g (scheme.rs:216-254) ---------------------
            float lv[NF], rv[NF];                           // columns c0 - 1 and c0 + 2
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                lv[f] = __shfl_up_sync(0xffffffffu, P0[f].y, 1);
                rv[f] = __shfl_down_sync(0xffffffffu, P0[f].x, 1);
                // the two outermost columns have no such neighbour: NaN in a
                // read-set check build (tma.cuh), whose states must not change
                if (lane == 0) lv[f] = poison_or(lv[f]);
                if (lane == 31) rv[f] = poison_or(rv[f]);
            }
            float2 gx[NF], gy[NF];                          // slopes over theta
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const float2 y = mul2(K[C_ITHETA2], add2(dP[f], dn[f]));
                gx[f] = make_float2(minmod3(dP[f].x, y.x, dn[f].x), minmod3(dP[f].y, y.y, dn[f].y));
                const float a0 = __fadd_rn(P0[f].x, -lv[f]), a1 = __fadd_rn(P0[f].y, -P0[f].x), a2 = __fadd_rn(rv[f], -P0[f].y);
                const float t = __fmul_rn(itheta2, a1);
                gy[f] = make_float2(minmod3(a0, fmaf(itheta2, a0, t), a1), minmod3(a1, fmaf(itheta2, a2, t), a2));
            }
            if (pdt > 0.0f) {   // (densities below 0 fail the advance before their slopes count)
                const int below = (trigger | trigger >> 2 | trigger >> 4) & 3, own = trigger >> 2 & 3;
                const bool yx = own || lv[0] < pdt, yy = own || rv[0] < pdt;
#pragma unroll
                for (int f = 0; f < NF; ++f) {
                    gx[f] = make_float2(below & 1 ? 0.0f : gx[f].x, below & 2 ? 0.0f : gx[f].y);
                    gy[f] = make_float2(yx ? 0.0f : gy[f].x, yy ? 0.0f : gy[f].y);
                }
            }
            const float2 cv = mul2(K[C_VISC], P0[NF == 4 && P.visc != 0 ? NF - 1 : 0]);
            const float2 txx = mul2(cv, fma2(K[C_TN], gx[1], mul2(K[C_TT], gy[2])));
            const float2 tyy = mul2(cv, fma2(K[C_TN], gy[2], mul2(K[C_TT], gx[1])));
            const float2 txy = mul2(cv, add2(gx[2], gy[1]));

            if (gr >= 0) {
                // ---- y fluxes of row g at the pair's left faces -------------------------
                float2 Fy[NF], dfy[NF];
                {
                    float2 pl[NF], pr[NF];
#pragma unroll
                    for (int f = 0; f < NF; ++f) {
                        const float2 e = fma2(gy[f], K[C_EDGE], P0[f]);
                        pl[f] = make_float2(__shfl_up_sync(0xffffffffu, e.y, 1), e.x);
                        pr[f] = fma2(gy[f], K[C_NEDGE], P0[f]);
                    }
                    const float2 tn = add2(make_float2(__shfl_up_sync(0xffffffffu, tyy.y, 1), tyy.x), tyy);
                    const float2 tt = add2(make_float2(__shfl_up_sync(0xffffffffu, txy.y, 1), txy.x), txy);
                    float2 cs2 = f2(0.0f), k = K[C_NHALF], vxs = f2(0.0f), vys = f2(0.0f);
                    const float2 dx1 = S.rows[R_C1][rt], dx2 = S.rows[R_C2][rt];
                    if constexpr (NF == 3) cs2 = sound2(dx1, dx2, 0);
                    else {
                        vxs = add2(make_float2(lv[1], P0[1].x), P0[1]);
                        vys = add2(make_float2(lv[2], P0[2].x), P0[2]);
                    }
                    if (P.visc != 0) {
                        k = alpha_nhalf_k2(K, dx1, dx2, S.dyv1[lane], S.dyv2[lane]);
                        if constexpr (NF == 3) k = mul2(k, cs2);
                    }
                    faces2<NF, 1>(K, pl, pr, cs2, k, tn, tt, vxs, vys, Fy);
#pragma unroll
                    for (int f = 0; f < NF; ++f) {
                        const float2 right = make_float2(Fy[f].y, __shfl_down_sync(0xffffffffu, Fy[f].x, 1));
                        dfy[f] = sub2(right, Fy[f]);
                    }
                }
                // ---- x fluxes between rows g - 1 and g ----------------------------------
                float2 Fx[NF];
                {
                    float2 pr[NF];
#pragma unroll
                    for (int f = 0; f < NF; ++f) pr[f] = fma2(gx[f], K[C_NEDGE], P0[f]);
                    float2 cs2 = f2(0.0f), k = K[C_NHALF], vxs = f2(0.0f), vys = f2(0.0f);
                    const float2 dx1 = S.rows[R_F1][rt], dx2 = S.rows[R_F2][rt];
                    if constexpr (NF == 3) cs2 = sound2(dx1, dx2, 2);
                    else {
                        vxs = add2(P0[1], sub2(P0[1], dP[1]));
                        vys = add2(P0[2], sub2(P0[2], dP[2]));
                    }
                    if (P.visc != 0) {
                        k = alpha_nhalf_k2(K, dx1, dx2, S.dyc1[lane], S.dyc2[lane]);
                        if constexpr (NF == 3) k = mul2(k, cs2);
                    }
                    faces2<NF, 0>(K, xl, pr, cs2, k, add2(xtn, txx), add2(xtt, txy), vxs, vys, Fx);
                }
                // ---- update of row g - 1 (side effects masked in the first iteration) ------
                {
                    const int ru = gr - 1;
                    const bool up_ok = ru >= 0;
                    const E* sb = my_stencil + ((ru + 2) & (SW_SLOTS - 1)) * T::STENCIL;
                    const E* q = my_update + (ru & 1) * T::UPDATE;
                    const E* qg = q + (STORE == 1 ? NF * T::U_PITCH : 0);                    // background
                    const E* qb = qg + NF * T::U_PITCH;                                      // RK base
                    float2 uc[NF], u0[NF];
                    pairs_of<NF, T::S_PITCH>(sb, uc);
                    pairs_of<NF, T::U_PITCH>(qg, u0);
                    // sources of the pair (Physics::source_terms, physics.rs:423-457;
                    // Isothermal 528-582, Euler 683-774)
                    float2 tot[NF];
                    const float2 dx1 = S.rows[R_C1][rt - 1], dx2 = S.rows[R_C2][rt - 1];
                    const float2 dy1 = S.dyc1[lane], dy2 = S.dyc2[lane];
                    // Plummer accelerations (kepler-two-body, restated): -m d / (d^2 + s^2)^(3/2)
                    const float2 t1 = fma2(dx1, dx1, NF == 3 ? S.part[2 % NPART][lane] : fma2(dy1, dy1, K[C_SOFT2]));
                    const float2 t2 = fma2(dx2, dx2, NF == 3 ? S.part[3 % NPART][lane] : fma2(dy2, dy2, K[C_SOFT2]));
                    const float2 r1 = rsqrt2(t1), r2 = rsqrt2(t2);
                    const float2 r13 = mul2(r1, mul2(r1, r1)), r23 = mul2(r2, mul2(r2, r2));
                    const float2 q1 = mul2(mul2(uc[0], K[C_NM1DT]), r13);
                    const float2 q2 = mul2(mul2(uc[0], K[C_NM2DT]), r23);
                    constexpr int G2 = NF - 1, BU = 2 * (NF - 1);
                    // buffer: 0.5 rate (1 + tanh(y)) Omega_outer, y = (r - R) / scale, 1 + tanh(y) = 2 / (1 + exp(-2y))
                    const float2 yc2 = S.yc[lane], rr2 = fma2(yc2, yc2, S.rows[R_XX][rt - 1]);
                    // (r - R first: r / scale - R / scale is NaN for a scale of 0, a sharp edge, and rounds twice)
                    const float2 yb = mul2(sub2(sqrt2(rr2), K[C_RADIUS]), K[C_BUF_SLOPE]);
                    const float2 den = add2(K[C_ONE], make_float2(exp2_fast(yb.x), exp2_fast(yb.y)));
                    const float2 kb = mul2(K[C_BUF_RATE], rcp2(den));
#pragma unroll
                    for (int f = 0; f < NF; ++f) {
                        tot[f] = mul2(sub2(uc[f], u0[f]), kb);
                        acc[BU + f] = add2(acc[BU + f], tot[f]);
                    }
                    if constexpr (NF == 3) {
                        tot[1] = fma2(q1, dx1, fma2(q2, dx2, tot[1]));
                        tot[2] = fma2(q1, dy1, fma2(q2, dy2, tot[2]));
                        acc[0] = fma2(q1, dx1, acc[0]);
                        acc[1] = fma2(q1, dy1, acc[1]);
                        acc[G2] = fma2(q2, dx2, acc[G2]);
                        acc[G2 + 1] = fma2(q2, dy2, acc[G2 + 1]);
                    }
                    if constexpr (NF == 4) {
                        // primitive velocities and specific internal energy (no floors, physics.rs:696)
                        const float2 ir = rcp2(uc[0]);
                        const float2 vx = mul2(uc[1], ir), vy = mul2(uc[2], ir);
                        const float2 v2 = fma2(vx, vx, mul2(vy, vy));
                        const float2 e0 = mul2(sub2(uc[3], mul2(mul2(K[C_HALF], uc[0]), v2)), ir);
                        // gravity and its work
                        const float2 g1x = mul2(q1, dx1), g1y = mul2(q1, dy1), g2x = mul2(q2, dx2), g2y = mul2(q2, dy2);
                        const float2 g1e = fma2(g1x, vx, mul2(g1y, vy)), g2e = fma2(g2x, vx, mul2(g2y, vy));
                        tot[1] = add2(add2(g1x, g2x), tot[1]);
                        tot[2] = add2(add2(g1y, g2y), tot[2]);
                        tot[3] = add2(add2(g1e, g2e), tot[3]);
                        acc[0] = add2(acc[0], g1x);
                        acc[1] = add2(acc[1], g1y);
                        acc[2] = add2(acc[2], g1e);
                        acc[3] = add2(acc[3], g2x);
                        acc[4] = add2(acc[4], g2y);
                        acc[5] = add2(acc[5], g2e);
                        // Cooling of the specific internal energy, de = e_cooled - e0 formed directly
                        // (e0 (exp(-c) - 1), e0 ((1 + x)^(-1/3) - 1) through expm1 and log1p): as a
                        // difference of two near-equal energies it loses ~1e-7 / (c or x) of its value.
                        // The item's mass and momentum are zero in FP32: in the reference they are
                        // only the rounding of a prim -> cons round trip.
                        float2 dec;
                        if (P.cooling_kind == 1) {
                            // beta-cooling (not in the reference): e -> e exp(-Omega dt / beta),
                            // Omega^2 = sum m / (d^2 + s^2)^(3/2)
                            const float2 om = sqrt2(fma2(K[C_M1], r13, mul2(K[C_M2], r23)));
                            const float2 c = mul2(om, K[C_COOL]);
                            if (__any_sync(0xffffffffu, fabsf(c.x) > 0.35f || fabsf(c.y) > 0.35f))
                                dec = mul2(e0, make_float2(expm1f(c.x), expm1f(c.y)));
                            else
                                dec = mul2(e0, expm1_small2(c));
                        } else {
                            // T^4 law: e -> e (1 + z)^(-1/3), z = 3 a e^3 dt, a = coefficient / rho^n x slow
                            // start.  With y = (1 + z)^(-1/3), y - 1 = (y^3 - 1) / (y^2 + y + 1) =
                            // -z / ((1 + z) (y^2 + y + 1)) without cancellation; y from the special
                            // functions and a Newton step for y^-3 = 1 + z.
                            float2 rho_n = K[C_ONE];
                            for (int m = 0; m < P.density_index; ++m) rho_n = mul2(rho_n, uc[0]);
                            const float2 ac = mul2(f2(__fmul_rn(P.cool_coef, slow)), rcp2(rho_n));
                            float2 z = mul2(mul2(f2(__fmul_rn(3.0f, dt)), ac), mul2(mul2(e0, e0), e0));
                            z = make_float2(z.x > 1e30f ? 1e30f : z.x, z.y > 1e30f ? 1e30f : z.y);   // y - 1 = -1
                            const float2 s = add2(K[C_ONE], z);
                            float2 y = make_float2(exp2_fast(__fmul_rn(log2_fast(s.x), -1.0f / 3.0f)),
                                                   exp2_fast(__fmul_rn(log2_fast(s.y), -1.0f / 3.0f)));
                            y = fma2(mul2(y, f2(1.0f / 3.0f)), sub2(K[C_ONE], mul2(mul2(s, y), mul2(y, y))), y);
                            const float2 q = mul2(s, fma2(y, add2(y, K[C_ONE]), K[C_ONE]));
                            dec = mul2(mul2(e0, mul2(z, rcp2(q))), f2(-1.0f));
                        }
                        if (P.has_mach_ceiling) {
                            // e >= 2 e_kinetic / (gamma (gamma - 1) M^2)
                            const float2 ek = mul2(f2(0.5f * P.k_mach_ceiling), v2);
                            const float eca = e0.x + dec.x, ecb = e0.y + dec.y;
                            const float ma = fmaxf(eca, ek.x), mb = fmaxf(ecb, ek.y);
                            if (ma != eca) dec.x = ma - e0.x;
                            if (mb != ecb) dec.y = mb - e0.y;
                        }
                        dec = mul2(uc[0], dec);
                        acc[10] = add2(acc[10], dec);
                        tot[3] = add2(tot[3], dec);
                    }
                    // sinks: only where a zone of the warp lies inside a sink radius
                    const bool near = inx && fminf(min3f(t1.x, t2.x, t1.y), t2.y) < near2;
                    if (__any_sync(0xffffffffu, near) && up_ok) {
                        if (!sinks_seen) {
#pragma unroll
                            for (int m = 0; m < 2 * NF; ++m) led[m] = f2(0.0f);
                            sinks_seen = true;
                        }
#pragma unroll
                        for (int side = 0; side < 2; ++side) {
                            float us[NF], s1[NF], s2[NF];
#pragma unroll
                            for (int f = 0; f < NF; ++f) us[f] = side ? uc[f].y : uc[f].x;
                            sink_items_exact<NF>(P, B, us, dx1.x, side ? dy1.y : dy1.x, dx2.x, side ? dy2.y : dy2.x, dt, s1, s2);
#pragma unroll
                            for (int f = 0; f < NF; ++f) {
                                const float sk = s1[f] + s2[f];
                                if (side) tot[f].y += sk;
                                else tot[f].x += sk;
                                (side ? led[f].y : led[f].x) += s1[f];
                                (side ? led[NF + f].y : led[NF + f].x) += s2[f];
                            }
                        }
                    }
                    // fake mass: u0 rate dt unless Sigma < Sigma_0 threshold
                    if (fake_on && up_ok) {
                        const bool offa = uc[0].x < u0[0].x * P.fake_thr, offb = uc[0].y < u0[0].y * P.fake_thr;
#pragma unroll
                        for (int f = 0; f < 3; ++f) {
                            const float2 fk = mul2(mul2(u0[f], f2(P.fake_rate)), f2(dt));
                            const float2 on = make_float2(offa ? 0.0f : fk.x, offb ? 0.0f : fk.y);
                            tot[f] = add2(tot[f], on);
                            float2& s = led[T::FAKE_AT - T::SINKS_AT + f];
                            s = fake_seen ? add2(s, on) : on;
                        }
                        fake_seen = true;
                    }
                    // flux divergence and the RK update (scheme.rs:290-305; state.rs:183-199)
                    float2 uo[NF], ulo[NF];                             // the result's high and low words
                    if constexpr (STORE == 1) {
                        df2 o[NF];
#pragma unroll
                        for (int f = 0; f < NF; ++f) {
                            const float2 inc = fma2(add2(Fx[f], div[f]), K[C_NDT_DX], tot[f]);
                            o[f] = two_sum2(uc[f], inc);
                            o[f].lo = add2(o[f].lo, pair_of(q + f * T::U_PITCH));
                        }
                        if (has_base) {
#pragma unroll
                            for (int f = 0; f < NF; ++f) {
                                const df2 b0{pair_of(qb + f * T::U_PITCH), pair_of(qb + (NF + f) * T::U_PITCH)};
                                if (half_avg) {
                                    const df2 sm = df_add2(o[f], b0);
                                    o[f] = {mul2(sm.hi, K[C_HALF]), mul2(sm.lo, K[C_HALF])};
                                } else {
                                    const df2 x1 = df_mul2(o[f], w1), x2 = df_mul2(b0, wb);
                                    o[f] = df_add2(x1, x2);
                                }
                            }
                        } else {
#pragma unroll
                            for (int f = 0; f < NF; ++f) o[f] = fast_two_sum2(o[f].hi, o[f].lo);
                        }
                        if (up_ok && inx) {
#pragma unroll
                            for (int f = 0; f < NF; ++f) {
                                E* oh = out + (size_t)(2 * f) * nn;
                                E* ol = out + (size_t)(2 * f + 1) * nn;
                                if constexpr (EVEN) {
                                    *(float2*)oh = o[f].hi;
                                    *(float2*)ol = o[f].lo;
                                } else {
                                    oh[0] = o[f].hi.x;
                                    ol[0] = o[f].lo.x;
                                    if (iny) { oh[1] = o[f].hi.y; ol[1] = o[f].lo.y; }
                                }
                            }
                        }
#pragma unroll
                        for (int f = 0; f < NF; ++f) { uo[f] = o[f].hi; ulo[f] = o[f].lo; }
                    } else {
                        double2 o[NF];
#pragma unroll
                        for (int f = 0; f < NF; ++f) {
                            const float2 inc = fma2(add2(Fx[f], div[f]), K[C_NDT_DX], tot[f]);
                            o[f] = *(const double2*)(sb + f * T::S_PITCH);
                            o[f].x += widen(inc.x);
                            o[f].y += widen(inc.y);
                        }
                        if (has_base) {
                            const double keep = -a.bf + 1.0;
#pragma unroll
                            for (int f = 0; f < NF; ++f) {
                                const double2 b0 = *(const double2*)(qb + f * T::U_PITCH);
                                if (half_avg) o[f] = make_double2(halve(o[f].x + b0.x), halve(o[f].y + b0.y));
                                else o[f] = make_double2(o[f].x * keep + b0.x * a.bf, o[f].y * keep + b0.y * a.bf);
                            }
                        }
                        if (want_amax) {
#pragma unroll
                            for (int f = 0; f < NF; ++f) {
                                split_double(o[f].x, uo[f].x, ulo[f].x);
                                split_double(o[f].y, uo[f].y, ulo[f].y);
                            }
                        }
                        if (up_ok && inx) {
#pragma unroll
                            for (int f = 0; f < NF; ++f) {
                                E* p = out + (size_t)f * nn;
                                if constexpr (EVEN) *(double2*)p = o[f];
                                else {
                                    p[0] = o[f].x;
                                    if (iny) p[1] = o[f].y;
                                }
                            }
                        }
                    }
                    if (up_ok) {
                        if (want_amax) {
                            float ua[NF], ub[NF], la[NF], lb[NF];
#pragma unroll
                            for (int f = 0; f < NF; ++f) { ua[f] = uo[f].x; ub[f] = uo[f].y; la[f] = ulo[f].x; lb[f] = ulo[f].y; }
                            if (inx) amax = fmaxf(max_speed_f32<NF>(P, ua, la), amax);
                            if (iny) amax = fmaxf(max_speed_f32<NF>(P, ub, lb), amax);
                        }
                        if (ru + 1 == next_flush || ru + 1 == TH) {   // the end of a block row, or of the chunk
                            if constexpr (!T::SUMS_OVER_OWN) __syncwarp();   // others may not have read theirs yet
                            float* sums = (float*)(update + (ru & 1) * T::UPDATE);   // this row's, which is done with
#pragma unroll
                            for (int m = 0; m < NACC; ++m) {
                                *(float2*)(sums + m * 64 + 2 * lane) = acc[m];
                                acc[m] = f2(0.0f);
                            }
                            flush_strip<NF, STORE, COPY>(rd, a.stage, strip, ti, brow, sums, led, sinks_seen, fake_seen);
                            sinks_seen = fake_seen = false;
                            ++brow;
                            next_flush += bs;
                        }
                        out += N;
                    } else {
#pragma unroll
                        for (int m = 0; m < NACC; ++m) acc[m] = f2(0.0f);   // the row above the chunk's first
                    }
                }
#pragma unroll
                for (int f = 0; f < NF; ++f) div[f] = sub2(dfy[f], Fx[f]);
            }
#pragma unroll
            for (int f = 0; f < NF; ++f) xl[f] = fma2(gx[f], K[C_EDGE], P0[f]);
            xtn = txx;
            xtt = txy;
        }
#pragma unroll
        for (int f = 0; f < NF; ++f) { dP[f] = dn[f]; P0[f] = pn[f]; }
    }

    if (NF == 4) let_next_start();

    if (want_amax) {
        const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));   // amax >= 0: its bits are in order
        if (lane == 0 && m) atomicMax(rd.amax, (unsigned long long)__double_as_longlong((double)__uint_as_float(m)));
    }
}

}  // namespace b2d
