// stage64.cuh — the FP64 RK-stage kernel (the parity path).
//
// One launch performs one call of try_advance_rk (src/scheme.rs:88-173) for
// every run of a context: cons→prim (try_block_primitive, scheme.rs:185-199),
// PLM slopes and HLLE + viscous fluxes (scheme.rs:216-268), flux divergence +
// sources + RK average (scheme.rs:290-305, state.rs:183-199), the per-block
// source ledger's pieces (scheme.rs:288-313) and, on the last stage of an advance, the
// max signal speed of the next dt (state.rs:121-133).
//
// What bounds it.  GB300 executes two FP64 lanes per clock and SM: one FP64
// warp instruction takes 16 clocks of the SM, 64 clocks of each scheduler's
// share.  So the kernel counts FP64 operations, and everything else (integer
// compares, selects, address arithmetic, shared-memory traffic) hides behind
// them.  Every result is the one that the reference's operation order gives;
// what is saved are operations whose result is known or can be had exactly
// in fewer:
//  * Divisions by a divisor that several quotients share (dx, Mach², the HLLE
//    wave-speed difference, a zone's density, a body's distance cubed) take
//    three operations each from the divisor's rounded reciprocal (Divisor),
//    and one where the divisor is a power of two.
//  * Minimum, maximum, sign tests and the limiter compare bit patterns as
//    integers: no FP64 compare.
//  * A difference of neighbouring zones, times theta, is formed once per face
//    and read by the two zones beside it.
//  * Products by ±1/2 are folded into a fused multiply-add: the product is
//    exact, so the rounding is the same.
//  * The x and y parts of the distances to the bodies are tables per row and
//    column of the tile; the stress of a constant viscosity is formed once
//    per zone instead of once per side of each of its four faces.
//  * The buffer's rate depends on the place only: it is a table of the context.
//  * A warp evaluates sinks only if one of its zones lies in a sink radius,
//    and only the upwind state of faces that are all supersonic, whose flux
//    times and over the wave speed takes three operations (ThereAndBack).
//
// Work decomposition.  A CTA takes sub-tiles of TH x TW zones of one mesh
// block (at most 16 x 32; blocks are split evenly, so any block size does) and
// goes through the phases with all its threads over the sub-tile's zones or
// faces, so the guard zones cost their share of warps only: marching down the
// rows of a column strip instead spends a whole warp's pass on the guard
// columns of every row.  Two CTAs per SM (128 registers) fill the phases' ends;
// three (85 registers) or one of 512 threads were 1-19 % slower.
//
// Measured per stage, against the marching kernel it took the place of (one
// thread per column of a block's 64 rows): isothermal 2048^2 10.6 -> 3.10 ms,
// 384^2 (6 x 6 blocks of 64^2) 2.97 -> 0.130 ms; Euler 256^2 with the T^4 law
// 3.79 -> 0.119 ms (of which the upwind fluxes' quotients and y loops that begin
// with the warps that had fewer x faces: 3.18 -> 3.15, 0.134 -> 0.131 and 0.123 ->
// 0.119 ms; one range test fewer in the quotients: 3.15 -> 3.10 ms).  With about
// 395 operations per zone 2.65 ms would be all of the FP64 pipe at 2048^2.
#pragma once

#include "stage.cuh"

namespace b2d {

constexpr int S64_THREADS = 256;

// Doubles of dynamic shared memory for sub-tiles of at most th x tw zones.
__host__ __device__ inline int s64_prim_doubles(int nf, int th, int tw) { return nf * (th + 4) * (tw + 4); }
__host__ __device__ inline int s64_rec_doubles(int nf, int th, int tw) { return (2 * nf + 4) * (th + 2) * (tw + 2); }
__host__ __device__ inline int s64_diff_doubles(int nf, int th, int tw)
{
    return nf * ((th + 3) * (tw + 2) + (th + 2) * (tw + 3));   // the faces' fluxes take its place later
}
// per row or column: centre and, per body, the signed distance, its square and
// -m times it at the centre, and the square at the face (n + 1 faces)
__host__ __device__ inline int s64_geo_doubles(int n) { return 7 * n + 5 * (n + 1); }
__host__ __device__ inline int s64_smem_bytes(int nf, int th, int tw)
{
    return 8 * (s64_prim_doubles(nf, th, tw) + s64_rec_doubles(nf, th, tw) + s64_diff_doubles(nf, th, tw) +
                s64_geo_doubles(th) + s64_geo_doubles(tw));
}

// ---------------------------------------------------------------------------
// Exact FP64 helpers.
__device__ __forceinline__ unsigned long long dbits(double x) { return (unsigned long long)__double_as_longlong(x); }
__device__ __forceinline__ double from_bits(unsigned long long b) { return __longlong_as_double((long long)b); }
constexpr unsigned long long D_SIGN = 0x8000000000000000ull;
constexpr unsigned long long D_INF = 0x7ff0000000000000ull;

// x < 0, false for NaN
__device__ __forceinline__ bool negative(double x) { return dbits(x) - (D_SIGN + 1) < D_INF; }
__device__ __forceinline__ bool zero(double x) { return (dbits(x) & ~D_SIGN) == 0ull; }
// zero, or a magnitude in [2^-400, 2^400)
__device__ __forceinline__ bool moderate(double x)
{
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return h - 0x26f00000u < 0x32000000u || (h | (unsigned)__double2loint(x)) == 0u;
}
// in [2^-400, 2^400)
__device__ __forceinline__ bool moderate_positive(double x) { return (unsigned)__double2hiint(x) - 0x26f00000u < 0x32000000u; }
// a magnitude below 2^100: neither infinite nor NaN, and products of a few such values are not either
__device__ __forceinline__ bool bounded(double x) { return ((unsigned)__double2hiint(x) & 0x7fffffffu) < 0x46300000u; }
// max(0, x), 0 for NaN
__device__ __forceinline__ unsigned long long positive_part(unsigned long long b) { return b <= D_INF ? b : 0ull; }
// max(0, a, b) and min(0, a, b) of fmax and fmin, which pass over NaN
__device__ __forceinline__ double max_0(double a, double b)
{
    const unsigned long long x = positive_part(dbits(a)), y = positive_part(dbits(b));
    return from_bits(x > y ? x : y);
}
__device__ __forceinline__ double min_0(double a, double b)
{
    const unsigned long long x = positive_part(dbits(a) ^ D_SIGN), y = positive_part(dbits(b) ^ D_SIGN);
    return from_bits((x > y ? x : y) ^ D_SIGN);
}

__device__ __noinline__ double plain_div(double a, double b) { return a / b; }

// Quotients by one divisor d: with r the rounded reciprocal of d, q = x r and
// the residual e = x - q d (exact in a fused step), q + e r rounds to x / d
// (Markstein 1990, IBM J. Res. Dev. 34; with the divisor known in advance:
// Brisebarre, Muller & Raina 2004, IEEE Trans. Comput. 53).  Equal to the
// division in each of 4e8 random quotients, among them divisors and dividends
// next to powers of two (tests/test_gpu_exact_helpers.py).  Negative divisors,
// magnitudes far from 1, infinities and NaN take the division itself.
struct Divisor {
    double d, r;
    bool ok;
    __device__ __forceinline__ explicit Divisor(double d_) : Divisor(d_, 1.0 / d_) {}
    __device__ __forceinline__ Divisor(double d_, double r_)
        : d(d_), r(r_), ok(moderate_positive(d_)) {}
    __device__ __forceinline__ double operator()(double x) const
    {
        if (!(ok && moderate(x))) return plain_div(x, d);
        const double q = __dmul_rn(x, r);
        return __fma_rn(-__fma_rn(q, d, -x), r, q);   // (as q + (x - q d) r, -0 / d would come out as +0)
    }
};

// (f w) / w, both rounded.  The quotient is f but for the rounding of x = f w:
// with e = x - f w (exact in a fused step) it is f + e / w, which one fused step
// rounds.  1 / w to rounding: the 20 bits of the approximate reciprocal and one
// cubic step, 1 + d + d^2 of the residual d (Householder).  Equal to the two
// operations in each of 2e8 random pairs (tests/test_gpu_exact_helpers.py); three
// operations a quotient and three for w in place of four and a division.
struct ThereAndBack {
    double w, r;
    bool ok;
    __device__ __forceinline__ explicit ThereAndBack(double w_) : w(w_), ok(moderate(w_) && w_ != 0.0)
    {
        double r0;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(w));
        const double d = __fma_rn(-w, r0, 1.0);
        r = __fma_rn(r0, __fma_rn(d, d, d), r0);
    }
    __device__ __forceinline__ double operator()(double f) const
    {
        if (!(ok && moderate(f))) return plain_div(f * w, w);
        const double x = __dmul_rn(f, w);
        const double q = __fma_rn(__fma_rn(-f, w, x), r, f);
        return zero(f) ? f : q;   // (the sign of a zero)
    }
};

__device__ __forceinline__ bool power_of_two(double x)
{
    const unsigned h = (unsigned)__double2hiint(x);
    return ((h & 0x000fffffu) | (unsigned)__double2loint(x)) == 0u && h - 0x26f00000u < 0x32000000u;
}

__device__ __noinline__ double minmod_nan(double x, double y, double z)
{
    return fmax(fmin(fmin(x, y), z), 0.0) + fmin(fmax(fmax(x, y), z), 0.0);
}

// The limiter of plm_gradient (godunov-core, restated) on x, y / 2 and z: the one of
// smallest magnitude if all share a sign, else 0.  Halving takes one off the
// exponent; NaN, infinite and subnormal arguments take the general form.
__device__ __forceinline__ double minmod_bits(double x, double y, double z)
{
    constexpr unsigned long long ONE = 1ull << 52;
    const unsigned long long a = dbits(x), b = dbits(y), c = dbits(z);
    const unsigned long long ma = a & ~D_SIGN, mc = c & ~D_SIGN;
    unsigned long long mb = b & ~D_SIGN;
    if (ma > D_INF || mc > D_INF || mb >= D_INF || (mb < 2 * ONE && mb != 0ull)) return minmod_nan(x, 0.5 * y, z);
    mb = mb != 0ull ? mb - ONE : 0ull;
    unsigned long long m = ma < mb ? ma : mb;
    m = m < mc ? m : mc;
    return (long long)((a ^ b) | (a ^ c)) < 0 ? 0.0 : from_bits(m | (a & D_SIGN));
}

// Sum K values (a power of two, K <= 32) over the warp by recursive halving.
template <int K> __device__ __forceinline__ double warp_sum_doubles(double (&v)[K], int lane)
{
#pragma unroll
    for (int half = K / 2, off = 16; half >= 1; half >>= 1, off >>= 1) {
        const bool upper = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const double send = upper ? v[i] : v[i + half];
            const double keep = upper ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
    double s = v[0];
    for (int off = 16 / K; off >= 1; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    return s;
}

// A warp's total of the K values into the K ledger words at `dst`, one lane each.
template <int K, int N>
__device__ __forceinline__ void warp_add(double (&v)[K], int lane, double* dst, const int (&slot)[N])
{
    const double s = warp_sum_doubles<K>(v, lane);
    if ((lane & (32 / K - 1)) != 0) return;
    int item = 0;
    for (int half = K / 2, off = 16; half >= 1; half >>= 1, off >>= 1)
        if (lane & off) item += half;
    if (item < N) dst[slot[item]] += s;
}

// One side of a face: the conserved state's momenta (and energy) and the
// physical flux along AXIS of the reconstructed primitives p.
template <int NF, int AXIS>
__device__ __forceinline__ void side64(const double* p, double pg, const Divisor& gm1, double* u, double* f)
{
    const double v = p[1 + AXIS];
    u[0] = p[0];
    u[1] = p[0] * p[1];
    u[2] = p[0] * p[2];
    f[0] = p[0] * v;
    f[1] = u[1] * v;
    f[2] = u[2] * v;
    f[1 + AXIS] = f[1 + AXIS] + pg;
    if constexpr (NF == 4) {
        u[3] = __fma_rn(0.5, p[0] * (p[1] * p[1] + p[2] * p[2]), gm1(p[3]));
        f[3] = (u[3] + pg) * v;
    }
}

// ---------------------------------------------------------------------------
template <int NF>
__global__ void __launch_bounds__(S64_THREADS, 2) stage64_kernel(const __grid_constant__ StageArgs a)
{
    constexpr int NL = NITEMS * NF;
    constexpr int NREC = 2 * NF + 4;   // slopes along x and y, then T or the shear: xx, yy, xy, bulk
    constexpr int GX = 0, GY = NF, TXX = 2 * NF, TYY = 2 * NF + 1, TXY = 2 * NF + 2, BULK = 2 * NF + 3;
    constexpr int K0 = NF == 3 ? 8 : 16;   // ledger items that are live everywhere: gravity, buffer, cooling
    constexpr int NT = S64_THREADS, NW = NT / 32;

    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int g = blockIdx.x;
    const int ri = a.nruns == 1 ? 0 : find_run(a, g);
    const RunDev& rd = a.runs[ri];

    __shared__ DevParams P;
    __shared__ double orb[10];
    __shared__ int skip;
    __shared__ double led[NW][NL];
    __shared__ double wmax[NW];
    for (int i = t; i < NW * NL; i += NT) led[i / NL][i % NL] = 0.0;
    if (t == 0) P = rd.p;
    if (t == 0) skip = left_out(a.failure, a.stage);   // (the caller keeps its state)
    __syncthreads();
    if (skip) return;
    if (t < 10) orb[t] = rd.orbit[a.stage * 10 + t];
    extern __shared__ __align__(128) unsigned char smem_raw[];   // one declaration for every stage kernel
    poison_dynamic_smem(smem_raw);
    __syncthreads();

    const int N = rd.N, bs = rd.bs;
    const size_t nn = (size_t)N * N;
    // this CTA's block and its sub-tiles [s0, s1) of it
    const int lt = g - rd.tile_base;
    const int block = lt / rd.tiles_per_block + (rd.slab_hi > 0 ? rd.slab_lo * rd.nb : 0);
    const int piece = lt % rd.tiles_per_block;
    const int bi = block / rd.nb, bj = block % rd.nb;
    const int s0 = piece * rd.sub_per_cta, s1 = min(s0 + rd.sub_per_cta, rd.sub_i * rd.sub_j);

    const double* uin = (const double*)rd.slot[a.in_slot];
    const double* ubase = a.base_slot >= 0 ? (const double*)rd.slot[a.base_slot] : nullptr;
    double* uout = (double*)rd.slot[a.out_slot];
    const double* ubg = (const double*)rd.bg;
    const double dt = *rd.dt, time = rd.stage_time[a.stage];
    const double keep = -a.bf + 1.0;
    const bool half_avg = a.bf == 0.5;

    const Divisor by_dx(P.dx, P.inv_dx), by_mach2(P.mach2, P.inv_mach2), by_gm1(P.gm1, P.inv_gm1);
    const bool dx2 = power_of_two(P.dx);   // x / dx is then x times 1 / dx, which commutes with rounding
    const double inv_dx = P.inv_dx;
    const bool const_nu = P.visc == 0, with_bulk = P.lambda != 0.0;
    const double lam_nu = P.lambda * P.nu;
    // this thread's first item of a loop that follows one of n items: the warps take turns on from its last
    auto after = [&](int n) { return (t - (n + 31) / 32 * 32 % NT + NT) % NT; };
    const bool trigger = P.pdt > 0.0;      // densities below 0 fail the advance before their slopes count

    double acc[K0];                        // this thread's zones' sums of the items that are live everywhere
#pragma unroll
    for (int k = 0; k < K0; ++k) acc[k] = 0.0;
    double amax = 0.0;

    for (int s = s0; s < s1; ++s) {
        const int si = s / rd.sub_j, sj = s % rd.sub_j;
        const int li0 = bs * si / rd.sub_i, TH = bs * (si + 1) / rd.sub_i - li0;
        const int lj0 = bs * sj / rd.sub_j, TW = bs * (sj + 1) / rd.sub_j - lj0;
        const int i0 = bi * bs + li0, j0 = bj * bs + lj0;
        const int PW = TW + 4, PS = (TH + 4) * PW;         // primitives: rows -2 .. TH+1, columns -2 .. TW+1
        const int CW = TW + 2, CS = (TH + 2) * CW;         // records: rows and columns -1 .. TH, TW
        double* sP = (double*)smem_raw;                    // [NF][PS]
        double* sC = sP + NF * PS;                         // [NREC][CS]
        double* sD = sC + NREC * CS;                       // theta differences, later the fluxes
        const int DXS = (TH + 3) * CW, DW = TW + 3, DYS = (TH + 2) * DW;
        double* sDX = sD;                                  // [NF][TH+3][CW]: x faces -3/2 .. , columns -1 .. TW
        double* sDY = sD + NF * DXS;                       // [NF][TH+2][DW]
        double* geo = sD + NF * (DXS + DYS);
        // rows: centre tables [TH] and face tables [TH+1]; then the same of the columns
        double* gr = geo;
        double* gc = geo + 7 * TH + 5 * (TH + 1);

        // Phase 1: primitives of the sub-tile and its 2-zone halo; the geometry tables.
        for (int e = t; e < PS; e += NT) {
            const int r = e / PW - 2, c = e % PW - 2;
            const int gi = wrap(wrap(i0 + r, N), N), gj = wrap(wrap(j0 + c, N), N);   // (twice: a mesh may be one zone wide)
            const size_t idx = (size_t)gi * N + gj;
            double u[NF], p[NF];
#pragma unroll
            for (int f = 0; f < NF; ++f) u[f] = __ldg(uin + f * nn + idx);
            int err = 0;
            if constexpr (NF == 3) {
                if (P.has_density_floor && u[0] < P.density_floor) {
                    u[0] = P.density_floor;
                    u[1] = u[2] = 0.0;
                }
                const Divisor by_rho(u[0]);
                p[0] = u[0];
                p[1] = by_rho(u[1]);
                p[2] = by_rho(u[2]);
                if (negative(u[0])) err = 1;
            } else {
                const Divisor by_rho(u[0]);
                p[0] = u[0];
                p[1] = by_rho(u[1]);
                p[2] = by_rho(u[2]);
                p[3] = __fma_rn(-0.5, u[0] * (p[1] * p[1] + p[2] * p[2]), u[3]) * P.gm1;
                if (P.has_density_floor && p[0] < P.density_floor) {
                    p[0] = P.density_floor;
                    p[1] = p[2] = 0.0;
                    p[3] = P.density_floor_pow_gamma;
                }
                if (negative(p[0])) err = 1;
                else {
                    if (P.has_pressure_floor && p[3] < P.pressure_floor) p[3] = P.pressure_floor;
                    if (p[3] <= 0.0) err = 2;
                }
            }
            if (err && r >= 0 && r < TH && c >= 0 && c < TW)
                atomicMin(&a.failure->key, error_key(a.stage, ri, rd, gi, gj, err));
#pragma unroll
            for (int f = 0; f < NF; ++f) sP[f * PS + e] = p[f];
        }
        for (int e = t; e < TH + TW + TH + 1 + TW + 1; e += NT) {
            // which table: row centres, column centres, row faces, column faces
            const bool face = e >= TH + TW;
            const int k = face ? e - TH - TW : e;
            const int split = face ? TH + 1 : TH;
            const bool col = k >= split;
            const int i = col ? k - split : k, n = col ? TW : TH, first = col ? j0 : i0;
            double* tab = col ? gc : gr;
            const double w = face ? rd.xv[(col ? bj : bi) * (bs + 1) + (col ? lj0 : li0) + i] : rd.xc[first + i];
            const double d1 = w - orb[col ? 2 : 1], d2 = w - orb[col ? 7 : 6];
            if (face) {
                double* q = tab + 7 * n + 5 * i;
                q[0] = d1 * d1;
                q[1] = d2 * d2;
                q[2] = w;
                q[3] = d1;
                q[4] = d2;
            } else {
                double* q = tab + 7 * i;
                q[0] = d1 * d1;
                q[1] = d2 * d2;
                q[2] = w;
                q[3] = d1;
                q[4] = d2;
                q[5] = -orb[0] * d1;
                q[6] = -orb[5] * d2;
            }
        }
        __syncthreads();

        // Phase 2: theta times the differences across x and y faces (where no
        // density trigger makes theta a zone's own).
        const double theta = P.plm;
        for (int e = t; e < DXS; e += NT) {
            const int r = e / CW, c = e % CW;               // face between record rows r - 2 and r - 1
            const int o = r * PW + c + 1;
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const double d = sP[f * PS + o + PW] - sP[f * PS + o];
                sDX[f * DXS + e] = trigger ? d : theta * d;
            }
        }
        for (int e = after(DXS); e < DYS; e += NT) {
            const int r = e / DW, c = e % DW;
            const int o = (r + 1) * PW + c;
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const double d = sP[f * PS + o + 1] - sP[f * PS + o];
                sDY[f * DYS + e] = trigger ? d : theta * d;
            }
        }
        __syncthreads();

        // Phase 3: slopes and stresses (scheme.rs:216-254; stress_field, physics.rs:322-340).
        for (int e = t; e < CS; e += NT) {
            const int r = e / CW, c = e % CW;
            const int o = (r + 1) * PW + c + 1;
            double thx = 1.0, thy = 1.0;
            if (trigger) {
                const double m = sP[o], pdt = P.pdt;
                thx = (sP[o - PW] < pdt || m < pdt || sP[o + PW] < pdt) ? 0.0 : theta;
                thy = (sP[o - 1] < pdt || m < pdt || sP[o + 1] < pdt) ? 0.0 : theta;
            }
            double gx[NF], gy[NF];
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const double* q = sP + f * PS + o;
                double xl = sDX[f * DXS + r * CW + c], xr = sDX[f * DXS + (r + 1) * CW + c];
                double yl = sDY[f * DYS + r * DW + c], yr = sDY[f * DYS + r * DW + c + 1];
                if (trigger) {
                    xl = thx * xl; xr = thx * xr;
                    yl = thy * yl; yr = thy * yr;
                }
                gx[f] = minmod_bits(xl, q[PW] - q[-PW], xr);
                gy[f] = minmod_bits(yl, q[1] - q[-1], yr);
                sC[(GX + f) * CS + e] = gx[f];
                sC[(GY + f) * CS + e] = gy[f];
            }
            double sxx, syy, sxy, bulk = 0.0;
            const double a43 = 4.0 / 3.0 * gx[1], a23 = -2.0 / 3.0 * gx[1];
            const double b43 = 4.0 / 3.0 * gy[2], b23 = 2.0 / 3.0 * gy[2];
            if (dx2) {
                sxx = (a43 - b23) * inv_dx;
                sxy = (gx[2] + gy[1]) * inv_dx;
                syy = (a23 + b43) * inv_dx;
                if (with_bulk) bulk = (gx[1] + gy[2]) * inv_dx;
            } else {
                sxx = by_dx(a43) - by_dx(b23);
                sxy = by_dx(gx[2]) + by_dx(gy[1]);
                syy = by_dx(a23) + by_dx(b43);
                if (with_bulk) bulk = by_dx(gx[1]) + by_dx(gy[2]);
            }
            if (const_nu) {
                const double rho = sP[o];
                sxx = P.nu * sxx;
                syy = P.nu * syy;
                if (with_bulk) {
                    sxx = sxx + lam_nu * bulk;
                    syy = syy + lam_nu * bulk;
                }
                sxx = rho * sxx;
                syy = rho * syy;
                sxy = rho * (P.nu * sxy);
            }
            sC[TXX * CS + e] = sxx;
            sC[TYY * CS + e] = syy;
            sC[TXY * CS + e] = sxy;
            sC[BULK * CS + e] = bulk;
        }
        __syncthreads();

        // Phase 4: fluxes through the x faces (TH + 1 rows of TW), then the y faces.
        double* sFX = sD;                                   // [NF][(TH+1) TW]
        const int FXS = (TH + 1) * TW, FW = TW + 1, FYS = TH * FW;
        double* sFY = sD + NF * FXS;                        // [NF][TH (TW+1)]
        auto face = [&](auto axis_c, int rec_l, int rec_r, int prim_l, int prim_r, double r1, double r2, double q1,
                        double q2, double* out, int stride) {
            constexpr int AX = decltype(axis_c)::value;
            constexpr int G = AX == 0 ? GX : GY;
            // r1 + q1 is the squared distance of the face to body 1
            const double s1 = r1 + q1, s2 = r2 + q2;
            double cl[NF], cr[NF], pl[NF], pr[NF];
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                cl[f] = sP[f * PS + prim_l];
                cr[f] = sP[f * PS + prim_r];
                pl[f] = __fma_rn(sC[(G + f) * CS + rec_l], 0.5, cl[f]);
                pr[f] = __fma_rn(sC[(G + f) * CS + rec_r], -0.5, cr[f]);
            }
            // sound speeds and gas pressures of the two sides
            double cs2 = 0.0, csl, csr, pgl, pgr;
            if constexpr (NF == 3) {
                const double f1 = orb[0] / sqrt(s1 + P.soft2), f2 = orb[5] / sqrt(s2 + P.soft2);
                cs2 = by_mach2(f1 + f2);
                csl = csr = sqrt(cs2);
                pgl = pl[0] * cs2;
                pgr = pr[0] * cs2;
            } else {
                csl = sqrt(P.gamma * pl[3] / pl[0]);
                csr = sqrt(P.gamma * pr[3] / pr[0]);
                pgl = pl[3];
                pgr = pr[3];
            }
            // viscous stresses along the normal and across it
            double ln, lt, rn, rt;
            constexpr int TN = AX == 0 ? TXX : TYY;
            if (const_nu) {
                ln = sC[TN * CS + rec_l];
                rn = sC[TN * CS + rec_r];
                lt = sC[TXY * CS + rec_l];
                rt = sC[TXY * CS + rec_r];
            } else {
                // the `nu` closure of compute_block_fluxes (scheme.rs:230-247)
                const double a1 = sqrt(s1) + P.eps_dx, a2 = sqrt(s2) + P.eps_dx;
                const double twofreq = sqrt(orb[0] / (a1 * a1 * a1) + orb[5] / (a2 * a2 * a2));
                const Divisor by_freq(twofreq), by_sg(P.sqrt_gm, P.inv_sqrt_gm);
                double nl, nr;
                if constexpr (NF == 3) nl = nr = by_sg(by_freq(P.nu * cs2));
                else {
                    nl = by_sg(by_freq(P.nu * (P.gamma * cl[3] / cl[0])));
                    nr = by_sg(by_freq(P.nu * (P.gamma * cr[3] / cr[0])));
                }
                double xl = nl * sC[TN * CS + rec_l], xr = nr * sC[TN * CS + rec_r];
                if (with_bulk) {
                    xl = xl + P.lambda * nl * sC[BULK * CS + rec_l];
                    xr = xr + P.lambda * nr * sC[BULK * CS + rec_r];
                }
                ln = cl[0] * xl;
                rn = cr[0] * xr;
                lt = cl[0] * (nl * sC[TXY * CS + rec_l]);
                rt = cr[0] * (nr * sC[TXY * CS + rec_r]);
            }
            const double tn2 = ln + rn, tt2 = lt + rt;      // twice the face's stresses
            const double vl = pl[1 + AX], vr = pr[1 + AX];
            const double ap = max_0(vl + csl, vr + csr), am = min_0(vl - csl, vr - csr);
            double F[NF];
            // All faces of the warp supersonic: (fl ap - fr am - (ul - ur) ap am) / (ap - am) is
            // then (fl ap) / ap with am = 0, (fr am) / am with ap = 0, and the other side drops out
            // (unless its terms are infinite or NaN: those times 0 are NaN).
            const bool from_l = zero(am);
            bool one_side = from_l || zero(ap);
#pragma unroll
            for (int f = 0; f < NF; ++f) one_side = one_side && bounded(pl[f]) && bounded(pr[f]);
            if (__all_sync(__activemask(), one_side)) {
                double pu[NF], u[NF], f[NF];
#pragma unroll
                for (int k = 0; k < NF; ++k) pu[k] = from_l ? pl[k] : pr[k];
                side64<NF, AX>(pu, from_l ? pgl : pgr, by_gm1, u, f);
                const ThereAndBack through(from_l ? ap : am);
#pragma unroll
                for (int k = 0; k < NF; ++k) F[k] = through(f[k]);
            } else {
                double ul[NF], ur[NF], fl[NF], fr[NF];
                side64<NF, AX>(pl, pgl, by_gm1, ul, fl);
                side64<NF, AX>(pr, pgr, by_gm1, ur, fr);
                const Divisor by_w(ap - am);
#pragma unroll
                for (int k = 0; k < NF; ++k) F[k] = by_w(fl[k] * ap - fr[k] * am - (ul[k] - ur[k]) * ap * am);
            }
            F[1] = __fma_rn(-0.5, AX == 0 ? tn2 : tt2, F[1]);
            F[2] = __fma_rn(-0.5, AX == 0 ? tt2 : tn2, F[2]);
            if constexpr (NF == 4) {
                const double tx = 0.5 * (AX == 0 ? tn2 : tt2), ty = 0.5 * (AX == 0 ? tt2 : tn2);
                const double vx = 0.5 * (cl[1] + cr[1]), vy = 0.5 * (cl[2] + cr[2]);
                F[3] = F[3] + -(tx * vx + ty * vy);
            }
#pragma unroll
            for (int f = 0; f < NF; ++f) out[f * stride] = F[f];
        };
        for (int e = t; e < FXS; e += NT) {
            const int r = e / TW, c = e % TW;               // face between rows r - 1 and r
            const double* q = gr + 7 * TH + 5 * r;
            const double* w = gc + 7 * c;
            const int rl = r * CW + c + 1, pl = (r + 1) * PW + c + 2;
            face(std::integral_constant<int, 0>(), rl, rl + CW, pl, pl + PW, q[0], q[1], w[0], w[1], sFX + e, FXS);
        }
        for (int e = after(FXS); e < FYS; e += NT) {
            const int r = e / FW, c = e % FW;               // face between columns c - 1 and c
            const double* q = gr + 7 * r;
            const double* w = gc + 7 * TW + 5 * c;
            const int rl = (r + 1) * CW + c, pl = (r + 2) * PW + c + 1;
            face(std::integral_constant<int, 1>(), rl, rl + 1, pl, pl + 1, q[0], q[1], w[0], w[1], sFY + e, FYS);
        }
        __syncthreads();

        // Phase 5: update (compute_block_updated_solution, scheme.rs:290-305) and the
        // RK weighted average (state.rs:183-199).  Whole warps, so that they can vote.
        const int nz = TH * TW;
        for (int e0 = warp * 32; e0 < nz; e0 += NT) {
            const bool on = e0 + lane < nz;
            const int e = min(e0 + lane, nz - 1);
            const int r = e / TW, c = e % TW;
            const size_t idx = (size_t)(i0 + r) * N + j0 + c;
            double u[NF], u0[NF];
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                u[f] = __ldg(uin + f * nn + idx);
                u0[f] = __ldg(ubg + f * nn + idx);
            }
            const double* q = gr + 7 * r;
            const double* w = gc + 7 * c;
            const double s1 = q[0] + w[0], s2 = q[1] + w[1];
            const double br = rd.buffer ? __ldg(rd.buffer + idx) : buffer_rate(P, q[2], w[2]);
            const double* fx = sFX + r * TW + c;
            const double* fy = sFY + r * FW + c;

            // gravity (Plummer accelerations, kepler-two-body)
            const double t1 = s1 + P.soft2, t2 = s2 + P.soft2;
            const Divisor c1(t1 * sqrt(t1)), c2(t2 * sqrt(t2));
            const double f1x = u[0] * c1(q[5]), f1y = u[0] * c1(w[5]);
            const double f2x = u[0] * c2(q[6]), f2y = u[0] * c2(w[6]);
            double tot[NF], it[K0];
            it[0] = f1x * dt;
            it[1] = f1y * dt;
            it[NF - 1] = f2x * dt;
            it[NF] = f2y * dt;
            double vx = 0.0, vy = 0.0, e_in = 0.0, v2 = 0.0;
            if constexpr (NF == 4) {
                const Divisor by_rho(u[0]);
                vx = by_rho(u[1]);
                vy = by_rho(u[2]);
                v2 = vx * vx + vy * vy;
                const double p3 = __fma_rn(-0.5, u[0] * v2, u[3]) * P.gm1;
                e_in = by_gm1(by_rho(p3));
                it[2] = (f1x * vx + f1y * vy) * dt;
                it[5] = (f2x * vx + f2y * vy) * dt;
            }
            constexpr int IB = 2 * (NF - 1);               // the buffer's items in acc
            const double kb = -dt * br;
            // items with a rate of 0 are left out where none of the warp's zones has another rate: not
            // where a zone's values could make NaN of that 0
            bool odd = false;
#pragma unroll
            for (int f = 0; f < NF; ++f) odd = odd || !bounded(u[f]) || !bounded(u0[f]);
            odd = __any_sync(0xffffffffu, odd);
            const bool buffer_on = odd || __any_sync(0xffffffffu, !zero(br));
#pragma unroll
            for (int f = 0; f < NF; ++f) it[IB + f] = buffer_on ? (u[f] - u0[f]) * kb : 0.0;
            // cooling (Euler::source_terms, physics.rs:701-738; beta-cooling is new)
            if constexpr (NF == 4) {
                double ec;
                if (P.cooling_kind == 1) {
                    const double om = sqrt(c1(orb[0]) + c2(orb[5]));
                    ec = e_in * exp(-om * dt / P.cool_beta);
                } else {
                    double f = 1.0;
                    if (P.cooling_slow_start) f = exp(-(2.0 * 3.14159265358979323846) / (time + dt));
                    double rho_n = 1.0;
                    for (int k = 0; k < P.density_index; ++k) rho_n *= u[0];
                    const double ca = P.cool_coef / rho_n * f;
                    ec = e_in * pow(1.0 + 3.0 * ca * (e_in * e_in * e_in) * dt, -1.0 / 3.0);
                }
                if (P.has_mach_ceiling) {
                    const double ek = 0.5 * v2;
                    ec = fmax(ec, 2.0 * ek / P.gamma / P.gm1 / P.mach_ceiling2);
                }
                const double pc3 = u[0] * ec * P.gm1;
                it[IB + 4] = u[0] * vx - u[1];
                it[IB + 5] = u[0] * vy - u[2];
                it[IB + 6] = __fma_rn(0.5, u[0] * v2, by_gm1(pc3)) - u[3];
                it[IB + 7] = 0.0;
                it[IB + 8] = 0.0;
                it[IB + 9] = 0.0;
            } else {
                it[IB + 3] = 0.0;
            }
            // the items' sum in the reference's order (sinks, gravity, buffer, cooling, fake mass), without
            // those that are zero
            const bool near = dbits(s1) < dbits(P.sink_r2) || dbits(s2) < dbits(P.sink_r2);
            tot[0] = it[IB];
            if (odd || __any_sync(0xffffffffu, near)) {
                // sink_kernel and the sink terms (physics.rs:388-397, 423-457)
                auto rate = [&](double r2) {
                    if (!(r2 < P.sink_r2)) return 0.0;
                    const double k = 1.0 - r2 / P.sink_r2;
                    return P.sink_rate * (k * k);
                };
                const double sr1 = rate(s1), sr2 = rate(s2);
                double a1[NF], a2[NF];
                if (P.sink_model == 0) {
#pragma unroll
                    for (int f = 0; f < NF; ++f) a1[f] = a2[f] = u[f];
                } else {
                    if constexpr (NF == 3) {
                        vx = u[1] / u[0];
                        vy = u[2] / u[0];
                    }
                    const PointMass<double> b1{orb[0], orb[1], orb[2], orb[3], orb[4]};
                    const PointMass<double> b2{orb[5], orb[6], orb[7], orb[8], orb[9]};
                    double x1, y1, x2, y2;
                    torque_free_velocity(P, b1, q[2], w[2], vx, vy, x1, y1);
                    torque_free_velocity(P, b2, q[2], w[2], vx, vy, x2, y2);
                    a1[0] = a2[0] = u[0];
                    a1[1] = u[0] * x1; a1[2] = u[0] * y1;
                    a2[1] = u[0] * x2; a2[2] = u[0] * y2;
                    if constexpr (NF == 4) {
                        a1[3] = u[0] * e_in + 0.5 * u[0] * (x1 * x1 + y1 * y1);
                        a2[3] = u[0] * e_in + 0.5 * u[0] * (x2 * x2 + y2 * y2);
                    }
                }
                double sk[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) sk[k] = 0.0;
#pragma unroll
                for (int f = 0; f < NF; ++f) {
                    sk[f] = a1[f] * -sr1 * dt;
                    sk[NF + f] = a2[f] * -sr2 * dt;
                    tot[f] = sk[f] + sk[NF + f];
                }
                tot[0] = tot[0] + it[IB];
#pragma unroll
                for (int f = 1; f < NF; ++f) tot[f] = tot[f] + it[f - 1] + it[NF - 2 + f] + it[IB + f];
                if (!on)
#pragma unroll
                    for (int k = 0; k < 8; ++k) sk[k] = 0.0;
                int slot[2 * NF];
#pragma unroll
                for (int k = 0; k < 2 * NF; ++k) slot[k] = (k < NF ? SINK1 : SINK2 - 1) * NF + k;
                warp_add<8>(sk, lane, led[warp], slot);
            } else {
#pragma unroll
                for (int f = 1; f < NF; ++f) tot[f] = it[f - 1] + it[NF - 2 + f] + it[IB + f];
            }
            if constexpr (NF == 4) {
#pragma unroll
                for (int f = 1; f < 4; ++f) tot[f] = tot[f] + it[IB + 3 + f];
            } else if (odd || P.fake_rate != 0.0) {
                double fk[4] = {0.0, 0.0, 0.0, 0.0};
                if (!(u[0] < u0[0] * P.fake_thr)) {
#pragma unroll
                    for (int f = 0; f < 3; ++f) {
                        fk[f] = u0[f] * P.fake_rate * dt;
                        tot[f] = tot[f] + fk[f];
                    }
                }
                if (!on) fk[0] = fk[1] = fk[2] = 0.0;
                const int slot[3] = {FAKE_MASS * 3, FAKE_MASS * 3 + 1, FAKE_MASS * 3 + 2};
                warp_add<4>(fk, lane, led[warp], slot);
            }
            double out[NF];
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const double ddx = fx[f * FXS + TW] - fx[f * FXS], ddy = fy[f * FYS + 1] - fy[f * FYS];
                const double du = (dx2 ? (ddx + ddy) * inv_dx : by_dx(ddx) + by_dx(ddy)) * -dt;
                out[f] = u[f] + du + tot[f];
                if (ubase) {
                    const double b = __ldg(ubase + f * nn + idx);
                    out[f] = half_avg ? __fma_rn(out[f], 0.5, b * 0.5) : out[f] * keep + b * a.bf;
                }
            }
            if (on) {
#pragma unroll
                for (int f = 0; f < NF; ++f) uout[f * nn + idx] = out[f];
#pragma unroll
                for (int k = 0; k < IB + (NF == 4 ? 7 : 3); ++k) acc[k] += it[k];
                if constexpr (NF == 4)
                    if (odd) acc[IB + 7] += u[0] - u[0];   // the mass of cooling
                if (a.amax_flag) {
                    // max(|vx|, |vy|) + c (physics.rs:521-526, 679-681); NaN speeds are passed over, as f64::max does
                    const Divisor by_rho(out[0]);
                    const double wx = by_rho(out[1]), wy = by_rho(out[2]);
                    const unsigned long long ax = positive_part(dbits(wx) & ~D_SIGN), ay = positive_part(dbits(wy) & ~D_SIGN);
                    double v = from_bits(ax > ay ? ax : ay);
                    if constexpr (NF == 4) {
                        const double p3 = __fma_rn(-0.5, out[0] * (wx * wx + wy * wy), out[3]) * P.gm1;
                        v = v + sqrt(by_rho(P.gamma * p3));
                    }
                    amax = max_0(v, amax);
                }
            }
        }
        if (s + 1 < s1) __syncthreads();
    }

    // --- ledger and max speed of the CTA's zones ---------------------------------
    {
        int slot[NF == 3 ? 7 : 14];
        int n = 0;
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int f = 1; f < NF; ++f) slot[n++] = (GRAV1 + k) * NF + f;
#pragma unroll
        for (int f = 0; f < NF; ++f) slot[n++] = BUFFER * NF + f;
        if constexpr (NF == 4) {
#pragma unroll
            for (int f = 1; f < 4; ++f) slot[n++] = COOLING * NF + f;
            slot[n++] = COOLING * NF;
        }
        warp_add<K0>(acc, lane, led[warp], slot);
    }
    if (a.amax_flag) {
        for (int off = 16; off >= 1; off >>= 1) amax = max_0(amax, __shfl_xor_sync(0xffffffffu, amax, off));
        if (lane == 0) wmax[warp] = amax;
    }
    __syncthreads();
    if (t < NL) {
        double v = 0.0;
        for (int w = 0; w < NW; ++w) v += led[w][t];
        // folded, in piece order, after the stages (b2d_advance's ledger kernels)
        stage_pieces(rd, a.stage, block, NL)[(size_t)piece * NL + t] = v;
    }
    if (a.amax_flag && t == 0) {
        double m = 0.0;
        for (int w = 0; w < NW; ++w) m = fmax(m, wmax[w]);
        if (m > 0.0) atomicMax(rd.amax, (unsigned long long)__double_as_longlong(m));
    }
}

}  // namespace b2d
