// physics.cuh — physics parameters in device form, and the per-zone formulas
// that several kernels share.
//
// R = double: the parity path.  Every expression is evaluated in the order
// of the reference's Rust source (this translation unit is compiled with
// --fmad=false), so the FP64 kernel reproduces the CPU restatement bit for
// bit apart from the last-ulp differences of tanh / sin / cos / pow / exp.
// R = float: the mixed-precision path.  Same formulas, reassociated for
// throughput (reciprocals, rsqrt, fused multiply-add), intrinsics for
// division and square roots.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

namespace b2d {

enum { SINK1 = 0, SINK2, GRAV1, GRAV2, BUFFER, COOLING, FAKE_MASS, NITEMS };

// Physics parameters in device form, built on the host from b2d_config.
// DevParamsT<double> serves the FP64 kernels, DevParamsT<float> the FP32
// kernels (no double arithmetic or conversion in their inner loops).
template <class T> struct DevParamsT {
    int hydro;            // 0 iso, 1 euler
    int visc;             // 0 constant nu, 1 alpha
    int sink_model;       // 0 impartial, 1 torque-free
    int one_body;
    int has_mach_ceiling, has_density_floor, has_pressure_floor, density_index;
    int cooling_kind, cooling_slow_start, has_dt_min, pad_;
    T dx, inv_dx;
    T cfl, dt_min;
    T plm, pdt;                       // θ and the PLM density trigger (0 if unset)
    T nu;                             // ν or α
    T lambda;                         // lambda_multiplier
    T mach2, inv_mach2;               // mach_number² (iso)
    T gamma, gm1, inv_gm1;            // γ, γ - 1 (euler; iso γ = 1)
    T sqrt_gm, inv_sqrt_gm;           // sqrt(γ) for α viscosity
    T soft2;                          // softening_length²
    T sink_r2, inv_sink_r2, sink_rate;
    T domain_radius, buffer_scale, inv_buffer_scale, half_buffer_rate, omega_outer, half_rate_omega;
    T fake_thr, fake_rate;
    T density_floor, pressure_floor, density_floor_pow_gamma;
    T mach_ceiling2;                  // mach_ceiling²
    T k_mach_ceiling;                 // 2 / (γ (γ - 1) mach_ceiling²)
    T cool_coef, cool_beta, inv_cool_beta;
    T eps_dx;                         // 1e-12 · dx (α viscosity)
};
using DevParams = DevParamsT<double>;
using DevParamsF = DevParamsT<float>;

template <class R> struct PointMass { R m, x, y, vx, vy; };
template <class R> struct Binary { PointMass<R> p1, p2; };

// ---------------------------------------------------------------------------
// Hydrodynamics::max_signal_speed (physics.rs:521-526, 679-681).
template <int NF> __device__ __forceinline__ double max_speed_f64(const DevParams& P, const double* u)
{
    const double vx = u[1] / u[0], vy = u[2] / u[0];
    const double v = fmax(fabs(vx), fabs(vy));
    if constexpr (NF == 4) {
        const double p = (u[3] - 0.5 * u[0] * (vx * vx + vy * vy)) * P.gm1;
        return v + sqrt(P.gamma * p / u[0]);
    }
    return v;
}

// The same in FP32, from a zone's words as double-floats hi + lo, every
// rounding written out: the kernels that call it are compiled with different
// flags and have to agree.  At Mach 30 the internal energy is 1/400 of the
// total: as a difference of FP32 words it is off by 2.5e-5, so it is formed
// from both words and the kinetic energy's remainders.
template <int NF> __device__ __forceinline__ float max_speed_f32(const DevParamsF& P, const float* hi, const float* lo)
{
    const float v = fmaxf(fabsf(__fdiv_rn(hi[1], hi[0])), fabsf(__fdiv_rn(hi[2], hi[0])));
    if constexpr (NF == 4) {
        // m^2 = a + b, a rounded
        const float a1 = __fmul_rn(hi[1], hi[1]), a2 = __fmul_rn(hi[2], hi[2]);
        const float b1 = __fmaf_rn(__fmul_rn(2.0f, hi[1]), lo[1], __fmaf_rn(hi[1], hi[1], -a1));
        const float b2 = __fmaf_rn(__fmul_rn(2.0f, hi[2]), lo[2], __fmaf_rn(hi[2], hi[2], -a2));
        const float big = fmaxf(a1, a2), small = fminf(a1, a2);
        const float a = __fadd_rn(big, small);
        const float b = __fadd_rn(__fadd_rn(small, -__fadd_rn(a, -big)), __fadd_rn(b1, b2));
        // k + r = (a + b) / (2 rho)
        const float ir = __frcp_rn(hi[0]), ha = __fmul_rn(0.5f, a);
        const float k = __fmul_rn(ha, ir);
        const float r = __fmul_rn(__fmaf_rn(-k, lo[0], __fmaf_rn(0.5f, b, __fmaf_rn(-k, hi[0], ha))), ir);
        const float e = __fadd_rn(__fadd_rn(hi[3], -k), __fadd_rn(lo[3], -r));
        return __fadd_rn(v, __fsqrt_rn(__fmul_rn(__fmul_rn(P.gamma, __fmul_rn(e, P.gm1)), ir)));
    }
    return v;
}

// ---------------------------------------------------------------------------
// Pieces of the source terms in the reference's FP64 operation order.
// The torque-free sink velocity (physics.rs:743-756).
__device__ __forceinline__ void torque_free_velocity(const DevParams& P, const PointMass<double>& b, double x, double y,
                                                     double vx, double vy, double& vxc, double& vyc)
{
    double vxb = P.one_body ? 0.0 : b.vx;
    double vyb = P.one_body ? 0.0 : b.vy;
    double r = sqrt((x - b.x) * (x - b.x) + (y - b.y) * (y - b.y));
    double rx = (x - b.x) / r, ry = (y - b.y) / r;
    double dvdotr = (vx - vxb) * rx + (vy - vyb) * ry;
    vxc = dvdotr * rx + vxb;
    vyc = dvdotr * ry + vyb;
}

// Buffer rate 0.5·rate·(1 + tanh((r - R)/scale))·Ω_outer (physics.rs:443-446).
__device__ __forceinline__ double buffer_rate(const DevParams& P, double x, double y)
{
    double r = sqrt(x * x + y * y);
    double yb = (r - P.domain_radius) / P.buffer_scale;
    return P.half_buffer_rate * (1.0 + tanh(yb)) * P.omega_outer;
}

}  // namespace b2d
