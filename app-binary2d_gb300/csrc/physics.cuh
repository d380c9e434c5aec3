// physics.cuh — physics parameters in device form, and the per-zone formulas
// that several kernels share, templated on the stencil arithmetic R.
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

template <class R> __device__ __forceinline__ R rmax(R a, R b) { return fmax(a, b); }
template <> __device__ __forceinline__ float rmax<float>(float a, float b) { return fmaxf(a, b); }
template <class R> __device__ __forceinline__ R rabs(R a) { return fabs(a); }
template <> __device__ __forceinline__ float rabs<float>(float a) { return fabsf(a); }
template <class R> __device__ __forceinline__ R rsqrt_(R a) { return sqrt(a); }
template <> __device__ __forceinline__ float rsqrt_<float>(float a) { return sqrtf(a); }

// ---------------------------------------------------------------------------
// Conserved -> primitive (hydro-iso2d / hydro-euler, restated).
template <int NF, class R> __device__ __forceinline__ void cons_to_prim_raw(const DevParamsT<R>& P, const R* u, R* p)
{
    p[0] = u[0];
    if constexpr (std::is_same<R, double>::value) {
        p[1] = u[1] / u[0];
        p[2] = u[2] / u[0];
        if constexpr (NF == 4) p[3] = (u[3] - 0.5 * u[0] * (p[1] * p[1] + p[2] * p[2])) * P.gm1;
    } else {
        float ir = __fdividef(1.0f, u[0]);
        p[1] = u[1] * ir;
        p[2] = u[2] * ir;
        if constexpr (NF == 4) p[3] = (u[3] - 0.5f * u[0] * (p[1] * p[1] + p[2] * p[2])) * P.gm1;
    }
}

// Hydrodynamics::max_signal_speed (physics.rs:521-526 iso; 679-681 euler).
template <int NF, class R> __device__ __forceinline__ R max_signal_speed(const DevParamsT<R>& P, const R* u)
{
    R p[NF];
    cons_to_prim_raw<NF, R>(P, u, p);
    R v = rmax(rabs(p[1]), rabs(p[2]));
    if constexpr (NF == 4) {
        R cs = rsqrt_(R(P.gamma) * p[3] / p[0]);
        return v + cs;
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
