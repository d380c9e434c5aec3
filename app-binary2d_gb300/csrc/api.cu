// api.cu — the C ABI of include/b2d.h: contexts, state transfer, and the
// advance driver (the role of scheme::advance, src/scheme.rs:323-349).
//
// Built with --fmad=false: the Kepler solve and the time bookkeeping of the
// prologue kernel round exactly like the FP64 CPU restatement.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "elements.cuh"
#include "runtime.cuh"
#include "split.cuh"

namespace b2d {
cudaError_t launch_stage_f64(int nf, const StageArgs& a, int grid, size_t smem, cudaStream_t s);
cudaError_t launch_buffer_rate(const RunDev* runs, int run, int N, double* out, cudaStream_t s);
size_t stage_f64_smem(int nf, int th, int tw);
cudaError_t launch_stage_f32_iso(int store, int divisor, const StageArgs& a, int grid, cudaStream_t s);
cudaError_t launch_stage_f32_euler(int store, int divisor, const StageArgs& a, int grid, cudaStream_t s);
int resident_f32_iso(int store, int divisor, int nruns);
int resident_f32_euler(int store, int divisor, int nruns);
void host_block_vertices(const b2d_config* c, int b, double* xv);
void host_cell_centers(const b2d_config* c, int b, double* xc);
}  // namespace b2d

using namespace b2d;

static thread_local std::string g_last_error;

static b2d_status fail(b2d_status s, const std::string& msg)
{
    g_last_error = msg;
    return s;
}

#define CUDA_TRY(expr)                                                                              \
    do {                                                                                            \
        cudaError_t e_ = (expr);                                                                    \
        if (e_ != cudaSuccess)                                                                      \
            return fail(B2D_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_));          \
    } while (0)

extern "C" const char* b2d_last_error(void) { return g_last_error.c_str(); }

// ---------------------------------------------------------------------------
// Device kernels of the runtime.

// Two-body orbit at time t: OrbitalElements::orbital_state_from_time
// (kepler-two-body, restated; called at physics.rs:419-421).  Elements
// (a, M, q, e) = (1, 1, q, e), or (1e-12, 1, 1, 0) for one_body
// (physics.rs:411-417).  Periapsis on +x at t = 0; Newton iteration on
// Kepler's equation E - e sin E = n t from E = n t.
__device__ void kepler_orbit(const RunDev& rd, double t, double* o)
{
    double a, M, q, e;
    if (rd.p.one_body) { a = 1e-12; M = 1.0; q = 1.0; e = 0.0; }
    else { a = 1.0; M = 1.0; q = rd.binary_q; e = rd.binary_e; }
    double n = sqrt(M / (a * a * a));
    double mean = n * t;
    double E = mean;
    for (int k = 0; k < 64; ++k) {
        double f = E - e * sin(E) - mean;
        if (fabs(f) < 1e-15) break;
        E = E - f / (1.0 - e * cos(E));
    }
    double cE = cos(E), sE = sin(E);
    double b = sqrt(1.0 - e * e);
    double x = a * (cE - e);
    double y = a * b * sE;
    double edot = n / (1.0 - e * cE);
    double vx = -a * sE * edot;
    double vy = a * b * cE * edot;
    double m1 = M / (1.0 + q);
    double m2 = M * q / (1.0 + q);
    double f1 = m2 / M, f2 = m1 / M;
    o[0] = m1; o[1] = -x * f1; o[2] = -y * f1; o[3] = -vx * f1; o[4] = -vy * f1;
    o[5] = m2; o[6] = x * f2; o[7] = y * f2; o[8] = vx * f2; o[9] = vy * f2;
}

// Start of an advance, one CTA per run: dt = cfl·dx / max signal speed
// (floored by dt_min, scheme.rs:336-340), the stage times of all `fold` RK
// steps (try_advance_rk stamps t + dt, scheme.rs:168-170; weighted_average
// averages time, state.rs:213-214), and the binary at each stage time.
__global__ void prologue_kernel(const RunDev* runs, int fold, int rk, int start, int final_slot,
                                Failure* failure, long long* adv_count)
{
    const RunDev& rd = runs[blockIdx.x];
    const int stages = rk;
    __shared__ int failed;
    // a failure is pending: this advance and every later one are abandoned.  Their kernels leave every
    // slot alone, since the one that the failing advance began from comes up again as an output slot.
    if (threadIdx.x == 0) {
        failed = (*(volatile unsigned long long*)&failure->key != ~0ull);
        if (blockIdx.x == 0) failure->abandoned = failed;
    }
    __syncthreads();
    if (failed) return;
    if (threadIdx.x == 0 && blockIdx.x == 0) *adv_count += 1;
    if (threadIdx.x == 0) {
        double amax = __longlong_as_double((long long)*rd.amax);
        double dt = rd.p.cfl * rd.p.dx / amax;
        if (rd.p.has_dt_min) dt = fmax(dt, rd.p.dt_min);
        *rd.dt = dt;
        *rd.amax = 0ull;
        double t = rd.time[start];
        int s = 0;
        for (int f = 0; f < fold; ++f) {
            const double t0 = t;
            if (rk == 1) {
                rd.stage_time[s++] = t0;
                t = t0 + dt;
            } else if (rk == 2) {
                rd.stage_time[s++] = t0;
                double t1 = t0 + dt;
                rd.stage_time[s++] = t1;
                double t2 = t1 + dt;
                t = t2 * (-0.5 + 1.) + t0 * 0.5;
            } else {
                rd.stage_time[s++] = t0;
                double t1 = t0 + dt;
                rd.stage_time[s++] = t1;
                double t2 = t1 + dt;
                double t2a = t2 * (-0.75 + 1.) + t0 * 0.75;
                rd.stage_time[s++] = t2a;
                double t3 = t2a + dt;
                const double bf = 1.0 / 3.0;
                t = t3 * (-bf + 1.) + t0 * bf;
            }
        }
        rd.time[final_slot] = t;
        rd.iter[final_slot] = rd.iter[start] + fold;
    }
    __syncthreads();
    for (int s = threadIdx.x; s < fold * stages; s += blockDim.x) kepler_orbit(rd, rd.stage_time[s], rd.orbit + 10 * s);
}

// State::max_signal_speed (state.rs:121-133) of one run's slot, in the
// precision the stage kernels use for it at the end of an advance: FP64 for
// the FP64 path, FP32 of the stored words for the FP32 paths (FP64
// divisions and roots on a whole mesh are slow on this GPU).
template <int NF, int STORE, class R>
__global__ void max_speed_kernel(const RunDev* runs, int run, int slot)
{
    const RunDev& rd = runs[run];
    const size_t nn = (size_t)rd.N * rd.N;
    // a row slab's zones only (its block rows are contiguous in the planes)
    const size_t z0 = rd.slab_hi > 0 ? (size_t)rd.slab_lo * rd.bs * rd.N : 0;
    const size_t z1 = rd.slab_hi > 0 ? (size_t)rd.slab_hi * rd.bs * rd.N : nn;
    R a = R(0);
    for (size_t z = z0 + blockIdx.x * (size_t)blockDim.x + threadIdx.x; z < z1; z += (size_t)gridDim.x * blockDim.x) {
        if constexpr (std::is_same<R, double>::value) {
            double u[NF];
            for (int f = 0; f < NF; ++f) u[f] = ((const double*)rd.slot[slot])[f * nn + z];
            a = fmax(max_speed_f64<NF>(rd.p, u), a);
        } else {
            float hi[NF], lo[NF];
            for (int f = 0; f < NF; ++f) {
                if (STORE == 0) {
                    const double v = ((const double*)rd.slot[slot])[f * nn + z];
                    hi[f] = (float)v;
                    lo[f] = (float)(v - (double)hi[f]);
                } else {
                    hi[f] = ((const float*)rd.slot[slot])[(2 * f) * nn + z];
                    lo[f] = ((const float*)rd.slot[slot])[(2 * f + 1) * nn + z];
                }
            }
            a = fmaxf(max_speed_f32<NF>(rd.pf, hi, lo), a);
        }
    }
    __shared__ double red[256];
    red[threadIdx.x] = a;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + s]);
        __syncthreads();
    }
    if (threadIdx.x == 0 && red[0] > 0.0) atomicMax(rd.amax, (unsigned long long)__double_as_longlong(red[0]));
}

// Block layout [nb][nb][bs][bs][nf] (host) <-> field planes (device).  A CTA
// takes LAYOUT_ZONES consecutive zones of the host layout: the host side
// (which may be a page-locked host buffer read or written in place over the
// CPU-GPU link) moves as one contiguous, coalesced sweep through shared
// memory, and each field plane is written (read) by one thread per zone, 32
// consecutive words per warp.
constexpr int LAYOUT_ZONES = 256;

// Plane index of host-layout zone q (block-major: block, row, column).  A
// run has at most 2^31 zones (validate), so 32-bit unsigned divisions do: a
// 64-bit division costs about 150 instructions.
__device__ __forceinline__ size_t plane_index(unsigned q, unsigned N, unsigned bs, unsigned nb)
{
    const unsigned r = q / bs, lj = q - r * bs;
    const unsigned b = r / bs, li = r - b * bs;
    const unsigned bi = b / nb, bj = b - bi * nb;
    return (size_t)(bi * bs + li) * N + bj * bs + lj;
}

__global__ void __launch_bounds__(LAYOUT_ZONES) scatter_kernel(const double* src, void* dst, int N, int bs, int nb,
                                                               int nf, int store)
{
    __shared__ double buf[LAYOUT_ZONES * 4];
    const size_t nn = (size_t)N * N;
    const int t = threadIdx.x;
    for (size_t q0 = (size_t)blockIdx.x * LAYOUT_ZONES; q0 < nn; q0 += (size_t)gridDim.x * LAYOUT_ZONES) {
        const int nz = (int)min((size_t)LAYOUT_ZONES, nn - q0);
        for (int e = t; e < nz * nf; e += LAYOUT_ZONES) buf[e] = src[q0 * nf + e];
        __syncthreads();
        if (t < nz) {
            const size_t z = plane_index((unsigned)(q0 + t), N, bs, nb);
            for (int f = 0; f < nf; ++f) {
                const double v = buf[t * nf + f];
                if (store == 0) {
                    ((double*)dst)[f * nn + z] = v;
                } else {
                    const float hi = (float)v;
                    const float lo = (float)(v - (double)hi);
                    ((float*)dst)[(2 * f) * nn + z] = hi;
                    ((float*)dst)[(2 * f + 1) * nn + z] = lo;
                }
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(LAYOUT_ZONES) gather_kernel(const void* src, double* dst, int N, int bs, int nb,
                                                              int nf, int store)
{
    __shared__ double buf[LAYOUT_ZONES * 4];
    const size_t nn = (size_t)N * N;
    const int t = threadIdx.x;
    for (size_t q0 = (size_t)blockIdx.x * LAYOUT_ZONES; q0 < nn; q0 += (size_t)gridDim.x * LAYOUT_ZONES) {
        const int nz = (int)min((size_t)LAYOUT_ZONES, nn - q0);
        if (t < nz) {
            const size_t z = plane_index((unsigned)(q0 + t), N, bs, nb);
            for (int f = 0; f < nf; ++f) {
                double v;
                if (store == 0) v = ((const double*)src)[f * nn + z];
                else v = (double)((const float*)src)[(2 * f) * nn + z] + (double)((const float*)src)[(2 * f + 1) * nn + z];
                buf[t * nf + f] = v;
            }
        }
        __syncthreads();
        for (int e = t; e < nz * nf; e += LAYOUT_ZONES) dst[q0 * nf + e] = buf[e];
        __syncthreads();
    }
}

// Launch shape of the layout kernels for one run: LAYOUT_ZONES threads, at
// most 4096 CTAs striding over the run's zones.
static unsigned layout_blocks(int N)
{
    const size_t nn = (size_t)N * N;
    return (unsigned)std::min<size_t>((nn + LAYOUT_ZONES - 1) / LAYOUT_ZONES, 4096);
}

// ---------------------------------------------------------------------------
// Host-side context.

namespace {

struct RunHost {
    b2d_config cfg;
    int N, bs, nb, nblocks;
    size_t state_bytes;
    void* slot[NSLOTS] = {};
    void* bg = nullptr;
    double* ledger[NSLOTS] = {};
    double* elements[NSLOTS] = {};
    double* partial = nullptr;
    size_t partial_bytes = 0;
    double *xc = nullptr, *xv = nullptr;
    float2 *xcf = nullptr, *xvf = nullptr;
    double* buffer = nullptr;   // FP64: the buffer's rate of every zone
    double* stage_time = nullptr;
    double* orbit = nullptr;
    double* stage_ds = nullptr;
    double* stage_de = nullptr;
    std::vector<double> hxc;
};

struct StagePlan {
    int in, base, out;
    double bf;
};

}  // namespace

struct b2d_ctx {
    int nruns = 0, nf = 3, precision = 0, hydro = 0, rk = 2;
    int tw = 64, th = 64;
    int sub_h = 16, sub_w = 32;   // FP64 kernel: the largest sub-tile (f64_sub_tile)
    int strip_rows = 0;   // > 0: the FP32 kernel's strips are cut into row chunks of at most this many rows
    // a slab advance in progress (b2d_slab_begin .. b2d_slab_end)
    std::vector<StagePlan> slab_plan;
    int slab_fold = 0, slab_start = -1, slab_final = -1, slab_next = -1;
    int cur = 0;
    std::vector<RunHost> runs;
    std::vector<RunDev> rdev_h;
    RunDev* rdev = nullptr;
    int* d_bases = nullptr;           // [nruns] first CTA of each run
    int stage_window = 1;             // stages whose ledger pieces fit their buffers
    // control arrays (device)
    // control words, 8 bytes each, one block on the device and its page-locked
    // mirror on the host, so that reading them is one copy (ControlRead)
    unsigned long long *d_ctl = nullptr, *h_ctl = nullptr;
    size_t ctl_words = 0;
    std::mutex ctl_mutex;
    double* d_dt = nullptr;           // [nruns]
    double* d_time = nullptr;         // [nruns][NSLOTS]
    long long* d_iter = nullptr;      // [nruns][NSLOTS]
    unsigned long long* d_amax = nullptr;  // [nruns]
    Failure* d_failure = nullptr;
    long long* d_adv_count = nullptr;       // advances begun without a pending failure
    long long adv_base = 0;
    std::vector<std::pair<int, std::vector<StagePlan>>> window;  // advances since the last check
    double* d_staging = nullptr;
    size_t staging_bytes = 0;
    // pipelined host transfers (b2d_upload_conserved_async / b2d_download_async):
    // copy streams, double-buffered device staging and their events
    cudaStream_t up_stream = nullptr, down_stream = nullptr;
    double* d_in[2] = {};
    double* d_out[2] = {};
    cudaEvent_t in_copied[2] = {}, in_used[2] = {}, out_ready[2] = {}, out_copied[2] = {};
    long long n_up = 0, n_down = 0;
    int max_stages = 0;
    cudaStream_t stream = nullptr;
    bool use_graphs = true;
    std::map<std::pair<int, int>, cudaGraphExec_t> graphs;
    long long launches = 0;
    int total_tiles = 0;
    // instrumentation
    bool instrument = false;
    std::vector<cudaEvent_t> ev;
    double stage_ms_total = 0.0;
    long long stage_count = 0;
};

template <class T> static DevParamsT<T> make_params(const b2d_config& c)
{
    DevParamsT<T> p;
    memset(&p, 0, sizeof p);
    p.hydro = c.hydro_kind;
    p.visc = c.viscosity_kind;
    p.sink_model = c.sink_model;
    p.one_body = c.one_body;
    p.has_mach_ceiling = c.has_mach_ceiling;
    p.has_density_floor = c.has_density_floor;
    p.has_pressure_floor = c.has_pressure_floor;
    p.density_index = c.density_index;
    p.cooling_kind = c.cooling_kind;
    p.cooling_slow_start = c.cooling_slow_start;
    p.has_dt_min = c.has_dt_min;
    double block_length = 2.0 * c.domain_radius / (double)c.num_blocks;  // mesh.rs:27-29
    double dx = block_length / (double)c.block_size;                     // mesh.rs:86-88
    p.dx = (T)dx;
    p.inv_dx = (T)(1.0 / dx);
    p.cfl = (T)c.cfl;
    p.dt_min = (T)c.dt_min;
    p.plm = (T)c.plm;
    p.pdt = (T)(c.has_plm_density_trigger ? c.plm_density_trigger : 0.0);  // scheme.rs:216-220
    p.nu = (T)c.viscosity;
    p.lambda = (T)c.lambda_multiplier;
    p.mach2 = (T)(c.mach_number * c.mach_number);
    p.inv_mach2 = (T)(1.0 / (c.mach_number * c.mach_number));
    double gamma = c.hydro_kind == B2D_EULER ? c.gamma_law_index : 1.0;  // physics.rs:477-479
    p.gamma = (T)gamma;
    p.gm1 = (T)(gamma - 1.0);
    p.inv_gm1 = (T)(1.0 / (gamma - 1.0));
    p.sqrt_gm = (T)sqrt(gamma);
    p.inv_sqrt_gm = (T)(1.0 / sqrt(gamma));
    double s = c.has_softening_length ? c.softening_length : c.sink_radius;  // physics.rs:399-405
    p.soft2 = (T)(s * s);
    p.sink_r2 = (T)(c.sink_radius * c.sink_radius);
    p.inv_sink_r2 = (T)(1.0 / (c.sink_radius * c.sink_radius));
    p.sink_rate = (T)c.sink_rate;
    p.domain_radius = (T)c.domain_radius;
    p.buffer_scale = (T)c.buffer_scale;
    p.inv_buffer_scale = (T)(1.0 / c.buffer_scale);
    p.half_buffer_rate = (T)(0.5 * c.buffer_rate);
    double q = c.one_body ? 1.0 : c.binary_mass_ratio;
    double m1 = 1.0 / (1.0 + q), m2 = 1.0 * q / (1.0 + q);
    double R = c.domain_radius;
    double omega_outer = sqrt((m1 + m2) / (R * R * R));                  // physics.rs:445
    p.omega_outer = (T)omega_outer;
    p.half_rate_omega = (T)(0.5 * c.buffer_rate * omega_outer);
    p.fake_thr = (T)c.fake_mass_threshold;
    p.fake_rate = (T)c.fake_mass_rate;
    p.density_floor = (T)c.density_floor;
    p.pressure_floor = (T)c.pressure_floor;
    p.density_floor_pow_gamma = (T)(c.has_density_floor ? pow(c.density_floor, gamma) : 0.0);
    p.mach_ceiling2 = (T)(c.mach_ceiling * c.mach_ceiling);
    p.k_mach_ceiling = (T)(c.has_mach_ceiling ? 2.0 / (gamma * (gamma - 1.0) * c.mach_ceiling * c.mach_ceiling) : 0.0);
    p.cool_coef = (T)c.cooling_coefficient;
    p.cool_beta = (T)c.cooling_beta;
    p.inv_cool_beta = (T)(c.cooling_beta != 0.0 ? 1.0 / c.cooling_beta : 0.0);
    p.eps_dx = (T)(1e-12 * dx);
    return p;
}

static b2d_status validate(const b2d_config& c, int hydro, int rk)
{
    if (c.num_blocks < 1 || c.block_size < 1) return fail(B2D_ERR_INVALID, "num_blocks and block_size must be positive");
    if (c.hydro_kind != hydro) return fail(B2D_ERR_INVALID, "all runs of a context must share the hydro kind");
    if (c.rk_order != rk) return fail(B2D_ERR_INVALID, "all runs of a context must share rk_order");
    if (rk < 1 || rk > 3) return fail(B2D_ERR_INVALID, "rk_order must be 1, 2 or 3");
    long long N = (long long)c.num_blocks * c.block_size;
    if (N * N > (1ll << 31)) return fail(B2D_ERR_INVALID, "mesh too large (more than 2^31 zones per run)");
    if (!(c.domain_radius > 0)) return fail(B2D_ERR_INVALID, "domain_radius must be positive");
    if (c.num_blocks > 256 || c.block_size > 4096)
        return fail(B2D_ERR_INVALID, "num_blocks must be at most 256 and block_size at most 4096");
    return B2D_OK;
}

static int default_tile_w(int bs)
{
    for (int w : {128, 64, 32})
        if (bs % w == 0) return w;
    return bs;
}

// The FP64 kernel's largest sub-tile for runs of the given block sizes and
// block counts: the shape whose sub-tiles, dealt evenly to the SMs, take the
// busiest SM the fewest FP64 operations.  The kernel is bound by each SM's FP64
// pipe, so large sub-tiles (few guard zones) win until the mesh is too small to
// give every SM the same share of them.  The weights are the kernel's FP64
// operations per guard-including zone, slope zone, face and updated zone, and
// 4000 for a sub-tile's latency between phases; a
// 16 x 32 sub-tile of Euler zones leaves room for one CTA per SM only, which
// costs 5 % (1024^2: 1.568 against 1.490 ms a stage).  Measured per stage, by
// shape 16x32 / 12x32 / 8x32 / 8x16 / 4x16: isothermal 2048^2 3.21 / 3.30 / 3.56
// / 4.16 / 5.80 ms, 384^2 140 / 182 / 152 / 173 / 236 us; Euler 256^2 129 / 167 /
// 135 / 149 / 193 us, 128^2 127 / 93 / 79 / 49 / 58 us.
struct BlockCount { int bs; long long blocks; };
static void f64_sub_tile(int nf, const std::vector<BlockCount>& runs, int* th, int* tw)
{
    constexpr int SMS = 152;
    const int shapes[5][2] = {{16, 32}, {12, 32}, {8, 32}, {8, 16}, {4, 16}};
    double best = 1e300;
    for (const auto& s : shapes) {
        long long n = 0;
        double cost = 0.0;
        for (const BlockCount& r : runs) {
            const int ni = (r.bs + s[0] - 1) / s[0], nj = (r.bs + s[1] - 1) / s[1];
            const int h = (r.bs + ni - 1) / ni, w = (r.bs + nj - 1) / nj;
            n += r.blocks * ni * nj;
            auto whole = [](int k) { return (k + 31) / 32 * 32; };   // lanes of whole warps
            cost = std::max(cost, 4000.0 + 15 * whole((h + 4) * (w + 4)) + 31 * whole((h + 2) * (w + 2)) +
                                      105 * (whole((h + 1) * w) + whole(h * (w + 1))) + 95 * whole(h * w));
        }
        if (nf == 4 && s[0] == 16) cost *= 1.05;
        cost *= n < 8 * SMS ? (double)((n + SMS - 1) / SMS) : (double)n / SMS;
        if (cost < best) {
            best = cost;
            *th = s[0];
            *tw = s[1];
        }
    }
}

// Split blocks of bs x bs zones evenly into sub-tiles of at most th x tw.
static void split_blocks(RunDev& d, int bs, int th, int tw, int per_cta)
{
    d.sub_i = (bs + th - 1) / th;
    d.sub_j = (bs + tw - 1) / tw;
    d.sub_per_cta = per_cta;
    d.tiles_per_block = (d.sub_i * d.sub_j + per_cta - 1) / per_cta;
}

static bool tile_ok(const b2d_ctx* ctx, int tw, int th)
{
    // (a width has no effect on the kernels: the FP64 kernel picks its own sub-tiles, the FP32 kernel's strips
    // are 60 columns.  128-, 256- and 512-column tiles may also span whole blocks side by side.)
    const bool span = ctx->precision == B2D_PREC_FP32_COMP && (tw == 128 || tw == 256 || tw == 512);
    if (tw < 1 || th < 1 || tw > (span ? 512 : 256)) return false;
    for (const RunHost& r : ctx->runs) {
        if (r.bs % th) return false;
        if (r.bs % tw && !(span && r.bs >= 64 && tw % r.bs == 0 && r.N % tw == 0)) return false;
    }
    if (tw % 32 != 0) {
        // a partial warp is allowed only when it is the whole block width
        for (const RunHost& r : ctx->runs)
            if (r.bs != tw) return false;
    }
    return true;
}

static void free_ctx(b2d_ctx* ctx)
{
    if (!ctx) return;
    for (auto& kv : ctx->graphs) cudaGraphExecDestroy(kv.second);
    for (RunHost& r : ctx->runs) {
        for (int s = 0; s < NSLOTS; ++s) { cudaFree(r.slot[s]); cudaFree(r.ledger[s]); cudaFree(r.elements[s]); }
        const size_t ri = &r - ctx->runs.data();
        if (ri < ctx->rdev_h.size())
            for (int s = 0; s < NSLOTS; ++s) cudaFree(ctx->rdev_h[ri].tracers[s]);
        cudaFree(r.buffer); cudaFree(r.bg); cudaFree(r.partial);
        cudaFree(r.xc); cudaFree(r.xv); cudaFree(r.xcf); cudaFree(r.xvf);
        cudaFree(r.stage_time); cudaFree(r.orbit); cudaFree(r.stage_ds); cudaFree(r.stage_de);
    }
    cudaFree(ctx->rdev); cudaFree(ctx->d_bases); cudaFree(ctx->d_ctl); cudaFree(ctx->d_staging);
    if (ctx->h_ctl) cudaFreeHost(ctx->h_ctl);
    for (cudaEvent_t e : ctx->ev) cudaEventDestroy(e);
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    if (ctx->up_stream) cudaStreamDestroy(ctx->up_stream);
    if (ctx->down_stream) cudaStreamDestroy(ctx->down_stream);
    for (int b = 0; b < 2; ++b) {
        cudaFree(ctx->d_in[b]);
        cudaFree(ctx->d_out[b]);
        for (cudaEvent_t e : {ctx->in_copied[b], ctx->in_used[b], ctx->out_ready[b], ctx->out_copied[b]})
            if (e) cudaEventDestroy(e);
    }
    delete ctx;
}

// Row chunks per column strip of a run: block-aligned tiles of height th, or,
// with strip rows set, ceil(N / rows) chunks that may cross block boundaries.
static int row_chunks(const b2d_ctx* ctx, const RunHost& r)
{
    if (ctx->strip_rows > 0) return (r.N + ctx->strip_rows - 1) / ctx->strip_rows;
    return r.N / ctx->th;
}

// 4, 2 or 1: the largest of them that divides the sides of all runs (how many
// columns the FP32 kernel can copy as one aligned word).
static int side_divisor(const b2d_ctx* ctx)
{
    int d = 4;
    for (const RunHost& r : ctx->runs)
        while (r.N % d) d /= 2;
    return d;
}

// Buffers for the ledger pieces of as many stages as PIECE_BYTES hold (at
// least one, at most an advance's capacity), and the run descriptors and first
// CTAs on the device.  Graphs that hold the old descriptors go.  Like every copy
// and clear of a context these go through its stream: that stream does not wait
// for the legacy one, and a stage that sees new first CTAs beside old
// descriptors would compute tiles out of range.
static b2d_status alloc_pieces(b2d_ctx* ctx)
{
    constexpr size_t PIECE_BYTES = 64u << 20;
    auto stage_bytes = [&](const RunDev& d) { return sizeof(double) * d.nblocks * d.tiles_per_block * NITEMS * ctx->nf; };
    size_t total = 0;
    std::vector<int> bases;
    for (const RunDev& d : ctx->rdev_h) {
        total += stage_bytes(d);
        bases.push_back(d.tile_base);
    }
    ctx->stage_window = (int)std::min<size_t>(std::max<size_t>(PIECE_BYTES / total, 1), std::max(ctx->max_stages, 1));
    for (int i = 0; i < ctx->nruns; ++i) {
        RunHost& r = ctx->runs[i];
        RunDev& d = ctx->rdev_h[i];
        const size_t bytes = stage_bytes(d) * ctx->stage_window;
        if (bytes > r.partial_bytes) {
            CUDA_TRY(cudaFree(r.partial));
            r.partial = nullptr;
            r.partial_bytes = 0;
            CUDA_TRY(cudaMalloc(&r.partial, bytes));
            r.partial_bytes = bytes;
        }
        CUDA_TRY(cudaMemsetAsync(r.partial, 0, bytes, ctx->stream));   // the words of items that are always zero are never written
        d.partial = r.partial;
        d.stage_window = ctx->stage_window;
    }
    CUDA_TRY(cudaMemcpyAsync(ctx->rdev, ctx->rdev_h.data(), sizeof(RunDev) * ctx->nruns, cudaMemcpyHostToDevice, ctx->stream));
    CUDA_TRY(cudaMemcpyAsync(ctx->d_bases, bases.data(), sizeof(int) * ctx->nruns, cudaMemcpyHostToDevice, ctx->stream));
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    for (auto& kv : ctx->graphs) cudaGraphExecDestroy(kv.second);
    ctx->graphs.clear();
    return B2D_OK;
}

// Rebuild the tile bookkeeping for the current tile shape and push the run
// descriptors to the device.
static b2d_status sync_rundev(b2d_ctx* ctx)
{
    int base = 0;
    for (int i = 0; i < ctx->nruns; ++i) {
        RunHost& r = ctx->runs[i];
        RunDev& d = ctx->rdev_h[i];
        // a slab launches the block-aligned chunks (tile height th) of its own block rows
        d.chunks = d.slab_hi > 0 ? r.N / ctx->th : row_chunks(ctx, r);
        d.chunk0 = d.slab_hi > 0 ? d.slab_lo * (r.bs / ctx->th) : 0;
        d.tiles_i = d.slab_hi > 0 ? (d.slab_hi - d.slab_lo) * (r.bs / ctx->th) : d.chunks;
        d.tile_base = base;
        if (ctx->precision == B2D_PREC_FP64) {
            // the FP64 kernel's CTAs take sub-tiles block by block
            split_blocks(d, r.bs, ctx->sub_h, ctx->sub_w, 1);
            d.ntiles = (d.slab_hi > 0 ? d.slab_hi - d.slab_lo : r.nb) * r.nb * d.tiles_per_block;
            base += d.ntiles;
        } else {
            // the FP32 kernel's one-warp CTAs take strips x row chunks
            d.tiles_j = (r.N + STRIP_COLS - 1) / STRIP_COLS;
            d.ntiles = d.tiles_i * d.tiles_j;
            base += d.ntiles;
            d.tiles_per_block = most_strip_pieces(r.bs, r.nb, d.chunks);
        }
    }
    ctx->total_tiles = base;
    return alloc_pieces(ctx);
}

static b2d_status ensure_stage_capacity(b2d_ctx* ctx, int fold)
{
    int need = fold * ctx->rk;
    if (need <= ctx->max_stages) return B2D_OK;
    int cap = std::max(need, 64);
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));   // queued advances use what is replaced here
    for (int i = 0; i < ctx->nruns; ++i) {
        RunHost& r = ctx->runs[i];
        CUDA_TRY(cudaFree(r.stage_time));
        CUDA_TRY(cudaFree(r.orbit));
        CUDA_TRY(cudaFree(r.stage_ds));
        CUDA_TRY(cudaFree(r.stage_de));
        r.stage_time = nullptr;
        r.orbit = nullptr;
        r.stage_ds = nullptr;
        r.stage_de = nullptr;
        CUDA_TRY(cudaMalloc(&r.stage_time, sizeof(double) * cap));
        CUDA_TRY(cudaMalloc(&r.orbit, sizeof(double) * 10 * cap));
        CUDA_TRY(cudaMalloc(&r.stage_ds, sizeof(double) * cap * r.nblocks * NITEMS * ctx->nf));
        CUDA_TRY(cudaMalloc(&r.stage_de, sizeof(double) * cap * r.nblocks * 16));
        ctx->rdev_h[i].stage_time = r.stage_time;
        ctx->rdev_h[i].orbit = r.orbit;
        ctx->rdev_h[i].stage_ds = r.stage_ds;
        ctx->rdev_h[i].stage_de = r.stage_de;
    }
    ctx->max_stages = cap;
    return alloc_pieces(ctx);
}

extern "C" b2d_ctx* b2d_create(const b2d_config* cfgs, int32_t nruns, int32_t precision, b2d_status* status)
{
    b2d_status st_dummy;
    if (!status) status = &st_dummy;
    if (!cfgs || nruns < 1 || nruns > 256) { *status = fail(B2D_ERR_INVALID, "need 1 to 256 runs"); return nullptr; }
    if (precision < 0 || precision > 2) { *status = fail(B2D_ERR_INVALID, "bad precision"); return nullptr; }
    int ndev = 0;
    cudaError_t ce = cudaGetDeviceCount(&ndev);
    if (ce != cudaSuccess || ndev == 0) {
        *status = fail(B2D_ERR_CUDA, std::string("no CUDA device: ") + cudaGetErrorString(ce));
        return nullptr;
    }
    b2d_ctx* ctx = new b2d_ctx;
    ctx->nruns = nruns;
    ctx->precision = precision;
    ctx->hydro = cfgs[0].hydro_kind;
    ctx->rk = cfgs[0].rk_order;
    ctx->nf = ctx->hydro == B2D_EULER ? 4 : 3;
    int min_bs = 1 << 30;
    for (int i = 0; i < nruns; ++i) {
        b2d_status v = validate(cfgs[i], ctx->hydro, ctx->rk);
        if (v != B2D_OK) { *status = v; free_ctx(ctx); return nullptr; }
        min_bs = std::min(min_bs, cfgs[i].block_size);
    }
#define CREATE_TRY(expr)                                                                         \
    do {                                                                                         \
        cudaError_t e_ = (expr);                                                                 \
        if (e_ != cudaSuccess) {                                                                 \
            *status = fail(B2D_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_));    \
            free_ctx(ctx);                                                                       \
            return nullptr;                                                                      \
        }                                                                                        \
    } while (0)
    CREATE_TRY(cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking));
    CREATE_TRY(cudaMalloc(&ctx->rdev, sizeof(RunDev) * nruns));
    CREATE_TRY(cudaMalloc(&ctx->d_bases, sizeof(int) * nruns));
    ctx->ctl_words = 3 + (size_t)nruns * (2 + 2 * NSLOTS);
    CREATE_TRY(cudaMalloc(&ctx->d_ctl, sizeof(unsigned long long) * ctx->ctl_words));
    CREATE_TRY(cudaMallocHost(&ctx->h_ctl, sizeof(unsigned long long) * ctx->ctl_words));
    CREATE_TRY(cudaMemsetAsync(ctx->d_ctl, 0, sizeof(unsigned long long) * ctx->ctl_words, ctx->stream));
    ctx->d_failure = (Failure*)ctx->d_ctl;
    ctx->d_adv_count = (long long*)(ctx->d_ctl + 2);
    ctx->d_amax = ctx->d_ctl + 3;
    ctx->d_dt = (double*)(ctx->d_amax + nruns);
    ctx->d_time = ctx->d_dt + nruns;
    ctx->d_iter = (long long*)(ctx->d_time + (size_t)nruns * NSLOTS);
    CREATE_TRY(cudaMemsetAsync(&ctx->d_failure->key, 0xff, sizeof(unsigned long long), ctx->stream));

    ctx->runs.resize(nruns);
    ctx->rdev_h.resize(nruns);
    const int store = precision == B2D_PREC_FP32_COMP ? 1 : 0;
    for (int i = 0; i < nruns; ++i) {
        RunHost& r = ctx->runs[i];
        RunDev& d = ctx->rdev_h[i];
        memset(&d, 0, sizeof d);
        r.cfg = cfgs[i];
        r.bs = cfgs[i].block_size;
        r.nb = cfgs[i].num_blocks;
        r.N = r.bs * r.nb;
        r.nblocks = r.nb * r.nb;
        size_t nn = (size_t)r.N * r.N;
        r.state_bytes = store == 1 ? nn * ctx->nf * 2 * sizeof(float) : nn * ctx->nf * sizeof(double);
        for (int s = 0; s < NSLOTS; ++s) {
            CREATE_TRY(cudaMalloc(&r.slot[s], r.state_bytes));
            CREATE_TRY(cudaMemsetAsync(r.slot[s], 0, r.state_bytes, ctx->stream));
            CREATE_TRY(cudaMalloc(&r.ledger[s], sizeof(double) * r.nblocks * NITEMS * ctx->nf));
            CREATE_TRY(cudaMemsetAsync(r.ledger[s], 0, sizeof(double) * r.nblocks * NITEMS * ctx->nf, ctx->stream));
            CREATE_TRY(cudaMalloc(&r.elements[s], sizeof(double) * r.nblocks * NITEMS * 4));
            CREATE_TRY(cudaMemsetAsync(r.elements[s], 0, sizeof(double) * r.nblocks * NITEMS * 4, ctx->stream));
        }
        CREATE_TRY(cudaMalloc(&r.bg, r.state_bytes));
        CREATE_TRY(cudaMemsetAsync(r.bg, 0, r.state_bytes, ctx->stream));
        // geometry tables
        std::vector<double> xc(r.N), xv((size_t)r.nb * (r.bs + 1));
        for (int b = 0; b < r.nb; ++b) {
            host_cell_centers(&cfgs[i], b, xc.data() + (size_t)b * r.bs);
            host_block_vertices(&cfgs[i], b, xv.data() + (size_t)b * (r.bs + 1));
        }
        // centres, and faces by global index (face k of block k / bs, the last
        // block's top face last), as FP32 high and low words
        auto split = [](double v) {
            const float hi = (float)v;
            return make_float2(hi, (float)(v - (double)hi));
        };
        std::vector<float2> xcf, xvf;
        for (int k = 0; k < r.N; ++k) {
            xcf.push_back(split(xc[k]));
            xvf.push_back(split(xv[(size_t)(k / r.bs) * (r.bs + 1) + k % r.bs]));
        }
        xvf.push_back(split(xv[(size_t)(r.nb - 1) * (r.bs + 1) + r.bs]));
        r.hxc = xc;
        CREATE_TRY(cudaMalloc(&r.xc, sizeof(double) * xc.size()));
        CREATE_TRY(cudaMalloc(&r.xv, sizeof(double) * xv.size()));
        CREATE_TRY(cudaMalloc(&r.xcf, sizeof(float2) * xcf.size()));
        CREATE_TRY(cudaMalloc(&r.xvf, sizeof(float2) * xvf.size()));
        CREATE_TRY(cudaMemcpyAsync(r.xc, xc.data(), sizeof(double) * xc.size(), cudaMemcpyHostToDevice, ctx->stream));
        CREATE_TRY(cudaMemcpyAsync(r.xv, xv.data(), sizeof(double) * xv.size(), cudaMemcpyHostToDevice, ctx->stream));
        CREATE_TRY(cudaMemcpyAsync(r.xcf, xcf.data(), sizeof(float2) * xcf.size(), cudaMemcpyHostToDevice, ctx->stream));
        CREATE_TRY(cudaMemcpyAsync(r.xvf, xvf.data(), sizeof(float2) * xvf.size(), cudaMemcpyHostToDevice, ctx->stream));

        d.N = r.N; d.bs = r.bs; d.nb = r.nb; d.nblocks = r.nblocks;
        d.xc = r.xc; d.xv = r.xv; d.xcf = r.xcf; d.xvf = r.xvf;
        for (int s = 0; s < NSLOTS; ++s) {
            d.slot[s] = r.slot[s];
            d.ledger[s] = r.ledger[s];
            d.elements[s] = r.elements[s];
        }
        // OrbitalElements of the run (physics.rs:411-417)
        if (cfgs[i].one_body) { d.el0[0] = 1e-12; d.el0[1] = 1.0; d.el0[2] = 1.0; d.el0[3] = 0.0; }
        else {
            d.el0[0] = 1.0;
            d.el0[1] = 1.0;
            d.el0[2] = cfgs[i].binary_mass_ratio;
            d.el0[3] = cfgs[i].binary_eccentricity;
        }
        d.bg = r.bg;
        d.time = ctx->d_time + (size_t)i * NSLOTS;
        d.iter = ctx->d_iter + (size_t)i * NSLOTS;
        d.dt = ctx->d_dt + i;
        d.amax = ctx->d_amax + i;
        d.binary_q = cfgs[i].binary_mass_ratio;
        d.binary_e = cfgs[i].binary_eccentricity;
        d.tracer_radius = split(cfgs[i].domain_radius);
        d.tracer_inv_dx = split(r.N / (2.0 * cfgs[i].domain_radius));
        d.p = make_params<double>(cfgs[i]);
        d.pf = make_params<float>(cfgs[i]);
        ctx->staging_bytes = std::max(ctx->staging_bytes, nn * ctx->nf * sizeof(double));
    }
    CREATE_TRY(cudaMalloc(&ctx->d_staging, ctx->staging_bytes));
    ctx->tw = default_tile_w(min_bs);
    ctx->th = std::min(64, min_bs);
    while (!tile_ok(ctx, ctx->tw, ctx->th) && ctx->th > 1) ctx->th /= 2;
    if (!tile_ok(ctx, ctx->tw, ctx->th)) {
        *status = fail(B2D_ERR_INVALID, "runs of a context need a common tile shape (block sizes must share a divisor)");
        free_ctx(ctx);
        return nullptr;
    }
    std::vector<BlockCount> counts;
    for (const RunHost& r : ctx->runs) counts.push_back({r.bs, r.nblocks});
    f64_sub_tile(ctx->nf, counts, &ctx->sub_h, &ctx->sub_w);
    if (sync_rundev(ctx) != B2D_OK) { *status = B2D_ERR_CUDA; free_ctx(ctx); return nullptr; }
    if (precision == B2D_PREC_FP64) {
        // the buffer's rate depends on the zone's place only, and takes an
        // FP64 root, division and tanh: a table, 8 bytes a zone beside the
        // run's 144 or 192 (without the memory for it, the stages compute it)
        size_t tables = 0, free_bytes = 0, total_bytes = 0;
        for (const RunHost& r : ctx->runs) tables += sizeof(double) * (size_t)r.N * r.N;
        CREATE_TRY(cudaMemGetInfo(&free_bytes, &total_bytes));
        for (int i = 0; i < nruns && room_for_tables(free_bytes, total_bytes, tables); ++i) {
            RunHost& r = ctx->runs[i];
            if (cudaMalloc(&r.buffer, sizeof(double) * (size_t)r.N * r.N) != cudaSuccess) {
                cudaGetLastError();
                r.buffer = nullptr;
                continue;
            }
            CREATE_TRY(launch_buffer_rate(ctx->rdev, i, r.N, r.buffer, ctx->stream));
            ctx->rdev_h[i].buffer = r.buffer;
        }
        CREATE_TRY(cudaStreamSynchronize(ctx->stream));
        CREATE_TRY(cudaMemcpyAsync(ctx->rdev, ctx->rdev_h.data(), sizeof(RunDev) * nruns, cudaMemcpyHostToDevice, ctx->stream));
    }
    if (ensure_stage_capacity(ctx, 16) != B2D_OK) { *status = B2D_ERR_CUDA; free_ctx(ctx); return nullptr; }
    *status = B2D_OK;
    return ctx;
#undef CREATE_TRY
}

extern "C" void b2d_destroy(b2d_ctx* ctx)
{
    if (ctx) cudaStreamSynchronize(ctx->stream);
    free_ctx(ctx);
}

extern "C" int32_t b2d_num_fields(const b2d_ctx* ctx) { return ctx ? ctx->nf : 0; }

// The control words, copied to the host after waiting for the stream; the
// mirror is this reader's until it goes out of scope.  One copy into
// page-locked memory: a copy of each word into pageable memory costs some
// 10 us, which is what a small mesh takes for two stages (128^2, measured:
// advance(1) 84 -> 64 us, synchronize 31 -> 12, download 41 -> 31).
class ControlRead {
  public:
    explicit ControlRead(b2d_ctx* c) : ctx(c), lock(c->ctl_mutex), status(copy()) {}
    template <class T> T operator()(const T* device_word) const
    {
        T v;
        memcpy(&v, ctx->h_ctl + ((const unsigned long long*)device_word - ctx->d_ctl), sizeof v);
        return v;
    }

  private:
    b2d_status copy()
    {
        CUDA_TRY(cudaMemcpyAsync(ctx->h_ctl, ctx->d_ctl, sizeof(unsigned long long) * ctx->ctl_words,
                                 cudaMemcpyDeviceToHost, ctx->stream));
        CUDA_TRY(cudaStreamSynchronize(ctx->stream));
        return B2D_OK;
    }
    b2d_ctx* ctx;
    std::lock_guard<std::mutex> lock;

  public:
    const b2d_status status;
};

static int store_of(const b2d_ctx* ctx) { return ctx->precision == B2D_PREC_FP32_COMP ? 1 : 0; }

static b2d_status launch_max_speed(b2d_ctx* ctx, int run, int slot)
{
    CUDA_TRY(cudaMemsetAsync(ctx->d_amax + run, 0, sizeof(unsigned long long), ctx->stream));
    int grid = 4 * 152;
    const bool f64 = ctx->precision == B2D_PREC_FP64;
    if (ctx->nf == 3) {
        if (f64) max_speed_kernel<3, 0, double><<<grid, 256, 0, ctx->stream>>>(ctx->rdev, run, slot);
        else if (store_of(ctx) == 0) max_speed_kernel<3, 0, float><<<grid, 256, 0, ctx->stream>>>(ctx->rdev, run, slot);
        else max_speed_kernel<3, 1, float><<<grid, 256, 0, ctx->stream>>>(ctx->rdev, run, slot);
    } else {
        if (f64) max_speed_kernel<4, 0, double><<<grid, 256, 0, ctx->stream>>>(ctx->rdev, run, slot);
        else if (store_of(ctx) == 0) max_speed_kernel<4, 0, float><<<grid, 256, 0, ctx->stream>>>(ctx->rdev, run, slot);
        else max_speed_kernel<4, 1, float><<<grid, 256, 0, ctx->stream>>>(ctx->rdev, run, slot);
    }
    ctx->launches++;
    CUDA_TRY(cudaGetLastError());
    return B2D_OK;
}

extern "C" b2d_status b2d_upload_state(b2d_ctx* ctx, int32_t run, const double* cons, const double* background,
                                       const double* ledger, double time, int64_t iteration_num, int64_t iteration_den)
{
    if (!ctx || run < 0 || run >= ctx->nruns || !cons) return fail(B2D_ERR_INVALID, "bad arguments");
    if (iteration_den != 1) return fail(B2D_ERR_INVALID, "iteration must be an integer at step boundaries");
    RunHost& r = ctx->runs[run];
    size_t n = (size_t)r.N * r.N * ctx->nf;
    int store = store_of(ctx);
    CUDA_TRY(cudaMemcpyAsync(ctx->d_staging, cons, n * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
    scatter_kernel<<<layout_blocks(r.N), LAYOUT_ZONES, 0, ctx->stream>>>(ctx->d_staging, r.slot[ctx->cur], r.N, r.bs, r.nb, ctx->nf, store);
    ctx->launches++;
    CUDA_TRY(cudaGetLastError());
    if (background) {
        CUDA_TRY(cudaMemcpyAsync(ctx->d_staging, background, n * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
        scatter_kernel<<<layout_blocks(r.N), LAYOUT_ZONES, 0, ctx->stream>>>(ctx->d_staging, r.bg, r.N, r.bs, r.nb, ctx->nf, store);
        ctx->launches++;
        CUDA_TRY(cudaGetLastError());
    }
    size_t nled = (size_t)r.nblocks * NITEMS * ctx->nf;
    if (ledger) CUDA_TRY(cudaMemcpyAsync(r.ledger[ctx->cur], ledger, nled * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
    else CUDA_TRY(cudaMemsetAsync(r.ledger[ctx->cur], 0, nled * sizeof(double), ctx->stream));
    CUDA_TRY(cudaMemsetAsync(r.elements[ctx->cur], 0, sizeof(double) * r.nblocks * NITEMS * 4, ctx->stream));
    long long it = iteration_num;
    CUDA_TRY(cudaMemcpyAsync(ctx->d_time + (size_t)run * NSLOTS + ctx->cur, &time, sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
    CUDA_TRY(cudaMemcpyAsync(ctx->d_iter + (size_t)run * NSLOTS + ctx->cur, &it, sizeof(long long), cudaMemcpyHostToDevice, ctx->stream));
    b2d_status s = launch_max_speed(ctx, run, ctx->cur);
    if (s != B2D_OK) return s;
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    return B2D_OK;
}

// Device address of a page-locked (cudaHostRegister / cudaMallocHost) host
// buffer that is 16-byte aligned, or nullptr.  The layout kernels read and
// write such buffers in place over the CPU-GPU link, so the copy and the
// layout change are one pass; other buffers go through the device staging
// buffer.
static void* mapped_host(const void* p)
{
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (at.type != cudaMemoryTypeHost || !at.devicePointer || ((uintptr_t)at.devicePointer & 15u)) return nullptr;
    return at.devicePointer;
}

extern "C" b2d_status b2d_upload_conserved(b2d_ctx* ctx, int32_t run, const double* cons)
{
    if (!ctx || run < 0 || run >= ctx->nruns || !cons) return fail(B2D_ERR_INVALID, "bad arguments");
    RunHost& r = ctx->runs[run];
    size_t n = (size_t)r.N * r.N * ctx->nf;
    const double* src = (const double*)mapped_host(cons);
    if (!src) {
        CUDA_TRY(cudaMemcpyAsync(ctx->d_staging, cons, n * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
        src = ctx->d_staging;
    }
    scatter_kernel<<<layout_blocks(r.N), LAYOUT_ZONES, 0, ctx->stream>>>(src, r.slot[ctx->cur], r.N, r.bs, r.nb, ctx->nf, store_of(ctx));
    ctx->launches++;
    CUDA_TRY(cudaGetLastError());
    b2d_status s = launch_max_speed(ctx, run, ctx->cur);
    if (s != B2D_OK) return s;
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    return B2D_OK;
}

// ---------------------------------------------------------------------------
// Pipelined host transfers.  Two copy streams move page-locked host buffers
// through double-buffered device staging while the context stream computes;
// the context stream only runs the layout kernels, so a step of a pipelined
// loop costs scatter + advance + gather on the device and the copies overlap
// the neighbouring steps' advances.

static b2d_status ensure_pipeline(b2d_ctx* ctx)
{
    if (ctx->up_stream) return B2D_OK;
    CUDA_TRY(cudaStreamCreateWithFlags(&ctx->up_stream, cudaStreamNonBlocking));
    CUDA_TRY(cudaStreamCreateWithFlags(&ctx->down_stream, cudaStreamNonBlocking));
    for (int b = 0; b < 2; ++b) {
        CUDA_TRY(cudaMalloc(&ctx->d_in[b], ctx->staging_bytes));
        CUDA_TRY(cudaMalloc(&ctx->d_out[b], ctx->staging_bytes));
        for (cudaEvent_t* e : {&ctx->in_copied[b], &ctx->in_used[b], &ctx->out_ready[b], &ctx->out_copied[b]})
            CUDA_TRY(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
    }
    return B2D_OK;
}

extern "C" b2d_status b2d_upload_conserved_async(b2d_ctx* ctx, int32_t run, const double* cons)
{
    if (!ctx || run < 0 || run >= ctx->nruns || !cons) return fail(B2D_ERR_INVALID, "bad arguments");
    b2d_status st = ensure_pipeline(ctx);
    if (st != B2D_OK) return st;
    RunHost& r = ctx->runs[run];
    const size_t n = (size_t)r.N * r.N * ctx->nf;
    const int b = (int)(ctx->n_up++ & 1);
    // the staging buffer is free once the scatter that last read it has run
    CUDA_TRY(cudaStreamWaitEvent(ctx->up_stream, ctx->in_used[b], 0));
    CUDA_TRY(cudaMemcpyAsync(ctx->d_in[b], cons, n * sizeof(double), cudaMemcpyHostToDevice, ctx->up_stream));
    CUDA_TRY(cudaEventRecord(ctx->in_copied[b], ctx->up_stream));
    CUDA_TRY(cudaStreamWaitEvent(ctx->stream, ctx->in_copied[b], 0));
    scatter_kernel<<<layout_blocks(r.N), LAYOUT_ZONES, 0, ctx->stream>>>(ctx->d_in[b], r.slot[ctx->cur], r.N, r.bs, r.nb, ctx->nf,
                                                       store_of(ctx));
    ctx->launches++;
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaEventRecord(ctx->in_used[b], ctx->stream));
    return launch_max_speed(ctx, run, ctx->cur);
}

extern "C" b2d_status b2d_download_async(b2d_ctx* ctx, int32_t run, double* cons)
{
    if (!ctx || run < 0 || run >= ctx->nruns || !cons) return fail(B2D_ERR_INVALID, "bad arguments");
    b2d_status st = ensure_pipeline(ctx);
    if (st != B2D_OK) return st;
    RunHost& r = ctx->runs[run];
    const size_t n = (size_t)r.N * r.N * ctx->nf;
    const int b = (int)(ctx->n_down++ & 1);
    // the staging buffer is free once the copy that last read it has finished
    CUDA_TRY(cudaStreamWaitEvent(ctx->stream, ctx->out_copied[b], 0));
    gather_kernel<<<layout_blocks(r.N), LAYOUT_ZONES, 0, ctx->stream>>>(r.slot[ctx->cur], ctx->d_out[b], r.N, r.bs, r.nb, ctx->nf,
                                                      store_of(ctx));
    ctx->launches++;
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaEventRecord(ctx->out_ready[b], ctx->stream));
    CUDA_TRY(cudaStreamWaitEvent(ctx->down_stream, ctx->out_ready[b], 0));
    CUDA_TRY(cudaMemcpyAsync(cons, ctx->d_out[b], n * sizeof(double), cudaMemcpyDeviceToHost, ctx->down_stream));
    CUDA_TRY(cudaEventRecord(ctx->out_copied[b], ctx->down_stream));
    return B2D_OK;
}

extern "C" b2d_status b2d_transfers_wait(b2d_ctx* ctx, int32_t pending)
{
    if (!ctx || pending < 0 || pending > 1) return fail(B2D_ERR_INVALID, "bad arguments");
    if (!ctx->up_stream) return B2D_OK;
    if (pending == 0) {
        CUDA_TRY(cudaStreamSynchronize(ctx->up_stream));
        CUDA_TRY(cudaStreamSynchronize(ctx->down_stream));
        return B2D_OK;
    }
    // every download but the newest has landed (downloads complete in order)
    if (ctx->n_down >= 2) CUDA_TRY(cudaEventSynchronize(ctx->out_copied[(ctx->n_down - 2) & 1]));
    return B2D_OK;
}

extern "C" b2d_status b2d_download_state(b2d_ctx* ctx, int32_t run, double* cons, double* time, int64_t* iteration_num,
                                         int64_t* iteration_den)
{
    if (!ctx || run < 0 || run >= ctx->nruns) return fail(B2D_ERR_INVALID, "bad arguments");
    RunHost& r = ctx->runs[run];
    size_t n = (size_t)r.N * r.N * ctx->nf;
    if (cons) {
        double* dst = (double*)mapped_host(cons);
        gather_kernel<<<layout_blocks(r.N), LAYOUT_ZONES, 0, ctx->stream>>>(r.slot[ctx->cur], dst ? dst : ctx->d_staging, r.N, r.bs, r.nb,
                                                         ctx->nf, store_of(ctx));
        ctx->launches++;
        CUDA_TRY(cudaGetLastError());
        if (!dst) CUDA_TRY(cudaMemcpyAsync(cons, ctx->d_staging, n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    }
    const ControlRead control(ctx);
    if (control.status != B2D_OK) return control.status;
    if (time) *time = control(ctx->d_time + (size_t)run * NSLOTS + ctx->cur);
    if (iteration_num) *iteration_num = control(ctx->d_iter + (size_t)run * NSLOTS + ctx->cur);
    if (iteration_den) *iteration_den = 1;
    return B2D_OK;
}

extern "C" b2d_status b2d_download_ledger(b2d_ctx* ctx, int32_t run, double* ledger)
{
    if (!ctx || run < 0 || run >= ctx->nruns || !ledger) return fail(B2D_ERR_INVALID, "bad arguments");
    RunHost& r = ctx->runs[run];
    size_t nled = (size_t)r.nblocks * NITEMS * ctx->nf;
    CUDA_TRY(cudaMemcpyAsync(ledger, r.ledger[ctx->cur], nled * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    return B2D_OK;
}

extern "C" b2d_status b2d_max_signal_speed(b2d_ctx* ctx, int32_t run, double* out)
{
    if (!ctx || run < 0 || run >= ctx->nruns || !out) return fail(B2D_ERR_INVALID, "bad arguments");
    const ControlRead control(ctx);
    if (control.status != B2D_OK) return control.status;
    const unsigned long long bits = control(ctx->d_amax + run);
    double v;
    memcpy(&v, &bits, sizeof v);
    *out = v;
    return B2D_OK;
}

// ---------------------------------------------------------------------------
// The advance.

__host__ __device__ static int free_slot(int a, int b, int c)
{
    for (int s = 0; s < NSLOTS; ++s)
        if (s != a && s != b && s != c) return s;
    return -1;
}

// Slot schedule of `fold` RK steps from slot `start`, which is left intact.
static std::vector<StagePlan> plan_advance(int rk, int fold, int start, int* final_slot)
{
    std::vector<StagePlan> plan;
    int base = start;
    for (int f = 0; f < fold; ++f) {
        if (rk == 1) {
            int a = free_slot(start, base, -1);
            plan.push_back({base, -1, a, 0.0});
            base = a;
        } else if (rk == 2) {
            int a = free_slot(start, base, -1);
            plan.push_back({base, -1, a, 0.0});
            int b = free_slot(start, base, a);
            plan.push_back({a, base, b, 0.5});
            base = b;
        } else {
            int a = free_slot(start, base, -1);
            plan.push_back({base, -1, a, 0.0});
            int b = free_slot(start, base, a);
            plan.push_back({a, base, b, 0.75});
            int c = free_slot(start, base, b);
            plan.push_back({b, base, c, 1.0 / 3.0});
            base = c;
        }
    }
    *final_slot = base;
    return plan;
}

// The ledgers of every block over one advance (compute_block_updated_solution,
// scheme.rs:307-314), after the stage kernels, which only write their pieces
// of each block's sums: folds and the serial FP64 perturbation stay out of
// their tails.  One CTA per block, in three steps:
//  * a thread per (stage, ledger word): the word's pieces, in order, to the
//    block's stage sums ds·dx·dy;
//  * a thread per (stage, gas item) for sink1, sink2, grav1 and grav2: the
//    perturbation (ItemizedChange::perturbation, state.rs:258-281).  An unbound
//    perturbed orbit fails its stage with OrbitalEvolutionError, reported at
//    position (0, 0) as in the reference.  The reference converts every block's
//    primitives before it updates any block, so within a stage a cons->prim
//    failure anywhere wins: the key's block field is saturated and the failing
//    block's index rides in the zone field; an earlier stage still wins through
//    the stage field;
//  * a thread per ledger word or element component: the stages in order,
//    x_out = x_in + change averaged like the state (state.rs:191-197), in the
//    slot schedule of plan_advance.
// Launched once per advance; meshes of very many pieces fold every stage_window
// stages, and the last launch sums.  It is all latency, at the end of every
// advance: as a launch of a thread per (stage, block, item) for the first two
// steps and another for the third an advance of one step of 128^2 took 49 us, with
// this 40 (a call of it 64 and 53).
template <int NF> __device__ __forceinline__ void fold_item(const RunDev& rd, int s, int block, int item, double* ds)
{
    constexpr int NL = NITEMS * NF;
    const double* p = stage_pieces(rd, s, block, NL) + item * NF;
    double v[NF] = {};
#pragma unroll 8
    for (int q = 0; q < rd.tiles_per_block; ++q)
#pragma unroll
        for (int f = 0; f < NF; ++f) v[f] += p[(size_t)q * NL + f];
    const double area = rd.p.dx * rd.p.dx;
#pragma unroll
    for (int f = 0; f < NF; ++f) ds[f] = v[f] * area;
}

__global__ void __launch_bounds__(256) ledger_kernel(const RunDev* runs, int first, int last, bool sum, int fold, int rk,
                                                     int start, Failure* failure)
{
    const int run = blockIdx.y, block = blockIdx.x;
    const RunDev& rd = runs[run];
    if (block >= rd.nblocks || failure->abandoned) return;
    if (rd.slab_hi > 0 && (block / rd.nb < rd.slab_lo || block / rd.nb >= rd.slab_hi)) return;   // another slab's
    const int nf = rd.p.hydro == B2D_EULER ? 4 : 3, nl = NITEMS * nf, pieces = rd.tiles_per_block;
    const size_t stride = (size_t)rd.nblocks * nl;
    double* stage_ds = rd.stage_ds + (size_t)block * nl;
    double* stage_de = rd.stage_de + (size_t)block * 16;
    const double area = rd.p.dx * rd.p.dx;
    for (int t = threadIdx.x; t < (last - first) * nl; t += blockDim.x) {
        const int s = first + t / nl, k = t % nl;
        const double* p = stage_pieces(rd, s, block, nl) + k;
        double v = 0.0;
#pragma unroll 16
        for (int q = 0; q < pieces; ++q) v += p[q * nl];
        stage_ds[s * stride + k] = v * area;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < (last - first) * 4; t += blockDim.x) {
        const int s = first + t / 4, item = t % 4;
        const double* orbit = rd.orbit + 10 * s;
        const double* ds = stage_ds + s * stride + item * nf;
        double* de = stage_de + (size_t)s * rd.nblocks * 16 + item * 4;
        // pert1 (body 1: sink1, grav1) and pert2 (body 2: sink2, grav2), state.rs:261-269
        const bool ok = (item == 0 || item == 2)
                            ? perturb_elements(orbit, rd.el0, -ds[0], 0.0, -ds[1], 0.0, -ds[2], 0.0, de)
                            : perturb_elements(orbit, rd.el0, 0.0, -ds[0], 0.0, -ds[1], 0.0, -ds[2], de);
        if (!ok) {
            de[0] = de[1] = de[2] = de[3] = 0.0;
            const unsigned long long key = ((unsigned long long)s << 54) | ((unsigned long long)run << 46) |
                                           (0xffffull << 30) | (0xfull << 26) | ((unsigned long long)block << 2) | 3ull;
            atomicMin(&failure->key, key);
        }
    }
    if (!sum) return;
    __syncthreads();
    for (int t = threadIdx.x; t < nl + NITEMS * 4; t += blockDim.x) {   // ledger words [7 nf], then elements [7][4]
        const bool elements = t >= nl;
        const int k = elements ? t - nl : t;
        const size_t w = (size_t)block * (elements ? NITEMS * 4 : nl) + k;
        double* const* slots = elements ? rd.elements : rd.ledger;
        // the change of each stage; only the gas items perturb the orbit
        const double* change = elements ? (k < 16 ? stage_de + k : nullptr) : stage_ds + k;
        const size_t stage_stride = (size_t)rd.nblocks * (elements ? 16 : nl);
        double e[NSLOTS];
        e[start] = slots[start][w];
        int s = 0;
        auto stage = [&](int in, int base_slot, int out, double bf) {
            double v = e[in] + (change ? change[s * stage_stride] : 0.0);
            if (base_slot >= 0) v = v * (-bf + 1.0) + e[base_slot] * bf;
            e[out] = v;
            ++s;
        };
        // the schedule of plan_advance
        int base = start;
        for (int f = 0; f < fold; ++f) {
            if (rk == 1) {
                const int a = free_slot(start, base, -1);
                stage(base, -1, a, 0.0);
                base = a;
            } else if (rk == 2) {
                const int a = free_slot(start, base, -1);
                stage(base, -1, a, 0.0);
                const int b = free_slot(start, base, a);
                stage(a, base, b, 0.5);
                base = b;
            } else {
                const int a = free_slot(start, base, -1);
                stage(base, -1, a, 0.0);
                const int b = free_slot(start, base, a);
                stage(a, base, b, 0.75);
                const int c = free_slot(start, base, b);
                stage(b, base, c, 1.0 / 3.0);
                base = c;
            }
        }
        slots[base][w] = e[base];
    }
}

static int max_blocks(const b2d_ctx* ctx)
{
    int m = 0;
    for (const RunHost& r : ctx->runs) m = std::max(m, r.nblocks);
    return m;
}

static df32w split_df(double v)
{
    float hi = (float)v;
    float lo = (float)(v - (double)hi);
    return {hi, lo};
}

static b2d_status launch_stage(b2d_ctx* ctx, const StagePlan& sp, int stage, int amax_flag)
{
    StageArgs a;
    a.runs = ctx->rdev;
    a.tile_bases = ctx->d_bases;
    a.nruns = ctx->nruns;
    a.pf1 = ctx->rdev_h[0].pf;
    a.in_slot = sp.in;
    a.base_slot = sp.base;
    a.out_slot = sp.out;
    a.stage = stage;
    a.amax_flag = amax_flag;
    a.bf = sp.bf;
    a.half_avg = sp.bf == 0.5;
    a.w1f = split_df(-sp.bf + 1.0);
    a.bff = split_df(sp.bf);
    a.failure = ctx->d_failure;
    cudaError_t e;
    if (ctx->precision == B2D_PREC_FP64)
        e = launch_stage_f64(ctx->nf, a, ctx->total_tiles, stage_f64_smem(ctx->nf, ctx->sub_h, ctx->sub_w), ctx->stream);
    else
        e = (ctx->nf == 3 ? launch_stage_f32_iso : launch_stage_f32_euler)(store_of(ctx), side_divisor(ctx), a,
                                                                           ctx->total_tiles, ctx->stream);
    if (e != cudaSuccess) return fail(B2D_ERR_CUDA, std::string("stage kernel launch: ") + cudaGetErrorString(e));
    return B2D_OK;
}

// ---------------------------------------------------------------------------
// Massless tracer particles (no counterpart in the reference's code; its
// README names them).  dx/dt = v(x, t) with v the gas velocity of the stage
// input, bilinear between the four surrounding cell centres of the uniform
// mesh, advanced by the same RK stages and weighted averages as the state and
// wrapped into the periodic domain [-R, R)^2.  Positions are FP64.
//
// tracer_kernel<0> is the FP64 parity arithmetic; tracer_kernel<1> and <2>
// serve the FP32 paths (FP64 state, compensated state).  What bounds them is
// the gathers and the positions' traffic (a position 16 bytes read, its base
// read, its result written; 12 state words around each tracer), so FP64 work,
// at two lanes per clock and SM, is kept out: cell and offset come from the
// position as a double-float, the displacement and the base's average too,
// and what is left are the additions to the FP64 positions, two per
// coordinate at most, and an integer compare for the periodic wrap.  Measured
// at 8192^2 with 1e7 tracers: a launch takes 146 us (179 with a base),
// about 600 when these steps were FP64 conversions and quotients.
template <int STORE> __device__ __forceinline__ float2 tracer_velocity_f32(const RunDev& rd, int slot, size_t idx)
{
    const size_t nn = (size_t)rd.N * rd.N;
    float u[3];
    for (int f = 0; f < 3; ++f) {
        if (STORE == 1) u[f] = narrow(((const double*)rd.slot[slot])[f * nn + idx]);
        else u[f] = ((const float*)rd.slot[slot])[(2 * f) * nn + idx];
    }
    const float ir = __fdividef(1.0f, u[0]);
    return make_float2(u[1] * ir, u[2] * ir);
}

// The cell centre below coordinate v (as hi + lo) and the offset from it in
// cells: (v + R) / dx - 1/2 = i + a.
__device__ __forceinline__ void tracer_cell(float hi, float lo, float2 R, float2 inv_dx, int& i, float& a)
{
    // s + e = v + R
    const float s = __fadd_rn(hi, R.x), bb = __fadd_rn(s, -hi);
    const float e = __fadd_rn(__fadd_rn(__fadd_rn(hi, -__fadd_rn(s, -bb)), __fadd_rn(R.x, -bb)), __fadd_rn(lo, R.y));
    const float p = __fmul_rn(s, inv_dx.x);
    const float q = __fmaf_rn(e, inv_dx.x, __fmaf_rn(s, inv_dx.y, __fmaf_rn(s, inv_dx.x, -p)));
    const float g = __fadd_rn(p, -0.5f), fl = floorf(g);
    i = (int)fl;
    a = __fadd_rn(__fadd_rn(g, -fl), q);
    // p's rounding can put a position on the wrong side of a cell's edge
    if (a < 0.0f) { --i; a += 1.0f; } else if (a >= 1.0f) { ++i; a -= 1.0f; }
}

static __device__ __noinline__ double tracer_wrap(double xo, double R)
{
    if (xo >= R) xo -= 2.0 * R;
    if (xo < -R) xo += 2.0 * R;
    return xo;
}

// x + (hi + lo), or with a base xb + w (x + (hi + lo) - xb) on the base's
// periodic image, wrapped into [-R, R).
__device__ __forceinline__ double tracer_move(double x, float xh, float xl, float d, bool has_base, double xb, float2 w,
                                              double R, float2 Rf)
{
    double xo;
    if (!has_base) xo = x + widen(d);
    else {
        float bh, bl;
        split_double(xb, bh, bl);
        // h + l = x - xb + d
        float dd = __fadd_rn(xh, -bh);
        const float ee = __fadd_rn(dd, -xh);
        float l = __fadd_rn(__fadd_rn(__fadd_rn(xh, -__fadd_rn(dd, -ee)), -__fadd_rn(bh, ee)), __fadd_rn(xl, -bl));
        // (exact in the high word; the radius has a low one too)
        if (dd > Rf.x) { dd = __fadd_rn(dd, -2.0f * Rf.x); l = __fadd_rn(l, -2.0f * Rf.y); }
        else if (dd < -Rf.x) { dd = __fadd_rn(dd, 2.0f * Rf.x); l = __fadd_rn(l, 2.0f * Rf.y); }
        const float h = __fadd_rn(dd, d), bb = __fadd_rn(h, -dd);
        l = __fadd_rn(l, __fadd_rn(__fadd_rn(dd, -__fadd_rn(h, -bb)), __fadd_rn(d, -bb)));
        // times w
        const float p = __fmul_rn(h, w.x);
        const float q = __fmaf_rn(l, w.x, __fmaf_rn(h, w.y, __fmaf_rn(h, w.x, -p)));
        xo = (xb + widen(p)) + widen(q);
    }
    const unsigned long long m = (unsigned long long)__double_as_longlong(xo) & 0x7fffffffffffffffull;
    return m >= (unsigned long long)__double_as_longlong(R) ? tracer_wrap(xo, R) : xo;
}

// MODE 0: FP64 arithmetic on the FP64 state; 1, 2: FP32 arithmetic on the FP64, compensated state.
// bf: the base's weight; w: 1 - bf as FP32 high and low words.
template <int MODE>
__global__ void __launch_bounds__(256) tracer_kernel(const RunDev* runs, int run, int in_slot, int base_slot, int out_slot,
                                                     double bf, float2 w, const Failure* failure)
{
    const RunDev& rd = runs[run];
    const long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (k >= rd.ntracers || failure->abandoned) return;
    const double R = rd.p.domain_radius, dx = rd.p.dx, dt = *rd.dt;
    const int N = rd.N;
    const double2 at = ((const double2*)rd.tracers[in_slot])[k];
    double2 base = make_double2(0.0, 0.0);
    if (base_slot >= 0) base = ((const double2*)rd.tracers[base_slot])[k];
    int i0, j0;
    double gx = 0.0, gy = 0.0;
    float ax = 0.0f, ay = 0.0f, xh = 0.0f, xl = 0.0f, yh = 0.0f, yl = 0.0f;
    if constexpr (MODE == 0) {
        // the oracle's arithmetic
        gx = (at.x + R) / dx - 0.5;
        gy = (at.y + R) / dx - 0.5;
        const double fi = floor(gx), fj = floor(gy);
        gx = gx - fi;
        gy = gy - fj;
        i0 = (int)fi;
        j0 = (int)fj;
    } else {
        split_double(at.x, xh, xl);
        split_double(at.y, yh, yl);
        tracer_cell(xh, xl, rd.tracer_radius, rd.tracer_inv_dx, i0, ax);
        tracer_cell(yh, yl, rd.tracer_radius, rd.tracer_inv_dx, j0, ay);
    }
    // positions are kept in [-R, R), so the cell index is in [-1, N - 1]: one
    // conditional wrap, then a clamp that keeps any other input in bounds
    i0 = i0 < 0 ? i0 + N : i0;
    j0 = j0 < 0 ? j0 + N : j0;
    i0 = min(max(i0, 0), N - 1);
    j0 = min(max(j0, 0), N - 1);
    const int i1 = i0 + 1 == N ? 0 : i0 + 1, j1 = j0 + 1 == N ? 0 : j0 + 1;
    const size_t c00 = (size_t)i0 * N + j0, c01 = (size_t)i0 * N + j1, c10 = (size_t)i1 * N + j0, c11 = (size_t)i1 * N + j1;
    double xo, yo;
    if constexpr (MODE == 0) {
        const size_t nn = (size_t)N * N;
        const double* u = (const double*)rd.slot[in_slot];
        auto vel = [&](size_t c, double& vx, double& vy) {
            vx = u[nn + c] / u[c];
            vy = u[2 * nn + c] / u[c];
        };
        double v00x, v00y, v10x, v10y, v01x, v01y, v11x, v11y;
        vel(c00, v00x, v00y);
        vel(c10, v10x, v10y);
        vel(c01, v01x, v01y);
        vel(c11, v11x, v11y);
        const double w00 = (1.0 - gx) * (1.0 - gy), w10 = gx * (1.0 - gy), w01 = (1.0 - gx) * gy, w11 = gx * gy;
        const double L = 2.0 * R;
        xo = at.x + dt * (w00 * v00x + w10 * v10x + w01 * v01x + w11 * v11x);
        yo = at.y + dt * (w00 * v00y + w10 * v10y + w01 * v01y + w11 * v11y);
        if (base_slot >= 0) {
            // average with the base position on the same periodic image
            if (xo - base.x > R) xo -= L;
            else if (xo - base.x < -R) xo += L;
            if (yo - base.y > R) yo -= L;
            else if (yo - base.y < -R) yo += L;
            xo = xo * (-bf + 1.0) + base.x * bf;
            yo = yo * (-bf + 1.0) + base.y * bf;
        }
        if (xo >= R) xo -= L;
        if (xo < -R) xo += L;
        if (yo >= R) yo -= L;
        if (yo < -R) yo += L;
    } else {
        const float2 v00 = tracer_velocity_f32<MODE>(rd, in_slot, c00), v10 = tracer_velocity_f32<MODE>(rd, in_slot, c10);
        const float2 v01 = tracer_velocity_f32<MODE>(rd, in_slot, c01), v11 = tracer_velocity_f32<MODE>(rd, in_slot, c11);
        const float bx = 1.0f - ax, by = 1.0f - ay;
        const float w00 = bx * by, w10 = ax * by, w01 = bx * ay, w11 = ax * ay;
        const float vx = w00 * v00.x + w10 * v10.x + w01 * v01.x + w11 * v11.x;
        const float vy = w00 * v00.y + w10 * v10.y + w01 * v01.y + w11 * v11.y;
        const float dtf = narrow(dt);
        const float2 Rf = rd.tracer_radius;
        xo = tracer_move(at.x, xh, xl, dtf * vx, base_slot >= 0, base.x, w, R, Rf);
        yo = tracer_move(at.y, yh, yl, dtf * vy, base_slot >= 0, base.y, w, R, Rf);
    }
    ((double2*)rd.tracers[out_slot])[k] = make_double2(xo, yo);
}

static b2d_status launch_tracers(b2d_ctx* ctx, const StagePlan& sp, bool count)
{
    const df32w keep = split_df(-sp.bf + 1.0);
    const float2 w = make_float2(keep.hi, keep.lo);   // the new position's weight
    for (int r = 0; r < ctx->nruns; ++r) {
        const long long n = ctx->rdev_h[r].ntracers;
        if (n <= 0) continue;
        const int threads = 256;
        const unsigned grid = (unsigned)((n + threads - 1) / threads);
        if (ctx->precision == B2D_PREC_FP64)
            tracer_kernel<0><<<grid, threads, 0, ctx->stream>>>(ctx->rdev, r, sp.in, sp.base, sp.out, sp.bf, w, ctx->d_failure);
        else if (ctx->precision == B2D_PREC_FP32_STATE64)
            tracer_kernel<1><<<grid, threads, 0, ctx->stream>>>(ctx->rdev, r, sp.in, sp.base, sp.out, sp.bf, w, ctx->d_failure);
        else
            tracer_kernel<2><<<grid, threads, 0, ctx->stream>>>(ctx->rdev, r, sp.in, sp.base, sp.out, sp.bf, w, ctx->d_failure);
        CUDA_TRY(cudaGetLastError());
        if (count) ctx->launches++;
    }
    return B2D_OK;
}

// Stages [first, last) of the advance's ledgers, and with `sum` the sums over its stages.
static b2d_status launch_ledgers(b2d_ctx* ctx, int first, int last, bool sum, int fold, int start, bool count)
{
    const int nl = NITEMS * ctx->nf, work = std::max((last - first) * nl, nl + NITEMS * 4);
    const int threads = std::min((work + 31) / 32 * 32, 256);
    ledger_kernel<<<dim3((unsigned)max_blocks(ctx), (unsigned)ctx->nruns), threads, 0, ctx->stream>>>(
        ctx->rdev, first, last, sum, fold, ctx->rk, start, ctx->d_failure);
    CUDA_TRY(cudaGetLastError());
    if (count) ctx->launches++;
    return B2D_OK;
}

// The first of the stages up to s whose pieces are to be folded after it, or -1.
static int fold_due(const b2d_ctx* ctx, int s, int nstages)
{
    const int first = s / ctx->stage_window * ctx->stage_window;
    return s + 1 == nstages || s + 1 == first + ctx->stage_window ? first : -1;
}

static b2d_status enqueue_advance(b2d_ctx* ctx, int fold, int start, int* final_slot, bool count)
{
    std::vector<StagePlan> plan = plan_advance(ctx->rk, fold, start, final_slot);
    prologue_kernel<<<ctx->nruns, 32, 0, ctx->stream>>>(ctx->rdev, fold, ctx->rk, start, *final_slot, ctx->d_failure,
                                                         ctx->d_adv_count);
    CUDA_TRY(cudaGetLastError());
    if (count) ctx->launches++;
    for (size_t s = 0; s < plan.size(); ++s) {
        bool timed = ctx->instrument;
        if (timed) {
            while (ctx->ev.size() < 2 * plan.size()) {
                cudaEvent_t e;
                CUDA_TRY(cudaEventCreate(&e));
                ctx->ev.push_back(e);
            }
            CUDA_TRY(cudaEventRecord(ctx->ev[2 * s], ctx->stream));
        }
        b2d_status st = launch_stage(ctx, plan[s], (int)s, s + 1 == plan.size());
        if (st != B2D_OK) return st;
        if (timed) CUDA_TRY(cudaEventRecord(ctx->ev[2 * s + 1], ctx->stream));
        if (count) ctx->launches++;
        st = launch_tracers(ctx, plan[s], count);
        if (st != B2D_OK) return st;
        const int first = fold_due(ctx, (int)s, (int)plan.size());
        if (first >= 0) st = launch_ledgers(ctx, first, (int)s + 1, s + 1 == plan.size(), fold, start, count);
        if (st != B2D_OK) return st;
    }
    return B2D_OK;
}

extern "C" b2d_status b2d_set_tracers(b2d_ctx* ctx, int32_t run, int64_t n, const double* xy)
{
    if (!ctx || run < 0 || run >= ctx->nruns || n < 0 || (n > 0 && !xy)) return fail(B2D_ERR_INVALID, "bad arguments");
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    RunDev& d = ctx->rdev_h[run];
    for (int s = 0; s < NSLOTS; ++s) {
        CUDA_TRY(cudaFree(d.tracers[s]));
        d.tracers[s] = nullptr;
    }
    d.ntracers = 0;
    if (n > 0) {
        for (int s = 0; s < NSLOTS; ++s) CUDA_TRY(cudaMalloc(&d.tracers[s], sizeof(double) * 2 * (size_t)n));
        CUDA_TRY(cudaMemcpyAsync(d.tracers[ctx->cur], xy, sizeof(double) * 2 * (size_t)n, cudaMemcpyHostToDevice, ctx->stream));
        d.ntracers = n;
    }
    CUDA_TRY(cudaMemcpyAsync(ctx->rdev, ctx->rdev_h.data(), sizeof(RunDev) * ctx->nruns, cudaMemcpyHostToDevice, ctx->stream));
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    for (auto& kv : ctx->graphs) cudaGraphExecDestroy(kv.second);
    ctx->graphs.clear();
    return B2D_OK;
}

extern "C" b2d_status b2d_get_tracers(b2d_ctx* ctx, int32_t run, double* xy)
{
    if (!ctx || run < 0 || run >= ctx->nruns || !xy) return fail(B2D_ERR_INVALID, "bad arguments");
    const RunDev& d = ctx->rdev_h[run];
    if (d.ntracers > 0)
        CUDA_TRY(cudaMemcpyAsync(xy, d.tracers[ctx->cur], sizeof(double) * 2 * (size_t)d.ntracers,
                                 cudaMemcpyDeviceToHost, ctx->stream));
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    return B2D_OK;
}

static b2d_status run_advance(b2d_ctx* ctx, int fold, int* final_slot)
{
    if (fold * ctx->rk > 1023) return fail(B2D_ERR_INVALID, "fold x rk_order must be at most 1023");
    b2d_status st = ensure_stage_capacity(ctx, fold);
    if (st != B2D_OK) return st;
    const int start = ctx->cur;
    {
        int fs;
        ctx->window.emplace_back(start, plan_advance(ctx->rk, fold, start, &fs));
    }
    if (!ctx->use_graphs || ctx->instrument) {
        st = enqueue_advance(ctx, fold, start, final_slot, true);
        if (st != B2D_OK) return st;
        if (ctx->instrument) {
            CUDA_TRY(cudaStreamSynchronize(ctx->stream));
            for (int s = 0; s < fold * ctx->rk; ++s) {
                float ms = 0;
                CUDA_TRY(cudaEventElapsedTime(&ms, ctx->ev[2 * s], ctx->ev[2 * s + 1]));
                ctx->stage_ms_total += ms;
                ctx->stage_count++;
            }
        }
        return B2D_OK;
    }
    auto key = std::make_pair(fold, start);
    auto it = ctx->graphs.find(key);
    if (it == ctx->graphs.end()) {
        cudaGraph_t g;
        CUDA_TRY(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        st = enqueue_advance(ctx, fold, start, final_slot, false);
        cudaError_t ec = cudaStreamEndCapture(ctx->stream, &g);
        if (st != B2D_OK) return st;
        if (ec != cudaSuccess) return fail(B2D_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(ec));
        cudaGraphExec_t ge;
        CUDA_TRY(cudaGraphInstantiate(&ge, g, 0));
        cudaGraphDestroy(g);
        it = ctx->graphs.emplace(key, ge).first;
    } else {
        plan_advance(ctx->rk, fold, start, final_slot);
    }
    CUDA_TRY(cudaGraphLaunch(it->second, ctx->stream));
    ctx->launches += b2d_launches_per_advance(ctx, fold);
    return B2D_OK;
}

// Host restatement of try_to_primitive's failure value (physics.rs:489-503,
// 631-660) for the zone named by a failure key.
static double failure_value(const b2d_config& c, const double* u, int code)
{
    if (c.hydro_kind == B2D_ISOTHERMAL) return u[0];
    double g = c.gamma_law_index;
    double p[4] = {u[0], u[1] / u[0], u[2] / u[0], 0.0};
    p[3] = (u[3] - 0.5 * u[0] * (p[1] * p[1] + p[2] * p[2])) * (g - 1.0);
    if (c.has_density_floor && p[0] < c.density_floor) {
        p[0] = c.density_floor; p[1] = 0.0; p[2] = 0.0; p[3] = pow(c.density_floor, g);
    }
    if (code == 1) return p[0];
    if (c.has_pressure_floor && p[3] < c.pressure_floor) p[3] = c.pressure_floor;
    return p[3];
}

// A copy to the host in the order of `stream`, waited for.
static cudaError_t read_back(void* dst, const void* src, size_t bytes, cudaStream_t stream)
{
    const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream);
    return e != cudaSuccess ? e : cudaStreamSynchronize(stream);
}

static b2d_status decode_failure(b2d_ctx* ctx, unsigned long long key, const std::vector<StagePlan>& plan,
                                 b2d_error* e)
{
    memset(e, 0, sizeof *e);
    const int stage = (int)(key >> 54);
    const int run = (int)((key >> 46) & 0xff);
    const int blk = (int)((key >> 30) & 0xffff);
    const int order = (int)((key >> 26) & 0xf);
    const int zone = (int)((key >> 2) & 0xffffff);
    e->code = (int)(key & 3);
    e->run = run;
    RunHost& r = ctx->runs[run];
    const int nb = r.nb, bs = r.bs;
    double orb[10];
    if (e->code == B2D_ERR_UNBOUND_ORBIT) {
        // OrbitalEvolutionError is reported at position (0, 0) (scheme.rs:308-309);
        // the failing block's index is carried in the zone field.
        e->block_i = zone / nb;
        e->block_j = zone % nb;
        CUDA_TRY(read_back(&e->time, r.stage_time + stage, sizeof(double), ctx->stream));
        CUDA_TRY(read_back(orb, r.orbit + 10 * stage, sizeof orb, ctx->stream));
        e->binary[0] = orb[1]; e->binary[1] = orb[2]; e->binary[2] = orb[6]; e->binary[3] = orb[7];
        return B2D_OK;
    }
    const int bi = blk / nb, bj = blk % nb, di = order / 3 - 1, dj = order % 3 - 1;
    e->block_i = (bi + di + nb) % nb;
    e->block_j = (bj + dj + nb) % nb;
    e->zone_i = zone / bs;
    e->zone_j = zone % bs;
    const int gi = e->block_i * bs + e->zone_i, gj = e->block_j * bs + e->zone_j;
    e->x = r.hxc[gi];
    e->y = r.hxc[gj];
    const size_t nn = (size_t)r.N * r.N, idx = (size_t)gi * r.N + gj;
    const int slot = plan.at(stage).in;
    double u[4] = {0, 0, 0, 0};
    for (int f = 0; f < ctx->nf; ++f) {
        if (store_of(ctx) == 0) {
            CUDA_TRY(read_back(&u[f], (const double*)r.slot[slot] + f * nn + idx, sizeof(double), ctx->stream));
        } else {
            float hl[2];
            CUDA_TRY(read_back(&hl[0], (const float*)r.slot[slot] + (2 * f) * nn + idx, sizeof(float), ctx->stream));
            CUDA_TRY(read_back(&hl[1], (const float*)r.slot[slot] + (2 * f + 1) * nn + idx, sizeof(float), ctx->stream));
            u[f] = (double)hl[0] + (double)hl[1];
        }
    }
    e->value = failure_value(r.cfg, u, e->code);
    CUDA_TRY(read_back(&e->time, r.stage_time + stage, sizeof(double), ctx->stream));
    CUDA_TRY(read_back(orb, r.orbit + 10 * stage, sizeof orb, ctx->stream));
    e->binary[0] = orb[1]; e->binary[1] = orb[2]; e->binary[2] = orb[6]; e->binary[3] = orb[7];
    return B2D_OK;
}

static b2d_status finish_advance(b2d_ctx* ctx, int final_slot, double* dt_out, b2d_error* err_out)
{
    const ControlRead control(ctx);
    if (control.status != B2D_OK) return control.status;
    const unsigned long long key = control(&ctx->d_failure->key);
    const long long count = control(ctx->d_adv_count);
    auto window = std::move(ctx->window);
    ctx->window.clear();
    const long long base = ctx->adv_base;
    ctx->adv_base = count;
    for (int r = 0; dt_out && r < ctx->nruns; ++r) dt_out[r] = control(ctx->d_dt + r);
    if (key != ~0ull) {
        // the failing advance is the last one whose prologue ran
        long long k = count - 1 - base;
        if (k < 0 || k >= (long long)window.size()) return fail(B2D_ERR_CUDA, "failure bookkeeping lost");
        const int start = window[k].first;
        b2d_error err;
        b2d_status s = decode_failure(ctx, key, window[k].second, &err);
        if (s != B2D_OK) return s;
        if (err_out) *err_out = err;
        CUDA_TRY(cudaMemsetAsync(&ctx->d_failure->key, 0xff, sizeof(unsigned long long), ctx->stream));
        ctx->cur = start;
        for (int r = 0; r < ctx->nruns; ++r) {
            s = launch_max_speed(ctx, r, start);
            if (s != B2D_OK) return s;
        }
        CUDA_TRY(cudaStreamSynchronize(ctx->stream));
        return fail((b2d_status)err.code, "hydro error during advance");
    }
    if (final_slot >= 0) ctx->cur = final_slot;
    return B2D_OK;
}

extern "C" b2d_status b2d_advance(b2d_ctx* ctx, int32_t fold, double* dt_out, b2d_error* err_out)
{
    if (!ctx || fold < 1) return fail(B2D_ERR_INVALID, "bad arguments");
    int final_slot = -1;
    b2d_status st = run_advance(ctx, fold, &final_slot);
    if (st != B2D_OK) return st;
    return finish_advance(ctx, final_slot, dt_out, err_out);
}

extern "C" b2d_status b2d_advance_async(b2d_ctx* ctx, int32_t fold)
{
    if (!ctx || fold < 1) return fail(B2D_ERR_INVALID, "bad arguments");
    int final_slot = -1;
    b2d_status st = run_advance(ctx, fold, &final_slot);
    if (st != B2D_OK) return st;
    ctx->cur = final_slot;
    return B2D_OK;
}

extern "C" b2d_status b2d_synchronize(b2d_ctx* ctx, double* dt_out, b2d_error* err_out)
{
    if (!ctx) return fail(B2D_ERR_INVALID, "bad arguments");
    return finish_advance(ctx, -1, dt_out, err_out);
}

extern "C" b2d_status b2d_set_tile(b2d_ctx* ctx, int32_t tile_w, int32_t tile_h)
{
    if (!ctx) return fail(B2D_ERR_INVALID, "bad arguments");
    int tw = tile_w ? tile_w : ctx->tw, th = tile_h ? tile_h : ctx->th;
    if (!tile_ok(ctx, tw, th)) return fail(B2D_ERR_INVALID, "tile must divide the block size (width a multiple of 32, at most 256)");
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    ctx->tw = tw;
    ctx->th = th;
    return sync_rundev(ctx);
}

extern "C" b2d_status b2d_get_tile(const b2d_ctx* ctx, int32_t* tile_w, int32_t* tile_h)
{
    if (!ctx) return fail(B2D_ERR_INVALID, "bad arguments");
    if (tile_w) *tile_w = ctx->tw;
    if (tile_h) *tile_h = ctx->th;
    return B2D_OK;
}

extern "C" b2d_status b2d_set_strip_rows(b2d_ctx* ctx, int32_t rows)
{
    if (!ctx || rows < 0) return fail(B2D_ERR_INVALID, "bad arguments");
    if (rows > 0) {
        if (rows < 8) return fail(B2D_ERR_INVALID, "strip rows must be 0 or at least 8");
        for (const RunHost& r : ctx->runs)
            if (rows > r.bs) return fail(B2D_ERR_INVALID, "strip rows must not exceed the block size");
    }
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    ctx->strip_rows = rows;
    return sync_rundev(ctx);
}

extern "C" b2d_status b2d_get_strip_rows(const b2d_ctx* ctx, int32_t* rows)
{
    if (!ctx || !rows) return fail(B2D_ERR_INVALID, "bad arguments");
    *rows = ctx->strip_rows;
    return B2D_OK;
}

extern "C" b2d_status b2d_set_graphs(b2d_ctx* ctx, int32_t enable)
{
    if (!ctx) return fail(B2D_ERR_INVALID, "bad arguments");
    ctx->use_graphs = enable != 0;
    return B2D_OK;
}

extern "C" int64_t b2d_launch_count(const b2d_ctx* ctx) { return ctx ? ctx->launches : 0; }

extern "C" int64_t b2d_launches_per_advance(const b2d_ctx* ctx, int32_t fold)
{
    if (!ctx) return 0;
    int with_tracers = 0;
    for (const RunDev& d : ctx->rdev_h) with_tracers += d.ntracers > 0 ? 1 : 0;
    const int64_t stages = (int64_t)fold * ctx->rk, window = std::min<int64_t>(ctx->stage_window, stages);
    return 1 + (stages + window - 1) / window + stages * (1 + with_tracers);
}

extern "C" b2d_status b2d_set_instrument(b2d_ctx* ctx, int32_t enable)
{
    if (!ctx) return fail(B2D_ERR_INVALID, "bad arguments");
    ctx->instrument = enable != 0;
    ctx->stage_ms_total = 0.0;
    ctx->stage_count = 0;
    return B2D_OK;
}

extern "C" b2d_status b2d_stage_stats(const b2d_ctx* ctx, int64_t* count, double* total_ms)
{
    if (!ctx) return fail(B2D_ERR_INVALID, "bad arguments");
    if (count) *count = ctx->stage_count;
    if (total_ms) *total_ms = ctx->stage_ms_total;
    return B2D_OK;
}

extern "C" b2d_status b2d_time_stages(b2d_ctx* ctx, int32_t fold, int32_t reps, double* ms_per_stage)
{
    if (!ctx || fold < 1 || reps < 1 || !ms_per_stage) return fail(B2D_ERR_INVALID, "bad arguments");
    bool was = ctx->instrument;
    b2d_set_instrument(ctx, 1);
    for (int r = 0; r < reps; ++r) {
        int fs;
        b2d_status st = run_advance(ctx, fold, &fs);
        if (st != B2D_OK) { ctx->instrument = was; return st; }
        ctx->cur = fs;
    }
    *ms_per_stage = ctx->stage_count ? ctx->stage_ms_total / ctx->stage_count : 0.0;
    ctx->instrument = was;
    return B2D_OK;
}

extern "C" b2d_status b2d_stream(const b2d_ctx* ctx, void** stream)
{
    if (!ctx || !stream) return fail(B2D_ERR_INVALID, "bad arguments");
    *stream = (void*)ctx->stream;
    return B2D_OK;
}

extern "C" b2d_status b2d_pin_host(void* ptr, uint64_t bytes)
{
    CUDA_TRY(cudaHostRegister(ptr, bytes, cudaHostRegisterDefault));
    return B2D_OK;
}

extern "C" b2d_status b2d_unpin_host(void* ptr)
{
    CUDA_TRY(cudaHostUnregister(ptr));
    return B2D_OK;
}

extern "C" b2d_status b2d_set_device(int32_t device)
{
    CUDA_TRY(cudaSetDevice(device));
    return B2D_OK;
}

// ---------------------------------------------------------------------------
// Tile autotuner: time every tile shape that divides the block size with CUDA
// events on the context's stream, keep the fastest.  The advances run from
// the current slot, which the slot schedule never overwrites, so the state is
// unchanged afterwards (the max signal speed is recomputed).  A tiling that is
// a quarter slower than `best` in its warm-up, or a twentieth in a repetition,
// is not repeated.
static b2d_status time_tile(b2d_ctx* ctx, int fold, int reps, double best, double* ms)
{
    ctx->instrument = true;
    ctx->stage_ms_total = 0.0;
    ctx->stage_count = 0;
    for (int r = 0; r < reps + 1; ++r) {
        int fs;
        std::vector<StagePlan> plan = plan_advance(ctx->rk, fold, ctx->cur, &fs);
        b2d_status st = enqueue_advance(ctx, fold, ctx->cur, &fs, true);
        if (st != B2D_OK) { ctx->instrument = false; return st; }
        CUDA_TRY(cudaStreamSynchronize(ctx->stream));
        double total = 0.0;
        for (size_t s = 0; s < plan.size(); ++s) {
            float m = 0;
            CUDA_TRY(cudaEventElapsedTime(&m, ctx->ev[2 * s], ctx->ev[2 * s + 1]));
            total += m;
        }
        if (r > 0) {
            ctx->stage_ms_total += total;
            ctx->stage_count += (long long)plan.size();
        }
        *ms = r > 0 ? ctx->stage_ms_total / ctx->stage_count : total / plan.size();
        if (*ms > best * (r > 0 ? 1.05 : 1.25)) break;
    }
    ctx->instrument = false;
    return B2D_OK;
}

// CTAs of the FP32 stage kernel that the GPU holds at once.
static long long resident_ctas(const b2d_ctx* ctx)
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return (long long)sms * (ctx->nf == 3 ? resident_f32_iso : resident_f32_euler)(store_of(ctx), side_divisor(ctx), ctx->nruns);
}

// CTAs of a launch with row chunks of at most `rows` rows.
static long long chunk_ctas(const b2d_ctx* ctx, int rows)
{
    long long n = 0;
    for (const RunHost& r : ctx->runs)
        n += (long long)((r.N + rows - 1) / rows) * ((r.N + STRIP_COLS - 1) / STRIP_COLS);
    return n;
}

// Strip rows to try: for the fewest whole waves of resident CTAs that chunks of
// at most a block's rows fill, and the next two, the shortest chunks that
// still fit in them.  Within a wave, so too for every whole number of one-warp
// CTAs per scheduler (four per SM): one warp more than that makes its scheduler
// the last (Euler 768^2: 27.2 us a stage in 1248 chunks of 8 rows, 26.1 in 1118
// of 9, with 1216 two to a scheduler; at 1024^2, 38.0 us in 11 rows, the wave's
// last, and 52.7 in 10).
static std::vector<int> strip_row_candidates(const b2d_ctx* ctx)
{
    std::vector<int> out;
    const long long slots = resident_ctas(ctx);
    if (slots <= 0) return out;
    int min_bs = 1 << 30;
    for (const RunHost& r : ctx->runs) min_bs = std::min(min_bs, r.bs);
    auto shortest = [&](long long ctas) {
        int best = 0;
        for (int rows = min_bs; rows >= 8 && chunk_ctas(ctx, rows) <= ctas; --rows) best = rows;
        if (best && std::find(out.begin(), out.end(), best) == out.end()) out.push_back(best);
    };
    long long waves = (chunk_ctas(ctx, min_bs) + slots - 1) / slots;
    for (int c = 0; c < 3; ++c, ++waves) shortest(waves * slots);
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return out;
    for (long long ctas = slots - 4 * sms; ctas > 0; ctas -= 4 * sms) shortest(ctas);
    return out;
}

// A candidate replaces the fastest so far only when it is faster by more than
// timing noise, so that the choice is the same from run to run.
constexpr double AUTOTUNE_MARGIN = 0.99;

extern "C" b2d_status b2d_autotune(b2d_ctx* ctx, int32_t fold, int32_t reps, int32_t* tile_w, int32_t* tile_h,
                                   double* ms_per_stage)
{
    if (!ctx || fold < 1 || reps < 1) return fail(B2D_ERR_INVALID, "bad arguments");
    b2d_status st = ensure_stage_capacity(ctx, fold);
    if (st != B2D_OK) return st;
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    int best_w = ctx->tw, best_h = ctx->th, best_rows = 0;
    double best = 1e300;
    auto trial = [&](int th, int rows) -> b2d_status {
        ctx->th = th;
        ctx->strip_rows = rows;
        b2d_status s = sync_rundev(ctx);
        double ms = 0;
        if (s == B2D_OK) s = time_tile(ctx, fold, reps, best, &ms);
        if (s == B2D_OK && ms < best * AUTOTUNE_MARGIN) { best = ms; best_h = th; best_rows = rows; }
        return s;
    };
    if (ctx->precision == B2D_PREC_FP64) {   // one tiling, whatever the tile shape
        st = trial(ctx->th, 0);
        if (st != B2D_OK) return st;
    } else {
        // block-aligned chunks: every height that divides the blocks, but not
        // so many chunks that they queue up behind one another, and none above
        // one whose chunks take up half the GPU (they would only be longer), nor
        // below a quarter of one that still fills it (four guard rows a chunk)
        const long long slots = resident_ctas(ctx);
        auto divides = [&](int h) {
            return std::all_of(ctx->runs.begin(), ctx->runs.end(), [h](const RunHost& r) { return r.bs % h == 0; });
        };
        int tallest = 128;   // of those that divide the blocks of every run: it is always tried
        while (!divides(tallest)) --tallest;
        for (int h = 1; h <= tallest; ++h) {
            if (!divides(h)) continue;
            if (h < 16 && 2 * h <= tallest && chunk_ctas(ctx, h) > 2 * slots) continue;
            if (4 * h <= tallest && chunk_ctas(ctx, 4 * h) > slots) continue;
            st = trial(h, 0);
            if (st != B2D_OK) return st;
            if (2 * chunk_ctas(ctx, h) <= slots) break;
        }
        // chunks that cross block rows and fill whole waves
        const int h = best_h;
        for (int rows : strip_row_candidates(ctx)) {
            st = trial(h, rows);
            if (st != B2D_OK) return st;
        }
    }
    // discard what the trial advances left behind
    long long count = 0;
    CUDA_TRY(read_back(&count, ctx->d_adv_count, sizeof count, ctx->stream));
    ctx->adv_base = count;
    ctx->window.clear();
    CUDA_TRY(cudaMemsetAsync(&ctx->d_failure->key, 0xff, sizeof(unsigned long long), ctx->stream));
    ctx->tw = best_w;
    ctx->th = best_h;
    ctx->strip_rows = best_rows;
    st = sync_rundev(ctx);
    if (st != B2D_OK) return st;
    for (int r = 0; r < ctx->nruns; ++r) {
        st = launch_max_speed(ctx, r, ctx->cur);
        if (st != B2D_OK) return st;
    }
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    if (tile_w) *tile_w = best_w;
    if (tile_h) *tile_h = best_h;
    if (ms_per_stage) *ms_per_stage = best;
    return B2D_OK;
}

// ---------------------------------------------------------------------------
// Row slabs: one run split across contexts (one per GPU or process), each of
// which advances the blocks of its own block rows.  No counterpart in the
// reference, which advances every block of a run in one process; its block
// dataflow joins each block with its 3x3 neighbours and extends a 2-zone
// halo (src/scheme.rs:119-133, periodic neighbours src/mesh.rs:101-110), so a
// slab needs the 2 zone rows on either side of it from the neighbouring slabs
// before every stage, the global maximum signal speed for dt once per
// advance, and its blocks' ledgers summed with the others' by the caller.

extern "C" b2d_status b2d_set_slab(b2d_ctx* ctx, int32_t run, int32_t block_row_lo, int32_t block_row_hi)
{
    if (!ctx || run < 0 || run >= ctx->nruns) return fail(B2D_ERR_INVALID, "bad arguments");
    RunDev& d = ctx->rdev_h[run];
    const bool whole = block_row_lo == 0 && block_row_hi == 0;
    if (!whole && (block_row_lo < 0 || block_row_hi > d.nb || block_row_lo >= block_row_hi))
        return fail(B2D_ERR_INVALID, "slab rows must satisfy 0 <= lo < hi <= num_blocks");
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    d.slab_lo = whole ? 0 : block_row_lo;
    d.slab_hi = whole ? 0 : block_row_hi;
    b2d_status st = sync_rundev(ctx);
    if (st != B2D_OK) return st;
    // the stored maximum signal speed becomes the slab's
    st = launch_max_speed(ctx, run, ctx->cur);
    if (st != B2D_OK) return st;
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    return B2D_OK;
}

extern "C" b2d_status b2d_slab_begin(b2d_ctx* ctx, int32_t fold, const double* amax)
{
    if (!ctx || fold < 1 || !amax) return fail(B2D_ERR_INVALID, "bad arguments");
    if (ctx->slab_next >= 0) return fail(B2D_ERR_INVALID, "a slab advance is already in progress");
    if (fold * ctx->rk > 1023) return fail(B2D_ERR_INVALID, "fold x rk_order must be at most 1023");
    b2d_status st = ensure_stage_capacity(ctx, fold);
    if (st != B2D_OK) return st;
    // dt comes from the maximum signal speed over every slab of each run
    std::vector<unsigned long long> bits(ctx->nruns);
    memcpy(bits.data(), amax, sizeof(double) * ctx->nruns);
    CUDA_TRY(cudaMemcpyAsync(ctx->d_amax, bits.data(), sizeof(unsigned long long) * ctx->nruns, cudaMemcpyHostToDevice,
                             ctx->stream));
    const int start = ctx->cur;
    ctx->slab_plan = plan_advance(ctx->rk, fold, start, &ctx->slab_final);
    ctx->slab_fold = fold;
    ctx->slab_start = start;
    ctx->slab_next = 0;
    ctx->window.emplace_back(start, ctx->slab_plan);
    prologue_kernel<<<ctx->nruns, 32, 0, ctx->stream>>>(ctx->rdev, fold, ctx->rk, start, ctx->slab_final, ctx->d_failure,
                                                         ctx->d_adv_count);
    CUDA_TRY(cudaGetLastError());
    ctx->launches++;
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));   // bits is host memory of this call
    return B2D_OK;
}

extern "C" b2d_status b2d_slab_stage(b2d_ctx* ctx)
{
    if (!ctx || ctx->slab_next < 0 || ctx->slab_next >= (int)ctx->slab_plan.size())
        return fail(B2D_ERR_INVALID, "no slab stage left to run");
    const int s = ctx->slab_next;
    b2d_status st = launch_stage(ctx, ctx->slab_plan[s], s, s + 1 == (int)ctx->slab_plan.size());
    if (st != B2D_OK) return st;
    ctx->launches++;
    st = launch_tracers(ctx, ctx->slab_plan[s], true);
    if (st != B2D_OK) return st;
    const int first = fold_due(ctx, s, (int)ctx->slab_plan.size());
    if (first >= 0) st = launch_ledgers(ctx, first, s + 1, false, ctx->slab_fold, ctx->slab_start, true);
    if (st != B2D_OK) return st;
    ctx->slab_next++;
    return B2D_OK;
}

extern "C" b2d_status b2d_slab_end(b2d_ctx* ctx, double* dt_out, b2d_error* err_out)
{
    if (!ctx || ctx->slab_next != (int)ctx->slab_plan.size() || ctx->slab_plan.empty())
        return fail(B2D_ERR_INVALID, "the slab advance has stages left to run");
    b2d_status st = launch_ledgers(ctx, 0, 0, true, ctx->slab_fold, ctx->slab_start, true);
    ctx->slab_next = -1;
    if (st != B2D_OK) return st;
    return finish_advance(ctx, ctx->slab_final, dt_out, err_out);
}

extern "C" b2d_status b2d_slab_rows(b2d_ctx* ctx, int32_t run, int32_t row0, int32_t nrows, double* rows, int32_t put)
{
    if (!ctx || run < 0 || run >= ctx->nruns || !rows || nrows < 1) return fail(B2D_ERR_INVALID, "bad arguments");
    RunHost& r = ctx->runs[run];
    if (nrows > r.N) return fail(B2D_ERR_INVALID, "more rows than the mesh has");
    // the next stage's input slot, or the current state between advances
    const int slot = ctx->slab_next >= 0 && ctx->slab_next < (int)ctx->slab_plan.size()
                         ? ctx->slab_plan[ctx->slab_next].in : ctx->cur;
    const size_t nn = (size_t)r.N * r.N;
    // the stored words as they are: FP64 planes (FP64 and FP64-state contexts),
    // or the hi and lo FP32 planes of the compensated state, so that the
    // receiving context continues with exactly the sender's words
    const int parts = store_of(ctx) == 1 ? 2 : 1;
    const size_t w = store_of(ctx) == 1 ? sizeof(float) : sizeof(double);
    unsigned char* planes = (unsigned char*)r.slot[slot];
    unsigned char* buf = (unsigned char*)rows;
    for (int f = 0; f < ctx->nf; ++f)
        for (int part = 0; part < parts; ++part)
            for (int k = 0; k < nrows; ++k) {
                const int gi = ((row0 + k) % r.N + r.N) % r.N;
                unsigned char* dev = planes + (((size_t)(f * parts + part)) * nn + (size_t)gi * r.N) * w;
                unsigned char* host = buf + (((size_t)(f * parts + part) * nrows + k) * r.N) * w;
                if (put) CUDA_TRY(cudaMemcpyAsync(dev, host, w * r.N, cudaMemcpyHostToDevice, ctx->stream));
                else CUDA_TRY(cudaMemcpyAsync(host, dev, w * r.N, cudaMemcpyDeviceToHost, ctx->stream));
            }
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    return B2D_OK;
}

// ---------------------------------------------------------------------------
// One RK stage that allocates nothing.
//
// Some callers cannot call cudaMalloc: a host code that owns a fixed device
// memory pool and forbids allocation by libraries, or an allocator-less
// embedded runtime.  They hand over every input and
// output buffer themselves; the scratch the stage kernel needs (its run
// descriptor, the binary at the stage time, per-tile ledger partials, block
// the max-speed word and the failure key) lives in the file-scope
// array below, which every GPU that loads this library holds until the
// process exits.
constexpr size_t B2D_NOALLOC_SCRATCH_BYTES = 4u << 20;   // 4 MiB
static __device__ __align__(256) unsigned char g_noalloc_scratch[B2D_NOALLOC_SCRATCH_BYTES];

namespace {
constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mutex;
unsigned char* g_noalloc_base[NOALLOC_MAX_DEVICES] = {};
}  // namespace

// Device address of the scratch array on the current device.  The host-side
// name g_noalloc_scratch is only a stand-in for the symbol, never a device
// address: the address comes from cudaGetSymbolAddress, once per device.
static b2d_status noalloc_scratch_base(unsigned char** base)
{
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return fail(B2D_ERR_INVALID, "device index out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_base[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return fail(B2D_ERR_CUDA, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
        g_noalloc_base[dev] = (unsigned char*)p;
    }
    *base = g_noalloc_base[dev];
    return B2D_OK;
}

// The binary at the stage time, dt and the stage time, written into scratch.
__global__ void noalloc_setup_kernel(RunDev* rd, double time, double dt)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        kepler_orbit(*rd, time, rd->orbit);
        *rd->dt = dt;
        rd->stage_time[0] = time;
    }
}

// The stage's ledger: pieces folded, added and averaged as compute_block_updated_solution
// and weighted_average do (scheme.rs:307-313, state.rs:196).
__global__ void noalloc_ledger_kernel(const RunDev* run, int base_slot, double bf)
{
    const RunDev& rd = *run;
    const int id = blockIdx.x * blockDim.x + threadIdx.x;   // block * 7 + item
    if (id >= rd.nblocks * NITEMS) return;
    const int nf = rd.p.hydro == B2D_EULER ? 4 : 3;
    double ds[4];
    if (nf == 3) fold_item<3>(rd, 0, id / NITEMS, id % NITEMS, ds);
    else fold_item<4>(rd, 0, id / NITEMS, id % NITEMS, ds);
    for (int f = 0; f < nf; ++f) {
        const size_t w = (size_t)id * nf + f;
        double v = rd.ledger[0][w] + ds[f];
        if (base_slot >= 0) v = v * (-bf + 1.0) + rd.ledger[base_slot][w] * bf;
        rd.ledger[2][w] = v;
    }
}

extern "C" b2d_status b2d_stage_noalloc(const b2d_config* cfg, const double* d_in, const double* d_background,
                                        const double* d_base, double* d_out, const double* d_ledger_in,
                                        const double* d_ledger_base, double* d_ledger_out, double time, double dt,
                                        double bf, double* d_max_speed, b2d_error* err_out, void* stream_ptr)
{
    if (!cfg || !d_in || !d_background || !d_out || !d_ledger_in || !d_ledger_out || (d_base && !d_ledger_base))
        return fail(B2D_ERR_INVALID, "b2d_stage_noalloc: missing buffer");
    b2d_status st = validate(*cfg, cfg->hydro_kind, cfg->rk_order);
    if (st != B2D_OK) return st;
    cudaStream_t stream = (cudaStream_t)stream_ptr;
    const int nf = cfg->hydro_kind == B2D_EULER ? 4 : 3;
    const int bs = cfg->block_size, nb = cfg->num_blocks, N = bs * nb, nblocks = nb * nb;
    if (bs % 32 != 0 && bs > 256)
        return fail(B2D_ERR_INVALID, "b2d_stage_noalloc: block_size " + std::to_string(bs) +
                                         " must be a multiple of 32 or at most 256");

    // scratch layout: run descriptor | control words | (unused, one word a block) | ledger pieces | geometry tables.  A CTA takes
    // several sub-tiles of a block where one piece per sub-tile would not fit.
    const size_t off_run = 0, off_ctl = 2048, off_cnt = 2304;
    const size_t off_part = off_cnt + ((sizeof(unsigned) * (size_t)nblocks + 255) / 256) * 256;
    const size_t geo_bytes = sizeof(double) * ((size_t)N + (size_t)nb * (bs + 1));
    int sub_h, sub_w;
    f64_sub_tile(nf, {{bs, nblocks}}, &sub_h, &sub_w);
    RunDev rd;
    memset(&rd, 0, sizeof rd);
    // the meshes taken are those whose pieces would fit at one per default tile
    int tile_h = std::min(64, bs);
    while (bs % tile_h) tile_h /= 2;
    size_t need = off_part + sizeof(double) * (size_t)nblocks * (bs / tile_h) * (bs / default_tile_w(bs)) * NITEMS * nf;
    const bool fits = (need + 255) / 256 * 256 + geo_bytes <= B2D_NOALLOC_SCRATCH_BYTES;
    for (int per_cta = 1; fits; per_cta *= 2) {
        split_blocks(rd, bs, sub_h, sub_w, per_cta);
        need = off_part + sizeof(double) * (size_t)nblocks * rd.tiles_per_block * NITEMS * nf;
        if (rd.tiles_per_block == 1 || (need + 255) / 256 * 256 + geo_bytes <= B2D_NOALLOC_SCRATCH_BYTES) break;
    }
    static_assert(sizeof(RunDev) <= 2048, "run descriptor outgrew its scratch slot");
    if (need > B2D_NOALLOC_SCRATCH_BYTES)
        return fail(B2D_ERR_INVALID, "b2d_stage_noalloc: this mesh needs " + std::to_string(need) +
                                         " bytes of scratch; the library holds " +
                                         std::to_string(B2D_NOALLOC_SCRATCH_BYTES) + " (use b2d_create instead)");
    unsigned char* base = nullptr;
    st = noalloc_scratch_base(&base);
    if (st != B2D_OK) return st;

    RunDev* d_run = (RunDev*)(base + off_run);
    double* orbit = (double*)(base + off_ctl);            // 10 doubles
    double* d_dt = orbit + 10;
    double* stime = orbit + 11;
    double* times = orbit + 12;                            // 4 doubles (unused by the stage)
    long long* iters = (long long*)(orbit + 16);           // 4 (unused by the stage)
    unsigned long long* amax = (unsigned long long*)(orbit + 20);
    Failure* failure = (Failure*)(amax + 1);
    double* partial = (double*)(base + off_part);

    std::vector<double> xc(N), xv((size_t)nb * (bs + 1));
    for (int b = 0; b < nb; ++b) {
        host_cell_centers(cfg, b, xc.data() + (size_t)b * bs);
        host_block_vertices(cfg, b, xv.data() + (size_t)b * (bs + 1));
    }
    // the FP64 kernel reads its geometry from the run descriptor's tables: place
    // them behind the partials in scratch
    const size_t off_geo = ((need + 255) / 256) * 256;
    const size_t need_geo = off_geo + sizeof(double) * (xc.size() + xv.size());
    if (need_geo > B2D_NOALLOC_SCRATCH_BYTES)
        return fail(B2D_ERR_INVALID, "b2d_stage_noalloc: mesh too large for the 4 MiB scratch (use b2d_create instead)");
    double* d_xc = (double*)(base + off_geo);
    double* d_xv = d_xc + xc.size();

    rd.N = N; rd.bs = bs; rd.nb = nb; rd.nblocks = nblocks;
    rd.ntiles = nblocks * rd.tiles_per_block;
    rd.xc = d_xc; rd.xv = d_xv;
    rd.slot[0] = (void*)d_in; rd.slot[1] = (void*)d_base; rd.slot[2] = d_out; rd.slot[3] = d_out;
    rd.bg = d_background;
    rd.ledger[0] = (double*)d_ledger_in; rd.ledger[1] = (double*)d_ledger_base;
    rd.ledger[2] = d_ledger_out; rd.ledger[3] = d_ledger_out;
    rd.time = times; rd.iter = iters;
    rd.partial = partial; rd.stage_window = 1;
    rd.dt = d_dt; rd.stage_time = stime; rd.orbit = orbit; rd.amax = amax;
    rd.binary_q = cfg->binary_mass_ratio; rd.binary_e = cfg->binary_eccentricity;
    rd.p = make_params<double>(*cfg);
    rd.pf = make_params<float>(*cfg);

    // every call shares the scratch: reset what must start from zero (or ~0)
    CUDA_TRY(cudaMemcpyAsync(d_run, &rd, sizeof rd, cudaMemcpyHostToDevice, stream));
    CUDA_TRY(cudaMemcpyAsync(d_xc, xc.data(), sizeof(double) * xc.size(), cudaMemcpyHostToDevice, stream));
    CUDA_TRY(cudaMemcpyAsync(d_xv, xv.data(), sizeof(double) * xv.size(), cudaMemcpyHostToDevice, stream));
    CUDA_TRY(cudaMemsetAsync(amax, 0, sizeof(unsigned long long), stream));
    CUDA_TRY(cudaMemsetAsync(failure, 0, sizeof(Failure), stream));
    CUDA_TRY(cudaMemsetAsync(&failure->key, 0xff, sizeof(unsigned long long), stream));
    noalloc_setup_kernel<<<1, 32, 0, stream>>>(d_run, time, dt);
    CUDA_TRY(cudaGetLastError());

    StageArgs a;
    a.runs = d_run;
    a.tile_bases = nullptr;
    a.nruns = 1;
    a.pf1 = rd.pf;
    a.in_slot = 0;
    a.base_slot = d_base ? 1 : -1;
    a.out_slot = 2;
    a.stage = 0;
    a.amax_flag = d_max_speed ? 1 : 0;
    a.bf = d_base ? bf : 0.0;
    a.half_avg = a.bf == 0.5;
    a.w1f = split_df(-a.bf + 1.0);
    a.bff = split_df(a.bf);
    a.failure = failure;
    cudaError_t e = launch_stage_f64(nf, a, rd.ntiles, stage_f64_smem(nf, sub_h, sub_w), stream);
    if (e != cudaSuccess) return fail(B2D_ERR_CUDA, std::string("stage kernel launch: ") + cudaGetErrorString(e));
    noalloc_ledger_kernel<<<(nblocks * NITEMS + 127) / 128, 128, 0, stream>>>(d_run, a.base_slot, a.bf);
    CUDA_TRY(cudaGetLastError());
    if (d_max_speed) CUDA_TRY(cudaMemcpyAsync(d_max_speed, amax, sizeof(double), cudaMemcpyDeviceToDevice, stream));

    unsigned long long key = ~0ull;
    CUDA_TRY(cudaMemcpyAsync(&key, &failure->key, sizeof key, cudaMemcpyDeviceToHost, stream));
    CUDA_TRY(cudaStreamSynchronize(stream));
    if (key == ~0ull) return B2D_OK;

    // decode the failure key of the stage (see error_key in stage.cuh)
    b2d_error err;
    memset(&err, 0, sizeof err);
    const int blk = (int)((key >> 30) & 0xffff), order = (int)((key >> 26) & 0xf);
    const int zone = (int)((key >> 2) & 0xffffff);
    err.code = (int)(key & 3);
    err.block_i = (blk / nb + order / 3 - 1 + nb) % nb;
    err.block_j = (blk % nb + order % 3 - 1 + nb) % nb;
    err.zone_i = zone / bs;
    err.zone_j = zone % bs;
    const int gi = err.block_i * bs + err.zone_i, gj = err.block_j * bs + err.zone_j;
    err.x = xc[gi];
    err.y = xc[gj];
    err.time = time;
    double u[4] = {0, 0, 0, 0}, orb[10];
    for (int f = 0; f < nf; ++f)
        CUDA_TRY(read_back(&u[f], d_in + (size_t)f * N * N + (size_t)gi * N + gj, sizeof(double), stream));
    CUDA_TRY(read_back(orb, orbit, sizeof orb, stream));
    err.value = failure_value(*cfg, u, err.code);
    err.binary[0] = orb[1]; err.binary[1] = orb[2]; err.binary[2] = orb[6]; err.binary[3] = orb[7];
    if (err_out) *err_out = err;
    return fail((b2d_status)err.code, "hydro error in b2d_stage_noalloc");
}

// ---------------------------------------------------------------------------
// Orbital-element change per block (BlockState::orbital_elements_change,
// src/state.rs:44-49): [nb][nb][7][4] of (a, M, q, e) per ItemizedChange item.
extern "C" b2d_status b2d_download_elements(b2d_ctx* ctx, int32_t run, double* elements)
{
    if (!ctx || run < 0 || run >= ctx->nruns || !elements) return fail(B2D_ERR_INVALID, "bad arguments");
    RunHost& r = ctx->runs[run];
    CUDA_TRY(cudaMemcpyAsync(elements, r.elements[ctx->cur], sizeof(double) * r.nblocks * NITEMS * 4,
                             cudaMemcpyDeviceToHost, ctx->stream));
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    return B2D_OK;
}

extern "C" b2d_status b2d_upload_elements(b2d_ctx* ctx, int32_t run, const double* elements)
{
    if (!ctx || run < 0 || run >= ctx->nruns || !elements) return fail(B2D_ERR_INVALID, "bad arguments");
    RunHost& r = ctx->runs[run];
    CUDA_TRY(cudaMemcpyAsync(r.elements[ctx->cur], elements, sizeof(double) * r.nblocks * NITEMS * 4,
                             cudaMemcpyHostToDevice, ctx->stream));
    CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    return B2D_OK;
}
