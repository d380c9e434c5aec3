// kernels_f64.cu — the FP64 stage kernel (the parity path).  Built with
// --fmad=false so that every FP64 operation rounds exactly as written.
#include "kernels.inc"
#include "stage64.cuh"

namespace b2d {

cudaError_t launch_stage_f64(int nf, const StageArgs& a, int grid, size_t smem, cudaStream_t s)
{
    void (*k)(StageArgs) = nf == 3 ? stage64_kernel<3> : stage64_kernel<4>;
    cudaError_t e = opt_in_smem((const void*)k, smem);
    if (e != cudaSuccess) return e;
    k<<<grid, S64_THREADS, smem, s>>>(a);
    return cudaGetLastError();
}

// The buffer's rate of every zone (Physics::source_terms, physics.rs:443-446),
// a function of its place only.
__global__ void buffer_rate_kernel(const RunDev* runs, int run, double* out)
{
    const RunDev& rd = runs[run];
    const size_t nn = (size_t)rd.N * rd.N;
    for (size_t z = blockIdx.x * (size_t)blockDim.x + threadIdx.x; z < nn; z += (size_t)gridDim.x * blockDim.x) {
        const unsigned i = (unsigned)z / (unsigned)rd.N, j = (unsigned)z - i * (unsigned)rd.N;
        out[z] = buffer_rate(rd.p, rd.xc[i], rd.xc[j]);
    }
}

cudaError_t launch_buffer_rate(const RunDev* runs, int run, int N, double* out, cudaStream_t s)
{
    const size_t blocks = ((size_t)N * N + 255) / 256;
    buffer_rate_kernel<<<(unsigned)(blocks < 16384 ? blocks : 16384), 256, 0, s>>>(runs, run, out);
    return cudaGetLastError();
}

// Shared memory of a launch with sub-tiles of at most th x tw zones.
size_t stage_f64_smem(int nf, int th, int tw) { return (size_t)s64_smem_bytes(nf, th, tw); }

}  // namespace b2d
