// runtime.cuh — device-side descriptors shared by the kernels and the C ABI.
#pragma once

#include <vector_types.h>

#include "../../include/b2d.h"
#include "physics.cuh"

namespace b2d {

constexpr int NSLOTS = 4;  // state slots: the advance input is kept intact until success

struct df32w { float hi, lo; };

// One run of a batch as the kernels see it.
struct RunDev {
    int N, bs, nb, nblocks;
    int tiles_i, tiles_j, ntiles, tile_base;
    int tiles_per_block, chunk0; // partial slots per block: the most ledger pieces a block receives;
                                 // the first row chunk the launch covers (a slab's; 0 for the whole run)
    int slab_lo, slab_hi;        // row slab: block rows [slab_lo, slab_hi) of the run are this context's
                                 // (slab_hi = 0: the whole run); the stage kernel's tiles, the max
                                 // speed and the orbital-element ledger cover only the slab
    int chunks, pad_;            // row chunks per column strip of the whole run (C of chunk_start);
                                 // tiles_i of them, from chunk0, are launched
    int sub_i, sub_j;        // FP64 kernel: sub-tiles per block along rows and columns
    int sub_per_cta;         // and how many of a block's sub-tiles (row-major) one CTA takes, the last one fewer
    const double* buffer;    // FP64 kernel: [N][N] buffer rate (nullptr: computed where it is used)
    const double* xc;        // [N] cell centres by global index (block formula, mesh.rs:49-54)
    const double* xv;        // [nb][bs+1] block vertices (mesh.rs:42-47)
    const float2* xcf;       // [N] the centres as FP32 high and low words
    const float2* xvf;       // [N+1] faces by global index (a block's first vertex at its lower boundary), likewise
    void* slot[NSLOTS];      // conserved state per slot (STORE layout)
    const void* bg;          // BlockData::initial_conserved (STORE layout)
    double* ledger[NSLOTS];  // [nblocks][7][nf] per slot
    double* time;            // [NSLOTS]
    long long* iter;         // [NSLOTS]
    double* partial;         // [stage_window][nblocks][tiles_per_block][7 nf] ledger pieces of the tiles over each block
    int stage_window;        // stages whose pieces are kept before they are folded
    double* dt;              // [1]
    double* stage_time;      // [max_stages]
    double* orbit;           // [max_stages][10]: m, x, y, vx, vy of body 1 then body 2
    unsigned long long* amax;
    double binary_q, binary_e;
    double* elements[NSLOTS];    // [nblocks][7][4] orbital-element change per slot (nullptr: not tracked)
    double* stage_ds;            // [max_stages][nblocks][7 nf] block sums ds·dx·dy of each stage (nullptr: none)
    double* stage_de;            // [max_stages][nblocks][4][4] element change of the gas items of each stage
    double el0[4];               // unperturbed elements (a, M, q, e), physics.rs:411-417
    long long ntracers;          // massless tracer particles of this run (0: none)
    double* tracers[NSLOTS];     // [ntracers][2] positions (x, y) per state slot
    float2 tracer_radius, tracer_inv_dx;   // domain radius and 1 / dx as FP32 high and low words
    DevParams p;     // FP64 kernels
    DevParamsF pf;   // FP32 kernels
};

// A context's failure words.
struct Failure {
    unsigned long long key;         // of the earliest failing zone (error_key, stage.cuh), ~0 when none failed
    unsigned long long abandoned;   // the advance found a failure pending when it began: it changes nothing
};

struct StageArgs {
    const RunDev* runs;
    const int* tile_bases;   // [nruns] first CTA of each run
    int nruns;
    int in_slot, base_slot, out_slot;
    int stage;
    int amax_flag;
    double bf;               // weight of the RK base state (br of godunov-core)
    int half_avg;            // bf is 1/2
    b2d::df32w w1f, bff;     // 1 - bf and bf as double-float
    Failure* failure;
    DevParamsF pf1;          // FP32 parameters of a single-run context, read as kernel arguments
};

// Row chunks of a column strip.  A run's N rows split into C chunks; chunk c
// covers rows [c N / C, (c + 1) N / C).  With C = N / th the chunks are the
// block-aligned tiles of height th; with C = ceil(N / rows) for rows <= bs a
// chunk crosses at most one block boundary.  C <= N and N^2 <= 2^31 (the
// mesh limit of validate, api.cu) keep c N and (r + 1) C below 2^32, so
// 32-bit unsigned arithmetic is exact (a 64-bit division costs the stage
// kernel about a thousand instructions).
__host__ __device__ inline int chunk_start(int c, int N, int C) { return (int)((unsigned)c * (unsigned)N / (unsigned)C); }
__host__ __device__ inline int chunk_of_row(int r, int N, int C)
{
    return (int)((((unsigned)r + 1u) * (unsigned)C - 1u) / (unsigned)N);
}
// chunks that cover rows of block row b (bs rows from b bs)
__host__ __device__ inline int chunks_in_block_row(int b, int bs, int N, int C)
{
    return chunk_of_row((b + 1) * bs - 1, N, C) - chunk_of_row(b * bs, N, C) + 1;
}

// The FP32 kernel's strips are this many columns wide.  Its ledger piece of a
// strip and chunk for a block under both: the block's strips from left to right,
// and the chunks of its rows (nc of them from `first`) in each.
constexpr int STRIP_COLS = 60;
__host__ __device__ inline int strip_piece(int strip, int chunk, int block_column, int bs, int nc, int first)
{
    return (strip - block_column * bs / STRIP_COLS) * nc + chunk - first;
}
// pieces of the block that has the most
inline int most_strip_pieces(int bs, int nb, int C)
{
    int rows = 0, cols = 0;
    for (int b = 0; b < nb; ++b) {
        const int n = chunks_in_block_row(b, bs, nb * bs, C), m = (b * bs + bs - 1) / STRIP_COLS - b * bs / STRIP_COLS + 1;
        if (n > rows) rows = n;
        if (m > cols) cols = m;
    }
    return rows * cols;
}

// Whether a context keeps tables that its stages can do without: where they
// leave half of the GPU's memory free.  Pipelined transfers allocate two thirds
// of what a context holds after it was made, tracers 64 bytes each; a mesh that
// fits with them must not fail for a table.
inline bool room_for_tables(size_t free_bytes, size_t total_bytes, size_t tables)
{
    return free_bytes >= tables && free_bytes - tables >= total_bytes / 2;
}

// The ledger pieces of a block in a stage.
__host__ __device__ inline double* stage_pieces(const RunDev& rd, int stage, int block, int words)
{
    return rd.partial + ((size_t)(stage % rd.stage_window) * rd.nblocks + block) * rd.tiles_per_block * words;
}

#ifdef __CUDACC__
// The run that CTA g belongs to: the last one whose first CTA is not beyond it
// (256 runs at most; the whole warp searches, so that a batch of many runs
// costs one load's latency).
__device__ __forceinline__ int find_run(const StageArgs& a, int g)
{
    int n = 0;
    for (int k = threadIdx.x & 31; k - (int)(threadIdx.x & 31) < a.nruns; k += 32)
        n += __popc(__ballot_sync(0xffffffffu, k < a.nruns && a.tile_bases[min(k, a.nruns - 1)] <= g));
    return n - 1;
}
#endif

}  // namespace b2d
