// Launch record of the warp-specialised Q8 kernel (k_q8w.cu), shared with the
// code that plans launches (k_q8s.cu).
#pragma once

#include <cuda.h>

#include "mv_device.cuh"

namespace mv {

typedef mv_q8_job Q8Job;

constexpr int kXQuads = 64;  // the longest segments, in quads, whose x the CUDA-core consumers' slots hold

struct Q8WLayout {  // byte offsets in shared memory
    uint32_t tiles, slots, red, bars, desc, ring, cnt, stage_o, stage_e, misc, total;
};

struct Q8WLaunch {
    Q8Job job0;         // the only job when jobs == nullptr
    const Q8Job *jobs;  // device array of njobs jobs, or nullptr
    int njobs;
    uint32_t nitems;
    int batch;  // valid vectors
    uint32_t *status;
    uint32_t spin_limit;
    int drop_copy;
    uint32_t slot_bytes;  // one stream slot: the largest block and the row after it
    int tbl_stage;        // staged table entries
    // chained pipeline (mv_q8_chain_matvec): job j's int8 output clamp(rn(y * chain_scales[j])) is job j+1's x
    // (the last job's goes to chain_out8); jobs[j].pad counts job j's finished work items
    const float *chain_scales;
    int8_t *chain_out8;
    uint32_t *queue;  // work queue of a stack (jobs[0].pad of the job table), or nullptr: static round robin
    // One job in even shares (nonzero: its number of units): CTA c of G takes units [c span / G, (c + 1) span / G),
    // whatever stripes they are of.  Sums of a stripe that several CTAs share are added to y (ys) unscaled.
    uint32_t span;
    int early;  // the launch before this one is this library's own, made in the same call (see q8w_kernel)
    int ragged;  // integer products, one job: x off the 16-byte grid, columns or segments not whole groups of 16 columns
    // set by the launcher
    int W, S;              // decode warps, stream slots
    uint32_t S_inv;        // ceil(2^32 / S): unit / S by multiplication
    uint32_t block_bytes;  // of a slot, its block's part
    uint32_t x_off;        // where a slot holds its segment's x (0: nowhere)
    uint32_t x_quad;       // bytes of a quad of x
    int xrows;  // MMA consumers: rows of the x tile (batch rounded up to 8)
    Q8WLayout lay;
    CUtensorMap xmap;  // x of a single matrix as tiles (XTiles)
};

// Integer product of L.batch vectors: on the tensor cores (up to 64 vectors) or, with dp4a, nv >= batch vectors
// (1, 2, 4, 8 or 16).  warps: decode warps per CTA (0: as many as fit); units: the most units a CTA can get.
mv_status q8w_launch_int(const Q8WLaunch &L, int nv, bool mma, int warps, int units, cudaStream_t st);
// Whether a ragged one (dp4a: of up to 8 vectors) finds room in shared memory at all.
bool q8w_ragged_fits(const Q8WLaunch &L, bool mma);
// Float forward: job0.x is bf16 [batch][cols], job0.ys fp32 [batch][rows].  On the tensor cores up to 64 vectors, on the CUDA
// cores (dot; one vector always) up to 8.
mv_status q8w_launch_fwd(const Q8WLaunch &L, bool dot, int warps, int units, cudaStream_t st);
// Float backward: job0.x is dY, bf16 [batch][rows], added to job0.ys, fp32 [batch][cols].  On the tensor cores up to 32
// vectors, on the CUDA cores (as above) up to 8.
mv_status q8w_launch_bwd(const Q8WLaunch &L, bool dot, int warps, int units, cudaStream_t st);

}  // namespace mv
