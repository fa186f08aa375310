// ss4d_loop.cuh — the persistent SOR loop (ss4d_loop.cu), used by the
// single-volume handle and the batch.
#pragma once

#include <string.h>

#include "ss4d_sweep.cuh"

namespace ss4d {

// one volume as the persistent loop sees it
struct LoopVol {
    FlatIndex F;
    int blk0, nblk;            // its group: blocks blk0 .. blk0 + nblk - 1
    SplitBufs b;
};

// a group's barrier: arrivals so far; err once a wait gave up
struct LoopGroup {
    unsigned count;
    int err;
    int pad_[30]; // one 128-byte line per group
};

LoopVol make_loop_vol(const Geo &g, const Split &sp, const SplitBufs &b);
// co-resident blocks of k_loop with that many threads on the device (0: unknown)
int loop_grid(int mixed, int nv, int threads, int sm_count);
// deals `grid` blocks out to the volumes in proportion to their targets
// (at least one each; nv <= grid)
void share_blocks(LoopVol *vols, int nv, int grid);
// vols (host memory), st, par, groups (zeroed by the caller) per volume;
// parts 4 doubles per block
cudaError_t launch_loop(int mixed, const LoopVol *vols, int nv, int grid, int threads, LoopState *st,
                        const DevParams *par, double *parts, LoopGroup *groups, int max_bodies, cudaStream_t stream);

} // namespace ss4d
