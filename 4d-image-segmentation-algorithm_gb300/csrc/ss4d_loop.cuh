// ss4d_loop.cuh — the persistent SOR loop (ss4d_loop.cu), used by the
// single-volume handle and the batch, and the group barrier it shares with
// the persistent presmoothing (ss4d_front.cuh).
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
    unsigned top; // presmoothing: upper word of the image's largest |value|
    int pad_[29]; // one 128-byte line per group
};

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Barrier of a group, thread 0 of each block, between two block barriers:
// arrive once the block's writes are made, then wait until `target` arrivals
// were.  The release and the acquire order the blocks' writes and reads (the
// block barriers carry the order to their other threads).  A wait is bounded
// (about a second); one that runs out marks the group.
__device__ __forceinline__ void group_arrive(LoopGroup *gr)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&gr->count) : "memory");
}
__device__ __forceinline__ bool group_wait(LoopGroup *gr, unsigned target)
{
    if ((int)(ld_acquire(&gr->count) - target) < 0) {
        const long long t0 = clock64();
        while ((int)(ld_acquire(&gr->count) - target) < 0) {
            if (clock64() - t0 > (1LL << 31)) {
                atomicExch(&gr->err, 1);
                return false;
            }
        }
    }
    return *(volatile int *)&gr->err == 0;
}

LoopVol make_loop_vol(const Geo &g, const Split &sp, const SplitBufs &b);
// co-resident blocks of k_loop with that many threads on the device (0: unknown)
int loop_grid(int mixed, int nv, int threads, int sm_count);
// the most blocks any form of one volume's k_loop has with that many threads
int loop_most_blocks(int threads, int sm_count);
// the grid of one volume's k_loop, and whether it is the AHEAD form (0: unknown)
int loop_plan(int mixed, const FlatIndex &F, int threads, int sm_count, bool *ahead);
// deals `grid` blocks out to the volumes in proportion to their targets
// (at least one each; nv <= grid)
void share_blocks(LoopVol *vols, int nv, int grid);
// vols (host memory), st, par, groups (zeroed by the caller) per volume;
// parts 4 doubles per block
cudaError_t launch_loop(int mixed, const LoopVol *vols, int nv, int grid, int threads, LoopState *st,
                        const DevParams *par, double *parts, LoopGroup *groups, int max_bodies, bool ahead,
                        cudaStream_t stream);

} // namespace ss4d
