// ss4d_loop.cu — the SOR loop of one or many volumes as one persistent
// cooperative launch (k_loop), in the plain FP64 and the mixed form.
//
// Every volume has a group of blocks of its own, in proportion to its
// targets; a group runs its volume's loop from the state the host left to
// the state that stops (or pauses) it and meets no other group.  A phase
// (half-sweep, refinement) walks the volume's targets in one flat index, so
// no lane is lost to partly filled tiles, and the volume's description stays
// in shared memory.  Between phases the group meets at a barrier of its own.
// The stopping test has no phase: after the barrier that ends a loop body
// every block of the group adds the group's partial sums in the same order
// and runs the controller (ctrl64_update, ctrl_mixed_update) on its own copy
// of the loop state, so all blocks of the group take the same next phase.
//
// What bounds it: for volumes that stay in L2 a body's two or three barriers
// and the latency of one round of loads per phase; for larger ones the
// stream of the records through HBM, as the separate kernels.  Per target
// the arithmetic is that of k_sweep64 / k_refine / k_sweep32, so results
// equal theirs bit for bit.
#include "ss4d_loop.cuh"

namespace ss4d {

namespace {

constexpr int LOOP_MAX_THREADS = 512;

template <int COL>
__device__ __forceinline__ double phase_sweep64(const LoopVol &V, int z, unsigned q0, unsigned dq)
{
    const double *src = COL == 0 ? V.b.R[z & 1] : V.b.Bk;
    double *dst = COL == 0 ? V.b.R[(z + 1) & 1] : V.b.Bk;
    const double *oth = COL == 0 ? V.b.Bk : V.b.R[z & 1];
    const double *cf = V.b.coef[COL], *pv = V.b.P[COL];
    double acc = 0.0;
    for (unsigned q = q0; q < V.F.ntargets; q += dq) {
        const Place a = place<1>(V.F, V.F.dX, COL, q);
        if (a.i > V.F.nx)
            continue;
        const double r = sweep64_at<true>(a.p, a.s, a.t, V.F.Hs, V.F.Hz, V.F.Hw, src, dst, oth, cf, pv);
        acc = fma(r, r, acc);
    }
    return acc;
}

// FP32 half-sweep, two adjacent targets per thread
template <int COL>
__device__ __forceinline__ double phase_sweep32(const LoopVol &V, int ds, float omega, unsigned q0, unsigned dq)
{
    const float *src = COL == 0 ? V.b.dR[ds] : V.b.dB;
    float *dst = COL == 0 ? V.b.dR[ds ^ 1] : V.b.dB;
    const float *oth = COL == 0 ? V.b.dB : V.b.dR[ds];
    float acc = 0.f;
    for (unsigned q = q0; q < V.F.npairs; q += dq) {
        const Place a = place<2>(V.F, V.F.dP, COL, q);
        if (a.i > V.F.nx)
            continue;
        acc = sweep32_pair<true>(a.p, a.s, a.t, a.i + 2 <= V.F.nx, V.F.Hs, V.F.Hz, V.F.Hw, src, dst, oth, V.b.coefq[COL],
                                 V.b.coefs[COL], V.b.r32[COL], omega, acc);
    }
    return (double)acc;
}

// The start of a round from zero corrections: k_zero_delta and the first red
// half-sweep at once.  With every correction zero the red update is
// (omega / diag) rhs, to the bit (r = -rhs, the products with zeros are
// zeros); the black corrections are set to zero, and the red array the sweep
// would read is not read again before it is written.  Ghost and padding
// cells of the three arrays are zero already.
__device__ __forceinline__ void phase_round_from_zero(const LoopVol &V, int ds, float omega, unsigned q0, unsigned dq)
{
    float *dst = V.b.dR[ds ^ 1];
    for (unsigned q = q0; q < V.F.npairs; q += dq) {
        const Place a = place<2>(V.F, V.F.dP, 0, q);
        if (a.i > V.F.nx)
            continue;
        const bool two = a.i + 2 <= V.F.nx;
        const float2 rh = __ldcg(reinterpret_cast<const float2 *>(V.b.r32[0] + a.s));
        float w[8], z8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, d;
        float sc = load_coef16(V.b.coefq[0], V.b.coefs[0], a.t, w);
        float r = resid32(w, sc, z8, 0.f, rh.x, d);
        dst[a.s] = fmaf(-__fdividef(omega, d), r, 0.f);
        if (two) {
            sc = load_coef16(V.b.coefq[0], V.b.coefs[0], a.t + 1, w);
            r = resid32(w, sc, z8, 0.f, rh.y, d);
            dst[a.s + 1] = fmaf(-__fdividef(omega, d), r, 0.f);
        }
    }
    for (unsigned q = q0; q < V.F.npairs; q += dq) {
        const Place a = place<2>(V.F, V.F.dP, 1, q);
        if (a.i > V.F.nx)
            continue;
        V.b.dB[a.s] = 0.f;
        if (a.i + 2 <= V.F.nx)
            V.b.dB[a.s + 1] = 0.f;
    }
}

__device__ __forceinline__ void phase_apply_black(const LoopVol &V, unsigned q0, unsigned dq)
{
    for (unsigned q = q0; q < V.F.ntargets; q += dq) {
        const Place a = place<1>(V.F, V.F.dX, 1, q);
        if (a.i <= V.F.nx)
            V.b.Bk[a.s] = __ldcg(V.b.Bk + a.s) + f2d_bits(__ldcg(V.b.dB + a.s));
    }
}

template <int COL>
__device__ __forceinline__ double phase_refine(const LoopVol &V, int ds, int pre, unsigned q0, unsigned dq)
{
    double *own = COL == 0 ? V.b.R[0] : V.b.Bk;
    const float *down = V.b.dR[ds];
    const double *oth = COL == 0 ? V.b.Bk : V.b.R[0];
    double acc = 0.0;
    for (unsigned q = q0; q < V.F.ntargets; q += dq) {
        const Place a = place<1>(V.F, V.F.dX, COL, q);
        if (a.i > V.F.nx)
            continue;
        double r;
        if (pre) {
            r = ld_stream(V.b.rpre[COL] + a.s);
        } else {
            const RefineOut o = refine_at<COL, true>(a.p, a.s, a.t, V.F.Hs, V.F.Hz, V.F.Hw, own, down, oth, V.b.coef[COL],
                                                     V.b.P[COL]);
            r = o.r;
            if (COL == 0)
                own[a.s] = o.u;
        }
        acc = fma(r, r, acc);
        V.b.r32[COL][a.s] = d2f_bits(-r);
    }
    return acc;
}

// The volumes are a kernel parameter: a target's index arithmetic takes its
// constants straight from the constant bank (from shared memory they are
// loads, for every target again, since the stores to u could alias them).
template <int NV>
struct LoopVols {
    LoopVol v[NV];
};

// 64 registers: two blocks of 512 (or four of 256) per SM
template <int MIXED, int NV>
__global__ void __launch_bounds__(LOOP_MAX_THREADS, 2) k_loop(const __grid_constant__ LoopVols<NV> vols, int nv,
                                                              LoopState *st, const DevParams *__restrict__ par,
                                                              double *parts, LoopGroup *groups, int max_bodies)
{
    __shared__ LoopState S;
    __shared__ DevParams P;
    __shared__ int ok, mine;
    const int tid = threadIdx.x;
    int v = 0;
    if (NV > 1) {
        if (tid == 0)
            mine = -1;
        __syncthreads();
        if (tid < nv && (unsigned)(blockIdx.x - vols.v[tid].blk0) < (unsigned)vols.v[tid].nblk)
            mine = tid;
        __syncthreads();
        v = mine;
        if (v < 0) // a block past the last group
            return;
    }
    const LoopVol &V = vols.v[v];
    if (tid == 0) {
        S = st[v];
        P = par[v];
    }
    __syncthreads();
    const unsigned rank = blockIdx.x - V.blk0, nb = V.nblk;
    const unsigned dq = nb * blockDim.x;
    // a volume of at most two rounds is dealt out warp by warp, so that its
    // last round is spread over all blocks; a larger one block by block (the
    // warps of a block then share neighbouring rows in L1)
    const unsigned q0 = (MIXED ? V.F.npairs : V.F.ntargets) <= 2 * dq ? ((tid >> 5) * nb + rank) * 32 + (tid & 31)
                                                                  : rank * blockDim.x + tid;
    LoopGroup *const gr = groups + v;
    unsigned target = 0;
    // partial sums of this group: [parity][colour][block]; two sets in turn,
    // since a block may still add one body's while another writes the next's
    double *const part = parts + 4 * (size_t)V.blk0;
    int par_set = 0;

    auto put = [&](int colour, double acc) {
        acc = block_sum(acc);
        if (tid == 0)
            part[(par_set * 2 + colour) * nb + rank] = acc;
    };
    // barrier of the group; false when a wait of the group gave up.  The
    // block's own sum `acc` of the phase it ends (partial `colour`, if >= 0)
    // is added up while the others arrive: it is read after the next barrier
    auto sync = [&](int colour, double acc) -> bool {
        target += nb;
        __syncthreads();
        if (tid == 0)
            group_arrive(gr);
        if (colour >= 0)
            put(colour, acc);
        if (tid == 0)
            ok = group_wait(gr, target);
        __syncthreads();
        return ok;
    };
    // the same, then every block runs the controller on the group's sums
    auto sync_ctrl = [&](bool sums) -> bool {
        target += nb;
        __syncthreads();
        if (tid < 32) {
            int good = 1;
            if (tid == 0) {
                group_arrive(gr);
                good = group_wait(gr, target);
            }
            good = __shfl_sync(0xffffffffu, good, 0);
            double a = 0.0, c = 0.0;
            if (sums && good) {
                const double *pa = part + par_set * 2 * nb;
                for (unsigned t = tid; t < nb; t += 32) {
                    a += __ldcg(pa + t);
                    c += __ldcg(pa + nb + t);
                }
                a = warp_sum(a);
                c = warp_sum(c);
            }
            if (tid == 0) {
                ok = good;
                if (good) {
                    if (MIXED)
                        ctrl_mixed_update(&S, a, c, &P);
                    else
                        ctrl64_update(&S, a, c, &P);
                }
            }
        }
        par_set ^= 1;
        __syncthreads();
        return ok;
    };

    bool good = true;
    if (!MIXED && S.z == 0) { // the first iteration's red half-sweep (no residual yet)
        phase_sweep64<0>(V, 0, q0, dq);
        good = sync(-1, 0.0);
        if (tid == 0)
            S.z = 1;
        __syncthreads();
    }
    for (int body = 0; good && body < max_bodies && !S.stop && !S.paused; ++body) {
        if (!MIXED) {
            if (!(good = sync(1, phase_sweep64<1>(V, S.z, q0, dq))))
                break;
            put(0, phase_sweep64<0>(V, S.z, q0, dq));
            good = sync_ctrl(true);
            continue;
        }
        const int mode = S.mode, ds = S.dsrc;
        const float omega = (float)P.omega;
        if (mode == 0) {
            const int pre = S.pre;
            if (!pre) { // (else the assembly applied the correction)
                phase_apply_black(V, q0, dq);
                if (!(good = sync(-1, 0.0)))
                    break;
            }
            const double red = phase_refine<0>(V, ds, pre, q0, dq);
            if (pre)
                put(0, red);
            else if (!(good = sync(0, red)))
                break;
            put(1, phase_refine<1>(V, ds, pre, q0, dq));
            good = sync_ctrl(true);
        } else if (mode == 1) {
            if (S.keep)
                phase_sweep32<0>(V, ds, omega, q0, dq);
            else
                phase_round_from_zero(V, ds, omega, q0, dq);
            good = sync_ctrl(false);
        } else {
            if (!(good = sync(1, phase_sweep32<1>(V, ds, omega, q0, dq))))
                break;
            put(0, phase_sweep32<0>(V, ds, omega, q0, dq));
            good = sync_ctrl(true);
        }
    }
    if (rank == 0 && tid == 0) {
        if (!good) {
            S.status = SS4D_ERR_TIMEOUT;
            S.stop = 1;
        }
        st[v] = S;
    }
}

} // namespace

LoopVol make_loop_vol(const Geo &g, const Split &sp, const SplitBufs &b)
{
    LoopVol V;
    memset(&V, 0, sizeof V);
    V.F = make_flat(g, sp);
    V.b = b;
    return V;
}

static const void *loop_kernel(int mixed, int nv)
{
    if (nv == 1)
        return mixed ? (const void *)k_loop<1, 1> : (const void *)k_loop<0, 1>;
    return mixed ? (const void *)k_loop<1, SS4D_BATCH_MAX_VOLUMES> : (const void *)k_loop<0, SS4D_BATCH_MAX_VOLUMES>;
}

int loop_grid(int mixed, int nv, int threads, int sm_count)
{
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, loop_kernel(mixed, nv), threads, 0) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return per * sm_count;
}

void share_blocks(LoopVol *vols, int nv, int grid)
{
    double total = 0.0;
    for (int v = 0; v < nv; ++v)
        total += vols[v].F.ntargets;
    int used = 0;
    for (int v = 0; v < nv; ++v) {
        const int n = (int)(grid * (vols[v].F.ntargets / total));
        vols[v].nblk = n < 1 ? 1 : n;
        used += vols[v].nblk;
    }
    // what rounding left over to the volumes with the most targets per
    // block; what small volumes took beyond the grid back from those with
    // the fewest
    while (used != grid) {
        int best = -1;
        for (int v = 0; v < nv; ++v) {
            const double load = (double)vols[v].F.ntargets / vols[v].nblk;
            if (used < grid) {
                if (best < 0 || load > (double)vols[best].F.ntargets / vols[best].nblk)
                    best = v;
            } else if (vols[v].nblk > 1 &&
                       (best < 0 || load < (double)vols[best].F.ntargets / vols[best].nblk)) {
                best = v;
            }
        }
        if (best < 0)
            break; // one block each and still too many: the caller checks
        vols[best].nblk += used < grid ? 1 : -1;
        used += used < grid ? 1 : -1;
    }
    int b0 = 0;
    for (int v = 0; v < nv; ++v) {
        vols[v].blk0 = b0;
        b0 += vols[v].nblk;
    }
}

cudaError_t launch_loop(int mixed, const LoopVol *vols, int nv, int grid, int threads, LoopState *st,
                        const DevParams *par, double *parts, LoopGroup *groups, int max_bodies, cudaStream_t stream)
{
    static_assert(sizeof(LoopVols<SS4D_BATCH_MAX_VOLUMES>) + 64 <= 32764, "kernel parameters");
    // the launch copies as many volumes as the kernel takes
    LoopVols<SS4D_BATCH_MAX_VOLUMES> all;
    if (nv > 1) {
        memset(&all, 0, sizeof all);
        memcpy(all.v, vols, sizeof(LoopVol) * nv);
    }
    void *args[] = {nv > 1 ? (void *)&all : (void *)vols, (void *)&nv, (void *)&st, (void *)&par, (void *)&parts,
                    (void *)&groups, (void *)&max_bodies};
    return cudaLaunchCooperativeKernel(loop_kernel(mixed, nv), dim3(grid), dim3(threads), args, 0, stream);
}

} // namespace ss4d
