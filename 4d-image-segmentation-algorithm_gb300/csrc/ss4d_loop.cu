// ss4d_loop.cu — the SOR loop of one or many volumes as one persistent
// cooperative launch (k_loop), in the plain FP64 and the mixed form.
//
// Every volume has a group of blocks of its own, in proportion to its
// targets; a group runs its volume's loop from the state the host left to
// the state that stops (or pauses) it and meets no other group.  A phase
// (half-sweep, refinement) walks the volume's targets in one flat index, so
// no lane is lost to partly filled tiles.  Between phases the group meets at a
// barrier of its own (1.2 to 1.4 us between 64 to 304 blocks).
// The stopping test has no phase: after the barrier that ends a loop body
// every block of the group adds the group's partial sums in the same order
// and runs the controller (ctrl64_update, ctrl_mixed_update) on its own copy
// of the loop state, so all blocks of the group take the same next phase.
//
// What bounds it: for volumes that stay in L2 a body's two or three barriers
// and the latency of one round of loads per phase (a step at 32^3 x 8 905 ->
// 526 us, of 45 x 37 x 29 x 7 in the mixed form 980 -> 476 us); for larger ones the
// stream of the records through HBM, as the separate kernels.  Per target
// the arithmetic is that of k_sweep64 / k_refine / k_sweep32, so results
// equal theirs bit for bit.
#include "ss4d_loop.cuh"

namespace ss4d {

namespace {

constexpr int LOOP_MAX_THREADS = 512;

// A half-sweep's first round of a thread, formed before it is known whether
// the loop goes on (nothing is stored)
struct Ahead64 {
    Sweep64Out o;
    unsigned s;
    bool any;
};
struct Ahead32 {
    Pair32Out o;
    unsigned s;
    bool any, two;
};

template <int COL> struct Sweep64 {
    const double *src, *oth, *cf, *pv;
    double *dst;
    __device__ __forceinline__ Sweep64(const LoopVol &V, int z)
    {
        src = COL == 0 ? V.b.R[z & 1] : V.b.Bk;
        dst = COL == 0 ? V.b.R[(z + 1) & 1] : V.b.Bk;
        oth = COL == 0 ? V.b.Bk : V.b.R[z & 1];
        cf = V.b.coef[COL];
        pv = V.b.P[COL];
    }
    __device__ __forceinline__ Ahead64 ahead(const LoopVol &V, unsigned q) const
    {
        Ahead64 h;
        h.any = q < V.F.ntargets;
        if (h.any) {
            const Place a = place<1>(V.F, V.F.dX, COL, q);
            h.any = a.i <= V.F.nx;
            h.s = a.s;
            if (h.any)
                h.o = sweep64_calc<true>(a.p, a.s, a.t, V.F.Hs, V.F.Hz, V.F.Hw, src, oth, cf, pv);
        }
        return h;
    }
    // the half-sweep; with `have` its first round is h
    __device__ __forceinline__ double run(const LoopVol &V, unsigned q0, unsigned dq, bool have, const Ahead64 &h) const
    {
        double acc = 0.0;
        unsigned q = q0;
        if (have) {
            if (h.any) {
                dst[h.s] = h.o.u;
                acc = h.o.r * h.o.r;
            }
            q += dq;
        }
        for (; q < V.F.ntargets; q += dq) {
            const Place a = place<1>(V.F, V.F.dX, COL, q);
            if (a.i > V.F.nx)
                continue;
            const double r = sweep64_at<true>(a.p, a.s, a.t, V.F.Hs, V.F.Hz, V.F.Hw, src, dst, oth, cf, pv);
            acc = fma(r, r, acc);
        }
        return acc;
    }
};

// FP32 half-sweep, two adjacent targets per thread
template <int COL> struct Sweep32 {
    const float *src, *oth;
    float *dst, omega;
    __device__ __forceinline__ Sweep32(const LoopVol &V, int ds, float w)
    {
        src = COL == 0 ? V.b.dR[ds] : V.b.dB;
        dst = COL == 0 ? V.b.dR[ds ^ 1] : V.b.dB;
        oth = COL == 0 ? V.b.dB : V.b.dR[ds];
        omega = w;
    }
    __device__ __forceinline__ Ahead32 ahead(const LoopVol &V, unsigned q) const
    {
        Ahead32 h;
        h.any = q < V.F.npairs;
        if (h.any) {
            const Place a = place<2>(V.F, V.F.dP, COL, q);
            h.any = a.i <= V.F.nx;
            h.two = a.i + 2 <= V.F.nx;
            h.s = a.s;
            if (h.any)
                h.o = sweep32_pair_calc<true>(a.p, a.s, a.t, h.two, V.F.Hs, V.F.Hz, V.F.Hw, src, oth, V.b.coefq[COL],
                                              V.b.coefs[COL], V.b.r32[COL], omega);
        }
        return h;
    }
    __device__ __forceinline__ float run(const LoopVol &V, unsigned q0, unsigned dq, bool have, const Ahead32 &h) const
    {
        float acc = 0.f;
        unsigned q = q0;
        if (have) {
            if (h.any)
                acc = sweep32_pair_put(h.o, h.s, h.two, dst, acc);
            q += dq;
        }
        for (; q < V.F.npairs; q += dq) {
            const Place a = place<2>(V.F, V.F.dP, COL, q);
            if (a.i > V.F.nx)
                continue;
            acc = sweep32_pair<true>(a.p, a.s, a.t, a.i + 2 <= V.F.nx, V.F.Hs, V.F.Hz, V.F.Hw, src, dst, oth,
                                     V.b.coefq[COL], V.b.coefs[COL], V.b.r32[COL], omega, acc);
        }
        return acc;
    }
};

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

// Sum over the block in thread 0 of the warp `to`: the threads' values go
// through shared memory and 128 threads add four (or two) each before they
// shuffle.  Shuffling in all 16 warps took 85 FP64 warp instructions, 1,300
// clocks of the SM's FP64 pipe with two blocks; this takes about 40 (a step at
// 32^3 x 8 619 -> 561 us, the mcf run of 40^4 3.95 -> 3.84 ms).  The batch's
// blocks of eight warps gain nothing by it and keep block_sum.
template <typename T>
__device__ __forceinline__ double block_total(T v, T *buf, double *part, int to)
{
    const int tid = threadIdx.x;
    buf[tid] = v;
    __syncthreads();
    if (tid < 128) {
        double s = (double)buf[tid];
        for (int q = tid + 128; q < blockDim.x; q += 128)
            s += (double)buf[q];
        s = warp_sum(s);
        if ((tid & 31) == 0)
            part[tid >> 5] = s;
    }
    __syncthreads();
    return tid == 32 * to ? (part[0] + part[1]) + (part[2] + part[3]) : 0.0;
}

// Two blocks of 512 (or four of 256) per SM, the mixed AHEAD form one (it
// takes 128 registers: within 64 it spilled and gained nothing).
// AHEAD (small volumes, loop_plan): the last warp of a block has no targets.
// It waits at the barrier that ends a body, adds the group's sums and runs the
// controller while the others already form (and keep in registers) their first
// round of the next body's black half-sweep, which they store once the
// controller lets the loop go on.
template <int MIXED, int NV, int AHEAD>
__global__ void __launch_bounds__(LOOP_MAX_THREADS, MIXED && AHEAD ? 1 : 2)
    k_loop(const __grid_constant__ LoopVols<NV> vols, int nv, LoopState *st, const DevParams *__restrict__ par,
           double *parts, LoopGroup *groups, int max_bodies)
{
    __shared__ LoopState S;
    __shared__ DevParams P;
    __shared__ int ok, mine;
    __shared__ double buf[LOOP_MAX_THREADS], bpart[4], own[2]; // own: this block's sums
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
    // the warp that meets the other blocks, and the threads with targets
    const int cwarp = AHEAD ? (int)(blockDim.x >> 5) - 1 : 0, ctid = 32 * cwarp;
    const unsigned wt = AHEAD ? blockDim.x - 32 : blockDim.x, dq = nb * wt;
    const bool works = (unsigned)tid < wt;
    // a volume of at most two rounds is dealt out warp by warp, so that its
    // last round is spread over all blocks; a larger one block by block (the
    // warps of a block then share neighbouring rows in L1)
    const unsigned n = MIXED ? V.F.npairs : V.F.ntargets;
    const unsigned q0 = !works ? 0xF0000000u : n <= 2 * dq ? ((tid >> 5) * nb + rank) * 32 + (tid & 31) : rank * wt + tid;
    LoopGroup *const gr = groups + v;
    unsigned target = 0;
    // partial sums (red, black) of this group's blocks, two sets in turn,
    // since a block may still add one body's while another writes the next's
    double2 *const part = reinterpret_cast<double2 *>(parts + 4 * (size_t)V.blk0);
    int par_set = 0;

    // this block's sum of a colour's squared residuals
    auto put = [&](int colour, auto acc) {
        double s;
        if (NV > 1)
            s = block_sum((double)acc);
        else
            s = block_total(acc, reinterpret_cast<decltype(acc) *>(buf), bpart, cwarp);
        if (tid == ctid)
            own[colour] = s;
    };
    // barrier of the group; false when a wait of the group gave up.  The
    // residuals `acc` of the phase it ends (`colour`, if >= 0) are added up
    // while the others arrive: the sum is needed after the next barrier
    auto sync = [&](int colour, auto acc) -> bool {
        target += nb;
        __syncthreads();
        if (tid == ctid)
            group_arrive(gr);
        if (colour >= 0)
            put(colour, acc);
        if (tid == ctid)
            ok = group_wait(gr, target);
        __syncthreads();
        return ok;
    };
    // the barrier that ends a body, and the controller on the group's sums;
    // meanwhile the other warps run `ahead`
    auto sync_ctrl = [&](bool sums, auto &&ahead) -> bool {
        target += nb;
        __syncthreads();
        if (tid == ctid) {
            if (sums)
                part[par_set * nb + rank] = make_double2(own[0], own[1]);
            group_arrive(gr);
            ok = group_wait(gr, target);
        }
        if (AHEAD)
            __syncthreads(); // the others go on to `ahead`
        else
            __syncwarp();
        if ((tid >> 5) == cwarp && ok) {
            double a = 0.0, c = 0.0;
            if (sums) {
                const double2 *pa = part + par_set * nb;
#pragma unroll 4
                for (unsigned t = tid & 31; t < nb; t += 32) {
                    const double2 x = __ldcg(pa + t);
                    a += x.x;
                    c += x.y;
                }
                a = warp_sum(a);
                c = warp_sum(c);
            }
            if (tid == ctid) {
                if (MIXED)
                    ctrl_mixed_update(&S, a, c, &P);
                else
                    ctrl64_update(&S, a, c, &P);
            }
        }
        if (AHEAD && works && ok)
            ahead();
        par_set ^= 1;
        __syncthreads();
        return ok;
    };

    bool good = true, have = false;
    if (!MIXED) {
        Ahead64 h = {};
        if (S.z == 0) { // the first iteration's red half-sweep (no residual yet)
            Sweep64<0>(V, 0).run(V, q0, dq, false, h);
            good = sync(-1, 0.0);
            if (tid == 0)
                S.z = 1;
            __syncthreads();
        }
        for (int body = 0; good && body < max_bodies && !S.stop; ++body) {
            const int z = S.z;
            if (!(good = sync(1, Sweep64<1>(V, z).run(V, q0, dq, have, h))))
                break;
            put(0, Sweep64<0>(V, z).run(V, q0, dq, false, h));
            good = sync_ctrl(true, [&] { h = Sweep64<1>(V, z + 1).ahead(V, q0); });
            have = AHEAD && works;
        }
    } else {
        Ahead32 h = {};
        for (int body = 0; good && body < max_bodies && !S.stop && !S.paused; ++body) {
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
                good = sync_ctrl(true, [] {});
                have = false;
            } else if (mode == 1) {
                if (S.keep)
                    Sweep32<0>(V, ds, omega).run(V, q0, dq, false, h);
                else
                    phase_round_from_zero(V, ds, omega, q0, dq);
                good = sync_ctrl(false, [&] { h = Sweep32<1>(V, ds ^ 1, omega).ahead(V, q0); });
                have = AHEAD && works;
            } else {
                if (!(good = sync(1, Sweep32<1>(V, ds, omega).run(V, q0, dq, have, h))))
                    break;
                put(0, Sweep32<0>(V, ds, omega).run(V, q0, dq, false, h));
                good = sync_ctrl(true, [&] { h = Sweep32<1>(V, ds ^ 1, omega).ahead(V, q0); });
                have = AHEAD && works;
            }
        }
    }
    if (rank == 0 && tid == 0) {
        if (!good || !(S.stop || (MIXED && S.paused))) { // a wait ran out, or the bodies did
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

static const void *loop_kernel(int mixed, int nv, bool ahead)
{
    if (nv > 1)
        return mixed ? (const void *)k_loop<1, SS4D_BATCH_MAX_VOLUMES, 0>
                     : (const void *)k_loop<0, SS4D_BATCH_MAX_VOLUMES, 0>;
    if (ahead)
        return mixed ? (const void *)k_loop<1, 1, 1> : (const void *)k_loop<0, 1, 1>;
    return mixed ? (const void *)k_loop<1, 1, 0> : (const void *)k_loop<0, 1, 0>;
}

static int resident(const void *kernel, int threads, int sm_count)
{
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, 0) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return per * sm_count;
}

int loop_grid(int mixed, int nv, int threads, int sm_count)
{
    return resident(loop_kernel(mixed, nv, false), threads, sm_count);
}

int loop_most_blocks(int threads, int sm_count)
{
    int most = 0;
    for (int q = 0; q < 4; ++q) {
        const int n = resident(loop_kernel(q & 1, 1, q & 2), threads, sm_count);
        most = n > most ? n : most;
    }
    return most;
}

// AHEAD up to three rounds per phase, in the FP64 form only where the warp it
// gives up costs no further round (us of a step, plain -> AHEAD):
//   FP64   32^3 x 8 (1 round) 571 -> 562, 45 x 37 x 29 x 7 (2) 722 -> 697,
//          48 x 48 x 36 x 10 (3) 1133 -> 1092, 48 x 48 x 32 x 8 (3 instead of
//          2) 884 -> 1005, 96 x 64 x 64 x 10 (14) 3874 -> 3886;
//   mixed  20^3 x 4 (1) 374 -> 325, 45 x 37 x 29 x 7 (2) 550 -> 476,
//          48 x 48 x 36 x 10 (3) 743 -> 650, 64 x 48 x 48 x 8 (4) 780 -> 791,
//          96 x 64 x 64 x 10 (14) 1711 -> 1931.
int loop_plan(int mixed, const FlatIndex &F, int threads, int sm_count, bool *ahead)
{
    const long long n = mixed ? F.npairs : F.ntargets;
    const int plain = resident(loop_kernel(mixed, 1, false), threads, sm_count);
    const int other = resident(loop_kernel(mixed, 1, true), threads, sm_count);
    if (plain <= 0 || other <= 0)
        return 0;
    auto rounds = [&](int grid, int work) { return (n + (long long)grid * work - 1) / ((long long)grid * work); };
    const long long r = rounds(other, threads - 32);
    *ahead = r <= 3 && (mixed || r <= rounds(plain, threads));
    const int work = *ahead ? threads - 32 : threads, grid = *ahead ? other : plain;
    const long long need = (n + work - 1) / work;
    return need < grid ? (int)need : grid;
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
                        const DevParams *par, double *parts, LoopGroup *groups, int max_bodies, bool ahead, cudaStream_t stream)
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
    return cudaLaunchCooperativeKernel(loop_kernel(mixed, nv, ahead), dim3(grid), dim3(threads), args, 0, stream);
}

} // namespace ss4d
