// ss4d_conv_tc.cu — the warm-start network's 3x3x3 convolution on the
// fifth-generation tensor cores: tcgen05.mma with BF16 operands in shared
// memory, FP32 accumulators in tensor memory (TMEM), input tiles brought in
// by the tensor memory accelerator (TMA).
//
// A convolution over every frame of [F][nz][ny][nx][CIN] BF16 activations
// (channels last) is an implicit GEMM: D[voxel][cout] = sum over the 27 taps
// and the input channels of X[voxel + tap][cin] W[tap][cout][cin].  A CTA
// takes output tiles of 8 (x) by 16 (y) voxels by TZ planes (z) of one
// frame; each plane is one M = 128 accumulator (row m = x + 8 y) of N
// output channels, the TZ accumulators of a tile side by side in tensor
// memory, plane p at column (TZ - 1 - p) N.  Activations are channel-group planar in global memory
// ([F][C/8][nz][ny][nx][8], ss4d_conv_tc.cuh), so the input halo tile,
// 10 x 18 x (TZ + 2) voxels, arrives in shared memory by one TMA box per
// group of 8 channels whose rows are 160 contiguous bytes (x and the 8
// channels merged into one dimension); a box lands as [z][y][x][8 channels],
// 16 bytes per voxel, which is the canonical K-major layout of the UMMA
// operands without swizzle: a core matrix is 8 consecutive voxels (rows) by
// 8 channels (16 bytes).  So the A operand of
// tap (dx, dy, dz) for output plane p is the halo tile itself, its
// descriptor starting at voxel (dx, dy, p + dz): rows x + 8 y step 16 bytes
// within a core matrix and the row stride of the halo (160 bytes) between
// the 8-row groups, channel groups a plane apart.  No operand is copied per
// tap.  The view at halo plane hz = p + dz serves the output planes hz,
// hz - 1 and hz - 2 (dz = 0, 1, 2) alike, so one MMA does them together:
// the weights of the three dz taps are stacked along N (3N rows per (dy, dx)
// block in shared memory) and, with the accumulators in descending plane
// order, the N blocks of taps dz_lo..dz_hi land on the accumulators of
// planes hz - dz_lo .. hz - dz_hi.  A tile of TZ planes then takes
// (TZ + 2) x 9 MMAs per K chunk instead of 27 TZ, each reading its A operand
// from shared memory once for up to three planes.  An accumulate flag is
// per MMA, not per column, so a first MMA of A = 0 clears all TZ
// accumulators and every MMA after it accumulates.
//
// Per CTA: one thread of the last warp issues the TMA loads and the MMAs, four
// or eight warps drain the accumulators (TMEM -> registers -> bias, ReLU, mask ->
// global); STAGES halo tiles and two accumulator buffers are in flight and
// the roles meet only at mbarriers, so the loads of the next tiles and the
// epilogue of tile i-1 run while the tensor core works on tile i.  Every wait on an
// mbarrier is bounded (about a second of clock cycles); one that runs out
// sets an error flag the host reads, the producer waits (bounded) for its own
// loads and MMAs in flight, and the CTA frees its tensor memory and returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ss4d_conv_tc.cuh"
#include "ss4d_tc_ptx.cuh"

namespace ss4d {
namespace tc {

// ---- the kernel ---------------------------------------------------------------

// warp roles: warps 0-3 (MASKED 0-7: warps w and w + 4 reach the same 32 lanes
// of tensor memory and take half of the planes each) read the accumulators
// and store; lane 0 of the last warp issues the loads and the MMAs.  Barriers,
// one phase per use: full[s] (the loads of the tile in halo stage s landed), done[b] (the MMAs of the tile in accumulator buffer
// b completed: tcgen05.commit), free[b] (the epilogue warps have read
// buffer b).  Tile it uses stage it % STAGES and buffer it % 2.
// A data gradient's epilogue loads its masks, 64 bytes a voxel: with eight
// warps and the masks loaded ahead 51 -> 30 us per hidden layer at 8 crops of
// 40x40x20 (four tiles per CTA).  A training step (three such convolutions
// among its eleven products) took with four and with eight, in us: 2 tiles per SM
// 234 and 228, 8 593 and 583, 16 1117 and 1086, 32 2112 and 2061, 63 4076 and
// 3980; 4 frames of 128x128x64 (54) 3595 and 3521.  Without masks the
// tensor core's operand reads set the pace and four warps, whose tensor-memory
// reads are spread out, disturb them less (a forward of 12 frames of
// 128x128x64 3.64 ms against 3.73).
__host__ __device__ constexpr int epi_warps(bool masked)
{
    return masked ? 8 : 4;
}
template <int CIN, int N, bool MASKED>
__global__ void __launch_bounds__(32 * (epi_warps(MASKED) + 1), 1)
    k_conv_tc(const __grid_constant__ CUtensorMap tmap, TcArgs a)
{
    constexpr int EPI_WARPS = epi_warps(MASKED);
    using C = TcCfg<CIN, N>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *halo0 = smem;
    unsigned char *wsm = smem + STAGES * C::HALO;
    unsigned char *zsm = wsm + C::WBYTES;                            // zeros: the clearing MMA's A operand
    uint64_t *bars = reinterpret_cast<uint64_t *>(zsm + C::ZBYTES); // full[STAGES], done[2], free[2]
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + STAGES + 4);
    int *abort_flag = reinterpret_cast<int *>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t full0 = smem_u32(bars), done0 = smem_u32(bars + STAGES), free0 = smem_u32(bars + STAGES + 2);

    // weights: global (already in core-matrix order) -> shared
    for (int q = tid; q < C::WBYTES / 16; q += blockDim.x)
        reinterpret_cast<uint4 *>(wsm)[q] = __ldg(reinterpret_cast<const uint4 *>(a.w) + q);
    for (int q = tid; q < C::ZBYTES / 16; q += blockDim.x)
        reinterpret_cast<uint4 *>(zsm)[q] = make_uint4(0, 0, 0, 0);
    if (tid == 0) {
        for (int q = 0; q < STAGES; ++q)
            mbar_init(full0 + 8 * q, 1);
        for (int b = 0; b < 2; ++b) {
            mbar_init(done0 + 8 * b, 1);
            mbar_init(free0 + 8 * b, EPI_WARPS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // the weights were written by the generic proxy; the MMAs read through the async proxy
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 0)
        tmem_alloc(smem_u32(tmem_slot), C::TCOLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    const int ntx = (a.nx + TX - 1) / TX, nty = (a.ny + TY - 1) / TY, ntz = (a.nz + TZ - 1) / TZ;
    const long long ntiles = (long long)ntx * nty * ntz * a.nf;
    const long long first = blockIdx.x;
    const int my_n = first < ntiles ? (int)((ntiles - 1 - first) / gridDim.x + 1) : 0;
    auto tile_xyzf = [&](int it, int &x0, int &y0, int &z0, int &f) {
        long long r = first + (long long)it * gridDim.x;
        x0 = (int)(r % ntx) * TX;
        r /= ntx;
        y0 = (int)(r % nty) * TY;
        r /= nty;
        z0 = (int)(r % ntz) * TZ;
        f = (int)(r / ntz);
    };

    if (warp == EPI_WARPS) {
        if (lane == 0) {
            // ---- producer: loads and MMAs ----
            // K-major operands without swizzle: LBO = stride of the core
            // matrices along K, SBO = stride of the 8-row groups along M (N)
            // instruction descriptor: D FP32, A and B BF16, M = 128, N = n
            auto idesc = [](int n) {
                return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
            };
            const uint64_t b0 = make_desc(smem_u32(wsm), (3 * N / 8) * 128, 128);
            // 128 rows x 16 K of zeros (16-row groups 128 B apart, K halves 2 KB apart)
            const uint64_t zdesc = make_desc(smem_u32(zsm), 16 * 128, 128);
            int loads = 0, mmas = 0; // issued
            auto load = [&](int it) {
                int x0, y0, z0, f;
                tile_xyzf(it, x0, y0, z0, f);
                const int q = it % STAGES;
                mbar_expect_tx(full0 + 8 * q, C::NCG * C::BOX_BYTES);
                const uint32_t dst = smem_u32(halo0 + q * C::HALO);
                // box {x and 8 channels merged: 80, y: 18, z: TZ + 2, plane: 1}
#pragma unroll
                for (int g = 0; g < C::NCG; ++g)
                    tma_load_4d(dst + g * PLANE, &tmap, full0 + 8 * q, 8 * (x0 - 1), y0 - 1, z0 - 1,
                                f * C::NCG + g);
                loads = it + 1;
            };
            bool ok = true;
            // withhold_loads (a test of the timeout path) issues no load:
            // the first wait below runs out and nothing is left in flight
            for (int it = 0; it < STAGES - 1 && it < my_n && !a.withhold_loads; ++it)
                load(it);
            for (int it = 0; it < my_n && ok; ++it) {
                const int q = it % STAGES, b = it & 1;
                // this tile's loads, and its accumulator buffer read out (tile it-2)
                if (!mbar_wait(full0 + 8 * q, (it / STAGES) & 1) ||
                    (it >= 2 && !mbar_wait(free0 + 8 * b, ((it - 2) >> 1) & 1))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                // descriptors differ only in their start address (the low 14
                // bits, in 16-byte units): one base each, plus constants
                const uint64_t a0 = make_desc(smem_u32(halo0 + q * C::HALO), PLANE, HX * 16);
                const uint32_t acc = tmem + (uint32_t)(b * TZ * N);
                // clear the TZ accumulators: A = 0 times any B rows (finite weights)
                umma_bf16(acc, zdesc, b0, idesc(TZ * N), 0);
#pragma unroll
                for (int hz = 0; hz < TZ + 2; ++hz) {
                    // the dz taps whose output plane hz - dz lies in the tile
                    const int dz_lo = hz - (TZ - 1) > 0 ? hz - (TZ - 1) : 0, dz_hi = hz < 2 ? hz : 2;
                    const uint32_t col = (uint32_t)((TZ - 1 - hz + dz_lo) * N);
#pragma unroll
                    for (int dd = 0; dd < 9; ++dd) {
                        const int dy = dd / 3, dx = dd % 3;
                        const uint32_t vox = (uint32_t)((hz * HY + dy) * HX + dx);
#pragma unroll
                        for (int kc = 0; kc < C::KC; ++kc)
                            umma_bf16(acc + col, a0 + ((2 * kc * PLANE + vox * 16) >> 4),
                                      b0 + (((dd * C::KC + kc) * C::WBLK + dz_lo * N * 16) >> 4),
                                      idesc((dz_hi - dz_lo + 1) * N), 1);
                    }
                }
                umma_commit(done0 + 8 * b);
                mmas = it + 1;
                // the next load goes to the halo stage that tile it-1 read:
                // wait for its MMAs while this tile's run behind them
                const int nxt = it + STAGES - 1;
                if (nxt < my_n && !a.withhold_loads) {
                    if (it >= 1 && !mbar_wait(done0 + 8 * ((it - 1) & 1), ((it - 1) >> 1) & 1)) {
                        ok = false;
                        break;
                    }
                    load(nxt);
                }
            }
            if (!ok) {
                *abort_flag = 1;
                atomicExch(a.err, 1);
                // the last loads and MMAs of each buffer may still be in
                // flight (earlier phases of their barriers have completed)
                for (int t = loads - STAGES; t < loads; ++t)
                    if (t >= mmas && t >= 0)
                        mbar_wait(full0 + 8 * (t % STAGES), (t / STAGES) & 1);
                for (int t = mmas - 2; t < mmas; ++t)
                    if (t >= 0)
                        mbar_wait(done0 + 8 * (t & 1), (t >> 1) & 1);
            }
        }
    } else {
        // ---- epilogue warps: accumulators -> bias, ReLU, mask -> global ----
        const int quad = warp & 3, m = quad * 32 + lane;
        constexpr int PL = TZ / (EPI_WARPS / 4); // planes per warp
        const int p0 = (warp >> 2) * PL;
        const long long vol = (long long)a.nx * a.ny * a.nz;
        for (int it = 0; it < my_n; ++it) {
            const int b = it & 1;
            int x0, y0, z0, f;
            tile_xyzf(it, x0, y0, z0, f);
            const int ox = x0 + (m & 7), oy = y0 + (m >> 3);
            MaskRegs<N> mask[MASKED ? PL : 1];
            if (MASKED) { // the masks come while the tensor core works on the tile
#pragma unroll
                for (int p = 0; p < PL; ++p) {
                    const int oz = z0 + p0 + p;
                    if (ox < a.nx && oy < a.ny && oz < a.nz)
                        load_masks<N>(a, mask[p], f, ((long long)oz * a.ny + oy) * a.nx + ox, vol);
                }
            }
            // one lane waits, so that the warp stays converged for the
            // .sync.aligned tensor-memory loads
            int ok = 0;
            if (lane == 0)
                ok = mbar_wait(done0 + 8 * b, (it >> 1) & 1);
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok || *(volatile int *)abort_flag) {
                if (lane == 0)
                    atomicExch(a.err, 1);
                break;
            }
            tc_fence_after();
            auto plane = [&](int p) {
                const uint32_t col =
                    tmem + (uint32_t)(b * TZ * N + (TZ - 1 - p0 - p) * N) + ((uint32_t)(quad * 32) << 16);
                float v[N];
#pragma unroll
                for (int h = 0; h < N / 16; ++h) {
                    uint32_t r[16];
                    tmem_ld_x16(col + 16 * h, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        v[16 * h + e] = __uint_as_float(r[e]);
                }
                const int oz = z0 + p0 + p;
                if (ox < a.nx && oy < a.ny && oz < a.nz)
                    epilogue_store<N, MASKED>(a, v, mask[MASKED ? p : 0], f,
                                              ((long long)oz * a.ny + oy) * a.nx + ox, vol);
            };
            if (MASKED) {
#pragma unroll
                for (int p = 0; p < PL; ++p)
                    plane(p);
            } else {
#pragma unroll 1
                for (int p = 0; p < PL; ++p)
                    plane(p);
            }
            // this warp is done with the buffer's tensor memory
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(free0 + 8 * b) : "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        tmem_dealloc(tmem, C::TCOLS);
}

// ---- host side ------------------------------------------------------------------

PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return (PFN_cuTensorMapEncodeTiled_v12000)p;
    }();
    return fn;
}

namespace {
template <int CIN, int N, bool MASKED>
cudaError_t launch_masked(const CUtensorMap &m, const TcArgs &a, long long tiles, int sm_count, cudaStream_t st)
{
    constexpr int threads = 32 * (epi_warps(MASKED) + 1);
    static const int per_sm = [] { // once, whichever thread comes first
        cudaFuncSetAttribute(k_conv_tc<CIN, N, MASKED>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcCfg<CIN, N>::SMEM);
        int p = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p, k_conv_tc<CIN, N, MASKED>, threads, TcCfg<CIN, N>::SMEM);
        return p < 1 ? 1 : (p > 2 ? 2 : p); // tensor memory: 2 x TCOLS <= 512 columns
    }();
    const long long cap = (long long)sm_count * per_sm;
    const int grid = (int)(tiles < cap ? tiles : cap);
    k_conv_tc<CIN, N, MASKED><<<grid, threads, TcCfg<CIN, N>::SMEM, st>>>(m, a);
    return cudaGetLastError();
}
} // namespace

// the 4-D map of a planar tensor ([nf * cin/8 planes][nz][ny][nx * 8] BF16,
// x and the 8 channels of a group merged) with boxes of the halo tile
static bool make_map(CUtensorMap *m, const void *x, int cin, int nx, int ny, int nz, int nf)
{
    PFN_cuTensorMapEncodeTiled_v12000 enc = encode_fn();
    if (!enc)
        return false;
    const cuuint64_t dims[4] = {(cuuint64_t)nx * 8, (cuuint64_t)ny, (cuuint64_t)nz, (cuuint64_t)nf * (cin / 8)};
    const cuuint64_t row = (cuuint64_t)nx * 16; // bytes of one x row of a plane
    const cuuint64_t strides[3] = {row, row * ny, row * ny * nz};
    const cuuint32_t box[4] = {HX * 8, HY, HZ, 1};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(x), dims, strides, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int CIN, int N>
static cudaError_t launch(const void *x, const TcArgs &a, int sm_count, cudaStream_t st)
{
    CUtensorMap m;
    if (!make_map(&m, x, CIN, a.nx, a.ny, a.nz, a.nf))
        return cudaErrorInvalidValue;
    const long long tiles = tc_tiles(a.nx, a.ny, a.nz, a.nf);
    return a.mask ? launch_masked<CIN, N, true>(m, a, tiles, sm_count, st)
                  : launch_masked<CIN, N, false>(m, a, tiles, sm_count, st);
}

cudaError_t conv_tc(int cin, int n, const void *x, const TcArgs &a, int sm_count, cudaStream_t st)
{
    if (cin == 16 && n == 32)
        return launch<16, 32>(x, a, sm_count, st);
    if (cin == 32 && n == 32)
        return launch<32, 32>(x, a, sm_count, st);
    if (cin == 32 && n == 16)
        return launch<32, 16>(x, a, sm_count, st);
    return cudaErrorInvalidValue;
}

// W[tap][cout][cin] FP32 (master layout, or the data-gradient layout with
// `reverse`: tap 26 - t and the channel roles swapped) -> B blocks
// [9 (dy, dx)][KC][2 K groups][3N/8 N groups][8 rows][8 K] BF16, row
// dz * N + co of block (dy, dx) holding tap 9 dz + 3 dy + dx; zero beyond
// cout/cin
// All of a network's blocks in one launch (blockIdx.y): seven of 3.3 us each
// were 5 % of a training step.
struct PackJobs {
    PackJob v[MAX_PACKS];
};
__global__ void __launch_bounds__(256) k_pack_tc(const __grid_constant__ PackJobs jobs)
{
    const PackJob &p = jobs.v[blockIdx.y];
    const int kc_n = p.cinp / 16, n = p.n;
    const int total = 9 * kc_n * 2 * 3 * n * 8;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < total; q += gridDim.x * blockDim.x) {
        int r = q;
        const int e = r % 8;
        r /= 8;
        const int row = r % 8;
        r /= 8;
        const int j = r % (3 * n / 8);
        r /= 3 * n / 8;
        const int h = r % 2;
        r /= 2;
        const int kc = r % kc_n;
        const int dd = r / kc_n;
        const int nr = 8 * j + row, dz = nr / n;
        const int tap = 9 * dz + dd, co = nr % n, ci = 16 * kc + 8 * h + e;
        float v = 0.f;
        if (!p.reverse) {
            if (co < p.cout && ci < p.cin)
                v = p.w[((size_t)tap * p.cout + co) * p.cin + ci];
        } else {
            // data gradient: output channel co = the forward's input channel,
            // input channel ci = the forward's output channel
            if (co < p.cin && ci < p.cout)
                v = p.w[((size_t)(26 - tap) * p.cout + ci) * p.cin + co];
        }
        p.out[q] = __float2bfloat16_rn(v);
    }
}

// after a convolution that gave up a wait: the prediction becomes NaN, which
// every consumer discards (the warm start's check) or shows (the loss)
__global__ void k_poison_if_err(const int *__restrict__ err, float *y, long long n)
{
    if (!*err)
        return;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        y[i] = __int_as_float(0x7fc00000);
}

void poison_if_err(const int *err, float *y, long long n, cudaStream_t st)
{
    k_poison_if_err<<<256, 256, 0, st>>>(err, y, n);
}

void pack_tc(const PackJob *jobs, int njobs, cudaStream_t st)
{
    PackJobs p = {};
    for (int q = 0; q < njobs && q < MAX_PACKS; ++q)
        p.v[q] = jobs[q];
    k_pack_tc<<<dim3(64, njobs), 256, 0, st>>>(p);
}

} // namespace tc
} // namespace ss4d
