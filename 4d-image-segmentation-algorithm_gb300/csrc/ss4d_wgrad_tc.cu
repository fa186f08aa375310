// ss4d_wgrad_tc.cu — the weight gradient of the warm-start network's 3x3x3
// convolutions on the fifth-generation tensor cores.
//
// dW[tap][co][ci] = sum over the voxels v of X[v + tap][ci] dY[v][co] is a
// matrix product whose contraction runs over the voxels: for each of the three
// dy taps D[(dz, ci)][(dx, co)], K = 16 voxels (8 along x, two rows of y) a
// multiply-add; along x the sum runs over w = v + dx, X[w] dY[w - dx], so that the
// dx taps are shifts of dY and lie in N.  The channel-group planar activations
// are what such operands want when the channels are the contiguous index
// (MN-major, no swizzle: a core matrix is 8 voxels by 8 channels, 128 contiguous bytes of a row of a
// channel group).  A tile of X, 8 x 18 x (WZ + 2) voxels, arrives by one TMA
// box with the channel groups inside the planes, [z][group][y][x][8], so
// that consecutive groups and then consecutive planes lie a constant stride
// apart: 128 rows of the A operand starting at plane p are the channels of
// planes p, p + 1, p + 2 (the three dz taps of output plane p) and beyond,
// whose rows of D nobody reads.  dY, 8 x 16 x WZ voxels at the three shifts,
// [z][dx][group][y][x][8], is the B operand.  Both operands are the tiles
// themselves; voxels outside the crop are zeros of the TMA's fill.  A fourth
// product with a matrix of ones adds up dY for the bias gradient.
//
// The accumulators stay in tensor memory over all tiles of a CTA
// (K = 256 voxels each); at its end a CTA writes its partial sums, which
// k_reduce_grad adds in CTA order.  One thread issues loads and
// multiply-adds, two tiles are in flight; waits are bounded as in
// ss4d_conv_tc.cu.
//
// What bounds it: the tensor core's operand reads from shared memory, 4 KB of
// A and 3 KB of B per multiply-add of M = 128, N = 96, K = 16, and the fill of a
// CTA's eight tiles (the tensor pipe is 35 % busy, DRAM 15 %).  With each of
// the nine (dy, dx) taps a multiply-add of its own (N = 32, 4 KB of A for 1 KB of
// B) a layer of 8 crops of 40 x 40 x 20 took 54 us, now 32.
#include <cuda_bf16.h>

#include "ss4d_conv_tc.cuh"
#include "ss4d_tc_ptx.cuh"

namespace ss4d {
namespace tc {

namespace {

constexpr int WG_WARPS = 4, WG_THREADS = 32 * (WG_WARPS + 1);
constexpr int WZ = 2; // planes of a tile: two tiles of X and of three dY's fit

// CIN input channels of X, NY channels of dY (N)
template <int CIN, int NY> struct WgCfg {
    static constexpr int XG = CIN / 8, YG = NY / 8; // channel groups
    static constexpr int XGS = TX * HY * 16;        // bytes of one group of one plane
    static constexpr int YGS = TX * TY * 16;
    static constexpr int XB = (WZ + 2) * XG * XGS, YB = WZ * 3 * YG * YGS; // one tile
    static constexpr int XS = (XB + 1023) / 1024 * 1024, YS = (YB + 1023) / 1024 * 1024;
    static constexpr int ONES = 4096; // 128 x 16 ones
    static constexpr int NACC = 10;
    static constexpr int TCOLS = 512; // 10 accumulators of NY columns: the next power of two for NY = 32
    // X tiles first: the rows of A past the tile's last plane stay inside
    static constexpr int SMEM = 1024 + 2 * XS + 2 * YS + ONES + 128;
    static_assert(NACC * NY <= TCOLS, "tensor memory");
    static_assert(XS + 2 * YS >= (WZ - 1) * XG * XGS + 16 * XGS,
                  "the A operand's unused rows must stay in shared memory");
    static_assert(SMEM <= 227 * 1024, "shared memory per CTA");
};

struct WgArgs {
    int nx, ny, nz, nf, cout;
    float *partial; // [CTA][27 cout CIN + cout]
    int *err;
    int withhold_loads; // test of the timeout path: issue no load, so that the wait for it runs out
};

template <int CIN, int NY>
__global__ void __launch_bounds__(WG_THREADS, 1)
    k_wgrad_tc(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap ymap, WgArgs a)
{
    using C = WgCfg<CIN, NY>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *ysm = smem + 2 * C::XS, *ones = ysm + 2 * C::YS;
    uint64_t *bars = reinterpret_cast<uint64_t *>(ones + C::ONES); // full[2], done[2], all
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 5);
    int *abort_flag = reinterpret_cast<int *>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t full0 = smem_u32(bars), done0 = smem_u32(bars + 2), all0 = smem_u32(bars + 4);

    for (int q = tid; q < C::ONES / 4; q += blockDim.x)
        reinterpret_cast<uint32_t *>(ones)[q] = 0x3F803F80u; // two BF16 ones
    if (tid == 0) {
        for (int b = 0; b < 2; ++b) {
            mbar_init(full0 + 8 * b, 1);
            mbar_init(done0 + 8 * b, 1);
        }
        mbar_init(all0, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // the ones, for the MMAs
    if (warp == 0)
        tmem_alloc(smem_u32(tmem_slot), C::TCOLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    const int ntx = (a.nx + TX - 1) / TX, nty = (a.ny + TY - 1) / TY, ntz = (a.nz + WZ - 1) / WZ;
    const long long ntiles = (long long)ntx * nty * ntz * a.nf;
    const long long first = blockIdx.x;
    const int my_n = (int)((ntiles - 1 - first) / gridDim.x + 1); // the grid has at most ntiles CTAs

    if (warp == WG_WARPS) {
        if (lane == 0) {
            // D FP32, A and B BF16 and both MN-major, M = 128, N = 3 NY (the ones' NY)
            const uint32_t type = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                                  ((uint32_t)(128 >> 4) << 24);
            const uint32_t idesc = type | ((uint32_t)(3 * NY >> 3) << 17), idesc1 = type | ((uint32_t)(NY >> 3) << 17);
            // MN-major without swizzle: LBO = stride of the core matrices along
            // K (the next row of 8 voxels), SBO = along M or N (the next group)
            const uint64_t odesc = make_desc(smem_u32(ones), 128, 256);
            auto load = [&](int it) {
                long long r = first + (long long)it * gridDim.x;
                const int x0 = (int)(r % ntx) * TX;
                r /= ntx;
                const int y0 = (int)(r % nty) * TY;
                r /= nty;
                const int z0 = (int)(r % ntz) * WZ, f = (int)(r / ntz), b = it & 1;
                mbar_expect_tx(full0 + 8 * b, C::XB + C::YB);
                tma_load_5d(smem_u32(smem + b * C::XS), &xmap, full0 + 8 * b, 8 * x0, y0 - 1, 0, z0 - 1, f);
                for (int q = 0; q < 3 * WZ; ++q) // plane q / 3, tap dx = q % 3 - 1: dY from x0 - dx on
                    tma_load_5d(smem_u32(ysm + b * C::YS + q * C::YG * C::YGS), &ymap, full0 + 8 * b,
                                8 * (x0 + 1 - q % 3), y0, 0, z0 + q / 3, f);
            };
            bool ok = true;
            int loads = 0, mmas = 0;
            for (int it = 0; it < 2 && it < my_n && !a.withhold_loads; ++it, ++loads)
                load(it);
            for (int it = 0; it < my_n; ++it) {
                const int b = it & 1;
                if (!mbar_wait(full0 + 8 * b, (it >> 1) & 1)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint64_t x0 = make_desc(smem_u32(smem + b * C::XS), TX * 16, C::XGS);
                const uint64_t y0 = make_desc(smem_u32(ysm + b * C::YS), TX * 16, C::YGS);
#pragma unroll 1
                for (int p = 0; p < WZ; ++p)
#pragma unroll
                    for (int y = 0; y < TY; y += 2) {
                        const uint64_t bd = y0 + ((p * 3 * C::YG * C::YGS + y * TX * 16) >> 4);
                        const uint64_t ad = x0 + ((p * C::XG * C::XGS + y * TX * 16) >> 4);
                        const uint32_t acc = (it | p | y) != 0;
#pragma unroll
                        for (int dy = 0; dy < 3; ++dy)
                            umma_bf16(tmem + dy * 3 * NY, ad + ((dy * TX * 16) >> 4), bd, idesc, acc);
                        umma_bf16(tmem + 9 * NY, odesc, bd + ((C::YG * C::YGS) >> 4), idesc1, acc);
                    }
                umma_commit(done0 + 8 * b);
                mmas = it + 1;
                if (it + 2 < my_n) { // this stage again once its multiply-adds are done
                    if (!mbar_wait(done0 + 8 * b, (it >> 1) & 1)) {
                        ok = false;
                        break;
                    }
                    load(it + 2);
                    ++loads;
                }
            }
            if (ok) {
                umma_commit(all0);
            } else {
                *abort_flag = 1;
                atomicExch(a.err, 1);
                // loads and multiply-adds still in flight
                for (int t = mmas; t < loads; ++t)
                    mbar_wait(full0 + 8 * (t & 1), (t >> 1) & 1);
                for (int t = mmas > 2 ? mmas - 2 : 0; t < mmas; ++t)
                    mbar_wait(done0 + 8 * (t & 1), (t >> 1) & 1);
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(all0) : "memory");
            }
        }
    } else {
        int ok = 0;
        // the producer's own bounded waits end before this one
        for (int t = 0; t < 8 && !ok; ++t) {
            if (lane == 0)
                ok = mbar_wait(all0, 0);
            ok = __shfl_sync(0xffffffffu, ok, 0);
        }
        if (ok && !*(volatile int *)abort_flag) {
            tc_fence_after();
            const int row = warp * 32 + lane, dz = row / CIN, ci = row % CIN;
            float *out = a.partial + (size_t)blockIdx.x * (27 * a.cout * CIN + a.cout);
#pragma unroll 1
            for (int dd = 0; dd < 10; ++dd)
#pragma unroll 1
                for (int h = 0; h < NY / 16; ++h) {
                    uint32_t r[16];
                    tmem_ld_x16(tmem + dd * NY + 16 * h + ((uint32_t)(warp * 32) << 16), r);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        const int co = 16 * h + e;
                        if (co >= a.cout)
                            break;
                        if (dd < 9) {
                            if (dz < 3)
                                out[((size_t)(9 * dz + dd) * a.cout + co) * CIN + ci] = __uint_as_float(r[e]);
                        } else if (row == 0) {
                            out[(size_t)27 * a.cout * CIN + co] = __uint_as_float(r[e]);
                        }
                    }
                }
        } else if (lane == 0) {
            atomicExch(a.err, 1);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        tmem_dealloc(tmem, C::TCOLS);
}

// the CTAs' partial sums, added in CTA order (eight interleaved runs of CTAs,
// then the runs in order), into the master layout [27][cout][cin], [cout]; all
// layers in one launch (blockIdx.y; one after the other they took 7 us each).
// A kernel of the step that gave up a wait (err) left rows, or what they were
// formed from, unwritten: the gradient is NaN then.
struct GradJobs {
    GradJob v[MAX_GRADS];
};
__global__ void __launch_bounds__(256) k_reduce_grad(const __grid_constant__ GradJobs jobs, int rows,
                                                     const int *__restrict__ err)
{
    const float *const partial = jobs.v[blockIdx.y].partial;
    float *const gw = jobs.v[blockIdx.y].gw, *const gb = jobs.v[blockIdx.y].gb;
    const int cout = jobs.v[blockIdx.y].cout, cinp = jobs.v[blockIdx.y].cin, cin = jobs.v[blockIdx.y].cin_real;
    const int failed = __ldg(err);
    __shared__ float part[8][33];
    const int n = 27 * cout * cin, cols = 27 * cout * cinp + cout;
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int q = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (q < n + cout) {
        const int c = q < n ? q / cin * cinp + q % cin : 27 * cout * cinp + (q - n);
        for (int r = g; r < rows; r += 8)
            s += __ldcs(partial + (size_t)r * cols + c);
    }
    part[g][lane] = s;
    __syncthreads();
    if (g == 0 && q < n + cout) {
        for (int k = 1; k < 8; ++k)
            s += part[k][lane];
        if (failed)
            s = __int_as_float(0x7fffffff);
        if (q < n)
            gw[q] = s;
        else
            gb[q - n] = s;
    }
}

// planar tensor [nf][C/8][nz][ny][nx][8] as (x and 8 channels, y, group, z, frame)
bool planar_map(CUtensorMap *m, const void *p, int c, int nx, int ny, int nz, int nf, int bx, int by, int bz)
{
    PFN_cuTensorMapEncodeTiled_v12000 enc = encode_fn();
    if (!enc)
        return false;
    const cuuint64_t row = (cuuint64_t)nx * 16, vol = row * ny * nz;
    const cuuint64_t dims[5] = {(cuuint64_t)nx * 8, (cuuint64_t)ny, (cuuint64_t)c / 8, (cuuint64_t)nz, (cuuint64_t)nf};
    const cuuint64_t strides[4] = {row, vol, row * ny, vol * (c / 8)};
    const cuuint32_t box[5] = {(cuuint32_t)bx * 8, (cuuint32_t)by, (cuuint32_t)c / 8, (cuuint32_t)bz, 1};
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void *>(p), dims, strides, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int CIN, int NY>
cudaError_t run(const void *x, const void *dy, const WgArgs &a, int grid, cudaStream_t st)
{
    using C = WgCfg<CIN, NY>;
    CUtensorMap xm, ym;
    if (!planar_map(&xm, x, CIN, a.nx, a.ny, a.nz, a.nf, TX, HY, WZ + 2) ||
        !planar_map(&ym, dy, NY, a.nx, a.ny, a.nz, a.nf, TX, TY, 1))
        return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(k_wgrad_tc<CIN, NY>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess)
        return e;
    k_wgrad_tc<CIN, NY><<<grid, WG_THREADS, C::SMEM, st>>>(xm, ym, a);
    return cudaGetLastError();
}

} // namespace

int wgrad_ctas(int nx, int ny, int nz, int nf, int sm_count)
{
    const long long tiles = (long long)((nx + TX - 1) / TX) * ((ny + TY - 1) / TY) * ((nz + WZ - 1) / WZ) * nf;
    return (int)(tiles < sm_count ? tiles : sm_count);
}

cudaError_t wgrad_tc(const GradJob &j, const void *x, const void *dy, int nx, int ny, int nz, int nf, int *err,
                     int withhold_loads, int sm_count, cudaStream_t st)
{
    WgArgs a;
    a.nx = nx;
    a.ny = ny;
    a.nz = nz;
    a.nf = nf;
    a.cout = j.cout;
    a.partial = j.partial;
    a.err = err;
    a.withhold_loads = withhold_loads;
    const int grid = wgrad_ctas(nx, ny, nz, nf, sm_count);
    if (j.cin == 16 && j.ycha == 32)
        return run<16, 32>(x, dy, a, grid, st);
    if (j.cin == 32 && j.ycha == 32)
        return run<32, 32>(x, dy, a, grid, st);
    if (j.cin == 32 && j.ycha == 16)
        return run<32, 16>(x, dy, a, grid, st);
    return cudaErrorInvalidValue;
}

cudaError_t reduce_grads(const GradJob *jobs, int njobs, int ctas, const int *err, cudaStream_t st)
{
    if (njobs < 1 || njobs > MAX_GRADS)
        return cudaErrorInvalidValue;
    GradJobs g = {};
    int most = 0;
    for (int q = 0; q < njobs; ++q) {
        g.v[q] = jobs[q];
        const int n = 27 * jobs[q].cout * jobs[q].cin_real + jobs[q].cout;
        most = n > most ? n : most;
    }
    k_reduce_grad<<<dim3((most + 31) / 32, njobs), 256, 0, st>>>(g, ctas, err);
    return cudaGetLastError();
}

} // namespace tc
} // namespace ss4d
