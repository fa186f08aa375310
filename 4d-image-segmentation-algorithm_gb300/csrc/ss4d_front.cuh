// ss4d_front.cuh — the presmoothing (segmentation4D.c:337-409) as one
// persistent launch, for the plain form's exact FP64 arithmetic
// (ss4d_front64.cu) and the mixed form's float-float one (ss4d_front_ff.cu).
//
// The image is split by colour like the solver's u, two adjacent columns of a
// row in one 16-byte unit, so a half-sweep reads its own colour and the
// other's once each and a thread's two targets share their index arithmetic.
// The launch runs, with barriers between: the reflection of the image's
// ghosts and the split copy; half-sweeps until the stop; the result back into
// the image.  No phase is spent on the residual: the red half-sweep of
// iteration z + 1 forms the red voxels' residual after iteration z from the
// neighbour sum it needs anyway (writing the other of two red buffers, so
// that the red values of z remain), and the black half-sweep forms the black
// voxels' after their own update.  Every block adds the partial sums in the
// same order and decides alike, as in ss4d_loop.cu.  A ghost next to an
// interior voxel holds that voxel's initial value all along (it is reflected
// once, before the iterations), which is the split copy's own value: ghosts
// need no storage.
#pragma once

#include "ss4d_exact.cuh"
#include "ss4d_loop.cuh"

namespace ss4d {

struct FrontState {
    int z, near, status, pad_;
    double R, R1;
};

// A stop test is reported as near the tolerance where the reference's sum
// R' of the same residuals could lie on its other side.  With n residuals r,
// R = h^4 sum r^2 and e the bound of what one residual's rounding may differ
// by, |R' - R| <= rel R + 2 h^4 e sum |r| + n h^4 e^2, and sum |r| <= sqrt(n)
// sqrt(sum r^2): rel stands for the order of the sum.  e = eps d U: a residual
// is formed from values of at most d U, with U the largest |u|.  Where the
// residuals are r, U <= max |image| + max |r| (the smoothing's matrix is
// diagonally dominant by 1), and max |r| <= sqrt(R / h^4).
struct FrontNear {
    double rel, eps, n;
};
__host__ __device__ inline double front_near_band(const FrontNear &f, double d, double h4, double most, double R)
{
    const double e = f.eps * d * (most + sqrt(R / h4));
    return f.rel * R + 2.0 * e * sqrt(f.n * R * h4) + f.n * h4 * e * e;
}

struct FrontArgs {
    Geo g;
    FlatIndex F;
    double *img;
    void *P[2], *R[2], *B; // split arrays of 8-byte values: initial image, red (two), black
    void *fold;            // float-float form: the smoothed image for the g faces (ss4d_front_ff.cu), or null
    int Hk;                // its fold
    float fold_scale;      // and the power of two it is scaled by
    double c, omega, d, y, h4, tol, maxit; // d = 1 + 8c, y its reciprocal (FP64 form: for div_by_const)
    FrontNear near;
    int last; // the residual after the last iteration is wanted
    double *parts;
    LoopGroup *group;
    FrontState *st;
};

template <int C>
struct FrontColour {
    static constexpr int value = C;
};

template <class A>
__device__ __forceinline__ void presmooth_body(const FrontArgs &a)
{
    typedef typename A::Q Q;
    const FlatIndex &F = a.F;
    const Geo &g = a.g;
    __shared__ FrontState S;
    __shared__ int ok, stop;
    __shared__ unsigned top;
    __shared__ double gap; // the least |R - tol| of the tests
    const int tid = threadIdx.x;
    const unsigned nb = gridDim.x, rank = blockIdx.x, dq = nb * blockDim.x;
    unsigned target = 0;
    const unsigned q0 = F.npairs <= 2 * dq ? ((tid >> 5) * nb + rank) * 32 + (tid & 31) : rank * blockDim.x + tid;
    int set = 0;
    if (tid == 0) {
        S.z = 1;
        S.near = S.status = 0;
        S.R = S.R1 = 0.0;
        stop = 0;
        top = 0;
        gap = INFINITY;
    }
    __syncthreads();
    auto put = [&](int colour, double acc) {
        acc = block_sum(acc);
        if (tid == 0)
            a.parts[(set * 2 + colour) * nb + rank] = acc;
    };
    auto sync = [&](int colour, double acc) -> bool {
        target += nb;
        __syncthreads();
        if (tid == 0)
            group_arrive(a.group);
        if (colour >= 0)
            put(colour, acc);
        if (tid == 0)
            ok = group_wait(a.group, target);
        __syncthreads();
        return ok;
    };

    // ghosts of the image: clamped coordinates (the reference's axis-by-axis
    // copies leave every ghost, edges included, with the nearest interior
    // voxel's value); a warp per padded row
    {
        const unsigned rows = (unsigned)(g.jM * g.kM * g.lM);
        const int lane = tid & 31;
        for (unsigned r = (rank * blockDim.x + tid) >> 5; r < rows; r += dq >> 5) {
            const unsigned rk = fdiv(r, g.fjM), l = fdiv(rk, g.fkM);
            const int j = (int)(r - rk * g.fjM.d), k = (int)(rk - l * g.fkM.d);
            const int jc = min(max(j, 1), g.ny), kc = min(max(k, 1), g.nz), lc = min(max((int)l, 1), g.nt);
            double *row = a.img + (size_t)r * g.iM;
            if (jc == j && kc == k && lc == (int)l) {
                if (lane < 2)
                    row[lane ? g.iM - 1 : 0] = row[lane ? g.nx : 1];
            } else {
                const double *src = a.img + nat_index(g, 0, jc, kc, lc);
                for (int i = lane; i < g.iM; i += 32)
                    row[i] = src[min(max(i, 1), g.nx)];
            }
        }
    }
    unsigned high = 0; // of the largest |value|: its upper word
    // split copy: columns x, x + 1 of both colours from the voxels 2x + 1 .. 2x + 4
    for (unsigned q = q0; q < F.npairs; q += dq) {
        int j, k, l;
        const Place t = place<2>(F, F.dP, 0, q, j, k, l);
        const int i = t.i - 1 + t.p; // 2x + 1: colour p == 1
        const double *src = a.img + nat_index(g, i, j, k, l);
        double v[4];
#pragma unroll
        for (int m = 0; m < 4; ++m)
            v[m] = i + m <= F.nx ? src[m] : 0.0;
#pragma unroll
        for (int m = 0; m < 4; ++m)
            high = max(high, (unsigned)__double2hiint(v[m]) & 0x7fffffffu);
        // colour 0 has row phase t.p here, colour 1 the other
        static_cast<Q *>(a.P[t.p ? 0 : 1])[t.s >> 1] = A::make(v[0], v[2]);
        static_cast<Q *>(a.P[t.p ? 1 : 0])[t.s >> 1] = A::make(v[1], v[3]);
    }
    high = __reduce_max_sync(0xffffffffu, high);
    if ((tid & 31) == 0)
        atomicMax(&top, high);
    __syncthreads();
    if (tid == 0)
        atomicMax(&a.group->top, top);
    if (!sync(-1, 0.0)) {
        if (rank == 0 && tid == 0)
            a.st->status = SS4D_ERR_TIMEOUT;
        return;
    }

    const typename A::Const C = A::constants(a);
    // one half-sweep of colour COL: own values from src to dst, neighbours
    // from oth; returns the sum of squared residuals (of the values before
    // the update for red, after it for black)
    auto half = [&](auto col_tag, const Q *src, const Q *oth, const Q *prev, Q *dst) -> double {
        constexpr int COL = decltype(col_tag)::value;
        typename A::Acc acc = A::zero();
        for (unsigned q = q0; q < F.npairs; q += dq) {
            int j, k, l;
            const Place t = place<2>(F, F.dP, COL, q, j, k, l);
            if (t.i > F.nx)
                continue;
            const unsigned s = t.s >> 1, Hy = F.Hs >> 1, Hz = F.Hz >> 1, Hw = F.Hw >> 1;
            const Q *const own0 = prev + s; // a ghost neighbour's value
            const Q u = A::live(src + s), pv = A::live(own0);
            const Q vx = A::live(oth + s);
            const auto ex = t.p ? A::second(oth + s - 1) : A::first(oth + s + 1);
            const Q ym = A::live(j == 1 ? own0 : oth + s - Hy), yp = A::live(j == F.ny ? own0 : oth + s + Hy);
            const Q zm = A::live(k == 1 ? own0 : oth + s - Hz), zp = A::live(k == F.nz ? own0 : oth + s + Hz);
            const Q wm = A::live(l == 1 ? own0 : oth + s - Hw), wp = A::live(l == g.nt ? own0 : oth + s + Hw);
            Q xr = t.p ? vx : A::up(vx, ex), xl = t.p ? A::down(ex, vx) : vx;
            const bool two = t.i + 2 <= F.nx;
            if (t.i == 1)
                xl = A::with_first(xl, pv);
            if (t.i == F.nx)
                xr = A::with_first(xr, pv);
            if (t.i + 2 == F.nx)
                xr = A::with_second(xr, pv);
            dst[s] = A::template update<COL>(C, u, pv, xr, xl, ym, yp, zm, zp, wm, wp, two, acc);
        }
        return A::template total<COL>(a, acc);
    };
    Q *const P0 = static_cast<Q *>(a.P[0]), *const P1 = static_cast<Q *>(a.P[1]);
    Q *const R0 = static_cast<Q *>(a.R[0]), *const R1 = static_cast<Q *>(a.R[1]), *const B = static_cast<Q *>(a.B);
    bool good = true;
    half(FrontColour<0>{}, P0, P1, P0, R1); // iteration 1
    good = sync(-1, 0.0);
    while (good && !stop) {
        const int z = S.z;
        Q *const cur = z & 1 ? R1 : R0, *const nxt = z & 1 ? R0 : R1;
        const double black = half(FrontColour<1>{}, z == 1 ? P1 : B, cur, P1, B);
        if (!a.last && z >= a.maxit) { // the last iteration, its residual not wanted
            good = sync(-1, 0.0);
            break;
        }
        if (!(good = sync(1, black)))
            break;
        put(0, half(FrontColour<0>{}, cur, B, P0, nxt));
        target += nb;
        __syncthreads();
        if (tid < 32) {
            int fine = 1;
            if (tid == 0) {
                group_arrive(a.group);
                fine = group_wait(a.group, target);
            }
            fine = __shfl_sync(0xffffffffu, fine, 0);
            double sum = 0.0;
            if (fine) {
                const double *pa = a.parts + set * 2 * nb;
                for (unsigned t = tid; t < 2 * nb; t += 32)
                    sum += __ldcg(pa + t);
                sum = warp_sum(sum);
            }
            if (tid == 0) {
                ok = fine;
                const double R = sum * a.h4;
                S.R = R;
                if (z == 1)
                    S.R1 = R;
                gap = fmin(gap, fabs(R - a.tol));
                if (R > a.tol && z < a.maxit)
                    S.z = z + 1;
                else
                    stop = 1;
            }
        }
        set ^= 1;
        __syncthreads();
        good = ok;
    }
    if (rank == 0 && tid == 0) {
        const double most = __hiloint2double((int)(__ldcg(&a.group->top) + 1), 0); // the next value above
        S.near = isfinite(gap) && gap <= front_near_band(a.near, a.d, a.h4, most, fmax(a.tol, 0.0) + gap);
        S.status = good ? (isfinite(S.R) ? SS4D_OK : SS4D_ERR_NONFINITE) : SS4D_ERR_TIMEOUT;
        *a.st = S;
    }
    if (!good)
        return;
    // the result: the red buffer of the last iteration and black
    const Q *const red = S.z & 1 ? R1 : R0;
    for (unsigned q = q0; q < F.npairs; q += dq) {
        int j, k, l;
        const Place t = place<2>(F, F.dP, 0, q, j, k, l);
        const int i = t.i - 1 + t.p;
        double *out = a.img + nat_index(g, i, j, k, l);
        const Q vr = A::live(red + (t.s >> 1)), vb = A::live(B + (t.s >> 1));
        double v[4], w[2];
        A::get(t.p ? vr : vb, w);
        v[0] = w[0];
        v[2] = w[1];
        A::get(t.p ? vb : vr, w);
        v[1] = w[0];
        v[3] = w[1];
#pragma unroll
        for (int m = 0; m < 4; ++m)
            if (i + m <= F.nx)
                out[m] = v[m];
    }
    A::fold(a, red, rank * blockDim.x + tid, dq);
}

// threads per block, co-resident blocks (4 partial sums each), and the launches
constexpr int FRONT64_THREADS = 256, FRONT_FF_THREADS = 512;
int presmooth64_grid(int sm_count);
int presmooth_ff_grid(int sm_count);
cudaError_t launch_presmooth64(const FrontArgs &a, int grid, cudaStream_t st);
cudaError_t launch_presmooth_ff(const FrontArgs &a, int grid, cudaStream_t st);

} // namespace ss4d
