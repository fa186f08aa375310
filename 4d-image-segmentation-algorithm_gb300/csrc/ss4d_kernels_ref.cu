// ss4d_kernels_ref.cu — natural-layout FP64 kernels in the reference's
// expression order.
//
// This translation unit is compiled with --fmad=false: every multiply and add
// is rounded separately, the way the x86-64 reference build rounds them, and
// division and square root are IEEE round-to-nearest.  The voxel updates here
// therefore reproduce the reference's arithmetic; only the order of the
// residual/norm summations differs (a parallel reduction instead of one
// serial sum).  They serve the SS4D_ARITH_REFERENCE form, the edge detector of
// every form (run once per segmentation), the MCF boundary and exact
// solution, the rescale, the mask and the norms.
#include <cooperative_groups.h>
#include <float.h>
#include <math.h>

#include "ss4d_exact.cuh"
#include "ss4d_kernels.cuh"

namespace ss4d {

// ---------------------------------------------------------------------------
// launch geometry over interior voxels: x along threadIdx.x, y along
// threadIdx.y, (k, l) along blockIdx.z.

__device__ inline bool interior_ijkl(const Geo &g, int &i, int &j, int &k, int &l)
{
    i = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    j = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    const int kl = blockIdx.z;
    k = 1 + kl % g.nz;
    l = 1 + kl / g.nz;
    return i <= g.nx && j <= g.ny;
}

// the voxels of one colour ((i + j + k + l) & 1 == colour), one per thread:
// thread x indexes the pairs (i, i+1) of a row, so every lane of a warp
// updates a voxel (a lane masked off by a colour test costs the FP64 pipe as
// much as an active one)
__device__ inline bool colour_ijkl(const Geo &g, int colour, int &i, int &j, int &k, int &l)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    j = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    const int kl = blockIdx.z;
    k = 1 + kl % g.nz;
    l = 1 + kl / g.nz;
    i = 1 + 2 * t + ((colour + j + k + l + 1) & 1);
    return i <= g.nx && j <= g.ny;
}

__device__ inline unsigned block_linear()
{
    return (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
}

__device__ inline int flat_tid()
{
    return threadIdx.y * blockDim.x + threadIdx.x;
}

// Block reduction over a 2D block (flattened thread order).
__device__ inline double block_sum2d(double v)
{
    __shared__ double s2[32];
    const int t = flat_tid();
    const int lane = t & 31, wid = t >> 5;
    const int nw = (blockDim.x * blockDim.y + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0)
        s2[wid] = v;
    __syncthreads();
    double r = 0;
    if (wid == 0) {
        r = lane < nw ? s2[lane] : 0.0;
        r = warp_sum(r);
    }
    return r;
}

// ---------------------------------------------------------------------------
// Neumann reflection (segmentation4D.c:826-864) in one launch: the
// reference's copies, axis by axis over full padded ranges, leave every ghost
// (edges and corners included) with the value of the nearest interior voxel,
// so a ghost reads it at its clamped coordinates.  A warp per padded row.

__global__ void k_reflect(Geo g, double *u)
{
    const unsigned rows = (unsigned)(g.jM * g.kM * g.lM), step = (gridDim.x * blockDim.x) >> 5;
    const int lane = threadIdx.x & 31;
    for (unsigned r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += step) {
        const unsigned rk = fdiv(r, g.fjM), l = fdiv(rk, g.fkM);
        const int j = (int)(r - rk * g.fjM.d), k = (int)(rk - l * g.fkM.d);
        const int jc = min(max(j, 1), g.ny), kc = min(max(k, 1), g.nz), lc = min(max((int)l, 1), g.nt);
        double *row = u + (size_t)r * g.iM;
        if (jc == j && kc == k && lc == (int)l) {
            if (lane < 2)
                row[lane ? g.iM - 1 : 0] = row[lane ? g.nx : 1];
        } else {
            const double *src = u + nat_index(g, 0, jc, kc, lc);
            for (int i = lane; i < g.iM; i += 32)
                row[i] = src[min(max(i, 1), g.nx)];
        }
    }
}

// ---------------------------------------------------------------------------
// residual passes: a thread sums RESID_K k-planes before the block reduction
#define RESID_K 4

__device__ inline bool resid_ijl(const Geo &g, int &i, int &j, int &k0, int &l)
{
    i = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    j = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    const int nkb = (g.nz + RESID_K - 1) / RESID_K;
    k0 = 1 + (blockIdx.z % nkb) * RESID_K;
    l = 1 + blockIdx.z / nkb;
    return i <= g.nx && j <= g.ny;
}

// explicit smoother (segmentation4D.c:422-441): one Jacobi-style step from
// prev over i = 1 .. iMax-3 (the reference's x loop stops one column short)
// and the interior j, k, l; the neighbours are summed in the reference's order

__global__ void k_presmooth_explicit(Geo g, double *v, const double *prev, double coeff)
{
    int i, j, k, l;
    if (!interior_ijkl(g, i, j, k, l) || i > g.nx - 1)
        return;
    const long long o = nat_index(g, i, j, k, l);
    v[o] = (1.0 - 8.0 * coeff) * prev[o]
           + coeff * (prev[o + 1] + prev[o - 1] + prev[o + g.sy] + prev[o - g.sy] + prev[o + g.sz] + prev[o - g.sz]
                      + prev[o + g.sw] + prev[o - g.sw]);
}

// ---------------------------------------------------------------------------
// separable Gaussian along one axis (an option beside the reference's
// implicit presmoothing, which is not a Gaussian): out = sum_{m=-R..R}
// w[|m|] in(c + m) in order of m, each term added by a fused multiply-add
// (explicit fma: one rounding, the same on the host, whatever --fmad says),
// the coordinate mirrored about the volume's faces as the reference's
// reflection does (ghost 0 = voxel 1: x < 1 -> 1 - x, x > n -> 2n + 1 - x);
// interior voxels only

__device__ inline int gauss_mirror(int x, int n)
{
    // each two reflections move x by 2n towards [1, n]: |x| <= R + n needs
    // fewer than 2 R / n + 2 steps (R <= SS4D_GAUSS_MAX_RADIUS)
    for (int q = 0; q < 4 * SS4D_GAUSS_MAX_RADIUS + 4; ++q) {
        if (x < 1)
            x = 1 - x;
        else if (x > n)
            x = 2 * n + 1 - x;
        else
            break;
    }
    return x;
}

template <int AXIS>
__global__ void k_gauss_axis(Geo g, const double *__restrict__ in, double *__restrict__ out, GaussWeights W)
{
    int i, j, k, l;
    if (!interior_ijkl(g, i, j, k, l))
        return;
    const int c[4] = {i, j, k, l};
    const int n[4] = {g.nx, g.ny, g.nz, g.nt};
    const long long st[4] = {1, g.sy, g.sz, g.sw};
    const long long o = nat_index(g, i, j, k, l);
    const long long base = o - (long long)c[AXIS] * st[AXIS];
    double acc = 0.0;
    for (int m = -W.R; m <= W.R; ++m)
        acc = fma(W.w[m < 0 ? -m : m], in[base + (long long)gauss_mirror(c[AXIS] + m, n[AXIS]) * st[AXIS]], acc);
    out[o] = acc;
}

// ---------------------------------------------------------------------------
// face gradients (segmentation4D.c:455-548, :594-821): normal component
// (v[nb]-v[c])/h, tangential ((v[nb+a]+v[c+a]) - (v[nb-a]+v[c-a]))/(4h),
// squares summed in x, y, z, w order.

__device__ inline double face_sq(const double *v, long long c, long long nb, const long long st[4], int d,
                                 double h, double q)
{
    double comp[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if (a == d)
            comp[a] = (v[nb] - v[c]) / h;
        else
            comp[a] = ((v[nb + st[a]] + v[c + st[a]]) - (v[nb - st[a]] + v[c - st[a]])) / q;
    }
    return (comp[0] * comp[0]) + (comp[1] * comp[1]) + (comp[2] * comp[2]) + (comp[3] * comp[3]);
}

// face_sq of the face between o and o + st[d], in the reference's expression
// order: through div_by_const (ih, iq: the reciprocals of h and q = 4h), or,
// POW2, times q^2 with h a power of two: the divisions then scale exactly, so
// the squares and their sum are formed unscaled (the normal difference times
// 4) and the caller scales once.
template <bool POW2, int D>
__device__ inline double face_sq_plus(const double *v, long long o, const long long st[4], double h, double q,
                                      double ih, double iq)
{
    const long long nb = o + st[D];
    double comp[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if (a == D) {
            const double t = v[nb] - v[o];
            comp[a] = POW2 ? t * 4.0 : div_by_const(t, h, ih);
        } else {
            const double t = (v[nb + st[a]] + v[o + st[a]]) - (v[nb - st[a]] + v[o - st[a]]);
            comp[a] = POW2 ? t : div_by_const(t, q, iq);
        }
    }
    return (comp[0] * comp[0]) + (comp[1] * comp[1]) + (comp[2] * comp[2]) + (comp[3] * comp[3]);
}

// The 8 g faces of every interior voxel, each shared face computed once.  The
// reference's value for the + face of voxel o along axis d and for the - face
// of voxel o + st[d] is the same number: the normal difference only changes
// sign (exactly) before it is squared, and the tangential sums add the same
// pairs (IEEE addition is commutative).  The thread at o computes the + face
// along d when o's other coordinates are interior, and stores it as g[2d][o]
// (o interior along d) and g[2d+1][o + st[d]] (o + st[d] interior along d).
// Threads cover coordinates 0..n along every axis.
template <bool POW2, int D>
__device__ inline void gface_plus(const Geo &g, const int c[4], const int n[4], long long o, const long long st[4],
                                  const double *i0, const double *ithr, GPtrs8 &gout, double h, double q, double ih,
                                  double iq, double K, double theta, double rho)
{
#pragma unroll
    for (int a = 0; a < 4; ++a)
        if (a != D && c[a] < 1)
            return;
    const double s0 = face_sq_plus<POW2, D>(i0, o, st, h, q, ih, iq);
    const double s1 = ithr ? face_sq_plus<POW2, D>(ithr, o, st, h, q, ih, iq) : 0.0;
    const double gv = 1.0 / (1 + K * (theta * s0 + rho * s1));
    if (c[D] >= 1)
        gout.p[2 * D][o] = gv;
    if (c[D] < n[D])
        gout.p[2 * D + 1][o + st[D]] = gv;
}

// One thread per voxel of a plane, i fastest across rows: bound by the FP64
// pipe, which a warp holds for the same time whatever lanes it uses, and a
// tile of 128 x 2 left a quarter of them empty at 97 x 101.  With that and the
// scaling (24 of about 230 FP64 instructions a voxel with two images) the edge
// detector of two images took, in us: 97 x 101 x 53 x 11 8846 -> 7859, 256^2 x
// 128 x 10 111.4e3 -> 103.3e3; h = 0.3: 11348 -> 10062, 142.8e3 -> 135.2e3.
// POW2: theta and rho hold the scale 1/(4h)^2.
template <bool POW2>
__global__ void __launch_bounds__(256) k_gfaces(Geo g, FastDiv row, FastDiv planes, const double *i0,
                                                const double *ithr, GPtrs8 gout, double h, double K, double theta,
                                                double rho, double ih, double iq)
{
    const unsigned at = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = (int)fdiv(at, row), i = (int)(at - j * row.d);
    const int l = (int)fdiv(blockIdx.y, planes), k = (int)(blockIdx.y - l * planes.d);
    if (j > g.ny)
        return;
    const int c[4] = {i, j, k, l};
    const int n[4] = {g.nx, g.ny, g.nz, g.nt};
    const long long o = nat_index(g, i, j, k, l);
    const long long st[4] = {1, g.sy, g.sz, g.sw};
    const double q = 4.0 * h;
    gface_plus<POW2, 0>(g, c, n, o, st, i0, ithr, gout, h, q, ih, iq, K, theta, rho);
    gface_plus<POW2, 1>(g, c, n, o, st, i0, ithr, gout, h, q, ih, iq, K, theta, rho);
    gface_plus<POW2, 2>(g, c, n, o, st, i0, ithr, gout, h, q, ih, iq, K, theta, rho);
    gface_plus<POW2, 3>(g, c, n, o, st, i0, ithr, gout, h, q, ih, iq, K, theta, rho);
}

// _gs_coefficients_ / _gs_coefficients_mcf in reference order
__global__ void k_coef_ref(Geo g, const double *u, CPtrs8 gin, int has_g, GPtrs8 coef, double h, double eps2)
{
    int i, j, k, l;
    if (!interior_ijkl(g, i, j, k, l))
        return;
    const long long o = nat_index(g, i, j, k, l);
    const long long st[4] = {1, g.sy, g.sz, g.sw};
    const double q = 4.0 * h;
    double nf[8];
#pragma unroll
    for (int f = 0; f < 8; ++f) {
        const int d = f >> 1;
        const long long nb = (f & 1) ? o - st[d] : o + st[d];
        nf[f] = sqrt(face_sq(u, o, nb, st, d, h, q) + eps2);
    }
    double mean = ((nf[0] + nf[1] + nf[2] + nf[3] + nf[4] + nf[5] + nf[6] + nf[7]) / 8.0);
    double vc = sqrt(mean * mean + eps2);
#pragma unroll
    for (int f = 0; f < 8; ++f)
        coef.p[f][o] = has_g ? vc * gin.p[f][o] * (1.0 / nf[f]) : vc * (1.0 / nf[f]);
}

// ---------------------------------------------------------------------------
// red-black SOR in reference order (segmentation4D.c:232-308)

__global__ void k_sor_half_ref(Geo g, double *u, const double *prev, CPtrs8 a, double c, double omega, int colour)
{
    int i, j, k, l;
    if (!colour_ijkl(g, colour, i, j, k, l))
        return;
    const long long o = nat_index(g, i, j, k, l);
    const double E = a.p[0][o], W = a.p[1][o], N = a.p[2][o], S = a.p[3][o];
    const double T = a.p[4][o], B = a.p[5][o], FW = a.p[6][o], BW = a.p[7][o];
    double gs = (prev[o] + c * ((E * u[o + 1]) + (W * u[o - 1]) + (S * u[o - g.sy]) + (N * u[o + g.sy])
                                + (B * u[o - g.sz]) + (T * u[o + g.sz]) + (BW * u[o - g.sw]) + (FW * u[o + g.sw])))
                / (1 + c * (E + W + N + S + T + B + FW + BW));
    u[o] = u[o] + omega * (gs - u[o]);
}

__global__ void k_sor_resid_ref(Geo g, const double *u, const double *prev, CPtrs8 a, double c, double h4,
                                double *partial)
{
    int i, j, k0, l;
    double acc = 0.0;
    if (resid_ijl(g, i, j, k0, l)) {
        for (int k = k0; k < k0 + RESID_K && k <= g.nz; ++k) {
            const long long o = nat_index(g, i, j, k, l);
            const double E = a.p[0][o], W = a.p[1][o], N = a.p[2][o], S = a.p[3][o];
            const double T = a.p[4][o], B = a.p[5][o], FW = a.p[6][o], BW = a.p[7][o];
            double r = u[o] * (1 + c * (E + W + N + S + T + B + FW + BW))
                       - c * ((E * u[o + 1]) + (W * u[o - 1]) + (S * u[o - g.sy]) + (N * u[o + g.sy])
                              + (B * u[o - g.sz]) + (T * u[o + g.sz]) + (BW * u[o - g.sw]) + (FW * u[o + g.sw]))
                       - prev[o];
            acc += (r * r) * h4;
        }
    }
    acc = block_sum2d(acc);
    if (flat_tid() == 0)
        partial[block_linear()] = acc;
}

// ---------------------------------------------------------------------------
// deterministic final reductions: one block, fixed order

// first stage of a long reduction: block b combines in[b*per, (b+1)*per)
__global__ void k_reduce_sum_part(const double *in, long long n, long long per, double *out)
{
    const long long beg = blockIdx.x * per, end = beg + per < n ? beg + per : n;
    double acc = 0.0;
    for (long long t = beg + threadIdx.x; t < end; t += blockDim.x)
        acc += in[t];
    acc = block_sum(acc);
    if (threadIdx.x == 0)
        out[blockIdx.x] = acc;
}

__global__ void k_reduce_sum(const double *partial, long long n, double *out)
{
    double acc = 0.0;
    for (long long t = threadIdx.x; t < n; t += blockDim.x)
        acc += partial[t];
    acc = block_sum(acc);
    if (threadIdx.x == 0)
        *out = acc;
}

// partial holds n (min, max) pairs; out[0] = min, out[1] = max,
// out[2] = min + level*(max-min)
__global__ void k_reduce_minmax(const double *partial, long long n, double level, double *out)
{
    double mn = 1e308, mx = -1e308;
    for (long long t = threadIdx.x; t < n; t += blockDim.x) {
        mn = fmin(mn, partial[2 * t]);
        mx = fmax(mx, partial[2 * t + 1]);
    }
    mn = block_min(mn);
    mx = block_max(mx);
    if (threadIdx.x == 0) {
        out[0] = mn;
        out[1] = mx;
        out[2] = mn + level * (mx - mn);
    }
}

// ---------------------------------------------------------------------------
// norms over every padded voxel (segmentation4D.c:194-213, :317-335)

__global__ void k_l2_partial(long long n, const double *a, const double *b, double h4, double *partial)
{
    double acc = 0.0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        double d = a[t] - b[t];
        acc += (d * d) * h4;
    }
    acc = block_sum(acc);
    if (threadIdx.x == 0)
        partial[blockIdx.x] = acc;
}

__global__ void k_mass_partial(long long n, const double *a, double h4, double *partial)
{
    double acc = 0.0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        acc += (a[t] * h4);
    acc = block_sum(acc);
    if (threadIdx.x == 0)
        partial[blockIdx.x] = acc;
}

// ---------------------------------------------------------------------------
// MCF exact solution and Dirichlet ghosts (mcf_4D.c:344-461)

__device__ inline double mcf_coord(int i, double h)
{
    return ((i - 1) * h) + (h / 2.) - 1.25;
}

// (x^2 + y^2 + z^2 + w^2 - 1) / 6 + t in the reference's order
__device__ __forceinline__ double mcf_value(double x, double y2, double z2, double w2, double t)
{
    return div_by_const(x * x + y2 + z2 + w2 - 1.0, 6.0, 1.0 / 6.0) + t;
}

// the coordinate of index q of an axis of M, on a face if asked for
__device__ __forceinline__ double mcf_axis(int q, int M, double h, bool face)
{
    return face ? (q == M - 1 ? (h / 2.) + 1.25 : -(h / 2.) - 1.25) : mcf_coord(q, h);
}

// On a ghost the reference's eight passes run x-lo, x-hi, ..., w-hi over full
// ranges: the last pass touching it decides its value, and it uses the special
// face coordinate on its own axis only: the last axis the voxel is a ghost on.
// With ghosts_only a thread per x ghost of the interior rows, then (as for
// the whole field) a warp per padded row that is all ghosts, y, z and w formed
// once per row.  A value costs tens of FP64 instructions, which a warp pays in
// full for one lane: walking every voxel, or a warp per interior row for its
// two ghosts, took 191-197 us at 40^4, every ghost with its own four coordinates 90.
__global__ void k_mcf_field(Geo g, double *u, double h, double t, int ghosts_only)
{
    const unsigned rows = (unsigned)(g.jM * g.kM * g.lM), threads = gridDim.x * blockDim.x;
    const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    auto coords = [&](unsigned r, int &j, int &k, int &l) {
        const unsigned rk = fdiv(r, g.fjM), q = fdiv(rk, g.fkM);
        j = (int)(r - rk * g.fjM.d);
        k = (int)(rk - q * g.fkM.d);
        l = (int)q;
        return j >= 1 && j <= g.ny && k >= 1 && k <= g.nz && l >= 1 && l <= g.nt;
    };
    auto square = [&](int q, int M, bool face) {
        const double c = mcf_axis(q, M, h, face);
        return c * c;
    };
    int j, k, l;
    if (ghosts_only)
        for (unsigned q = tid; q < 2 * rows; q += threads) {
            const unsigned r = q >> 1;
            const int i = (q & 1) ? g.iM - 1 : 0;
            if (coords(r, j, k, l))
                u[(size_t)r * g.iM + i] = mcf_value(mcf_axis(i, g.iM, h, true), square(j, g.jM, false),
                                                    square(k, g.kM, false), square(l, g.lM, false), t);
        }
    for (unsigned r = tid >> 5; r < rows; r += threads >> 5) {
        const bool inner = coords(r, j, k, l);
        if (inner && ghosts_only)
            continue;
        const bool fl = ghosts_only && (l == 0 || l == g.lM - 1), fk = ghosts_only && !fl && (k == 0 || k == g.kM - 1),
                   fj = ghosts_only && !fl && !fk;
        const double y2 = square(j, g.jM, fj), z2 = square(k, g.kM, fk), w2 = square(l, g.lM, fl);
        for (int i = lane; i < g.iM; i += 32)
            u[(size_t)r * g.iM + i] = mcf_value(mcf_coord(i, h), y2, z2, w2, t);
    }
}

// ---------------------------------------------------------------------------
// rescale to [0,1] per ball (segmentation4D.c:1020-1104): one block per
// frame; the balls of a frame are processed in their order because each
// ball's min/max sees the values the earlier balls rescaled.

// The test sqrt(dx^2 + dy^2 + dz^2) <= R is made on the squares: t2 is the
// largest double whose square root, correctly rounded, is at most R (found on
// the host), and the square root is monotonic; the squares per axis come from
// tables of the box, and what only compares runs on the integer pipe.  A
// frame's balls are a serial chain, and on one SM the FP64 pipe set its pace
// (414 us for five balls of radius 8 per frame with a square root per voxel and
// pass): a cluster of RESCALE_CTAS blocks shares a frame's rows and exchanges
// the extrema through distributed shared memory.

// tables of one ball's box; an axis longer than the table is formed in place
constexpr int BALL_TABLE = 256;
constexpr int RESCALE_CTAS = 8;

__device__ __forceinline__ double sq_at(const double *tab, int q, int i0, double c)
{
    if (q < BALL_TABLE)
        return tab[q];
    const double d = (i0 + q) - c;
    return d * d;
}

// a signed comparison of two keys compares the numbers (-0 below +0); its own inverse
__device__ inline long long dkey(long long b)
{
    return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}

// minimum of a and maximum of b over the block, in every thread
__device__ __forceinline__ void block_minmax_keys(long long &a, long long &b)
{
    __shared__ long long sa[32], sb[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const long long x = __shfl_xor_sync(0xffffffffu, a, o), y = __shfl_xor_sync(0xffffffffu, b, o);
        a = x < a ? x : a;
        b = y > b ? y : b;
    }
    __syncthreads();
    if (lane == 0) {
        sa[warp] = a;
        sb[warp] = b;
    }
    __syncthreads();
    for (int w = 0; w < nw; ++w) {
        a = sa[w] < a ? sa[w] : a;
        b = sb[w] > b ? sb[w] : b;
    }
}

__global__ void __cluster_dims__(RESCALE_CTAS, 1, 1) __launch_bounds__(256)
    k_rescale_balls(Geo g, double *v, const int *frame_first, const int *frame_count, const double *bx,
                    const double *by, const double *bz, double R, double t2, int l0)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ double tx[BALL_TABLE], ty[BALL_TABLE], tz[BALL_TABLE];
    __shared__ long long ext[2][RESCALE_CTAS][2]; // per parity of the ball: every block's extrema
    const int l = l0 + blockIdx.x / RESCALE_CTAS, rank = (int)cluster.block_rank();
    const int first = frame_first[l], count = frame_count[l];
    const int lane = threadIdx.x & 31, nw = (blockDim.x >> 5) * RESCALE_CTAS;
    const int warp = (threadIdx.x >> 5) * RESCALE_CTAS + rank;
    const long long t2b = __double_as_longlong(t2);
    // the other blocks' shared memory may be written only once they have all
    // started, which a barrier of the cluster alone establishes
    cluster.sync();
    for (int c = 0; c < count; ++c) {
        const double cx = bx[first + c], cy = by[first + c], cz = bz[first + c];
        const int k0 = (int)(cz - R - 0.5), j0 = (int)(cy - R - 0.5), i0 = (int)(cx - R - 0.5);
        const int nk = (int)(cz + R + 0.5) - k0 + 1, nj = (int)(cy + R + 0.5) - j0 + 1,
                  ni = (int)(cx + R + 0.5) - i0 + 1;
        const int most = max(ni, max(nj, nk)) < BALL_TABLE ? max(ni, max(nj, nk)) : BALL_TABLE;
        for (int q = threadIdx.x; q < most; q += blockDim.x) {
            const double dx = (i0 + q) - cx, dy = (j0 + q) - cy, dz = (k0 + q) - cz;
            tx[q] = dx * dx;
            ty[q] = dy * dy;
            tz[q] = dz * dz;
        }
        __syncthreads();
        // a warp of the cluster per row of the box; d2 <= t2 as a comparison of
        // bit patterns (d2 >= +0 or NaN; a negative or NaN t2 admits nothing)
        auto rows = [&](auto &&body) {
            if (!(t2 >= 0.0))
                return;
            for (int r = warp; r < nj * nk; r += nw) {
                const int kk = r / nj, jj = r - kk * nj;
                const double y2 = sq_at(ty, jj, j0, cy), z2 = sq_at(tz, kk, k0, cz);
                double *row = v + nat_index(g, i0, j0 + jj, k0 + kk, l);
                for (int ii = lane; ii < ni; ii += 32)
                    if (__double_as_longlong((sq_at(tx, ii, i0, cx) + y2) + z2) <= t2b)
                        body(row + ii);
            }
        };
        // the reference's starting bounds 100000 and 0; a NaN changes neither
        long long mn = dkey(__double_as_longlong(100000.0)), mx = dkey(__double_as_longlong(0.0));
        rows([&](double *p) {
            const long long b = __double_as_longlong(__ldcg(p));
            if ((b & 0x7fffffffffffffffLL) <= 0x7ff0000000000000LL) {
                const long long k = dkey(b);
                mn = k < mn ? k : mn;
                mx = k > mx ? k : mx;
            }
        });
        block_minmax_keys(mn, mx);
        if (threadIdx.x < RESCALE_CTAS) {
            long long(*to)[2] = cluster.map_shared_rank(ext[c & 1], threadIdx.x);
            to[rank][0] = mn;
            to[rank][1] = mx;
        }
        cluster.sync();
        for (int q = 0; q < RESCALE_CTAS; ++q) {
            mn = ext[c & 1][q][0] < mn ? ext[c & 1][q][0] : mn;
            mx = ext[c & 1][q][1] > mx ? ext[c & 1][q][1] : mx;
        }
        const double lo = __longlong_as_double(dkey(mn)), hi = __longlong_as_double(dkey(mx));
        const double quot = 1. / (hi - lo), off = lo * quot;
        rows([&](double *p) {
            const double val = __ldcg(p), nv = (quot * val) - off;
            if (c == 0 || val < nv)
                *p = nv;
        });
        cluster.sync(); // the next ball may cover the same voxels
    }
}

// ---------------------------------------------------------------------------
// initial segmentation (segmentation4D.c:876-1018, 1106-1147).  One block per
// frame walks that frame's balls in order, as k_rescale_balls does.

// minimum (from 100000) and maximum (from 0) of frame l inside the ball of
// radius R: _get3DMinWithinR_ / _get3DMaxWithinR_ (segmentation4D.c:897-969);
// the results in every thread
__device__ void ball_min_max(const Geo &g, const double *v, int l, double cx, double cy, double cz, double R,
                             double &mn_out, double &mx_out)
{
    const int k0 = (int)(cz - R - 0.5), k1 = (int)(cz + R + 0.5);
    const int j0 = (int)(cy - R - 0.5), j1 = (int)(cy + R + 0.5);
    const int i0 = (int)(cx - R - 0.5), i1 = (int)(cx + R + 0.5);
    const int ni = i1 - i0 + 1, nj = j1 - j0 + 1, nk = k1 - k0 + 1;
    const long long cnt = (long long)ni * nj * nk;
    double mn = 100000, mx = 0;
    for (long long t = threadIdx.x; t < cnt; t += blockDim.x) {
        const int i = i0 + (int)(t % ni), j = j0 + (int)((t / ni) % nj), k = k0 + (int)(t / ((long long)ni * nj));
        const double dx = i - cx, dy = j - cy, dz = k - cz;
        if (sqrt((dx * dx) + (dy * dy) + (dz * dz)) <= R) {
            const double val = v[nat_index(g, i, j, k, l)];
            mn = val < mn ? val : mn;
            mx = val > mx ? val : mx;
        }
    }
    mn = block_min(mn);
    mx = block_max(mx);
    __shared__ double r2[2];
    if (threadIdx.x == 0) {
        r2[0] = mn;
        r2[1] = mx;
    }
    __syncthreads();
    mn_out = r2[0];
    mx_out = r2[1];
    __syncthreads();
}

__global__ void k_ball_min_max(Geo g, const double *v, int l, double cx, double cy, double cz, double R, double *out)
{
    double mn, mx;
    ball_min_max(g, v, l, cx, cy, cz, R, mn, mx);
    if (threadIdx.x == 0) {
        out[0] = mn;
        out[1] = mx;
    }
}

// _locallyThreshold4Ddata_ (segmentation4D.c:971-1018): per ball the level
// alpha min + beta max of the input inside it; thr = the global maximum
// (from 0, _get4DMax_) wherever the input inside the ball exceeds it
__global__ void k_local_threshold(Geo g, const double *in, double *thr, const int *frame_first, const int *frame_count,
                                  const double *bx, const double *by, const double *bz, double R, double alpha,
                                  double beta, const double *minmax)
{
    const int l = 1 + blockIdx.x;
    const double gmax = minmax[1] > 0 ? minmax[1] : 0;
    const int first = frame_first[l], count = frame_count[l];
    for (int c = 0; c < count; ++c) {
        const double cx = bx[first + c], cy = by[first + c], cz = bz[first + c];
        double mn, mx;
        ball_min_max(g, in, l, cx, cy, cz, R, mn, mx);
        const double level = alpha * mn + beta * mx;
        const int k0 = (int)(cz - R - 0.5), k1 = (int)(cz + R + 0.5);
        const int j0 = (int)(cy - R - 0.5), j1 = (int)(cy + R + 0.5);
        const int i0 = (int)(cx - R - 0.5), i1 = (int)(cx + R + 0.5);
        const int ni = i1 - i0 + 1, nj = j1 - j0 + 1, nk = k1 - k0 + 1;
        const long long cnt = (long long)ni * nj * nk;
        for (long long t = threadIdx.x; t < cnt; t += blockDim.x) {
            const int i = i0 + (int)(t % ni), j = j0 + (int)((t / ni) % nj), k = k0 + (int)(t / ((long long)ni * nj));
            const double dx = i - cx, dy = j - cy, dz = k - cz;
            if (sqrt((dx * dx) + (dy * dy) + (dz * dz)) <= R) {
                const long long o = nat_index(g, i, j, k, l);
                if (in[o] > level)
                    thr[o] = gmax;
            }
        }
    }
}

// _generate4DsegmFunct_ (segmentation4D.c:1106-1147): in each ball's box
// (half-width R + 0.5) and within the fixed distance 12 of its centre,
// u = max(u, |1/(r + 0.5) - 1/12.5|) and Mmask = 1; balls in order
__global__ void k_generate_segm(Geo g, double *u, double *Mmask, const int *frame_first, const int *frame_count,
                                const double *bx, const double *by, const double *bz, double R)
{
    const int l = 1 + blockIdx.x;
    const double v = 0.5, Rf = 12.;
    const int first = frame_first[l], count = frame_count[l];
    for (int c = 0; c < count; ++c) {
        const double cx = bx[first + c], cy = by[first + c], cz = bz[first + c];
        const int k0 = (int)(cz - R - 0.5), k1 = (int)(cz + R + 0.5);
        const int j0 = (int)(cy - R - 0.5), j1 = (int)(cy + R + 0.5);
        const int i0 = (int)(cx - R - 0.5), i1 = (int)(cx + R + 0.5);
        const int ni = i1 - i0 + 1, nj = j1 - j0 + 1, nk = k1 - k0 + 1;
        const long long cnt = (long long)ni * nj * nk;
        for (long long t = threadIdx.x; t < cnt; t += blockDim.x) {
            const int i = i0 + (int)(t % ni), j = j0 + (int)((t / ni) % nj), k = k0 + (int)(t / ((long long)ni * nj));
            const double dx = i - cx, dy = j - cy, dz = k - cz;
            if (sqrt((dx * dx) + (dy * dy) + (dz * dz)) <= Rf) {
                const double nv = fabs((1. / (sqrt((dx * dx) + (dy * dy) + (dz * dz)) + v)) - (1. / (Rf + v)));
                const long long o = nat_index(g, i, j, k, l);
                if (u[o] < nv)
                    u[o] = nv;
                Mmask[o] = 1.;
            }
        }
        __syncthreads(); // the next ball may cover the same voxels
    }
}

// ---------------------------------------------------------------------------
// one frame's interior <-> the bytes of its file (x fastest, then y, z):
// _load3dDataArrayVTK_ (segmentation4D.c:1317-1320), _writeData_ (:1250-1254),
// _writeData_mpi_ (segmentation4D_mpi.c:1466-1473)

// byte / 255. from a table of the 256 quotients (the same IEEE divisions),
// built once per block; a block walks FRAME_Z_PER_BLOCK planes
#define FRAME_Z_PER_BLOCK 32
__global__ void k_frame_from_bytes(Geo g, double *img, int l, const uint8_t *__restrict__ bytes)
{
    __shared__ double lut[256];
    const int t = threadIdx.y * blockDim.x + threadIdx.x;
    if (t < 256)
        lut[t] = t / 255.;
    __syncthreads();
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= g.nx || y >= g.ny)
        return;
    for (int z = blockIdx.z; z < g.nz; z += gridDim.z) {
        const long long q = ((long long)z * g.ny + y) * g.nx + x;
        img[nat_index(g, x + 1, y + 1, z + 1, l)] = lut[bytes[q]];
    }
}

// mode 0: (unsigned char)(255 v + 0.5), clamped to [0, 255] (the reference's
// conversion is undefined outside); mode 1: 1 where v >= 0.5, else 0
__global__ void k_frame_to_bytes(Geo g, const double *img, int l, int mode, uint8_t *__restrict__ bytes)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y, z = blockIdx.z;
    if (x >= g.nx || y >= g.ny)
        return;
    const long long q = ((long long)z * g.ny + y) * g.nx + x;
    const double v = img[nat_index(g, x + 1, y + 1, z + 1, l)];
    uint8_t out;
    if (mode == 1) {
        out = v >= 0.5 ? 1 : 0;
    } else {
        const double w = 255 * v + 0.5;
        out = w >= 255. ? 255 : (w > 0. ? (uint8_t)(int)w : 0);
    }
    bytes[q] = out;
}

__global__ void k_mask_zero(Geo g, double *v, const double *Mmask, int l_off)
{
    int i, j, k, l;
    if (!interior_ijkl(g, i, j, k, l))
        return;
    l += l_off;
    const long long o = nat_index(g, i, j, k, l);
    if (Mmask[o] == 0)
        v[o] = 0;
}

// ---------------------------------------------------------------------------
// threshold to mask (segmentation4D_mpi.c:1470-1478)

#define MINMAX_BLOCKS 2048
// interior min and max of u per block, as (min, max) pairs in partial; a
// block walks whole rows (threads along x), comparing integer keys so the
// FP64 pipe is not used; a block without a number reports (1e308, -1e308)
__global__ void k_minmax_partial(Geo g, const double *u, double *partial)
{
    long long mn = 0x7fffffffffffffffLL, mx = -0x7fffffffffffffffLL - 1;
    const int rows = g.ny * g.nz * g.nt;
    for (int r = blockIdx.x * blockDim.y + threadIdx.y; r < rows; r += gridDim.x * blockDim.y) {
        const int j = r % g.ny, kl = r / g.ny;
        const long long base = nat_index(g, 0, j + 1, 1 + kl % g.nz, 1 + kl / g.nz);
        for (int i = 1 + threadIdx.x; i <= g.nx; i += blockDim.x) {
            const long long b = __double_as_longlong(u[base + i]);
            if ((b & 0x7fffffffffffffffLL) <= 0x7ff0000000000000LL) {
                const long long key = dkey(b);
                mn = key < mn ? key : mn;
                mx = key > mx ? key : mx;
            }
        }
    }
    __shared__ long long smn[32], smx[32];
    const int t = flat_tid(), lane = t & 31, wid = t >> 5, nw = (blockDim.x * blockDim.y + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const long long a = __shfl_down_sync(0xffffffffu, mn, o), b = __shfl_down_sync(0xffffffffu, mx, o);
        mn = a < mn ? a : mn;
        mx = b > mx ? b : mx;
    }
    if (lane == 0) {
        smn[wid] = mn;
        smx[wid] = mx;
    }
    __syncthreads();
    if (wid == 0) {
        mn = lane < nw ? smn[lane] : 0x7fffffffffffffffLL;
        mx = lane < nw ? smx[lane] : -0x7fffffffffffffffLL - 1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const long long a = __shfl_down_sync(0xffffffffu, mn, o), b = __shfl_down_sync(0xffffffffu, mx, o);
            mn = a < mn ? a : mn;
            mx = b > mx ? b : mx;
        }
        if (lane == 0) {
            const bool none = mn == 0x7fffffffffffffffLL;
            partial[2 * blockIdx.x] = none ? 1e308 : __longlong_as_double(dkey(mn));
            partial[2 * blockIdx.x + 1] = none ? -1e308 : __longlong_as_double(dkey(mx));
        }
    }
}

__global__ void k_threshold(Geo g, const double *u, const double *level_dev, double level, uint8_t *mask)
{
    int i, j, k, l;
    if (!interior_ijkl(g, i, j, k, l))
        return;
    const double lev = level_dev ? level_dev[2] : level;
    const long long m = ((((long long)(l - 1) * g.nz + (k - 1)) * g.ny + (j - 1)) * g.nx) + (i - 1);
    mask[m] = u[nat_index(g, i, j, k, l)] >= lev ? 1 : 0;
}

// ---------------------------------------------------------------------------
// host-side launch wrappers

static inline void interior_cfg(const Geo &g, dim3 &grid, dim3 &block)
{
    const int bx = g.nx >= 128 ? 128 : (g.nx >= 64 ? 64 : 32);
    const int by = 256 / bx;
    block = dim3(bx, by, 1);
    grid = dim3((g.nx + bx - 1) / bx, (g.ny + by - 1) / by, g.nz * g.nt);
}

long long interior_blocks(const Geo &g)
{
    dim3 gr, bl;
    interior_cfg(g, gr, bl);
    return (long long)gr.x * gr.y * gr.z;
}

void launch_reflect(const Geo &g, double *u, cudaStream_t st)
{
    const long long warps = (long long)g.jM * g.kM * g.lM;
    k_reflect<<<(unsigned)(warps < 8 * 1216 ? (warps + 7) / 8 : 1216), 256, 0, st>>>(g, u);
}

// one colour: ceil(nx/2) threads along a row
static inline void colour_cfg(const Geo &g, dim3 &grid, dim3 &block)
{
    const int nxh = (g.nx + 1) / 2;
    const int bx = nxh >= 128 ? 128 : (nxh >= 64 ? 64 : 32);
    const int by = 256 / bx;
    block = dim3(bx, by, 1);
    grid = dim3((nxh + bx - 1) / bx, (g.ny + by - 1) / by, g.nz * g.nt);
}

static inline void resid_cfg(const Geo &g, dim3 &grid, dim3 &block)
{
    interior_cfg(g, grid, block);
    grid.z = ((g.nz + RESID_K - 1) / RESID_K) * g.nt;
}

long long resid_blocks(const Geo &g)
{
    dim3 gr, bl;
    resid_cfg(g, gr, bl);
    return (long long)gr.x * gr.y * gr.z;
}

void launch_gauss_axis(const Geo &g, int axis, const double *in, double *out, const GaussWeights &W,
                       cudaStream_t st)
{
    dim3 gr, bl;
    interior_cfg(g, gr, bl);
    if (axis == 0)
        k_gauss_axis<0><<<gr, bl, 0, st>>>(g, in, out, W);
    else if (axis == 1)
        k_gauss_axis<1><<<gr, bl, 0, st>>>(g, in, out, W);
    else if (axis == 2)
        k_gauss_axis<2><<<gr, bl, 0, st>>>(g, in, out, W);
    else
        k_gauss_axis<3><<<gr, bl, 0, st>>>(g, in, out, W);
}

void launch_presmooth_explicit(const Geo &g, double *v, const double *prev, double coeff, cudaStream_t st)
{
    dim3 gr, bl;
    interior_cfg(g, gr, bl);
    k_presmooth_explicit<<<gr, bl, 0, st>>>(g, v, prev, coeff);
}

void launch_gfaces(const Geo &g, const double *i0, const double *ithr, GPtrs8 gout, double h, double K, double theta,
                   double rho, cudaStream_t st)
{
    const int planes = (g.nz + 1) * (g.nt + 1); // grids of at most 65,535 planes
    int e = 0;
    const double m = frexp(h, &e);
    const double ih = 1.0 / h, iq = 1.0 / (4.0 * h);
    const FastDiv row = make_fastdiv((unsigned)g.nx + 1), pl = make_fastdiv((unsigned)g.nz + 1);
    const dim3 gr(((unsigned)(g.nx + 1) * (g.ny + 1) + 255) / 256, planes);
    // a power of two far from the ends of the range, and weights that stay
    // normal with its scale
    const double s0 = theta * (iq * iq), s1 = rho * (iq * iq);
    if (m == 0.5 && abs(e) < 128 && (theta == 0.0 || isnormal(s0)) && (rho == 0.0 || isnormal(s1)))
        k_gfaces<true><<<gr, 256, 0, st>>>(g, row, pl, i0, ithr, gout, h, K, s0, s1, ih, iq);
    else
        k_gfaces<false><<<gr, 256, 0, st>>>(g, row, pl, i0, ithr, gout, h, K, theta, rho, div_const_recip(h),
                                            div_const_recip(4.0 * h));
}

void launch_coef_ref(const Geo &g, const double *u, CPtrs8 gin, int has_g, GPtrs8 coef, double h, double eps2,
                     cudaStream_t st)
{
    dim3 gr, bl;
    interior_cfg(g, gr, bl);
    k_coef_ref<<<gr, bl, 0, st>>>(g, u, gin, has_g, coef, h, eps2);
}

void launch_sor_half_ref(const Geo &g, double *u, const double *prev, CPtrs8 a, double c, double omega, int colour,
                         cudaStream_t st)
{
    dim3 gr, bl;
    colour_cfg(g, gr, bl);
    k_sor_half_ref<<<gr, bl, 0, st>>>(g, u, prev, a, c, omega, colour);
}

void launch_sor_resid_ref(const Geo &g, const double *u, const double *prev, CPtrs8 a, double c, double h4,
                          double *partial, cudaStream_t st)
{
    dim3 gr, bl;
    resid_cfg(g, gr, bl);
    k_sor_resid_ref<<<gr, bl, 0, st>>>(g, u, prev, a, c, h4, partial);
}

// n partials: one block when n is small; else up to 1024 blocks first, their
// results written behind the partials (partial[n ..]), then one block.
// Returns the number of launches.
static long long reduce_split(long long n, long long &per)
{
    per = 4096;
    long long nb = (n + per - 1) / per;
    if (nb > 1024) {
        per = (n + 1023) / 1024;
        nb = (n + per - 1) / per;
    }
    return nb;
}

int launch_reduce_sum(double *partial, long long n, double *out, cudaStream_t st)
{
    if (n <= 16384) {
        k_reduce_sum<<<1, 1024, 0, st>>>(partial, n, out);
        return 1;
    }
    long long per;
    const long long nb = reduce_split(n, per);
    k_reduce_sum_part<<<(unsigned)nb, 256, 0, st>>>(partial, n, per, partial + n);
    k_reduce_sum<<<1, 1024, 0, st>>>(partial + n, nb, out);
    return 2;
}

void launch_l2(const Geo &g, const double *a, const double *b, double h4, double *partial, int nblk, cudaStream_t st)
{
    k_l2_partial<<<nblk, 256, 0, st>>>(g.n, a, b, h4, partial);
}

void launch_mass(const Geo &g, const double *a, double h4, double *partial, int nblk, cudaStream_t st)
{
    k_mass_partial<<<nblk, 256, 0, st>>>(g.n, a, h4, partial);
}

void launch_mcf_field(const Geo &g, double *u, double h, double t, int ghosts_only, cudaStream_t st)
{
    const long long warps = (long long)g.jM * g.kM * g.lM;
    k_mcf_field<<<(unsigned)(warps < 8 * 1216 ? (warps + 7) / 8 : 1216), 256, 0, st>>>(g, u, h, t, ghosts_only);
}

void launch_rescale_balls(const Geo &g, double *v, const int *frame_first, const int *frame_count, const double *bx,
                          const double *by, const double *bz, double R, cudaStream_t st)
{
    launch_rescale_balls_range(g, v, frame_first, frame_count, bx, by, bz, R, 1, g.lM - 1, st);
}

// the largest double t with sqrt(t) <= R (both rounded to nearest); negative
// or NaN where there is none, which no square is at most
static double largest_square(double R)
{
    if (!(R >= 0.0) || isinf(R))
        return R;
    double t = R * R;
    if (isinf(t))
        t = DBL_MAX;
    while (sqrt(t) > R)
        t = nextafter(t, -1.0);
    while (t < DBL_MAX && sqrt(nextafter(t, HUGE_VAL)) <= R)
        t = nextafter(t, HUGE_VAL);
    return t;
}

void launch_rescale_balls_range(const Geo &g, double *v, const int *frame_first, const int *frame_count,
                                const double *bx, const double *by, const double *bz, double R, int l0, int l1,
                                cudaStream_t st)
{
    k_rescale_balls<<<(l1 - l0) * RESCALE_CTAS, 256, 0, st>>>(g, v, frame_first, frame_count, bx, by, bz, R,
                                                              largest_square(R), l0);
}

void launch_mask_zero(const Geo &g, double *v, const double *Mmask, cudaStream_t st)
{
    launch_mask_zero_range(g, v, Mmask, 1, g.lM - 1, st);
}

void launch_mask_zero_range(const Geo &g, double *v, const double *Mmask, int l0, int l1, cudaStream_t st)
{
    dim3 gr, bl;
    interior_cfg(g, gr, bl);
    gr.z = g.nz * (l1 - l0);
    k_mask_zero<<<gr, bl, 0, st>>>(g, v, Mmask, l0 - 1);
}

void launch_ball_min_max(const Geo &g, const double *v, int l, double cx, double cy, double cz, double R, double *out2,
                         cudaStream_t st)
{
    k_ball_min_max<<<1, 256, 0, st>>>(g, v, l, cx, cy, cz, R, out2);
}

void launch_local_threshold(const Geo &g, const double *in, double *thr, const int *frame_first, const int *frame_count,
                            const double *bx, const double *by, const double *bz, double R, double alpha, double beta,
                            const double *minmax, cudaStream_t st)
{
    k_local_threshold<<<g.nt, 256, 0, st>>>(g, in, thr, frame_first, frame_count, bx, by, bz, R, alpha, beta, minmax);
}

void launch_generate_segm(const Geo &g, double *u, double *Mmask, const int *frame_first, const int *frame_count,
                          const double *bx, const double *by, const double *bz, double R, cudaStream_t st)
{
    k_generate_segm<<<g.nt, 256, 0, st>>>(g, u, Mmask, frame_first, frame_count, bx, by, bz, R);
}

void launch_frame_bytes(const Geo &g, double *img_out, const double *img_in, int l, int mode, const uint8_t *bytes_in,
                        uint8_t *bytes_out, cudaStream_t st)
{
    const int bx = g.nx >= 128 ? 128 : (g.nx >= 64 ? 64 : 32);
    dim3 bl(bx, 256 / bx, 1), gr((g.nx + bx - 1) / bx, (g.ny + 256 / bx - 1) / (256 / bx), g.nz);
    if (img_out) {
        gr.z = (g.nz + FRAME_Z_PER_BLOCK - 1) / FRAME_Z_PER_BLOCK;
        k_frame_from_bytes<<<gr, bl, 0, st>>>(g, img_out, l, bytes_in);
    } else {
        k_frame_to_bytes<<<gr, bl, 0, st>>>(g, img_in, l, mode, bytes_out);
    }
}

int launch_minmax(const Geo &g, const double *u, double *partial, double level, double *out3, cudaStream_t st)
{
    const long long rows = (long long)g.ny * g.nz * g.nt;
    const int nb = (int)(rows / 2 < MINMAX_BLOCKS ? (rows + 1) / 2 : MINMAX_BLOCKS);
    k_minmax_partial<<<nb, dim3(128, 2, 1), 0, st>>>(g, u, partial);
    k_reduce_minmax<<<1, 1024, 0, st>>>(partial, nb, level, out3);
    return 2;
}

void launch_threshold(const Geo &g, const double *u, const double *level_dev, double level, uint8_t *mask,
                      cudaStream_t st)
{
    dim3 gr, bl;
    interior_cfg(g, gr, bl);
    k_threshold<<<gr, bl, 0, st>>>(g, u, level_dev, level, mask);
}

} // namespace ss4d
