// ss4d_front_ff.cu — the edge detector of the mixed form in float-float
// arithmetic: the presmoothing's red-black SOR (segmentation4D.c:337-409) and
// the 8 face g values (segmentation4D.c:594-821, _gFunction_ :67-70), with
// about 48 significant bits on the FP32 pipe instead of FP64.  The plain and
// reference forms keep the reference's FP64 rounding (ss4d_front64.cu,
// ss4d_kernels_ref.cu).
//
// Both work on two values per instruction (ss4d_ff2.cuh).  The presmoothing
// (ss4d_front.cuh) pairs two adjacent columns of a colour.  The g faces read
// the image folded in k: a 16-byte unit holds voxel k = m and voxel
// k = m + Hk of the same (i, j, l), so every neighbour of both is in one
// unit too, and addresses, loads and arithmetic serve two voxels; planes 0
// and Hk + 1 of the fold are both halves' halo.  Relative error of the
// results against the FP64 forms: about 1e-14.
#include <math.h>

#include "ss4d_ff2.cuh"
#include "ss4d_front.cuh"

namespace ss4d {

using namespace ffa;

namespace {

__device__ __forceinline__ ff split_d(double v)
{
    const float h = (float)v;
    return ff_make(h, (float)(v - (double)h));
}

__device__ __forceinline__ unsigned fold_index(const Geo &g, int Hk, int i, int j, int m, int l)
{
    return (((unsigned)l * (Hk + 2) + m) * g.jM + j) * g.iM + i;
}

struct PairFF {
    typedef float4 Q;
    // sum of squares per lane: its rounding errors are kept beside it
    struct Acc {
        f2 s, e;
    };
    struct Const {
        ff2 c, inv_d, omega;
    };
    static __device__ __forceinline__ Const constants(const FrontArgs &a)
    {
        return Const{both(split_d(a.c)), both(split_d(a.y)), both(split_d(a.omega))};
    }
    static __device__ __forceinline__ Acc zero()
    {
        return Acc{both(0.f), both(0.f)};
    }
    template <int COL>
    static __device__ __forceinline__ double total(const FrontArgs &f, Acc a)
    {
        const double k = COL == 0 ? f.d : (1.0 - f.omega) * f.d;
        return k * k * ( ((double)lo2(a.s) + (double)hi2(a.s)) + ((double)lo2(a.e) + (double)hi2(a.e)));
    }
    static __device__ __forceinline__ Q make(double x, double y)
    {
        const ff a = ff_from_d(x), b = ff_from_d(y);
        return make_float4(a.h, b.h, a.l, b.l);
    }
    static __device__ __forceinline__ void get(Q v, double *w)
    {
        w[0] = ff_to_d(ff_make(v.x, v.z));
        w[1] = ff_to_d(ff_make(v.y, v.w));
    }
    static __device__ __forceinline__ Q live(const Q *p)
    {
        Q v;
        asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
        return v;
    }
    static __device__ __forceinline__ ff first(const Q *p)
    {
        return ff_make(ld_oth<true>(&p->x), ld_oth<true>(&p->z));
    }
    static __device__ __forceinline__ ff second(const Q *p)
    {
        return ff_make(ld_oth<true>(&p->y), ld_oth<true>(&p->w));
    }
    static __device__ __forceinline__ Q up(Q v, ff e)
    {
        return make_float4(v.y, e.h, v.w, e.l);
    }
    static __device__ __forceinline__ Q down(ff e, Q v)
    {
        return make_float4(e.h, v.x, e.l, v.z);
    }
    static __device__ __forceinline__ Q with_first(Q v, Q w)
    {
        return make_float4(w.x, v.y, w.z, v.w);
    }
    static __device__ __forceinline__ Q with_second(Q v, Q w)
    {
        return make_float4(v.x, w.y, v.z, w.w);
    }
    // gs = (prev + c sum_8 v_nb) / (1 + 8c), v = u + omega (gs - u).  The
    // residual u (1 + 8c) - c sum - prev is (1 + 8c) (u - gs), and after a
    // target's own update (1 - omega) of that (its neighbours do not move):
    // the squares of gs - u are summed and scaled once.  The neighbours are
    // added in pairs without renormalising (positive terms): against 64 bits an
    // update's error is 3.0e-15 where renormalising after every operation of
    // the reference's order left 3.3e-15, with two thirds of the instructions.
    template <int COL>
    static __device__ __forceinline__ Q update(const Const &C, Q u4, Q pv4, Q xr, Q xl, Q ym, Q yp, Q zm, Q zp, Q wm,
                                               Q wp, bool two, Acc &acc)
    {
        const ff2 x = ff_add_nr2(unpack4(xr), unpack4(xl)), y = ff_add_nr2(unpack4(ym), unpack4(yp));
        const ff2 z = ff_add_nr2(unpack4(zm), unpack4(zp)), w = ff_add_nr2(unpack4(wm), unpack4(wp));
        const ff2 s = ff_norm2(ff_add_nr2(ff_add_nr2(x, y), ff_add_nr2(z, w)));
        const ff2 u = unpack4(u4);
        const ff2 gs = ff_mul2(C.inv_d, ff_norm2(ff_add_nr2(unpack4(pv4), ff_mul_nr2(C.c, s))));
        const ff2 r = ff_sub2(gs, u);
        const ff2 v = ff_add2(u, ff_mul_nr2(C.omega, r));
        f2 rh = r.h;
        if (!two)
            rh = mk2(lo2(rh), 0.f);
        const ff2 q = two_sum2(acc.s, mul2(rh, rh));
        acc.s = q.h;
        acc.e = add2(acc.e, q.l);
        return pack4(v);
    }
    // the smoothed image folded in k for the g faces: the result inside, the
    // reflected initial image (at its clamped coordinates) on the ghosts
    static __device__ __forceinline__ ff value(const FrontArgs &a, const Q *red, int i, int j, int k, int l)
    {
        const Geo &g = a.g;
        const int ic = min(max(i, 1), g.nx), jc = min(max(j, 1), g.ny), kc = min(max(k, 1), g.nz),
                  lc = min(max(l, 1), g.nt);
        const int col = (ic + jc + kc + lc) & 1;
        const bool in = ic == i && jc == j && kc == k && lc == l;
        const float *v = static_cast<const float *>(in ? (col ? a.B : (const void *)red) : a.P[col]);
        const unsigned s = (((unsigned)lc * g.kM + kc) * g.jM + jc) * a.F.Hs + ((ic + 1) >> 1) + a.F.A - 1;
        const size_t e = 4 * (size_t)(s >> 1) + (s & 1);
        return ff_make(ld_oth<true>(v + e), ld_oth<true>(v + e + 2));
    }
    static __device__ __forceinline__ void fold(const FrontArgs &a, const Q *red, unsigned t0, unsigned dt)
    {
        if (!a.fold)
            return;
        const Geo &g = a.g;
        const unsigned planes = (unsigned)a.Hk + 2, rows = (unsigned)g.lM * planes * g.jM;
        // a warp per row
        for (unsigned r = t0 >> 5; r < rows; r += dt >> 5) {
            const unsigned rk = fdiv(r, g.fjM), l = rk / planes;
            const int j = (int)(r - rk * g.fjM.d), m = (int)(rk - l * planes);
            for (int i = (int)(t0 & 31); i < g.iM; i += 32) {
                const ff x = value(a, red, i, j, m, (int)l), y = value(a, red, i, j, m + a.Hk, (int)l);
                const float S = a.fold_scale;
                __stcs(static_cast<float4 *>(a.fold) + ((size_t)r * g.iM + i),
                       make_float4(x.h * S, y.h * S, x.l * S, y.l * S));
            }
        }
    }
};

// 62 registers, two blocks of 512 per SM.  At 256^2 x 128 x 20 an image takes
// 13.1 ms; among launch shapes tried side by side two blocks of 512 took 12.4,
// three of 256 14.0, four of them 12.8, five (48 registers) 13.6.  A half-sweep
// has to move 2.7 GB (0.40 ms at the copy rate); at 192^2 x 96 x 12 the launch
// runs at 83 % of the copy rate in DRAM bytes, its issue slots 48 % busy.  The
// kernels it replaces (one thread per target, a residual pass) took 28 ms per
// image.
__global__ void __launch_bounds__(FRONT_FF_THREADS, 2) k_presmooth_ff(const __grid_constant__ FrontArgs a)
{
    presmooth_body<PairFF>(a);
}

// a double image, ghosts included, folded in k
__global__ void k_to_fold(Geo g, int Hk, float S, const double *__restrict__ img, float4 *__restrict__ out)
{
    const unsigned planes = (unsigned)Hk + 2, rows = (unsigned)g.lM * planes * g.jM;
    const int lane = threadIdx.x & 31;
    for (unsigned r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += (gridDim.x * blockDim.x) >> 5) {
        const unsigned rk = fdiv(r, g.fjM), l = rk / planes;
        const int j = (int)(r - rk * g.fjM.d), m = (int)(rk - l * planes);
        const double *a = img + nat_index(g, 0, j, min(m, g.kM - 1), (int)l);
        const double *b = img + nat_index(g, 0, j, min(m + Hk, g.kM - 1), (int)l);
        for (int i = lane; i < g.iM; i += 32) {
            const ff x = ff_from_d(__ldg(a + i)), y = ff_from_d(__ldg(b + i));
            out[(size_t)r * g.iM + i] = make_float4(x.h * S, y.h * S, x.l * S, y.l * S);
        }
    }
}

// --- g faces ----------------------------------------------------------------

struct FaceConst {
    FFc n[2], t[2]; // per image: K weight / (h S)^2 (normal) and K weight / (4 h S)^2 (tangential)
};

__device__ __forceinline__ ff2 ldv(const float4 *__restrict__ v, unsigned x)
{
    return unpack4(__ldg(v + x));
}
// central difference along a stride
__device__ __forceinline__ ff2 cdiff2(const float4 *__restrict__ v, unsigned x, unsigned sa)
{
    return ff_sub_nr2(ldv(v, x + sa), ldv(v, x - sa));
}
__device__ __forceinline__ ff2 konst(FFc c)
{
    return both(ff_make(c.h, c.l));
}

// K weight |grad v|^2 at the face between x and x + st[D] from the central
// differences own[] at x: the reference's face formula with its tangential
// pairs exchanged, (v[nb+a] + v[o+a]) - (v[nb-a] + v[o-a]) = D_a(nb) + D_a(o),
// so that D_a(o) serves three faces
template <int D>
__device__ __forceinline__ ff2 face_term(const float4 *__restrict__ v, unsigned x, const unsigned st[4],
                                         const ff2 own[4], ff2 vx, ff2 kn, ff2 kt)
{
    const unsigned nb = x + st[D];
    ff2 tt;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if (a == D)
            continue;
        const ff2 q = ff_sqr_nr2(ff_add_nr2(cdiff2(v, nb, st[a]), own[a]));
        tt = a == (D == 0 ? 1 : 0) ? q : ff_add_nr2(tt, q);
    }
    const ff2 nn = ff_sqr_nr2(ff_sub_nr2(ldv(v, nb), vx));
    return ff_add_nr2(ff_mul_nr2(kt, tt), ff_mul_nr2(kn, nn));
}

// g = 1/(1 + s): FP32 seeds y0, one Newton step y = y0 + y0 (1 - x y0) with x y0
// formed to float-float: error about that of y0 squared
__device__ __forceinline__ void g_of(ff2 s, double out[2])
{
    const ff2 x = ff_add2(both(ff_make(1.f, 0.f)), ff_norm2(s));
    const f2 y0 = mk2(__frcp_rn(lo2(x.h)), __frcp_rn(hi2(x.h)));
    const f2 q = mul2(x.h, y0);
    const f2 qe = fma2(x.l, y0, fma2(x.h, y0, neg2(q)));
    const f2 r = sub2(sub2(both(1.f), q), qe);
    const f2 c = mul2(y0, r), ce = fma2(y0, r, neg2(c));
    ff2 y = fast_two_sum2(y0, c);
    y.l = add2(y.l, ce);
    out[0] = ff_to_d(ff_make(lo2(y.h), lo2(y.l)));
    out[1] = ff_to_d(ff_make(hi2(y.h), hi2(y.l)));
}

// Face between o (coordinate cD along D) and o + st[D]: g[2D] at o where o
// is interior along D, g[2D+1] at o + st[D] where that is.
__device__ __forceinline__ void put_face(double *__restrict__ lo, double *__restrict__ hi, size_t o, size_t sd, int cD,
                                         int nD, double gv)
{
    if (cD >= 1)
        __stcs(lo + o, gv);
    if (cD < nD)
        __stcs(hi + o + sd, gv);
}

template <int D, bool TWO>
__device__ __forceinline__ void boundary_gface(const float4 *__restrict__ v0, const float4 *__restrict__ v1, unsigned x,
                                               const unsigned st[4], const FaceConst &F, double out[2])
{
    ff2 s;
#pragma unroll
    for (int im = 0; im < (TWO ? 2 : 1); ++im) {
        const float4 *__restrict__ v = im ? v1 : v0;
        ff2 own[4];
#pragma unroll
        for (int a = 0; a < 4; ++a)
            own[a] = a == D ? ff2{both(0.f), both(0.f)} : cdiff2(v, x, st[a]);
        const ff2 t = face_term<D>(v, x, st, own, ldv(v, x), konst(F.n[im]), konst(F.t[im]));
        s = im ? ff_add_nr2(s, t) : t;
    }
    g_of(s, out);
}

// One folded voxel per thread (voxels (i, j, m, l) and (i, j, m + Hk, l)):
// the faces towards +x, +y, +z, +t of both, and at the volume's lower
// boundaries also the face towards the ghost.  The flat index has i fastest,
// m slowest: blocks at work together cover a few planes of all frames, whose
// neighbouring frames and planes are then read from L2.
// Bound by latency: about 950 instructions per voxel with two images, in chains
// of float-float operations and loads, issue 41 % busy and DRAM at 31 % of the
// copy rate with the 28 % of the warps that 96 registers leave (192^2 x 96 x 12).
// At 256^2 x 128 x 20: two images 9.8 ms; among register limits tried side by
// side 9.5 ms at five blocks of 128 threads (96 registers, some spilled), 10.4 at
// 128 registers, 11.0 at 80; one image 5.1 ms at 80 registers, 5.5 at 96.  The kernel it replaces (scalar float-float, every
// difference formed at each of its faces) took 14.5 ms for two.
constexpr int GFACES_THREADS = 128;
template <bool TWO>
__global__ void __launch_bounds__(GFACES_THREADS, TWO ? 5 : 6)
    k_gfaces_ff(Geo g, int Hk, FastDiv dnx, FastDiv dny, FastDiv dnt, unsigned n, const float4 *__restrict__ v0,
                const float4 *__restrict__ v1, GPtrs8 gout, const __grid_constant__ FaceConst F)
{
    const unsigned q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n)
        return;
    unsigned h = fdiv(q, dnx);
    const int i = 1 + (int)(q - h * dnx.d);
    unsigned r = h;
    h = fdiv(r, dny);
    const int j = 1 + (int)(r - h * dny.d);
    r = h;
    h = fdiv(r, dnt);
    const int l = 1 + (int)(r - h * dnt.d);
    const int m = 1 + (int)h;
    const unsigned st[4] = {1u, (unsigned)g.iM, (unsigned)(g.iM * g.jM), (unsigned)(g.iM * g.jM) * (Hk + 2)};
    const unsigned x = fold_index(g, Hk, i, j, m, l);
    ff2 s[4];
#pragma unroll
    for (int im = 0; im < (TWO ? 2 : 1); ++im) {
        const float4 *__restrict__ v = im ? v1 : v0;
        const ff2 kn = konst(F.n[im]), kt = konst(F.t[im]);
        ff2 own[4];
#pragma unroll
        for (int a = 0; a < 4; ++a)
            own[a] = cdiff2(v, x, st[a]);
        const ff2 vx = ldv(v, x);
        ff2 t = face_term<0>(v, x, st, own, vx, kn, kt);
        s[0] = im ? ff_add_nr2(s[0], t) : t;
        t = face_term<1>(v, x, st, own, vx, kn, kt);
        s[1] = im ? ff_add_nr2(s[1], t) : t;
        t = face_term<2>(v, x, st, own, vx, kn, kt);
        s[2] = im ? ff_add_nr2(s[2], t) : t;
        t = face_term<3>(v, x, st, own, vx, kn, kt);
        s[3] = im ? ff_add_nr2(s[3], t) : t;
    }
    const bool b1 = m + Hk <= g.nz; // the second voxel exists
    const size_t oa = (size_t)nat_index(g, i, j, m, l), ob = oa + (size_t)Hk * g.sz;
    const int c[4] = {i, j, m, l}, nn[4] = {g.nx, g.ny, g.nz, g.nt};
    const size_t sd[4] = {1, (size_t)g.sy, (size_t)g.sz, (size_t)g.sw};
    double gv[2];
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        g_of(s[d], gv);
        put_face(gout.p[2 * d], gout.p[2 * d + 1], oa, sd[d], c[d], nn[d], gv[0]);
        if (b1)
            put_face(gout.p[2 * d], gout.p[2 * d + 1], ob, sd[d], d == 2 ? m + Hk : c[d], nn[d], gv[1]);
    }
    // the faces between a ghost and the first voxel along an axis
    if (i == 1) {
        boundary_gface<0, TWO>(v0, v1, x - st[0], st, F, gv);
        __stcs(gout.p[1] + oa, gv[0]);
        if (b1)
            __stcs(gout.p[1] + ob, gv[1]);
    }
    if (j == 1) {
        boundary_gface<1, TWO>(v0, v1, x - st[1], st, F, gv);
        __stcs(gout.p[3] + oa, gv[0]);
        if (b1)
            __stcs(gout.p[3] + ob, gv[1]);
    }
    if (m == 1) { // k = 0 | 1; the second half's lower face is the first half's upper one
        boundary_gface<2, TWO>(v0, v1, x - st[2], st, F, gv);
        __stcs(gout.p[5] + oa, gv[0]);
    }
    if (l == 1) {
        boundary_gface<3, TWO>(v0, v1, x - st[3], st, F, gv);
        __stcs(gout.p[7] + oa, gv[0]);
        if (b1)
            __stcs(gout.p[7] + ob, gv[1]);
    }
}

FFc split_ff(double v)
{
    FFc c;
    c.h = (float)v;
    c.l = (float)(v - (double)c.h);
    return c;
}

} // namespace

int fold_of(const Geo &g)
{
    return (g.nz + 1) / 2;
}

size_t fold_units(const Geo &g)
{
    return (size_t)g.lM * (fold_of(g) + 2) * g.jM * g.iM;
}

int presmooth_ff_grid(int sm_count)
{
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_presmooth_ff, FRONT_FF_THREADS, 0);
    return per * sm_count;
}

cudaError_t launch_presmooth_ff(const FrontArgs &a, int grid, cudaStream_t st)
{
    void *args[] = {(void *)&a};
    return cudaLaunchCooperativeKernel((const void *)k_presmooth_ff, dim3(grid), dim3(FRONT_FF_THREADS), args, 0, st);
}

// The folded image is scaled by the power of two nearest above 1/h, exactly,
// so that its differences are of the gradient's size whatever h is: their
// squares then stay in FP32's range as long as the gradient's do.
float fold_scale(double h)
{
    int e = 0;
    frexp(h, &e);
    e = e < -100 ? -100 : (e > 100 ? 100 : e);
    return (float)ldexp(1.0, 1 - e);
}

void launch_to_fold(const Geo &g, const double *img, float4 *out, double h, cudaStream_t st)
{
    k_to_fold<<<2432, 256, 0, st>>>(g, fold_of(g), fold_scale(h), img, out);
}

void launch_gfaces_ff(const Geo &g, const float4 *i0, const float4 *ithr, GPtrs8 gout, double h, double K,
                      double theta, double rho, cudaStream_t st)
{
    const int Hk = fold_of(g);
    FaceConst F;
    const double w[2] = {theta, rho};
    const double hs = h * fold_scale(h), hs2 = hs * hs;
    for (int im = 0; im < 2; ++im) {
        F.n[im] = split_ff(K * w[im] / hs2);
        F.t[im] = split_ff(K * w[im] / (16.0 * hs2));
    }
    const unsigned n = (unsigned)g.nx * g.ny * g.nt * Hk;
    const unsigned nb = (n + GFACES_THREADS - 1) / GFACES_THREADS;
    const FastDiv dx = make_fastdiv((unsigned)g.nx), dy = make_fastdiv((unsigned)g.ny), dt = make_fastdiv((unsigned)g.nt);
    if (ithr)
        k_gfaces_ff<true><<<nb, GFACES_THREADS, 0, st>>>(g, Hk, dx, dy, dt, n, i0, ithr, gout, F);
    else
        k_gfaces_ff<false><<<nb, GFACES_THREADS, 0, st>>>(g, Hk, dx, dy, dt, n, i0, i0, gout, F);
}

} // namespace ss4d
