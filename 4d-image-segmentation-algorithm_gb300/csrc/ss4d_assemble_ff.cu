// ss4d_assemble_ff.cu — coefficient assembly of the mixed form in
// float-float arithmetic.
//
// The FP64 assembly (k_faces + k_voxel_coef, ss4d_kernels_fast.cu) executes
// about 125 FP64 instructions per voxel and is bounded by GB300's FP64 pipe
// (roughly 1/70 of its FP32 rate).  Here every quantity after the first
// differences of u is carried as an unevaluated sum of two floats (h + l,
// 48 significant bits; Dekker's and Knuth's error-free transformations: the
// rounding error of a float sum is recovered with the two-sum of Knuth, that
// of a product with one fused multiply-add), so the work runs on the FP32
// pipe.  FP64 instructions are left only where a double enters or leaves
// the float-float form: one subtraction per first difference of u and one
// addition per coefficient written (a double is split into two floats by
// integer operations).
//
//   k_fdiff:          F_a(v) = u(v + e_a) - u(v) for the 4 axes (FP64
//                     difference, split into two floats), folded in k;
//   k_faces_ff:       per face between v and v + e_d, from F only:
//                     |grad u|^2 = F_d^2/h^2 + sum_{a != d} (D_a(v+e_d) + D_a(v))^2/(4h)^2
//                     with D_a(x) = F_a(x) + F_a(x - e_a) the central difference
//                     (the reference's face formula, segmentation4D.c:446-580),
//                     s2 = |grad u|^2 + eps2, fn = s2 / sqrt(s2), fq = g / sqrt(s2);
//   k_voxel_coef_ff:  vc = sqrt(mean(fn)^2 + eps2), c a_f = c vc fq_f,
//                     diag = 1 + sum c a_f; written as FP64 records
//                     (refinement) and the FP32 sweeps' records (16-bit
//                     fractions of sum c a_f and that sum, store_coef16).
//
// Relative error of the coefficients: below 1e-12 (1/sqrt from an FP32 seed
// and one Newton step, about 1.5 (2^-22)^2 each; sums and products to 2^-46).  The mixed form's refinement passes measure the FP64 residual
// against these coefficients; the residual of its result against exact FP64
// coefficients meets the same tolerance (tested), the coefficient error
// entering it only squared, far below any tolerance.
#include <math.h>

#include "ss4d_ff2.cuh"

namespace ss4d {

using namespace ffa;


struct FFConst {
    float ih2h, ih2l;   // 1/h^2
    float iq2h, iq2l;   // 1/(4h)^2
    float eps2h, eps2l; // eps2
    float ch, cl;       // tau/h^2
    int pow2;           // 1/h^2 and 1/(4h)^2 are powers of two (h is): exact scaling
};

// The differences are folded in k, as the edge detector's images
// (ss4d_front_ff.cu): a 16-byte unit holds the float pairs of voxel k = m and
// of voxel k = m + Hk of the same (i, j, l), high parts first, so that in the
// faces kernel one address, one load and the packed FP32 instructions
// (ss4d_ff2.cuh) serve two voxels.  Planes 0 and Hk + 1 of the fold are both
// halves' halo.  The face quantities are natural again: the coefficient
// kernel is bound by the FP64 pipe and by latency, and with two voxels per
// thread (80 registers) it took 7.6 ms at 256^2 x 128 x 20 instead of 6.4.

template <int D> struct Axis {
    static constexpr int value = D;
};

__device__ __forceinline__ ff2 pair_of(ff a, ff b)
{
    return ff2{mk2(a.h, b.h), mk2(a.l, b.l)};
}
__device__ __forceinline__ ff2 ldf(const float4 *__restrict__ p, unsigned x)
{
    return unpack4(__ldg(p + x));
}

// forward differences of every voxel that has a neighbour along the axis, of
// frames [l0, l1).  With PACK also the split copies of u that k_pack makes
// when prev is u (red voxels into both red buffers, black ones into the black
// buffer, every voxel into prev of its colour): the FP64 subtractions leave
// memory bandwidth for the copy, and u is read once for both.  PACK 2 also
// adds the first refinement pass's start correction to the interior of the u
// copies the pass would update (red: R[0], black: Bk) with the pass's own
// FP64 addition: the correction in dR[0] / dB (withd) or zero.
template <int PACK>
__global__ void __launch_bounds__(256) k_fdiff(Geo g, int Hk, FastDiv fpl, Split sp, const double *__restrict__ u,
                                               SplitBufs b, unsigned o0, unsigned o1, int withd)
{
    const unsigned st[4] = {1u, (unsigned)g.sy, (unsigned)g.sz, (unsigned)g.sw};
    for (unsigned o = o0 + blockIdx.x * blockDim.x + threadIdx.x; o < o1; o += gridDim.x * blockDim.x) {
        unsigned q = fdiv(o, g.fiM);
        const int i = (int)(o - q * g.fiM.d);
        unsigned r = fdiv(q, g.fjM);
        const int j = (int)(q - r * g.fjM.d);
        const unsigned l = fdiv(r, fpl);
        const int m = (int)(r - l * fpl.d), kb = m + Hk;
        const bool vb = kb < g.kM;
        const unsigned oa = ((l * g.kM + m) * g.jM + j) * g.iM + i, ob = vb ? oa + Hk * st[2] : oa;
        const bool up[4] = {i < g.iM - 1, j < g.jM - 1, true, (int)l < g.lM - 1};
        const double ua = u[oa], ub = u[ob];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const bool na = a == 2 ? m < g.kM - 1 : up[a], nb = a == 2 ? kb < g.kM - 1 : up[a] && vb;
            const ff da = na ? ff_from_d(u[oa + st[a]] - ua) : ff_make(0.f, 0.f);
            const ff db = nb ? ff_from_d(u[ob + st[a]] - ub) : ff_make(0.f, 0.f);
            __stcs(reinterpret_cast<float4 *>(b.fd[a]) + o, make_float4(da.h, db.h, da.l, db.l));
        }
        if (PACK) {
            const bool ij = i >= 1 && i <= g.nx && j >= 1 && j <= g.ny && l >= 1 && (int)l <= g.nt;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                // each plane once: k = 0 .. Hk by the first half, the rest by the second
                const int k = h ? kb : m;
                if (h ? m < 1 || !vb : m > Hk)
                    continue;
                const double uc = h ? ub : ua;
                const unsigned s = ((l * g.kM + k) * g.jM + j) * (unsigned)sp.Hs + ((i + 1) >> 1) + sp.A - 1;
                const bool red = ((i + j + k + (int)l) & 1) == 0;
                double u0 = uc;
                if (PACK == 2 && ij && k >= 1 && k <= g.nz)
                    u0 = uc + (withd ? f2d_bits(red ? b.dR[0][s] : b.dB[s]) : 0.0);
                if (red) {
                    b.R[0][s] = u0;
                    b.R[1][s] = uc;
                    b.P[0][s] = uc;
                } else {
                    b.Bk[s] = u0;
                    b.P[1][s] = uc;
                }
            }
        }
    }
}

// --- faces ------------------------------------------------------------------
// A block takes a tile of FTX (32 or 16) x FTY folded voxels (i, j) of one (m, l) plane.
// The central differences D_a of every voxel are formed once, by its own thread,
// and the i- and j-faces read those of their upper neighbour from shared
// memory (the tile plus one column and one row of halo); the k- and l-faces
// form them at v + e_k and v + e_l.  Offsets are 32-bit (padded volumes below
// 2^31 voxels).
constexpr int FTY = 8;

// D_a(x) = F_a(x) + F_a(x - e_a), unnormalised (it is added again)
__device__ __forceinline__ ff2 cdiff(const float4 *__restrict__ fa, unsigned x, unsigned sa)
{
    return ff_add_nr2(ldf(fa, x), ldf(fa, x - sa));
}

__device__ __forceinline__ ff2 konst(float h, float l)
{
    return both(ff_make(h, l));
}

// 1/sqrt (ff_rsqrt)
__device__ __forceinline__ ff2 ff_rsqrt2(ff2 x)
{
    const f2 y0 = mk2(rsqrtf(lo2(x.h)), rsqrtf(hi2(x.h)));
    const f2 p = mul2(y0, y0), pe = fma2(y0, y0, neg2(p)); // y0^2 = p + pe exactly
    const f2 q = mul2(x.h, p);
    const f2 qe = fma2(x.l, p, fma2(x.h, pe, fma2(x.h, p, neg2(q)))); // x y0^2 = q + qe
    const f2 hr = mul2(both(0.5f), sub2(sub2(both(1.f), q), qe));    // 1 - q is exact (q near 1)
    const f2 c = mul2(y0, hr), ce = fma2(y0, hr, neg2(c));           // y0 hr = c + ce exactly
    ff2 y = fast_two_sum2(y0, c);
    y.l = add2(y.l, ce);
    return y;
}

// the face between v and v + e_D: Dv, Dn the central differences at v and
// v + e_D along the axes a != D, cn = F_D(v), gv its g; gives
// r = |grad u|_eps and q = g / |grad u|_eps
template <int D>
__device__ __forceinline__ void face_val(const FFConst &K, const ff2 Dv[4], const ff2 Dn[4], ff2 cn, ff2 gv, ff2 &r,
                                         ff2 &q)
{
    // sum of squares of the tangential central differences: positive terms,
    // renormalised once
    ff2 tt;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if (a == D)
            continue;
        const ff2 t = ff_add2(Dn[a], Dv[a]); // may cancel: renormalised before squaring
        const f2 p = mul2(t.h, t.h);
        const ff2 sq = ff2{p, fma2(add2(t.h, t.h), t.l, fma2(t.h, t.h, neg2(p)))};
        tt = a == (D == 0 ? 1 : 0) ? sq : ff_add_nr2(tt, sq);
    }
    tt = ff_norm2(tt);
    const f2 p = mul2(cn.h, cn.h);
    const ff2 cn2 = fast_two_sum2(p, fma2(add2(cn.h, cn.h), cn.l, fma2(cn.h, cn.h, neg2(p))));
    const ff2 a1 = K.pow2 ? ff2{mul2(cn2.h, both(K.ih2h)), mul2(cn2.l, both(K.ih2h))}
                          : ff_mul2(cn2, konst(K.ih2h, K.ih2l));
    const ff2 a2 = K.pow2 ? ff2{mul2(tt.h, both(K.iq2h)), mul2(tt.l, both(K.iq2h))}
                          : ff_mul2(tt, konst(K.iq2h, K.iq2l));
    const ff2 s2 = ff_add2(ff_add_nr2(a1, a2), konst(K.eps2h, K.eps2l));
    const ff2 y = ff_rsqrt2(s2);
    r = ff_mul2(s2, y);
    q = ff_mul2(gv, y);
}

// face_val, written as fn and fq at the natural offsets of both voxels
template <int D>
__device__ __forceinline__ void face_ff(const FFConst &K, const ff2 Dv[4], const ff2 Dn[4], ff2 cn, ff2 gv,
                                        const SplitBufs &b, unsigned oa, unsigned ob, bool vb)
{
    ff2 r, q;
    face_val<D>(K, Dv, Dn, cn, gv, r, q);
    float2 *fn = reinterpret_cast<float2 *>(b.fn[D]), *fq = reinterpret_cast<float2 *>(b.fq[D]);
    __stcs(fn + oa, make_float2(lo2(r.h), lo2(r.l)));
    __stcs(fq + oa, make_float2(lo2(q.h), lo2(q.l)));
    if (vb) {
        __stcs(fn + ob, make_float2(hi2(r.h), hi2(r.l)));
        __stcs(fq + ob, make_float2(hi2(q.h), hi2(q.l)));
    }
}

// g of the face between a ghost v along D (of the second half too: vb) and
// v + e_D: stored at v + e_D (g_w, g_s, ...)
template <int D>
__device__ __forceinline__ ff2 ghost_face_g(const CPtrs8 &gin, int has_g, unsigned oa, unsigned ob, bool vb,
                                            unsigned sd)
{
    ff a = ff_make(1.f, 0.f), c = a;
    if (has_g) {
        a = ff_from_pos_d(__ldg(gin.p[2 * D + 1] + oa + sd));
        if (vb)
            c = ff_from_pos_d(__ldg(gin.p[2 * D + 1] + ob + sd));
    }
    return pair_of(a, c);
}

// the faces of every voxel v with all indices in [0, n_a] whose faces
// between v and v + e_d have v and v + e_d in the extended box: all four for
// interior v, the one along a where v's index along a is 0 (and none where
// two indices are); frames l_off .. l_off + gridDim.z / (Hk + 1) - 1.
// Bound by the latency of its loads (at 128 x 128 x 64 x 8 issue 45 % busy, 64 %
// of the copy rate in DRAM bytes, 46 % of the warps): 64 registers, four blocks per SM, 5.3 ms at 256^2 x 128 x 20; three blocks (80) or
// five (48) took 0.2 and 0.6 ms more.  One voxel per thread, scalar, it took 5.9.
template <int FTX>
__global__ void __launch_bounds__(FTX *FTY, 128 / FTX) k_faces_ff(Geo g, int Hk, CPtrs8 gin, int has_g, FFConst K,
                                                                  SplitBufs b, int l_off, PlaneOrder po)
{
    __shared__ float4 sD[4][FTY + 1][FTX + 1];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int i0 = 1 + blockIdx.x * FTX, j0 = 1 + blockIdx.y * FTY;
    const int i = i0 + tx, j = j0 + ty;
    int m, lf;
    plane_frame(blockIdx.z, po, m, lf);
    const int l = l_off + lf;
    const unsigned st[4] = {1u, (unsigned)g.iM, (unsigned)(g.iM * g.jM), (unsigned)(g.iM * g.jM) * (Hk + 2)};
    const unsigned nst[4] = {1u, (unsigned)g.sy, (unsigned)g.sz, (unsigned)g.sw}; // natural strides
    const float4 *const F[4] = {reinterpret_cast<const float4 *>(b.fd[0]), reinterpret_cast<const float4 *>(b.fd[1]),
                                reinterpret_cast<const float4 *>(b.fd[2]), reinterpret_cast<const float4 *>(b.fd[3])};
    const unsigned x = (((unsigned)l * (Hk + 2) + m) * g.jM + j) * g.iM + i;
    const unsigned oa = (((unsigned)l * g.kM + m) * g.jM + j) * g.iM + i, ob = oa + Hk * nst[2];
    const bool vb = m + Hk <= g.nz; // the second half's voxel exists
    const ff2 zero = ff2{both(0.f), both(0.f)};
    // the single face along D of the voxels x, whose index along D is 0 (and
    // >= 1 along the others; for D = 2 in the first half only): the face
    // between them and x + e_D, where the differences Dn hold
    auto boundary = [&](auto tag, unsigned xv, unsigned na, unsigned nb, const ff2 Dn[4], bool second_too) {
        constexpr int D = decltype(tag)::value;
        ff2 Dv[4];
#pragma unroll
        for (int a = 0; a < 4; ++a)
            Dv[a] = a == D ? zero : cdiff(F[a], xv, st[a]);
        const bool v2 = vb && second_too;
        face_ff<D>(K, Dv, Dn, ldf(F[D], xv), ghost_face_g<D>(gin, has_g, na, nb, v2, nst[D]), b, na, nb, v2);
    };
    if (m == 0 || l == 0) { // ghost plane or frame: its one face along k or l
        if (m == l || i > g.nx || j > g.ny)
            return;
        ff2 Dn[4];
        if (m == 0) {
#pragma unroll
            for (int a = 0; a < 4; ++a)
                Dn[a] = a == 2 ? zero : cdiff(F[a], x + st[2], st[a]);
            boundary(Axis<2>{}, x, oa, ob, Dn, false);
        } else {
#pragma unroll
            for (int a = 0; a < 4; ++a)
                Dn[a] = a == 3 ? zero : cdiff(F[a], x + st[3], st[a]);
            boundary(Axis<3>{}, x, oa, ob, Dn, true);
        }
        return;
    }
    // g of the four faces, on its way from the start: each face waiting for
    // its own took 15.3 ms per assembly at 256^2 x 128 x 20 against 14.3
    double ga[4], gb[4];
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        const bool in = has_g && i <= g.nx && j <= g.ny;
        ga[d] = in ? __ldg(gin.p[2 * d] + oa) : 1.0;
        gb[d] = in && vb ? __ldg(gin.p[2 * d] + ob) : 1.0;
    }
    // central differences of the tile (ghost column / row included) ...
    ff2 Dv[4];
    if (i <= g.nx + 1 && j <= g.ny + 1) {
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            Dv[a] = cdiff(F[a], x, st[a]);
            sD[a][ty][tx] = pack4(Dv[a]);
        }
    }
    // ... and of its halo: row j0 + FTY (for the j-faces of the tile's last
    // row) and column i0 + FTX (for the i-faces of its last column), where
    // those faces exist
    if (ty == 0) {
        if (i <= g.nx && j0 + FTY <= g.ny + 1) {
            const unsigned xh = x + FTY * st[1];
#pragma unroll
            for (int a = 0; a < 4; ++a)
                if (a != 1)
                    sD[a][FTY][tx] = pack4(cdiff(F[a], xh, st[a]));
        }
    } else if (ty == 1 && tx < FTY) {
        if (i0 + FTX <= g.nx + 1 && j0 + tx <= g.ny) {
            const unsigned xh = (((unsigned)l * (Hk + 2) + m) * g.jM + (j0 + tx)) * g.iM + (i0 + FTX);
#pragma unroll
            for (int a = 1; a < 4; ++a)
                sD[a][tx][FTX] = pack4(cdiff(F[a], xh, st[a]));
        }
    }
    __syncthreads();
    if (i > g.nx || j > g.ny)
        return;
    ff2 Dn[4];
    // i-face and j-face: the upper neighbour's differences from the tile
#pragma unroll
    for (int a = 1; a < 4; ++a)
        Dn[a] = unpack4(sD[a][ty][tx + 1]);
    face_ff<0>(K, Dv, Dn, ldf(F[0], x), pair_of(ff_from_pos_d(ga[0]), ff_from_pos_d(gb[0])), b, oa, ob, vb);
#pragma unroll
    for (int a = 0; a < 4; ++a)
        if (a != 1)
            Dn[a] = unpack4(sD[a][ty + 1][tx]);
    face_ff<1>(K, Dv, Dn, ldf(F[1], x), pair_of(ff_from_pos_d(ga[1]), ff_from_pos_d(gb[1])), b, oa, ob, vb);
    // k-face and l-face: the differences at v + e_k and v + e_l
#pragma unroll
    for (int a = 0; a < 4; ++a)
        if (a != 2)
            Dn[a] = cdiff(F[a], x + st[2], st[a]);
    face_ff<2>(K, Dv, Dn, ldf(F[2], x), pair_of(ff_from_pos_d(ga[2]), ff_from_pos_d(gb[2])), b, oa, ob, vb);
#pragma unroll
    for (int a = 0; a < 4; ++a)
        if (a != 3)
            Dn[a] = cdiff(F[a], x + st[3], st[a]);
    face_ff<3>(K, Dv, Dn, ldf(F[3], x), pair_of(ff_from_pos_d(ga[3]), ff_from_pos_d(gb[3])), b, oa, ob, vb);
    // the faces between the ghosts i = 0 / j = 0 and the first voxel: the
    // thread of that voxel (its differences are the upper side's)
    if (i == 1)
        boundary(Axis<0>{}, x - st[0], oa - nst[0], ob - nst[0], Dv, true);
    if (j == 1)
        boundary(Axis<1>{}, x - st[1], oa - nst[1], ob - nst[1], Dv, true);
}

// Memory-bound, its warps waiting on loads: 8 blocks per SM (32 registers)
// rather than 7 took the assembly from 13.5 to 13.0 ms at 256^2 x 128 x 20.
// With PRE it also forms the first refinement pass's FP64 residual at the
// target exactly as k_refine forms it (prev, then the products of the eight
// coefficients just written with the other colour's u in record order, then
// diag u0, with the same fused multiply-adds) on the split copies of u whose
// start correction the first-difference kernel added, into rpre.
// The records of interior voxel (i, j, k, l) (and with PRE the first pass's
// residual) from its 8 faces: fp[d], fm[d] the |grad u|_eps of its faces
// towards v + e_d and v - e_d, q[2d], q[2d+1] their g / |grad u|_eps
template <int PRE>
__device__ __forceinline__ void voxel_coef(const Geo &g, const Split &sp, const FFConst &K, const SplitBufs &b, int i,
                                           int j, int k, int l, const ff fp[4], const ff fm[4], const ff q[8])
{
    ff sum = ff_make(0.f, 0.f);
#pragma unroll
    for (int d = 0; d < 4; ++d) // positive terms: renormalised once
        sum = ff_add_nr(sum, ff_add_nr(fp[d], fm[d]));
    sum = ff_norm(sum);
    // mean^2 + eps2 with mean = sum / 8 (exact scaling)
    const ff m = ff_make(sum.h * 0.125f, sum.l * 0.125f);
    const ff x = ff_add(ff_sqr(m), ff_make(K.eps2h, K.eps2l));
    const ff cv = ff_mul(ff_make(K.ch, K.cl), ff_mul(x, ff_rsqrt(x))); // c * vc
    const int col = (i + j + k + l) & 1;
    double *cf = pick(b.coef, col);
    const long long t = coef_index(g, sp, i, j, k, l);
    // split index of the target and its neighbours (row phase p = i & 1)
    const long long Hy = sp.Hs, Hz = Hy * g.jM, Hw = Hz * g.kM;
    const long long sx = (((long long)l * g.kM + k) * g.jM + j) * Hy + ((i + 1) >> 1) + sp.A - 1;
    const int p = i & 1;
    const long long nb[8] = {sx - p + 1, sx - p, sx + Hy, sx - Hy, sx + Hz, sx - Hz, sx + Hw, sx - Hw};
    const double *__restrict__ oth = col == 0 ? b.Bk : b.R[0];
    double S = PRE ? __ldg(pick(b.P, col) + sx) : 0.0;
    ff diag = ff_make(1.f, 0.f);
    float a32[8];
#pragma unroll
    for (int f = 0; f < 8; ++f) {
        const ff a = ff_mul(cv, q[f]);
        diag = ff_add_nr(diag, a); // positive terms: renormalised after the loop
        const double ad = ff_to_d(a);
        __stcs(cf + coef_at(t, f, 10), ad);
        a32[f] = a.h;
        if (PRE)
            S = fma(ad, __ldg(oth + nb[f]), S);
    }
    diag = ff_norm(diag);
    const double dd = ff_to_d(diag);
    __stcs(cf + coef_at(t, 8, 10), dd);
    if (PRE)
        pick(b.rpre, col)[sx] = fma(dd, __ldg((col == 0 ? b.R[0] : b.Bk) + sx), -S);
    // component 9 (omega/diag) serves only the FP64 sweep, whose form always
    // assembles its own records: not written here
    store_coef16(pick(b.coefq, col), pick(b.coefs, col), t, a32);
}

// One thread per voxel of a plane, i fastest across rows: blocks of rows'
// chunks left 37 % of the lanes idle at nx = 161 (the step of 161 x 143 x 61 x 9
// 6.15 ms, now 6.09).
template <int PRE>
__global__ void __launch_bounds__(256, PRE ? 6 : 8) k_voxel_coef_ff(Geo g, Split sp, FFConst K, SplitBufs b, int l_off,
                                                                    FastDiv row, PlaneOrder po)
{
    const unsigned at = blockIdx.x * blockDim.x + threadIdx.x, jr = fdiv(at, row);
    const int i = 1 + (int)(at - jr * row.d), j = 1 + (int)jr;
    int kk, lf;
    plane_frame(blockIdx.z, po, kk, lf);
    const int k = 1 + kk, l = 1 + l_off + lf;
    if (j > g.ny)
        return;
    const long long o = nat_index(g, i, j, k, l);
    const long long st[4] = {1, g.sy, g.sz, g.sw};
    ff fp[4], fm[4], q[8];
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        fp[d] = ld_ff(b.fn[d], o);
        fm[d] = ld_ff(b.fn[d], o - st[d]);
        q[2 * d] = ld_ff(b.fq[d], o);
        q[2 * d + 1] = ld_ff(b.fq[d], o - st[d]);
    }
    voxel_coef<PRE>(g, sp, K, b, i, j, k, l, fp, fm, q);
}

static void split_host(double v, float &h, float &l)
{
    h = (float)v;
    l = (float)(v - (double)h);
}

template <int PACK>
static void run_fdiff(const Geo &g, const Split &s, const double *u, const SplitBufs &b, int l0, int l1, int sm_count,
                      cudaStream_t st, int withd)
{
    static const int per_sm = [] { // once, whichever thread steps first
        int a = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_fdiff<PACK>, 256, 0);
        return a > 0 ? a : 1;
    }();
    const int Hk = fold_of(g);
    const unsigned frame = (unsigned)(g.iM * g.jM) * (Hk + 2), n = frame * (unsigned)(l1 - l0);
    const unsigned need = (n + 255) / 256, most = (unsigned)(sm_count * per_sm);
    k_fdiff<PACK><<<need < most ? need : most, 256, 0, st>>>(g, Hk, make_fastdiv((unsigned)Hk + 2), s, u, b,
                                                             frame * (unsigned)l0, frame * (unsigned)l1, withd);
}

void launch_fdiff_range(const Geo &g, const double *u, SplitBufs b, int l0, int l1, int sm_count, cudaStream_t st)
{
    run_fdiff<0>(g, Split{}, u, b, l0, l1, sm_count, st, 0);
}

void launch_fdiff_pack_range(const Geo &g, const Split &s, const double *u, SplitBufs b, int l0, int l1, int sm_count,
                             cudaStream_t st, int pre)
{
    if (pre)
        run_fdiff<2>(g, s, u, b, l0, l1, sm_count, st, pre == 2);
    else
        run_fdiff<1>(g, s, u, b, l0, l1, sm_count, st, 0);
}

void launch_assemble_ff(const Geo &g, const Split &s, const double *u, CPtrs8 gin, int has_g, const ss4d_params &p,
                        SplitBufs b, int pack, int sm_count, cudaStream_t st, int pre, int kblock)
{
    if (pack)
        launch_fdiff_pack_range(g, s, u, b, 0, g.lM, sm_count, st, pre);
    else
        launch_fdiff_range(g, u, b, 0, g.lM, sm_count, st);
    launch_assemble_ff_faces(g, s, gin, has_g, p, b, st, pack ? pre : 0, kblock);
}

void launch_assemble_ff_faces(const Geo &g, const Split &s, CPtrs8 gin, int has_g, const ss4d_params &p, SplitBufs b,
                              cudaStream_t st, int pre, int kblock)
{
    launch_assemble_ff_faces_range(g, s, gin, has_g, p, b, 0, g.nt + 1, 1, g.nt + 1, st, pre, kblock);
}

static FFConst make_ffconst(const ss4d_params &p)
{
    FFConst K;
    split_host(1.0 / (p.h * p.h), K.ih2h, K.ih2l);
    split_host(1.0 / (16.0 * p.h * p.h), K.iq2h, K.iq2l);
    split_host(p.eps2, K.eps2h, K.eps2l);
    split_host(p.tau / (p.h * p.h), K.ch, K.cl);
    int e1 = 0, e2 = 0;
    K.pow2 = K.ih2l == 0.f && K.iq2l == 0.f && frexp((double)K.ih2h, &e1) == 0.5 && frexp((double)K.iq2h, &e2) == 0.5;
    return K;
}

void launch_assemble_ff_faces_range(const Geo &g, const Split &s, CPtrs8 gin, int has_g, const ss4d_params &p,
                                    SplitBufs b, int f0, int f1, int v0, int v1, cudaStream_t st, int pre, int kblock)
{
    const FFConst K = make_ffconst(p);
    const int Hk = fold_of(g);
    const int kb = kblock <= 0 ? 0 : (kblock + 1) / 2; // folded planes
    if (f1 > f0) {
        // tiles 16 wide where they leave fewer lanes idle: 48 volumes of 24-48
        // 19.0 -> 18.6 ms a run, a step of 161 x 143 x 61 x 9 6.09 -> 6.08; at 256
        // wide their larger halo costs 0.5 % (228.4 -> 229.5 ms)
        const bool narrow = (g.nx + 15) / 16 % 2 != 0;
        const int w = narrow ? 16 : 32;
        const dim3 gr((g.nx + w - 1) / w, (g.ny + FTY - 1) / FTY, (Hk + 1) * (f1 - f0)), bl(w, FTY, 1);
        const PlaneOrder po = make_plane_order(Hk + 1, f1 - f0, kb);
        if (narrow)
            k_faces_ff<16><<<gr, bl, 0, st>>>(g, Hk, gin, has_g, K, b, f0, po);
        else
            k_faces_ff<32><<<gr, bl, 0, st>>>(g, Hk, gin, has_g, K, b, f0, po);
    }
    if (v1 > v0) {
        const dim3 gr(((unsigned)g.nx * g.ny + 255) / 256, 1, g.nz * (v1 - v0));
        const FastDiv row = make_fastdiv((unsigned)g.nx);
        const PlaneOrder po = make_plane_order(g.nz, v1 - v0, kblock);
        if (pre)
            k_voxel_coef_ff<1><<<gr, 256, 0, st>>>(g, s, K, b, v0 - 1, row, po);
        else
            k_voxel_coef_ff<0><<<gr, 256, 0, st>>>(g, s, K, b, v0 - 1, row, po);
    }
}

} // namespace ss4d
