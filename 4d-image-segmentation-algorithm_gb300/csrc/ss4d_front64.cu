// ss4d_front64.cu — the presmoothing in the reference's FP64 arithmetic
// (ss4d_front.cuh).  Compiled with --fmad=false: every multiply and add is
// rounded as in the reference's build, and the voxel update keeps its
// expression order (segmentation4D.c:366-384), so after the same number of
// iterations the image equals the reference's bit for bit.  The stop test's
// sum differs in rounding: a residual is formed with one rounding from the
// update's own sum instead of three, and the terms are added in another
// order (and unscaled by h^4 until their sum is complete).  Where that could
// decide a test the other way it is reported (FrontNear).
//
// Bound by the FP64 pipe (80 % busy): 16 instructions per target for the update and 2 for
// its residual, which the separate residual pass formed with 15.4 per voxel
// (the edge detector of two images of 97 x 101 x 53 x 11: 7.84 ms with 4, 7.39 with 2).
// Two blocks of 256 per SM (90 registers, none spilled): 6.96 ms; three 7.16,
// four 7.39, five 7.43; one of 384 7.10, one of 512 7.20.
#include "ss4d_front.cuh"

namespace ss4d {

namespace {

struct Exact64 {
    typedef double2 Q;
    typedef double Acc;
    struct Const {
        double c, d, y, omega;
    };
    static __device__ __forceinline__ Const constants(const FrontArgs &a)
    {
        return Const{a.c, a.d, a.y, a.omega};
    }
    static __device__ __forceinline__ Acc zero()
    {
        return 0.0;
    }
    template <int COL>
    static __device__ __forceinline__ double total(const FrontArgs &, Acc a)
    {
        return a;
    }
    static __device__ __forceinline__ Q make(double x, double y)
    {
        return make_double2(x, y);
    }
    static __device__ __forceinline__ void get(Q v, double *w)
    {
        w[0] = v.x;
        w[1] = v.y;
    }
    static __device__ __forceinline__ Q live(const Q *p)
    {
        Q v;
        asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
        return v;
    }
    static __device__ __forceinline__ double first(const Q *p)
    {
        return ld_oth<true>(&p->x);
    }
    static __device__ __forceinline__ double second(const Q *p)
    {
        return ld_oth<true>(&p->y);
    }
    static __device__ __forceinline__ Q up(Q v, double e)
    {
        return make_double2(v.y, e);
    }
    static __device__ __forceinline__ Q down(double e, Q v)
    {
        return make_double2(e, v.x);
    }
    static __device__ __forceinline__ Q with_first(Q v, Q w)
    {
        return make_double2(w.x, v.y);
    }
    static __device__ __forceinline__ Q with_second(Q v, Q w)
    {
        return make_double2(v.x, w.y);
    }
    template <int COL>
    static __device__ __forceinline__ double one(const Const &C, double u, double pv, double xr, double xl, double ym,
                                                 double yp, double zm, double zp, double wm, double wp, double &acc)
    {
        const double cs = C.c * (xr + xl + ym + yp + zm + zp + wm + wp);
        const double t = pv + cs;
        const double gs = div_by_const(t, C.d, C.y);
        const double v = u + C.omega * (gs - u);
        const double r = fma(COL == 0 ? u : v, C.d, -t); // one rounding instead of three
        acc = fma(r, r, acc);
        return v;
    }
    template <int COL>
    static __device__ __forceinline__ Q update(const Const &C, Q u, Q pv, Q xr, Q xl, Q ym, Q yp, Q zm, Q zp, Q wm,
                                               Q wp, bool two, Acc &acc)
    {
        Q v = u;
        v.x = one<COL>(C, u.x, pv.x, xr.x, xl.x, ym.x, yp.x, zm.x, zp.x, wm.x, wp.x, acc);
        if (two)
            v.y = one<COL>(C, u.y, pv.y, xr.y, xl.y, ym.y, yp.y, zm.y, zp.y, wm.y, wp.y, acc);
        return v;
    }
    static __device__ __forceinline__ void fold(const FrontArgs &, const Q *, unsigned, unsigned)
    {
    }
};

__global__ void __launch_bounds__(FRONT64_THREADS, 2) k_presmooth64(const __grid_constant__ FrontArgs a)
{
    presmooth_body<Exact64>(a);
}

} // namespace

int presmooth64_grid(int sm_count)
{
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_presmooth64, FRONT64_THREADS, 0);
    return per * sm_count;
}

cudaError_t launch_presmooth64(const FrontArgs &a, int grid, cudaStream_t st)
{
    void *args[] = {(void *)&a};
    return cudaLaunchCooperativeKernel((const void *)k_presmooth64, dim3(grid), dim3(FRONT64_THREADS), args, 0, st);
}

} // namespace ss4d
