// Shared device/host helpers of the dadi_gb300 kernels.
//
// The implicit ADI sweep of dadi (dadi/integration_shared.c:4-93,
// dadi/tridiag.c:14-34) is restated here in a form that costs ~10 FP64
// pipe instructions per grid point per sweep:
//
//  * Every tridiagonal row is multiplied by dt, so r = phi and the diagonal
//    is 1 + dt*(...); no per-point division by dt.
//  * With delta_j = 0.5 (dadi's default, use_delj_trick False), the
//    coefficients of a line are affine in W = sum_k m_k o_k, the only
//    quantity that depends on the line's other coordinates o_k:
//        a'_i = W*A1_i + A0_i,  c'_i = W*C1_i + C0_i,
//        b'_i = B0_i  (interior rows; W cancels),  b'_0 and b'_{L-1} carry W*B1.
//    A1..B0 are per-axis vectors rebuilt once per step (O(L) work) from
//    dx, dfactor, xInt, V = x(1-x)/nu and the selection term, following
//    compute_abc_nobc (dadi/integration_shared.c:72-93).
//  * 1/bet uses the hardware reciprocal seed (rcp.approx.ftz.f64) refined by
//    one third-order Newton-Raphson step r(1 + e + e^2), e = 1 - x r, which
//    is accurate to about one ulp; quotients become products.
//  * The reciprocal and the products with it are formed on the integer pipes
//    (pivot, below), which leaves 5 of the 10 on the FP64 pipe.
// These reassociations move results by a few ulps per step relative to the
// reference C, far inside the 1e-9 relative bar on extrapolated spectra.
//
// Under the delj trick (Chang-Cooper delta_j, dadi/integration_shared.c:
// 52-70) none of this is done.  delta_j = (-e w + e V - V) / (w - e w),
// e = exp(w / V), cancels catastrophically as w / V -> 0, so any rounding
// of MInt or of delta_j's own terms is amplified; the delj path therefore
// follows the reference operation by operation: unscaled rows (b starts at
// 1/dt, r = phi/dt), every product and sum rounded on its own (the __d*_rn
// intrinsics, which the compiler never fuses into a multiply-add, where C
// compiled for x86-64 has no fused multiply-add either), IEEE division, and
// the Numerical-Recipes recurrence as written.  Only exp is CUDA's (an
// error bound of one ulp rather than the C library's half ulp).
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/dadi_gb300.h"

namespace dgb {

#define DGB_HD __host__ __device__ __forceinline__

// ---------------------------------------------------------------- arithmetic

__device__ __forceinline__ double rcp_seed(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}

// Reciprocal to ~1 ulp: seed refined by one cubic Newton-Raphson step.
// rcp_newton is not inlined: it is the rare other side of rcp_full and pivot
// below, and a predicated-off FP64 instruction takes the pipe like one that
// runs.
__device__ __forceinline__ double rcp_newton_here(double x)
{
    double r = rcp_seed(x);
    double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
static __device__ __noinline__ double rcp_newton(double x) { return rcp_newton_here(x); }

// The same reciprocal, and products with it, on the integer pipes.
//
// The SM has one FP64 pipe: an FP64 instruction of a warp takes it 16 cycles
// (64 issue slots of a sub-partition; DMUL and DADD 19), and one warp issues
// at most one per 64 cycles.  A sweep is bound by its count of FP64
// instructions, whatever their dependencies, while the integer pipes stand
// idle.  So of the 10 FP64 instructions of a grid point the three of the
// reciprocal and the products t * inv and c * inv are done with 32 x 32 -> 64
// bit multiply-adds instead (about 110 instructions), which leaves 5.
// Measured, Thomas lines of 48 points on one SM, cycles per point and warp of
// lines: 171 -> 88 with 16 warps, 175 -> 110 with 7, 844 -> 634 for one warp
// (its chain: 134 cycles for the reciprocal, 108 for a product).  1,000 IM
// spectra at pts 80/90/100: 1.08 -> 0.73 s.  The
// results are the same bits as those of rcp_newton and of IEEE multiplication:
// every value is rounded from one that carries 32 or more further bits, and
// where these cannot tell which way the rounding on doubles goes (one pivot
// in 8,000), or a value leaves the range handled here, the doubles decide.
//
// rcp_mant: for x = m 2^E, X = m 2^52 (53 bits) and the seed r0 of 1/m as rho
// = r0 2^21 (21 bits), -X rho mod 2^64 is the residual e = 1 - m r0 (|e| <
// 2^-19) in units of 2^-73, exactly; then 1/m = r0 (1 + e + e^2) is built in
// units of 2^-96 with an error below 2^-67, and rounded to 53 bits.
struct Mant {
    unsigned h, l; // 2^64 / m rounded to 53 bits: the top bit of h is set
};

__device__ __forceinline__ Mant rcp_mant(double x, bool &bad)
{
    const unsigned xh = (unsigned)__double2hiint(x), xl = (unsigned)__double2loint(x);
    const unsigned hx = (xh & 0xfffffu) | 0x100000u;
    const double seed = rcp_seed(__hiloint2double((int)(hx + 0x3fe00000u), (int)xl));
    const unsigned rho = (unsigned)__double2hiint(seed) - 0x3fd00000u;
    const unsigned nr = 0u - rho; // xl * nr counts xl 2^32 too much
    const unsigned long long t = (unsigned long long)xl * nr;
    const unsigned eh = (unsigned)(t >> 32) + hx * nr - xl;
    const unsigned long long e = (unsigned long long)eh << 32 | (unsigned)t;
    const int s = (int)__funnelshift_r((unsigned)t, eh, 23);
    const unsigned long long f = (unsigned long long)(unsigned)__mulhi(s, s) * 32u + e;
    const unsigned r4 = rho << 2;
    const unsigned long long w = (unsigned long long)r4 * (unsigned)f;
    const unsigned long long r =
        (unsigned long long)((long long)(int)r4 * (int)(f >> 32)) +
        ((unsigned long long)(rho << 11) << 32 | (unsigned)(w >> 32));
    // the bits below the 53rd, against one half, within the error
    const unsigned v = __funnelshift_l((unsigned)w, (unsigned)r, 21);
    const unsigned long long y = r + 0x400u;
    Mant o;
    o.h = (unsigned)(y >> 32);
    o.l = (unsigned)y & ~0x7ffu;
    // (the top bit is clear for m = 1; exponents from -128 to 127)
    bad = (v - 0x7ffc0000u < 0x80000u) | ((int)o.h >= 0) |
          ((xh & 0x7fffffffu) - 0x37f00000u >= 0x10000000u);
    return o;
}

// x * (1/b) for the mantissa y of 1/b, rounded as IEEE multiplication rounds;
// exps = exponent field of 1/b less the bias and one.
__device__ __forceinline__ double mul_mant(double x, const Mant &y, unsigned exps, bool &bad)
{
    const unsigned xh = (unsigned)__double2hiint(x), xl = (unsigned)__double2loint(x);
    const unsigned mh = (xh & 0xfffffu) | 0x100000u;
    const unsigned long long t1 = (unsigned long long)mh * y.l + __umulhi(xl, y.l);
    const unsigned long long t2 = (unsigned long long)xl * y.h + (unsigned)t1;
    const unsigned long long p = (unsigned long long)mh * y.h +
                                 ((unsigned long long)(unsigned)(t1 >> 32) + (unsigned)(t2 >> 32));
    const unsigned w1 = (unsigned)t2, w2 = (unsigned)p, w3 = (unsigned)(p >> 32);
    const unsigned sh = (w3 >> 20) ^ 1u; // mantissa in [1, 2): one bit up
    const unsigned m1 = w1 << sh;
    const unsigned long long m = ((unsigned long long)__funnelshift_l(w2, w3, sh) << 32 |
                                  __funnelshift_l(w1, w2, sh)) +
                                 (m1 >> 31);
    // (a tie, or a value whose product may leave the normal range)
    bad = bad | (m1 == 0x80000000u) | ((xh & 0x7fffffffu) - 0x0c800000u >= 0x66000000u);
    return __hiloint2double(
        (int)((unsigned)(m >> 32) + (xh & 0xfff00000u) + exps + (w3 & 0x100000u)),
        (int)(unsigned)m);
}

__device__ __forceinline__ unsigned rcp_exps(double x)
{
    return 0x3fd00000u - ((unsigned)__double2hiint(x) & 0xfff00000u);
}

// The double of mantissa y and exps (as mul_mant takes them).
__device__ __forceinline__ double mant_double(const Mant &y, unsigned exps)
{
    return __hiloint2double((int)((y.h >> 11) + 0x3ff00000u + exps),
                            (int)__funnelshift_r(y.l, y.h, 11));
}

__device__ __forceinline__ double rcp_full(double x)
{
    bool bad;
    const Mant y = rcp_mant(x, bad);
    double r = mant_double(y, rcp_exps(x));
    if (bad)
        r = rcp_newton(x);
    return r;
}

// 1/x for x = m 2^E to 67 bits: r[2]:r[1]:r[0] = 2^96 / m (rcp_mant's, with
// one more term of the series, before its rounding).
__device__ __forceinline__ void rcp_wide(double x, unsigned (&r)[3])
{
    const unsigned xh = (unsigned)__double2hiint(x), xl = (unsigned)__double2loint(x);
    const unsigned hx = (xh & 0xfffffu) | 0x100000u;
    const double seed = rcp_seed(__hiloint2double((int)(hx + 0x3fe00000u), (int)xl));
    const unsigned rho = (unsigned)__double2hiint(seed) - 0x3fd00000u;
    const unsigned nr = 0u - rho;
    const unsigned long long t = (unsigned long long)xl * nr;
    const unsigned eh = (unsigned)(t >> 32) + hx * nr - xl;
    const unsigned long long e = (unsigned long long)eh << 32 | (unsigned)t;
    const int s = (int)__funnelshift_r((unsigned)t, eh, 23);
    const int q = __mulhi(s, s);
    const unsigned long long f = (unsigned long long)(unsigned)q * 32u + e +
                                 (unsigned long long)(long long)(__mulhi(s, q) >> 13);
    const unsigned r4 = rho << 2;
    const unsigned long long w = (unsigned long long)r4 * (unsigned)f;
    const unsigned long long y =
        (unsigned long long)((long long)(int)r4 * (int)(f >> 32)) +
        ((unsigned long long)(rho << 11) << 32 | (unsigned)(w >> 32));
    r[0] = (unsigned)w;
    r[1] = (unsigned)y;
    r[2] = (unsigned)(y >> 32);
}

static __device__ __noinline__ double mul_fp64(double x, double y) { return x * y; }

// The rare sides of functions among whose operands zero is an ordinary value
// (a model without migration or selection: every coupling to the row before the
// first segment of a partitioned line, every mean change under the delj trick):
// a zero's product or quotient is formed off the FP64 pipe, all else by it.
// Not inlined, see rcp_newton.  Without migration and selection, milliseconds
// with every zero on the FP64 pipe / so: 60 steps under the delj trick at 100
// points 25.2 / 15.4 (with migration 17.1 / 17.0), 300 steps on clusters at 128
// points 11.8 / 10.0, 60 steps of three populations at 90 points 5.42 / 4.99.
// The lines' other products (pivot, mul_full) keep the plain call: they meet a
// zero once a line, and in k_integrate2d_ws these sides cost 1-10 %.
__device__ __forceinline__ bool is_zero(double x)
{
    return ((unsigned)__double2hiint(x) << 1 | (unsigned)__double2loint(x)) == 0;
}

__device__ __forceinline__ bool is_finite(double x)
{
    return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000;
}

// Zero with the sign of x * y.
__device__ __forceinline__ double zero_of(double x, double y)
{
    return __hiloint2double((__double2hiint(x) ^ __double2hiint(y)) & (int)0x80000000u, 0);
}

static __device__ __noinline__ double mul_rare(double x, double y)
{
    if ((is_zero(x) && is_finite(y)) || (is_zero(y) && is_finite(x)))
        return zero_of(x, y);
    return x * y;
}

static __device__ __noinline__ double div_rare(double x, double y)
{
    if (is_zero(x) && !is_zero(y) && is_finite(y))
        return zero_of(x, y);
    return __ddiv_rn(x, y);
}

// (The delj rows have five divisions a point: 64 IM sets at pts 40/50/60 took
// 1.33 s with them on the FP64 pipe, 0.89 with div_full.)

// x / y rounded as IEEE division rounds, from y's rcp_wide.  A quotient is
// never half way between two doubles, and one within the error of it (one in
// 2^11), or out of range, is left to the FP64 pipe (some 10 instructions).
__device__ __forceinline__ double div_wide(double x, double y, const unsigned (&r)[3])
{
    const unsigned xh = (unsigned)__double2hiint(x), xl = (unsigned)__double2loint(x);
    const unsigned yh = (unsigned)__double2hiint(y);
    const unsigned mh = (xh & 0xfffffu) | 0x100000u;
    const unsigned long long t1 = (unsigned long long)mh * r[1] + __umulhi(xl, r[1]);
    const unsigned long long t2 = (unsigned long long)xl * r[2] +
                                  ((unsigned long long)(unsigned)t1 + __umulhi(mh, r[0]));
    const unsigned long long p = (unsigned long long)mh * r[2] +
                                 ((unsigned long long)(unsigned)(t1 >> 32) + (unsigned)(t2 >> 32));
    const unsigned w1 = (unsigned)t2, w2 = (unsigned)p, w3 = (unsigned)(p >> 32);
    const unsigned sh = (w3 >> 20) ^ 1u;
    const unsigned m1 = w1 << sh;
    const unsigned long long m = ((unsigned long long)__funnelshift_l(w2, w3, sh) << 32 |
                                  __funnelshift_l(w1, w2, sh)) +
                                 (m1 >> 31);
    const bool bad = (m1 - 0x7ff00000u < 0x200000u) | ((int)r[2] >= 0) |
                     ((yh & 0x7fffffffu) - 0x37f00000u >= 0x10000000u) |
                     ((xh & 0x7fffffffu) - 0x0c800000u >= 0x66000000u);
    double q = __hiloint2double((int)((unsigned)(m >> 32) + (xh & 0xfff00000u) + 0x3fd00000u -
                                      (yh & 0xfff00000u) + (w3 & 0x100000u)),
                                (int)(unsigned)m);
    if (bad)
        q = div_rare(x, y);
    return q;
}

__device__ __forceinline__ double div_full(double x, double y)
{
    unsigned r[3];
    rcp_wide(y, r);
    return div_wide(x, y, r);
}

// x * y rounded as IEEE multiplication rounds (y an unpacked double); ZEROS:
// for operands of which zero is an ordinary value.
template <bool ZEROS = false> __device__ __forceinline__ double mul_full(double x, double y)
{
    const unsigned yh = (unsigned)__double2hiint(y), yl = (unsigned)__double2loint(y);
    Mant m;
    m.h = __funnelshift_l(yl, (yh & 0xfffffu) | 0x100000u, 11);
    m.l = yl << 11;
    bool bad = (yh & 0x7fffffffu) - 0x37f00000u >= 0x10000000u;
    double r = mul_mant(x, m, (yh & 0xfff00000u) - 0x40000000u, bad);
    if (bad)
        r = ZEROS ? mul_rare(x, y) : mul_fp64(x, y);
    return r;
}

static __device__ __noinline__ double2 pivot_fp64(double bet, double t, double c)
{
    const double inv = rcp_newton(bet);
    return make_double2(t * inv, c * inv);
}

// u = t * (1/bet) and g = c * (1/bet).
__device__ __forceinline__ void pivot(double bet, double t, double c, double &u, double &g)
{
    bool bad;
    const Mant y = rcp_mant(bet, bad);
    const unsigned exps = rcp_exps(bet);
    u = mul_mant(t, y, exps, bad);
    g = mul_mant(c, y, exps, bad);
    if (bad) {
        const double2 ug = pivot_fp64(bet, t, c);
        u = ug.x;
        g = ug.y;
    }
}

// The same, on the FP64 pipe if FP64.
template <bool FP64>
__device__ __forceinline__ void pivot_as(double bet, double t, double c, double &u, double &g)
{
    if (FP64) {
        const double inv = rcp_newton_here(bet);
        u = t * inv;
        g = c * inv;
    } else {
        pivot(bet, t, c, u, g);
    }
}

static __device__ __noinline__ double3 pivot3_fp64(double bet, double t, double c, double d)
{
    const double inv = rcp_newton(bet);
    return make_double3(t * inv, c * inv, d * inv);
}

// A product with 1/bet that mul_mant refused: a zero put right, or not all are.
__device__ __forceinline__ void pivot_zero(double bet, double x, int bad, double &v, bool &all)
{
    if (bad) {
        v = zero_of(x, bet);
        all = all && is_zero(x);
    }
}

// (bad, bit by bit: 1/bet, and its products with t, c and d)
static __device__ __noinline__ double3 pivot3_rare(double bet, double t, double c, double d,
                                                   double u, double g, double w, int bad)
{
    bool all = !(bad & 1);
    pivot_zero(bet, t, bad & 2, u, all);
    pivot_zero(bet, c, bad & 4, g, all);
    pivot_zero(bet, d, bad & 8, w, all);
    return all ? make_double3(u, g, w) : pivot3_fp64(bet, t, c, d);
}

// u = t * (1/bet), g = c * (1/bet) and w = d * (1/bet): the rows of the
// partitioned solves.
__device__ __forceinline__ void pivot3(double bet, double t, double c, double d, double &u,
                                       double &g, double &w)
{
    bool bb, bt = false, bc = false, bd = false;
    const Mant y = rcp_mant(bet, bb);
    const unsigned exps = rcp_exps(bet);
    u = mul_mant(t, y, exps, bt);
    g = mul_mant(c, y, exps, bc);
    w = mul_mant(d, y, exps, bd);
    if (bb | bt | bc | bd) {
        const double3 r = pivot3_rare(bet, t, c, d, u, g, w,
                                      (int)bb | (int)bt << 1 | (int)bc << 2 | (int)bd << 3);
        u = r.x;
        g = r.y;
        w = r.z;
    }
}

// ------------------------------------------------------- parameter schedule

// Parametric time dependence (see dgb_pform in dadi_gb300.h).
DGB_HD double pform_eval(const dgb_pform &f, double t)
{
    switch (f.kind) {
    case DGB_PF_EXPGROW:
        return f.a * pow(f.b / f.a, t / f.c);
    case DGB_PF_EXPLOG:
        return f.a * exp(log(f.b / f.a) * t / f.c);
    case DGB_PF_LINEAR:
        return f.a + f.b * t;
    default:
        return f.a;
    }
}

// Timestep from one population's current parameters, as
// dadi/Integration.py:147-176 (Python max/min keep the first extreme).
DGB_HD double compute_dt(double nu, double msum, double gamma, double h,
                         const dgb_settings &s, double dx0)
{
    if (s.use_old_timestep)
        return s.old_timescale_factor * dx0;
    double v1 = 0.25 / nu;
    double t1 = fabs(h + (1 - 2 * h) * 0.5) * 0.5 * (1 - 0.5);
    double t2 = fabs(h + (1 - 2 * h) * 0.25) * 0.25 * (1 - 0.25);
    double tm = t1;
    if (t2 > tm)
        tm = t2;
    double v3 = fabs(gamma) * 2 * tm;
    double mx = v1;
    if (msum > mx)
        mx = msum;
    if (v3 > mx)
        mx = v3;
    if (mx > 0)
        return s.timescale_factor / mx;
    return INFINITY;
}

// Python min(a, b): a unless b < a.
DGB_HD double pymin(double a, double b) { return (b < a) ? b : a; }

// Selection part of M (dadi/integration_shared.c:12-14).
DGB_HD double msel(double x, double gamma, double h)
{
    return gamma * 2 * (h + (1. - 2 * h) * x) * x * (1. - x);
}

// Table-row layout (see dadi_gb300.h).
DGB_HD int row_stride(int P) { return 3 + 3 * P + P * (P - 1); }
DGB_HD int row_nu(int P, int k) { return 2 + k; }
DGB_HD int row_gamma(int P, int k) { return 2 + P + k; }
DGB_HD int row_h(int P, int k) { return 2 + 2 * P + k; }
DGB_HD int row_beta(int P) { return 2 + 3 * P; }
DGB_HD int row_mig(int P, int k, int j)
{
    return 3 + 3 * P + k * (P - 1) + (j < k ? j : j - 1);
}

// Mutation mass added at the unit corner of population k: the value of
// dadi/Integration.py:70-122 with the common grid xx (x0, x1, x2 = xx[0..2]).
DGB_HD double inject_value(int P, double dt, double theta0, double x0,
                           double x1, double x2)
{
    double denom = x2 - x0;
    for (int j = 1; j < P; j++)
        denom = denom * x1;
    double num = dt / x1 * theta0 / 2;
    return num * (double)(1 << P) / denom;
}

// ------------------------------------------------------ per-axis vectors

// Per-grid constants of one axis held in shared memory.
struct GridVecs {
    double *x;    // xx[i]
    double *xv;   // x(1-x)
    double *dfac; // dfactor[i]
    double *xInt; // midpoints
    double *ih;   // 1/(2 dx[i])
    double *dx;   // dx[i]
};

// Per-step coefficient vectors of one axis (see the header comment).
struct AxisVecs {
    double *A1, *A0, *C1, *C0, *B0;
    // delj-trick path only: per-interval selection term, V[i]/(2dx),
    // V[i+1]/(2dx), VInt, and per-row dfactor
    double *G, *Pv, *Qv, *VI, *DF;
};

// Scalars of one axis for one step (written by one thread, read by all).
struct AxisScalars {
    double dt, nu, inv_nu, msum, gamma, h;
    double B1s, B1e; // W multipliers of b'_0 and b'_{L-1}
    double bcs, bce; // dt-scaled corner boundary terms (0 if not applied)
    double mig[DGB_MAX_DIM];
};

// Corner boundary terms of dadi/integration2D.c:67-70 (and the 3-D/4-D
// equivalents): M at x = xx[0] with every other coordinate 0, and at
// x = xx[L-1] with every other coordinate 1, summed in increasing axis order.
DGB_HD void corner_bc(int P, int axis, const double *mig, double nu, double gamma,
                      double h, double x0, double xl, double dx0, double dxl,
                      double dt, double &bcs, double &bce)
{
    double mf = 0, ml = 0;
    bool first = true;
    for (int k = 0; k < P; k++) {
        if (k == axis)
            continue;
        double tf = mig[k] * (0.0 - x0), tl = mig[k] * (1.0 - xl);
        mf = first ? tf : mf + tf;
        ml = first ? tl : ml + tl;
        first = false;
    }
    mf = first ? msel(x0, gamma, h) : mf + msel(x0, gamma, h);
    ml = first ? msel(xl, gamma, h) : ml + msel(xl, gamma, h);
    bcs = (mf <= 0) ? dt * ((0.5 / nu - mf) * 2. / dx0) : 0.0;
    bce = (ml >= 0) ? dt * (-(-0.5 / nu - ml) * 2. / dxl) : 0.0;
}

// Scalars of axis a for one step from a parameter row (called by one lane
// per axis so both axes cost one warp-wide instruction stream).
__device__ __forceinline__ void axis_scalars_2d(AxisScalars &s, int a, const double *row,
                                                const GridVecs &g, int L)
{
    double dt = row[0];
    s.dt = dt;
    s.nu = row[row_nu(2, a)];
    s.inv_nu = 1.0 / s.nu;
    s.gamma = row[row_gamma(2, a)];
    s.h = row[row_h(2, a)];
    double m = row[row_mig(2, a, 1 - a)];
    s.msum = m;
    s.mig[a] = 0;
    s.mig[1 - a] = m;
    s.B1s = 0.5 * (dt * g.dfac[0]);
    s.B1e = -0.5 * (dt * g.dfac[L - 1]);
    corner_bc(2, a, s.mig, s.nu, s.gamma, s.h, g.x[0], g.x[L - 1], g.dx[0], g.dx[L - 2], dt,
              s.bcs, s.bce);
}

// Pitch of a density of L x L points in shared memory.
__host__ __device__ inline int odd_pitch(int L) { return (L % 2) ? L : L + 1; }

// Barrier of n threads of a CTA.
__device__ __forceinline__ void bar_group(int id, int n)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// ------------------------------------------- the delj path's exact operations

__device__ __forceinline__ double xm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double xa(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double xs(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double xd(double a, double b) { return div_full(a, b); }
// xm on the integer pipes (b of ordinary size), for products that no chain
// waits for.
__device__ __forceinline__ double xmi(double a, double b) { return mul_full<true>(a, b); }

// Selection part of Mfunc (dadi/integration_shared.c:12-14) in the
// reference's order: gamma * 2*(h + (1.-2*h)*x) * x*(1.-x).
__device__ __forceinline__ double msel_ref(double x, double gamma, double h)
{
    return xm(xm(xm(xm(gamma, 2.0), xa(h, xm(xs(1.0, xm(2.0, h)), x))), x), xs(1.0, x));
}

// Vfunc (dadi/integration_shared.c:4-6), or Vfunc_beta (:8-10) when beta > 0
// (one population): 1./nu * x*(1.-x) [* pow(beta+1, 2)/(4*beta)].
__device__ __forceinline__ double vfunc_ref(double x, double nu, double beta)
{
    double v = xm(xm(xd(1.0, nu), x), xs(1.0, x));
    if (beta > 0) {
        const double b1 = xa(beta, 1.0);
        v = xd(xm(v, xm(b1, b1)), xm(4.0, beta));
    }
    return v;
}

// Entry i of one axis for the default delta_j (see the header comment): the
// affine coefficients of row i and its interior diagonal.  vscale multiplies V
// (the breeding-ratio factor of Vfunc_beta in 1-D, 1 otherwise).
struct AxisEntry {
    double A1, A0, C1, C0, B0;
};

__device__ __forceinline__ AxisEntry axis_entry(int i, int L, const GridVecs &g,
                                                const AxisScalars &s, double vscale)
{
    const double iv = s.inv_nu * vscale;
    auto Gk = [&](int k) { return msel(g.xInt[k], s.gamma, s.h) - s.msum * g.xInt[k]; };
    const double dfi = s.dt * g.dfac[i];
    AxisEntry e = {0, 0, 0, 0, 0};
    double p_i = 0, q_im1 = 0;
    if (i < L - 1) {
        double G = Gk(i);
        double P = iv * g.xv[i] * g.ih[i];
        double Q = iv * g.xv[i + 1] * g.ih[i];
        p_i = fma(0.5, G, P);
        e.C1 = 0.5 * dfi;
        e.C0 = -dfi * fma(-0.5, G, Q);
    }
    if (i > 0) {
        double G = Gk(i - 1);
        double P = iv * g.xv[i - 1] * g.ih[i - 1];
        double Q = iv * g.xv[i] * g.ih[i - 1];
        q_im1 = fma(-0.5, G, Q);
        e.A1 = -0.5 * dfi;
        e.A0 = -dfi * fma(0.5, G, P);
    }
    e.B0 = fma(dfi, p_i + q_im1, 1.0);
    return e;
}

// Build entry i of the per-step vectors of one axis (called for i = 0..L-1
// by different threads).  beta1 is the breeding ratio itself for one
// population and 0 otherwise (the delj path evaluates Vfunc_beta as written).
__device__ __forceinline__ void build_axis_entry(int i, int L, const GridVecs &g,
                                                 const AxisScalars &s, double vscale,
                                                 bool delj, AxisVecs &v, double beta1 = 0.0)
{
    const AxisEntry e = axis_entry(i, L, g, s, vscale);
    v.A1[i] = e.A1;
    v.A0[i] = e.A0;
    v.C1[i] = e.C1;
    v.C0[i] = e.C0;
    v.B0[i] = e.B0;
    if (delj) {
        // the delj path rebuilds MInt per point in the reference order; per
        // interval it needs the selection term, V[i]/(2 dx[i]),
        // V[i+1]/(2 dx[i]) and VInt (dadi/integration2D.c:42-49,
        // integration_shared.c:72-93), each rounded as the reference does
        if (i < L - 1) {
            const double d2 = xm(2.0, g.dx[i]);
            v.G[i] = msel_ref(g.xInt[i], s.gamma, s.h);
            v.Pv[i] = xd(vfunc_ref(g.x[i], s.nu, beta1), d2);
            v.Qv[i] = xd(vfunc_ref(g.x[i + 1], s.nu, beta1), d2);
            v.VI[i] = vfunc_ref(g.xInt[i], s.nu, beta1);
        }
        v.DF[i] = g.dfac[i]; // unscaled: the delj rows are the reference's
    }
}

// ------------------------------------------------------------ line solvers

// Back substitution u_i = u'_i - gam_{i+1} u_{i+1} for i = L-2..0, where
// u holds u_{L-1}.  The gam and u' of 16 rows are loaded before their
// dependent FMA chain runs, so scratch that lives in global memory (L2) does
// not stall the chain on every row.
template <typename TP, typename TG>
__device__ __forceinline__ void back_substitute(TP *__restrict__ ph, int sp,
                                                TG *__restrict__ gm, int gs, int L, double u)
{
    constexpr int B = 16;
    int i = L - 2;
    for (; i >= B - 1; i -= B) {
        double gv[B], pv[B];
#pragma unroll
        for (int k = 0; k < B; k++) {
            gv[k] = gm[(i - k + 1) * gs];
            pv[k] = ph[(i - k) * sp];
        }
#pragma unroll
        for (int k = 0; k < B; k++) {
            u = fma(-gv[k], u, pv[k]);
            ph[(i - k) * sp] = u;
        }
    }
    for (; i >= 0; i--) {
        u = fma(-(double)gm[(i + 1) * gs], u, ph[i * sp]);
        ph[i * sp] = u;
    }
}

// Thomas solve of one line, delta_j = 0.5.  Element p of the line is
// ph[p*sp]; gam scratch element p is gm[p*gs].  W is the line's migration
// weight, bs/be the corner boundary terms for this line (0 if none).
// FP64: the pivots on the FP64 pipe (the same bits), for lines in global memory
// on full SMs, where the rare call of the integer ones would hold up the loads.
template <bool FP64 = false, typename TP, typename TG>
__device__ __forceinline__ void solve_line(TP *__restrict__ ph, int sp, TG *__restrict__ gm,
                                           int gs, int L, double W, double bs, double be,
                                           const AxisVecs &v, const AxisScalars &s)
{
    double u, g, none;
    pivot_as<FP64>(fma(W, s.B1s, v.B0[0]) + bs, ph[0], fma(W, v.C1[0], v.C0[0]), u, g);
    ph[0] = u;
    gm[gs] = g;
    // row i's coefficients and right-hand side are formed while row i - 1's
    // pivot is still in the integer pipes
    double a = fma(W, v.A1[1], v.A0[1]), c = fma(W, v.C1[1], v.C0[1]);
    double b0 = v.B0[1], p = ph[sp];
    for (int i = 1; i < L - 1; i++) {
        const double bet = fma(-a, g, b0), t = fma(-a, u, p), ci = c;
        a = fma(W, v.A1[i + 1], v.A0[i + 1]);
        c = fma(W, v.C1[i + 1], v.C0[i + 1]);
        b0 = v.B0[i + 1];
        p = ph[(i + 1) * sp];
        pivot_as<FP64>(bet, t, ci, u, g);
        ph[i * sp] = u;
        gm[(i + 1) * gs] = g;
    }
    pivot_as<FP64>(fma(-a, g, fma(W, s.B1e, b0) + be), fma(-a, u, p), 1.0, u, none);
    ph[(L - 1) * sp] = u;
    back_substitute(ph, sp, gm, gs, L, u);
}

// Chang-Cooper delta_j (dadi/integration_shared.c:52-70) for one interval,
// in the reference's order.
__device__ __forceinline__ double delj_of(double MInt, double VInt, double dx)
{
    const double wj = xmi(MInt, 2.0 * dx); // (2 MInt) dx: doubling is exact
    const double epsj = exp(xd(wj, VInt));
    // epsj != 1.0 && wj != 0 (not on the FP64 pipe, which a comparison takes
    // longer than a fused multiply-add)
    if (__double_as_longlong(epsj) != 0x3ff0000000000000ll && __double_as_longlong(wj) << 1 != 0)
    {
        const double ew = xmi(wj, epsj);
        return xd(xs(xa(-ew, xmi(VInt, epsj)), VInt), xs(wj, ew));
    }
    return 0.5;
}

// Thomas solve of one line with the delj trick, as the reference computes
// it: MInt per interval as Mfunc{1..5}D (dadi/integration_shared.c:12-30:
// the migration terms m_k (o_k - x) summed in increasing axis order, then
// the selection term), delta_j, the unscaled rows of compute_abc_nobc
// (:72-93, b = 1/dt + ...), the corner terms of dadi/integration2D.c:67-70
// when c0 / c1 (this line's other coordinates are all 0 / all 1; always in
// one dimension, integration1D.c:47-51), r = phi/dt, and tridiag_premalloc
// (dadi/tridiag.c:14-34).  The gam scratch holds element p at gm[p*gs].
template <typename TP, typename TG>
__device__ __forceinline__ void solve_line_delj(TP *__restrict__ ph, int sp, TG *__restrict__ gm,
                                                int gs, int L, const double *mo,
                                                const double *oo, int nother, bool c0, bool c1,
                                                const GridVecs &gv, const AxisVecs &v,
                                                const AxisScalars &s)
{
    auto mfun = [&](double x, double sel) {
        if (nother == 0)
            return sel;
        double acc = xm(mo[0], xs(oo[0], x));
        for (int j = 1; j < nother; j++)
            acc = xa(acc, xm(mo[j], xs(oo[j], x)));
        return xa(acc, sel);
    };
    const double dt = s.dt;
    const double idt = xd(1.0, dt);
    // interval 0: atemp, ctemp (compute_abc_nobc)
    double Mk = mfun(gv.xInt[0], v.G[0]);
    double d = delj_of(Mk, v.VI[0], gv.dx[0]);
    double at = xa(xm(Mk, d), v.Pv[0]);
    double ct = xa(xm(-Mk, xs(1.0, d)), v.Qv[0]);
    double b = xa(idt, xm(v.DF[0], at));
    if (c0) {
        const double mf = mfun(gv.x[0], msel_ref(gv.x[0], s.gamma, s.h));
        if (mf <= 0)
            b = xa(b, xd(xm(xs(xd(0.5, s.nu), mf), 2.0), gv.dx[0]));
    }
    double bet = b;
    double u = xd(xd((double)ph[0], dt), bet);
    ph[0] = u;
    double cprev = -xm(v.DF[0], ct);
    for (int i = 1; i < L; i++) {
        const double a = -xm(v.DF[i], at);
        double bb = xa(idt, xm(v.DF[i], ct));
        double cnext = 0;
        if (i < L - 1) {
            Mk = mfun(gv.xInt[i], v.G[i]);
            d = delj_of(Mk, v.VI[i], gv.dx[i]);
            at = xa(xm(Mk, d), v.Pv[i]);
            ct = xa(xm(-Mk, xs(1.0, d)), v.Qv[i]);
            bb = xa(bb, xm(v.DF[i], at));
            cnext = -xm(v.DF[i], ct);
        } else if (c1) {
            const double ml = mfun(gv.x[L - 1], msel_ref(gv.x[L - 1], s.gamma, s.h));
            if (ml >= 0)
                bb = xa(bb, xd(xm(-xs(-xd(0.5, s.nu), ml), 2.0), gv.dx[L - 2]));
        }
        const double g = xd(cprev, bet);
        gm[i * gs] = g;
        bet = xs(bb, xm(a, g));
        u = xd(xs(xd((double)ph[i * sp], dt), xm(a, u)), bet);
        ph[i * sp] = u;
        cprev = cnext;
    }
    for (int i = L - 2; i >= 0; i--) {
        u = xs((double)ph[i * sp], xm((double)gm[(i + 1) * gs], u));
        ph[i * sp] = u;
    }
}

} // namespace dgb
