// A Thomas sweep's factors and its solve apart, for kernels that run them on
// different warps: the factors (a, 1/bet, g of every row of a line) follow from
// the coefficient vectors alone, the solve takes them from global memory (L2).
// Used by the forward integration (dgb_integrate2d.cu) and by the adjoint's
// backward walk (dgb_adjoint2d.cu); per line the arithmetic is solve_line's.
#pragma once

#include "dgb_common.cuh"

namespace dgb {

constexpr int K2W_STEPS = 16; // steps whose scalars are formed at once

// Workspace of one CTA: [axis][inv, g, a][row][line] (keep_a), lines padded to
// 128 bytes.
__host__ __device__ inline int k2w_pitch(int L) { return (L + 15) / 16 * 16; }

__host__ __device__ inline size_t k2w_slice_doubles(int L, bool keep_a)
{
    return (size_t)(keep_a ? 6 : 4) * L * k2w_pitch(L);
}

// 1/bet and c * (1/bet).
__device__ __forceinline__ void pivot_inv(double bet, double c, double &inv, double &g)
{
    bool bad;
    const Mant y = rcp_mant(bet, bad);
    const unsigned exps = rcp_exps(bet);
    g = mul_mant(c, y, exps, bad);
    inv = mant_double(y, exps);
    if (bad) {
        inv = rcp_newton(bet);
        g = mul_fp64(c, inv);
    }
}

// The factors of one line: f[0][i] = 1/bet_i, f[1][i] = g_i and, where KEEP_A,
// f[2][i] = a_i; array k at f + k * stride, row i at i * LP.
template <bool KEEP_A>
__device__ __forceinline__ void k2w_factor(const AxisVecs &v, const AxisScalars &s, int L,
                                           double W, double bs, double be, double *f,
                                           size_t stride, int LP)
{
    double *fi = f, *fg = f + stride, *fa = f + 2 * stride;
    double inv, g;
    pivot_inv(fma(W, s.B1s, v.B0[0]) + bs, fma(W, v.C1[0], v.C0[0]), inv, g);
    fi[0] = inv;
    fg[0] = g;
    double a = fma(W, v.A1[1], v.A0[1]), c = fma(W, v.C1[1], v.C0[1]), b0 = v.B0[1];
    for (int i = 1; i < L - 1; i++) {
        const double bet = fma(-a, g, b0), ai = a, ci = c;
        a = fma(W, v.A1[i + 1], v.A0[i + 1]);
        c = fma(W, v.C1[i + 1], v.C0[i + 1]);
        b0 = v.B0[i + 1];
        pivot_inv(bet, ci, inv, g);
        if (KEEP_A)
            fa[i * LP] = ai;
        fi[i * LP] = inv;
        fg[i * LP] = g;
    }
    if (KEEP_A)
        fa[(L - 1) * LP] = a;
    fi[(L - 1) * LP] = rcp_full(fma(-a, g, fma(W, s.B1e, b0) + be));
}

// The solve of one line from its factors (as k2w_factor leaves them); element
// p at src[p * sp], the result at ph[p * sp] (which may be src).  The factors of the next rows are loaded ahead of the rows
// that use them.
template <bool KEEP_A>
__device__ __forceinline__ void k2w_solve(const double *src, double *ph, int sp, int L,
                                          const AxisVecs &v, double W,
                                          const double *__restrict__ f, size_t stride, int LP)
{
    constexpr int B = 4, C = 8;
    const double *fi = f, *fg = f + stride, *fa = f + 2 * stride;
    double av[B], iv[B], gv[C];
#pragma unroll
    for (int k = 0; k < B; k++) {
        const int r = min(1 + k, L - 1);
        iv[k] = __ldcg(fi + r * LP);
        if (KEEP_A)
            av[k] = __ldcg(fa + r * LP);
    }
    double u = mul_full(src[0], __ldcg(fi));
    ph[0] = u;
    int i = 1;
    for (; i + B <= L; i += B) {
        double an[B], in[B], pv[B];
#pragma unroll
        for (int k = 0; k < B; k++) {
            const int r = min(i + B + k, L - 1);
            in[k] = __ldcg(fi + r * LP);
            if (KEEP_A)
                an[k] = __ldcg(fa + r * LP);
            else
                av[k] = fma(W, v.A1[i + k], v.A0[i + k]);
            pv[k] = src[(i + k) * sp];
        }
#pragma unroll
        for (int k = 0; k < B; k++) {
            u = mul_full(fma(-av[k], u, pv[k]), iv[k]);
            ph[(i + k) * sp] = u;
        }
#pragma unroll
        for (int k = 0; k < B; k++) {
            if (KEEP_A)
                av[k] = an[k];
            iv[k] = in[k];
        }
    }
#pragma unroll
    for (int k = 0; k < C; k++)
        gv[k] = __ldcg(fg + max(L - 2 - k, 0) * LP);
#pragma unroll
    for (int k = 0; k < B - 1; k++)
        if (i + k < L) {
            const double a = KEEP_A ? av[k] : fma(W, v.A1[i + k], v.A0[i + k]);
            u = mul_full(fma(-a, u, src[(i + k) * sp]), iv[k]);
            ph[(i + k) * sp] = u;
        }
    i = L - 2;
    for (; i >= C - 1; i -= C) {
        double gn[C], pv[C];
#pragma unroll
        for (int k = 0; k < C; k++) {
            gn[k] = __ldcg(fg + max(i - C - k, 0) * LP);
            pv[k] = ph[(i - k) * sp];
        }
#pragma unroll
        for (int k = 0; k < C; k++) {
            u = fma(-gv[k], u, pv[k]);
            ph[(i - k) * sp] = u;
        }
#pragma unroll
        for (int k = 0; k < C; k++)
            gv[k] = gn[k];
    }
#pragma unroll
    for (int k = 0; k < C - 1; k++)
        if (i - k >= 0) {
            u = fma(-gv[k], u, ph[(i - k) * sp]);
            ph[(i - k) * sp] = u;
        }
}

} // namespace dgb
