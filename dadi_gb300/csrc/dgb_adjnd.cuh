// The transposed per-axis sweep of the N-dimensional adjoint and its
// contraction with the derivatives of the sweep's matrix (the method is
// described in dgb_adjointnd.cu): shared by the one-integration kernel there
// and the batched one in dgb_batchnd.cu.
#pragma once
#include "dgb_nd.cuh"

namespace dgb {

// A line's contraction is summed in ADN_RUNS runs of intervals, and 32 lines
// make one partial row.  The contraction is bound by one warp's FP64 issue
// (13 instructions per interval, 64 cycles apart), so a tile is 32 lines with
// ADN_RUNS threads each: one warp solves, four contract, and a lone grid of 40
// points has 50 CTAs.  Against one thread per line on tiles of 64-128 lines, a
// step backwards of the three-population growth model (two recomputing sweeps
// and three of these) takes 163 us instead of 236 for one set at 40 points,
// 173 instead of 237 for six, 298 instead of 394 for one at 80 points, 355
// instead of 407 for four at 70, and 1749 instead of 1703 for 24 at 80.  Loads
// of u and r four points ahead change nothing here.
constexpr int ADN_RUNS = 4;

inline long adn_rows(long nlines) { return (nlines + 31) / 32; }

// This axis' entries of the row: dt, nu, gamma, h, then the migration rates
// into it in ascending order.
constexpr int ADN_NG = 4 + DGB_MAX_DIM - 1;

struct ADNArgs {
    NDArgs nd;          // lam as nd.phi; axis, strides, table row
    const double *out;  // this sweep's forward output s_j
    const double *rhs;  // this sweep's forward input s_{j-1} (psi without injection)
    double *gpart;      // per 32 lines: row_stride(P) doubles
    const double *coef; // coefficient records of the chunk from step0 (null: build inline)
    long step0;
    long rec_off;       // offset of this integration's records after the grid constants
};

// Shared memory of an adjoint sweep CTA of nt lines: the forward sweep's
// (tile, gam unless it sits in a workspace slice, grid constants, vectors), the
// transposed vectors and four per-interval contraction factors; at the end the
// sums of the runs, in the same place.
__host__ __device__ inline size_t adn_smem_doubles(int L, int nt, bool gsmem = true)
{
    const size_t lines = (size_t)L * (nt + 1) + (gsmem ? (size_t)L * nt : 0) + 20 * (size_t)L;
    const size_t sums = (size_t)(ADN_RUNS - 1) * ADN_NG * 32;
    return lines > sums ? lines : sums;
}

// Whether an adjoint sweep takes lines of L points: what a tile of the forward
// sweep's lines (nd_threads) would leave of shared memory decides, though
// tiles of 32 lines need less.
static bool adn_fits(int L, long nlines, bool gsmem)
{
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) !=
            cudaSuccess)
        return false;
    return adn_smem_doubles(L, nd_threads(L, nlines), gsmem) * sizeof(double) +
               sizeof(NDShared) + 2432 <=
           (size_t)optin;
}

// Whether a launch over `tiles` tiles of 32 lines gives each line one thread,
// which takes the runs in turn (the same sums in the same order), on tiles of
// 128 lines: from eight tiles per SM on, if lines of 48 points or fewer let an
// SM hold four such CTAs (16 solving warps, where 32-line tiles give six).
// 32 sets at 40 points: 373 us a step backwards, 425 with ADN_RUNS threads;
// on tiles of 64 lines 24 sets at 80 points take 1807 and 1794.
static bool adn_wide(int L, long tiles)
{
    int dev = 0, sms = 152;
    if (cudaGetDevice(&dev) == cudaSuccess)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return L <= 48 && tiles >= 8L * sms;
}

// The transposed sweep and contraction of the 32 * WL lines from
// tile_idx * 32 * WL of one integration, SG (1 or ADN_RUNS) threads per line:
// the body of k_adjoint_sweep_nd and of the batched k_adjoint_sweep_batch.
// Called by the whole CTA of 32 * WL * SG threads; red is shared.
template <int WL, int SG>
__device__ __forceinline__ void adn_tile(const ADNArgs &A, long tile_idx, double *smem,
                                         NDShared &Sh, double (*red)[ADN_NG],
                                         double *gam_slice = nullptr)
{
    static_assert(SG == 1 || (SG == ADN_RUNS && WL == 1), "");
    constexpr int nt = 32 * WL, bt = nt * SG;
    const NDArgs &N = A.nd;
    const int L = N.L, P = N.ndim, ax = N.axis, tid = threadIdx.x;
    const int ln = tid % nt, seg = tid / nt;
    const int stride = row_stride(P);
    double *tile, *gam;
    GridVecs g;
    AxisVecs v, vt;
    if (gam_slice) {
        // the Thomas scratch in this CTA's workspace slice: the shared
        // memory holds the tile and the vectors only
        tile = smem;
        gam = gam_slice;
        double *q = smem + (size_t)L * (nt + 1);
        g.x = q; q += L;
        g.xv = q; q += L;
        g.dfac = q; q += L;
        g.xInt = q; q += L;
        g.ih = q; q += L;
        g.dx = q; q += L;
        nd_vecs_at(q, L, false, v);
    } else {
        nd_carve(smem, L, nt, false, tile, gam, g, v);
    }
    double *p = v.B0 + L;
    vt.A1 = p; p += L;
    vt.A0 = p; p += L;
    vt.C1 = p; p += L;
    vt.C0 = p; p += L;
    vt.B0 = p; p += L;
    // per interval i, for the contraction below: cP, cQ (the nu terms), gS,
    // hS (the selection terms' gamma and h factors)
    double *cP = p, *cQ = p + L, *gS = p + 2 * L, *hS = p + 3 * L;
    if (A.coef) {
        // the grid constants and this step's record, in the carve order
        const double *rec = A.coef + nd_grid_doubles(L) + A.rec_off +
                            ((size_t)(N.step - A.step0) * P + ax) * nd_rec_doubles(L, false);
        constexpr int NS = (int)(sizeof(AxisScalars) / sizeof(double));
        double *sp = reinterpret_cast<double *>(&Sh.s);
        for (int i = tid; i < nd_grid_doubles(L); i += bt)
            g.x[i] = A.coef[i];
        for (int i = tid; i < 5 * L; i += bt)
            v.A1[i] = rec[ND_HEAD + i];
        for (int i = tid; i < ND_HEAD; i += bt) {
            if (i < NS)
                sp[i] = rec[i];
            else
                Sh.inj[i - NS] = rec[i];
        }
    } else {
        nd_grid_consts(N, g);
        if (tid == 0)
            nd_load_params(N, Sh, g);
        __syncthreads();
        for (int i = tid; i < L; i += bt)
            build_axis_entry(i, L, g, Sh.s, Sh.vscale, false, v);
    }
    __syncthreads();
    for (int i = tid; i < L; i += bt) {
        vt.A1[i] = (i > 0) ? v.C1[i - 1] : 0.0;
        vt.A0[i] = (i > 0) ? v.C0[i - 1] : 0.0;
        vt.C1[i] = (i < L - 1) ? v.A1[i + 1] : 0.0;
        vt.C0[i] = (i < L - 1) ? v.A0[i + 1] : 0.0;
        vt.B0[i] = v.B0[i];
        if (i < L - 1) {
            // with w = D_i (u_i + u_{i+1}) (twice D_i times the mean density):
            // d/dnu: D_i (Q_i u_{i+1} - P_i u_i) / nu = D_i (cQ u_{i+1} - cP u_i);
            // d/dgamma, d/dh of the selection term times D_i hp: w gS, w hS
            const double inu = Sh.s.inv_nu, hh = Sh.s.h, gm = Sh.s.gamma;
            const double xi = g.xInt[i], xx1 = xi * (1. - xi);
            cP[i] = inu * inu * g.xv[i] * g.ih[i];
            cQ[i] = inu * inu * g.xv[i + 1] * g.ih[i];
            gS[i] = (hh + (1. - 2 * hh) * xi) * xx1;
            hS[i] = gm * (1. - 2 * xi) * xx1;
        }
    }
    const long l0 = tile_idx * nt;
    const int n = (int)min((long)nt, N.nlines - l0);
    nd_tile_io<SG>(N, tile, nt, l0, n, false);
    __syncthreads();
    const int j0 = (g.x[0] == 0.0) ? 0 : -1;
    const int j1 = (g.x[L - 1] == 1.0) ? L - 1 : -1;
    const AxisScalars &s = Sh.s;
    const int ng = 4 + P - 1;
    double G[ADN_NG] = {};
    const int tp = nt + 1;
    long base = 0;
    double W = 0, oo[DGB_MAX_DIM], bs = 0, be = 0;
    int n1 = 0, k1 = -1;
    if (ln < n) {
        int coord[DGB_MAX_DIM];
        base = nd_line_base(N, l0 + ln, coord);
        bool all0 = true, all1 = true;
        for (int k = 0; k < P; k++) {
            oo[k] = g.x[coord[k]];
            if (k == ax)
                continue;
            W = fma(s.mig[k], g.x[coord[k]], W);
            all0 = all0 && coord[k] == j0;
            all1 = all1 && coord[k] == j1;
            if (coord[k] == 1) {
                n1++;
                k1 = k;
            } else if (coord[k] != 0) {
                n1 = 99;
            }
        }
        if (P == 1)
            all0 = all1 = true;
        bs = all0 ? s.bcs : 0.0;
        be = all1 ? s.bce : 0.0;
        // mu = X^{-T} lambda on this line, in place in the tile
        if (seg == 0)
            solve_line(tile + ln, tp, gam + ln, nt, L, W, bs, be, vt, s);
    }
    __syncthreads();
    if (ln < n) {
        const double *mu = tile + ln;
        // contraction with u (forward output) and r (forward input)
        const double *u = A.out + base, *rhs = A.rhs + base;
        const long S = N.S;
        const double dt = s.dt, inu = s.inv_nu, gm = s.gamma, hh = s.h;
        const double inj0 = (n1 == 1 && k1 >= 0) ? Sh.inj[k1] : 0.0; // point 0 of this line
        const double inj1 = (n1 == 0) ? Sh.inj[ax] : 0.0;             // point 1 of this line
        // the corner terms, which few lines have (a branch of the warp's: FP64
        // instructions switched off for a lane would cost the same)
        double bnu = 0, bg = 0, bh = 0, bmf = 0, bml = 0;
        if (seg == 0 && __any_sync(__activemask(), bs != 0.0 || be != 0.0)) {
            if (bs != 0.0) {
                const double x0 = g.x[0], f = dt * 2. / g.dx[0], w = mu[0] * u[0];
                bnu += w * f * (-0.5 * inu * inu);
                bmf = w * f * x0;
                bg -= w * f * (2 * (hh + (1. - 2 * hh) * x0) * x0 * (1. - x0));
                bh -= w * f * (gm * 2 * (1. - 2 * x0) * x0 * (1. - x0));
            }
            if (be != 0.0) {
                const double xl = g.x[L - 1], f = dt * 2. / g.dx[L - 2];
                const double w = mu[(L - 1) * tp] * u[(L - 1) * S];
                bnu += w * f * (-0.5 * inu * inu);
                bml = w * f * (1. - xl);
                bg += w * f * (2 * (hh + (1. - 2 * hh) * xl) * xl * (1. - xl));
                bh += w * f * (gm * 2 * (1. - 2 * xl) * xl * (1. - xl));
            }
        }
        const int run = (L + ADN_RUNS - 1) / ADN_RUNS;
        for (int r0 = seg; r0 < ADN_RUNS; r0 += SG) {
            // the migration terms D_i (x_k - xInt_i) hp of every other population
            // k from two sums: s1 = sum w, s2 = sum w xInt_i
            double smr = 0, smp = 0, snu = 0, sg = 0, sh = 0, s1 = 0, s2 = 0;
            // the points [i0, i1) of the line, and the intervals from them
            const int i0 = min(r0 * run, L), i1 = min(i0 + run, L), ib = min(i0, L - 1);
            double mi = mu[ib * tp], ui = u[ib * S];
            double dmi = g.dfac[ib] * mi;
            for (int i = i0; i < i1; i++) {
                double ri = rhs[i * S];
                if (i == 0)
                    ri += inj0;
                if (i == 1)
                    ri += inj1;
                smr = fma(mi, ri, smr);
                smp = fma(mi, ui, smp);
                if (i < L - 1) {
                    const double mn = mu[(i + 1) * tp], un = u[(i + 1) * S];
                    const double dmn = g.dfac[i + 1] * mn;
                    const double Di = dmi - dmn;
                    const double w = Di * (ui + un);
                    snu = fma(Di, fma(-cP[i], ui, cQ[i] * un), snu);
                    s1 += w;
                    s2 = fma(w, g.xInt[i], s2);
                    sg = fma(w, gS[i], sg);
                    sh = fma(w, hS[i], sh);
                    mi = mn;
                    ui = un;
                    dmi = dmn;
                }
            }
            const bool corner = r0 == 0;
            double Q[ADN_NG] = {smp - smr, -fma(dt, snu, corner ? bnu : 0.0),
                                -fma(dt, sg, corner ? bg : 0.0), -fma(dt, sh, corner ? bh : 0.0)};
#pragma unroll
            for (int k = 0; k < DGB_MAX_DIM; k++)
                if (k < P && k != ax) {
                    const double m = -fma(0.5 * dt, fma(oo[k], s1, -s2), corner ? bmf + bml : 0.0);
#pragma unroll
                    for (int e = 4; e < ADN_NG; e++)
                        if (e == 4 + k - (k > ax))
                            Q[e] = m;
                }
#pragma unroll
            for (int q = 0; q < ADN_NG; q++)
                G[q] = (SG > 1 || r0 == 0) ? Q[q] : G[q] + Q[q];
        }
    }
    nd_tile_io<SG>(N, tile, nt, l0, n, true);
    // fixed-order sums of G: the runs of each line (in the tile's place), then
    // the 32 lines of a warp
    if (SG > 1) {
        __syncthreads();
        if (seg > 0)
            for (int q = 0; q < ng; q++)
                smem[((seg - 1) * ADN_NG + q) * nt + ln] = G[q];
        __syncthreads();
        if (seg > 0)
            return;
    }
    const int lw = ln >> 5, lane = ln & 31;
#pragma unroll
    for (int q = 0; q < ADN_NG; q++) {
        if (q >= ng)
            break;
        double x = G[q];
        for (int r = 0; r < SG - 1; r++)
            x += smem[(r * ADN_NG + q) * nt + ln];
        for (int off = 16; off > 0; off >>= 1)
            x += __shfl_down_sync(0xffffffffu, x, off);
        if (lane == 0)
            red[lw][q] = q ? x : x / s.dt;
    }
    __syncwarp();
    const long at = tile_idx * WL + lw;
    if (at * 32 >= N.nlines)
        return;
    double *row = A.gpart + (size_t)at * stride;
    for (int q = lane; q < stride; q += 32) {
        double x = 0;
        if (q == 0)
            x = red[lw][0];
        else if (q == row_nu(P, ax))
            x = red[lw][1];
        else if (q == row_gamma(P, ax))
            x = red[lw][2];
        else if (q == row_h(P, ax))
            x = red[lw][3];
        else
            for (int k = 0; k < P; k++)
                if (k != ax && q == row_mig(P, ax, k))
                    x = red[lw][4 + k - (k > ax)];
        row[q] = x;
    }
}

// The injection's part of dJ/d(dt) and dJ/d(theta0) for one step (one
// thread): lambda (the adjoint at the start of the step) at the injected
// points times d(injected amount)/d(dt, theta0).
__device__ __forceinline__ void adn_inject_terms(const double *lam, const double *xx,
                                                 const double *row, int P, int L, int active,
                                                 double *gout)
{
    double lin = 0;
    for (int k = 0; k < P; k++) {
        if (!(active >> k & 1))
            continue;
        long idx = 0;
        for (int j = 0; j < P; j++)
            idx = idx * L + (j == k ? 1 : 0);
        lin += lam[idx];
    }
    const double dt = row[0], th = row[1];
    gout[0] = lin * inject_value(P, 1.0, th, xx[0], xx[1], xx[2]);
    gout[1] = lin * inject_value(P, dt, 1.0, xx[0], xx[1], xx[2]);
}

} // namespace dgb
