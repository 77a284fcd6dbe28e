// Shared-memory-resident 2-D integrator and the batched 2-population engine.
//
// One CTA owns one (instance, grid) work item for its whole time loop: phi
// (L x L doubles, odd row pitch so both sweep directions are bank-conflict
// free) is loaded once into shared memory; every step injects mutations,
// rebuilds the per-axis coefficient vectors and runs the x sweep (lines are
// columns) and the y sweep (lines are rows) with one thread per line; phi is
// written back once at the end.  The Thomas gam scratch lives in shared
// memory when it fits next to phi, otherwise in a per-CTA slice of a global
// workspace (L2-resident).
//
// The integrator only reads per-step parameter rows (see dadi_gb300.h).  For
// the drop-in path the host evaluates them from Python callables; for the
// batched engine a separate pass (k_sched2d, one thread per instance, so the
// scalar pow/exp/divide chain of the schedule runs on full warps instead of
// serialising inside every integrating CTA) evaluates the parametric forms
// with the reference's operation order: one fill pass into room reserved
// from host bounds on the rows, or count rows, scan, fill rows.
// The batched integration is a persistent launch whose CTAs pull work items
// longest-first from an atomic counter (one launch over all grids, or one
// per grid size with a CTA shaped for it), or one CTA per item.  Under the
// default delta_j the factorisations of a sweep run on other warps than its
// solves (k_integrate2d_ws), under the delj trick its coefficients
// (k_integrate2d_delj), up to 159 points; k_integrate2d, one warp for both,
// serves an explicit CTA size, the scratch in shared memory, one CTA per item,
// larger grids, and callers without workspace.
//
// Reference: the time loop of Integration.two_pops (dadi/Integration.py:
// 340-386) with implicit_2Dx / implicit_2Dy (dadi/integration2D.c:19-160).
#include <algorithm>
#include <mutex>
#include <vector>

#include "dgb_common.cuh"
#include "dgb_internal.h"
#include "dgb_split.cuh"

namespace dgb {

constexpr int K2_THREADS = 128;
constexpr int K2_MAXG = DGB_B2_MAXG;
constexpr int K2_ROW = 11; // DGB_ROW_STRIDE(2)
constexpr int K2_AUTO_SHARED = -2; // dgb_settings.threads: as 0, beside other launches

struct K2Args {
    int ngrids;
    int L[K2_MAXG];
    long xx_off[K2_MAXG];
    long phi0_off[K2_MAXG];
    long out_off[K2_MAXG];
    const double *xx_all;
    const double *phi0_all; // null: phi_out holds the initial density
    double *phi_out;
    const double *table;   // parameter rows
    const long *row_off;   // first row of each schedule (null: one schedule at row 0)
    const int *row_cnt;    // rows of each schedule
    int fixed_cnt;         // rows of the single schedule when row_off is null
    int sched_per_grid;    // schedule index = inst*ngrids+g (1) or inst (0)
    const int *masks;      // per instance: frozen | nomut << 8 (null: use fixed)
    int frozen_mask, nomut_mask;
    const int *order;      // null: work id = position
    int nwork;
    int *counter;          // null: one item per CTA (blockIdx.x)
    int Lmax;
    int gam_smem;          // 1: gam in shared memory
    double *gam_glob;      // per-CTA slices of Lmax*Lmax doubles
    int use_delj;
    double *ckpt;          // optional: phi before every ckpt_every-th step
    const long *ckpt_off;  // first checkpoint double of each work id
    int ckpt_every;
    const dgb_item2d *items; // optional explicit work items (grid, slot, schedule each)
    int *live;               // k_integrate2d_ws, CHOSEN: CTAs per SM that run, then the
                             // number of CTAs started on each SM
};

struct K2Layout {
    int pitch;
    size_t total;
};

static K2Layout k2_layout(int Lmax, bool gam_smem, bool delj)
{
    K2Layout l;
    l.pitch = odd_pitch(Lmax);
    size_t d = (size_t)Lmax * l.pitch + (gam_smem ? (size_t)Lmax * Lmax : 0) + 6 * (size_t)Lmax +
               2 * (size_t)(delj ? 10 : 5) * Lmax;
    l.total = d * sizeof(double);
    return l;
}

struct K2Shared {
    AxisScalars ax[2];
    double inj;
    int item;
};

__device__ __forceinline__ void k2_carve(double *smem, int Lmax, int pitch, bool gam_smem,
                                         bool delj, double *&phi, double *&gam, GridVecs &g,
                                         AxisVecs (&v)[2])
{
    double *p = smem;
    phi = p;
    p += (size_t)Lmax * pitch;
    gam = nullptr;
    if (gam_smem) {
        gam = p;
        p += (size_t)Lmax * Lmax;
    }
    g.x = p; p += Lmax;
    g.xv = p; p += Lmax;
    g.dfac = p; p += Lmax;
    g.xInt = p; p += Lmax;
    g.ih = p; p += Lmax;
    g.dx = p; p += Lmax;
    for (int a = 0; a < 2; a++) {
        v[a].A1 = p; p += Lmax;
        v[a].A0 = p; p += Lmax;
        v[a].C1 = p; p += Lmax;
        v[a].C0 = p; p += Lmax;
        v[a].B0 = p; p += Lmax;
        if (delj) {
            v[a].G = p; p += Lmax;
            v[a].Pv = p; p += Lmax;
            v[a].Qv = p; p += Lmax;
            v[a].VI = p; p += Lmax;
            v[a].DF = p; p += Lmax;
        }
    }
}

// Work item wid of a launch.
struct K2Item {
    int wid, L, frozen, nomut, nsteps;
    const double *xx, *src, *rows;
    double *out;
};

__device__ __forceinline__ K2Item k2_item(const K2Args &A, int wid)
{
    K2Item I;
    int sidx;
    I.wid = wid;
    if (A.items) {
        // explicit item: its own grid, output slot (holding the initial
        // density) and schedule
        const dgb_item2d &it = A.items[wid];
        I.L = it.L;
        I.xx = A.xx_all + it.xx_off;
        I.out = A.phi_out + it.out_off;
        I.src = I.out;
        sidx = (int)it.sched;
        I.frozen = it.masks & 0xff;
        I.nomut = it.masks >> 8 & 0xff;
    } else {
        const int inst = wid / A.ngrids, gi = wid - inst * A.ngrids;
        I.L = A.L[gi];
        I.xx = A.xx_all + A.xx_off[gi];
        I.out = A.phi_out + A.out_off[gi] + (size_t)inst * I.L * I.L;
        I.src = A.phi0_all ? A.phi0_all + A.phi0_off[gi] : I.out;
        sidx = A.sched_per_grid ? wid : inst;
        I.frozen = A.masks ? (A.masks[inst] & 0xff) : A.frozen_mask;
        I.nomut = A.masks ? (A.masks[inst] >> 8 & 0xff) : A.nomut_mask;
    }
    I.rows = A.row_off ? A.table + A.row_off[sidx] * K2_ROW : A.table;
    I.nsteps = A.row_off ? A.row_cnt[sidx] : A.fixed_cnt;
    return I;
}

template <bool DELJ>
__global__ void __launch_bounds__(K2_THREADS) k_integrate2d(K2Args A)
{
    extern __shared__ __align__(16) double smem[];
    __shared__ K2Shared S;
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int nwarps = blockDim.x >> 5;
    const int pitch = odd_pitch(A.Lmax);
    double *phi, *gam_s;
    GridVecs g;
    AxisVecs v[2];
    k2_carve(smem, A.Lmax, pitch, A.gam_smem, DELJ, phi, gam_s, g, v);
    double *gam_g = A.gam_glob ? A.gam_glob + (size_t)blockIdx.x * A.Lmax * A.Lmax : nullptr;

    // S.item is written by thread 0 and read by all between the barrier that
    // follows the write and the next barrier thread 0 must pass to write again.
    for (int iter = 0;; iter++) {
        if (tid == 0)
            S.item = A.counter ? atomicAdd(A.counter, 1) : (iter == 0 ? (int)blockIdx.x : A.nwork);
        __syncthreads();
        const int w = S.item;
        if (w >= A.nwork)
            break;
        const int wid = A.order ? A.order[w] : w;
        const K2Item I = k2_item(A, wid);
        const int L = I.L, frozen = I.frozen, nomut = I.nomut, nsteps = I.nsteps;
        const double *xx = I.xx, *src = I.src, *rows = I.rows;
        double *out = I.out;

        // grid constants and initial density
        for (int i = tid; i < L; i += blockDim.x) {
            double x = xx[i];
            g.x[i] = x;
            g.xv[i] = x * (1. - x);
            if (i < L - 1) {
                double d = xx[i + 1] - x;
                g.dx[i] = d;
                g.ih[i] = 1.0 / (2 * d);
                g.xInt[i] = 0.5 * (xx[i + 1] + x);
            }
        }
        for (int idx = tid; idx < L * L; idx += blockDim.x) {
            int r = idx / L, c = idx - r * L;
            phi[r * pitch + c] = src[idx];
        }
        __syncthreads();
        for (int i = tid; i < L; i += blockDim.x) {
            if (i == 0)
                g.dfac[i] = 2. / g.dx[0];
            else if (i == L - 1)
                g.dfac[i] = 2. / g.dx[L - 2];
            else
                g.dfac[i] = 2. / (g.dx[i] + g.dx[i - 1]);
        }
        __syncthreads();
        // grid index of the corner lines (other coordinate exactly 0 / 1)
        const int j0 = (g.x[0] == 0.0) ? 0 : -1;
        const int j1 = (g.x[L - 1] == 1.0) ? L - 1 : -1;
        const int lpw = (L + nwarps - 1) / nwarps;

        for (int step = 0; step < nsteps; step++) {
            const double *row = rows + (size_t)step * K2_ROW;
            if (A.ckpt && step % A.ckpt_every == 0) {
                // checkpoint for the adjoint: phi before this step, row-major
                double *c = A.ckpt + A.ckpt_off[wid] + (size_t)(step / A.ckpt_every) * L * L;
                for (int idx = tid; idx < L * L; idx += blockDim.x) {
                    int r = idx / L, q = idx - r * L;
                    c[idx] = phi[r * pitch + q];
                }
            }
            // ---- step scalars: lane a of warp 0 handles axis a, lane 2 the injection
            if (warp == 0) {
                if (lane < 2)
                    axis_scalars_2d(S.ax[lane], lane, row, g, L);
                else if (lane == 2)
                    S.inj = inject_value(2, row[0], row[1], g.x[0], g.x[1], g.x[2]);
            }
            __syncthreads();
            // ---- per-axis vectors (both axes) and mutation injection
            for (int t = tid; t < 2 * L; t += blockDim.x) {
                int a = t >= L, i = t - a * L;
                build_axis_entry(i, L, g, S.ax[a], 1.0, DELJ, v[a]);
            }
            if (tid == 0) {
                if (!(frozen & 1) && !(nomut & 1))
                    phi[1 * pitch + 0] += S.inj;
                if (!(frozen & 2) && !(nomut & 2))
                    phi[0 * pitch + 1] += S.inj;
            }
            __syncthreads();
            // ---- x sweep (axis 0): line = column j, element i at phi[i*pitch + j]
            // ---- y sweep (axis 1): line = row i, element j at phi[i*pitch + j]
            for (int a = 0; a < 2; a++) {
                if (frozen & (1 << a))
                    continue;
                const AxisScalars &s = S.ax[a];
                const int sp = (a == 0) ? pitch : 1;
                const int sl = (a == 0) ? 1 : pitch;
                const double mo = s.mig[1 - a];
                for (int k = lane; k < lpw; k += 32) {
                    int line = warp * lpw + k;
                    if (line >= L)
                        break;
                    double W = mo * g.x[line];
                    double bs = (line == j0) ? s.bcs : 0.0;
                    double be = (line == j1) ? s.bce : 0.0;
                    double *ph = phi + (size_t)line * sl;
                    if (A.gam_smem) {
                        double *gm = gam_s + line;
                        if (DELJ)
                            solve_line_delj(ph, sp, gm, L, L, &s.mig[1 - a], &g.x[line], 1,
                                            line == j0, line == j1, g, v[a], s);
                        else
                            solve_line(ph, sp, gm, L, L, W, bs, be, v[a], s);
                    } else {
                        double *gm = gam_g + line;
                        if (DELJ)
                            solve_line_delj(ph, sp, gm, L, L, &s.mig[1 - a], &g.x[line], 1,
                                            line == j0, line == j1, g, v[a], s);
                        else
                            solve_line(ph, sp, gm, L, L, W, bs, be, v[a], s);
                    }
                }
                __syncthreads();
            }
        }
        for (int idx = tid; idx < L * L; idx += blockDim.x) {
            int r = idx / L, c = idx - r * L;
            out[idx] = phi[r * pitch + c];
        }
        __syncthreads();
    }
}

// ------------------------------------- factors and solves on their own warps

// k_integrate2d with each sweep's factorisation on other warps than its
// solves.  Of a line's Thomas recurrence only t = phi - a u, u = t inv and
// the back substitution need the density; the pivots, their reciprocals inv
// and the couplings g = c inv follow from the parameter row alone.  So while
// the solve warps (one line per lane) run a sweep, as many factor warps form
// a, inv and g of the next one and hand them over through the workspace (one
// set per axis, in L2), with one barrier per sweep.  Per grid point the chain
// of the solve is a fused multiply-add, a product on the integer pipes and a
// back substitution, and the chain of the factors a fused multiply-add, a
// reciprocal and a product, where the fused sweep's warps run one after the
// other.  The arithmetic per line is solve_line's, so the results are bitwise
// the same.  Measured, microseconds per step with one warp for both / with
// this kernel: one grid alone, L = 31 25 / 14, 64 45 / 25, 100 69 / 45, 128
// 83 / 56, 133 (two rounds of lines on four warps / five warps) 168 / 72; 8
// grids per SM, per grid and SM, L = 45 18.6 / 11.6, 80 30 / 24, 90 38 / 30,
// 100 42 / 43, 133 169 / 81.
constexpr int K2W_MAXWARPS = 5; // of lines

struct K2WShared {
    AxisScalars ax[2 * K2W_STEPS][2]; // ring over the steps
    double inj[2 * K2W_STEPS];
    int item;
};

__host__ __device__ inline size_t k2w_smem_doubles(int L)
{
    return (size_t)L * odd_pitch(L) + 6 * (size_t)L + 10 * (size_t)L;
}

// Groups of W warps of a CTA: solves, factors, and (few lines, where the
// vectors would hold up the solves) the vectors.  Milliseconds of 200 steps of
// one grid with two groups / with three: L = 31 3.61 / 3.09, 45 4.68 / 4.08, 64
// 5.01 / 4.95, 80 6.92 / 7.22, 96 8.23 / 8.57.
__host__ __device__ constexpr int k2w_groups(int W) { return W <= 2 ? 3 : 2; }

// How much one of k CTAs of W warps of lines on an SM is slower than one alone
// (grids of 24 and 31 points, k = 2 .. 5: 1.12 1.18 1.30 1.60 and 1.05 1.07
// 1.12 1.24; of 45 and 64, k = 2 .. 4: 1.14 1.38 1.79 and 1.22 1.60 2.14).
__host__ __device__ constexpr float k2w_slowdown(int W, int k)
{
    return 1.0f + (W == 1 ? 0.1f : 0.3f) * (k - 1);
}

// k2w_live serves launches of fewer than K2W_HEADS - 1 items per SM (from there
// on k2w_per_sm gives all the CTAs that fit).
constexpr int K2W_HEADS = 16;
constexpr int K2W_LIVE_THREADS = 256;
constexpr int K2W_SMIDS = 1023; // (SMs are told apart by their number below this)

// Whether a CTA, asked once at its start, is beyond those of its SM that run.
__device__ __forceinline__ bool k2w_leaves(int *live)
{
    unsigned sm;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
    return atomicAdd(live + 1 + sm % K2W_SMIDS, 1) >= *live;
}

// How many CTAs per SM of a launch with a few items per SM run: `most` are
// launched, and those beyond leave (k2w_leaves; going by SM and not by
// blockIdx, as the first CTAs need not be on different SMs).  Such a batch ends
// with its longest item, and further CTAs on an SM slow that one down; but
// items of like length end sooner the more of them run at once.  With k CTAs
// per SM it takes, in units of an item's cost alone, at least its work spread
// evenly, and j + 1 times the cost of the item at place j k sms of the order
// (longest first); to that comes what they slow each other down while all of
// them have work.  The k with the least runs.  A kernel of its own, and asked
// where a CTA takes its items: more code at the head of k_integrate2d_ws gave
// its loop other registers and cost 4-6 %.  For one and two warps of lines; at
// three, where an SM holds two CTAs, 320 sets of 100 steps at 80 points would
// gain (10.1 and 7.9 ms), but IM sets lose (400 at 70/75/80 201-208 and
// 207-213).
// Milliseconds with k2w_per_sm's count and so: 320 sets of 100 steps at 31
// points 4.01 and 1.63, at 64 7.16 and 3.87; 160 such at 40/50/60 points 7.44
// and 4.05; 320 sets of 30 to 170 steps at 31/38/45 6.13 and 5.00; IM sets,
// whose longest schedule is a dozen times the mean: 257 at 31/38/45 90 and 88,
// 700 131 and 107, 320 at 40/50/60 126 and 108, 700 170 and 135.
__global__ void __launch_bounds__(K2W_LIVE_THREADS)
    k2w_live(K2Args A, int warps, int sms, int most, int *live)
{
    __shared__ float head[K2W_HEADS], part[K2W_LIVE_THREADS / 32];
    const int tid = threadIdx.x;
    for (int i = tid; i < K2W_SMIDS; i += K2W_LIVE_THREADS)
        live[1 + i] = 0;
    auto cost = [&](int w) {
        const K2Item I = k2_item(A, A.order[w]);
        return (float)(I.nsteps + 2) * (float)I.L; // (2: an item's set-up)
    };
    float sum = 0;
    for (int w = tid; w < A.nwork; w += K2W_LIVE_THREADS)
        sum += cost(w);
    for (int off = 16; off > 0; off >>= 1)
        sum += __shfl_down_sync(0xffffffffu, sum, off);
    if ((tid & 31) == 0)
        part[tid >> 5] = sum;
    if (tid < K2W_HEADS)
        head[tid] = ((long)tid * sms < A.nwork) ? cost(tid * sms) : 0.0f;
    __syncthreads();
    if (tid > 0)
        return;
    sum = 0;
    for (int w = 0; w < K2W_LIVE_THREADS / 32; w++)
        sum += part[w];
    int best = 1;
    float shortest = INFINITY;
    for (int k = 1; k <= most; k++) {
        const float even = sum / (float)(k * sms);
        float t = even;
        for (int j = 0; j * k < K2W_HEADS; j++)
            t = fmaxf(t, (float)(j + 1) * head[j * k]);
        t += (k2w_slowdown(warps, k) - 1.0f) * even;
        if (t < shortest) {
            best = k;
            shortest = t;
        }
    }
    *live = best;
}

// (CTAs per SM of the launch bounds: with 4, 2 and 1 grids of 45 points, 3000
// sets of 40 steps, take 12.0 ms and with 6, 4 and 2 10.3, against 10.2; one
// grid alone 4.08 and 4.38 ms for 200 steps, against 4.07.)
template <int W, bool KEEP_A, bool CHOSEN = false>
__global__ void __launch_bounds__(32 * W * k2w_groups(W), W == 1 ? 5 : W == 2 ? 3 : 2)
    k_integrate2d_ws(K2Args A)
{
    extern __shared__ __align__(16) double smem[];
    __shared__ K2WShared S;
    constexpr int ng = 32 * W; // threads of a group
    const int tid = threadIdx.x;
    constexpr bool P = k2w_groups(W) == 3;
    static_assert(KEEP_A || !P, "a third group rebuilds the vectors that the solves would read");
    const int group = tid / ng, q = tid - group * ng;
    const int pitch = odd_pitch(A.Lmax);
    double *phi = smem;
    GridVecs g;
    double *p = smem + (size_t)A.Lmax * pitch;
    g.x = p; p += A.Lmax;
    g.xv = p; p += A.Lmax;
    g.dfac = p; p += A.Lmax;
    g.xInt = p; p += A.Lmax;
    g.ih = p; p += A.Lmax;
    g.dx = p; p += A.Lmax;
    auto vecs = [&](int a) {
        double *w = p + (size_t)a * 5 * A.Lmax;
        AxisVecs v;
        v.A1 = w;
        v.A0 = w + A.Lmax;
        v.C1 = w + 2 * A.Lmax;
        v.C0 = w + 3 * A.Lmax;
        v.B0 = w + 4 * A.Lmax;
        v.G = v.Pv = v.Qv = v.VI = v.DF = nullptr;
        return v;
    };
    double *slice = A.gam_glob + (size_t)blockIdx.x * k2w_slice_doubles(A.Lmax, KEEP_A);

    for (int iter = 0;; iter++) {
        if (tid == 0)
            S.item = (CHOSEN && iter == 0 && k2w_leaves(A.live)) ? A.nwork
                     : A.counter                                 ? atomicAdd(A.counter, 1)
                     : iter == 0                                 ? (int)blockIdx.x
                                                                 : A.nwork;
        __syncthreads();
        const int w = S.item;
        if (w >= A.nwork)
            break;
        const K2Item I = k2_item(A, A.order ? A.order[w] : w);
        const int L = I.L, LP = k2w_pitch(L);
        const size_t stride = (size_t)L * LP;
        for (int i = tid; i < L; i += blockDim.x) {
            double x = I.xx[i];
            g.x[i] = x;
            g.xv[i] = x * (1. - x);
            if (i < L - 1) {
                double d = I.xx[i + 1] - x;
                g.dx[i] = d;
                g.ih[i] = 1.0 / (2 * d);
                g.xInt[i] = 0.5 * (I.xx[i + 1] + x);
            }
        }
        for (int idx = tid; idx < L * L; idx += blockDim.x) {
            int r = idx / L, c = idx - r * L;
            phi[r * pitch + c] = I.src[idx];
        }
        __syncthreads();
        for (int i = tid; i < L; i += blockDim.x) {
            if (i == 0)
                g.dfac[i] = 2. / g.dx[0];
            else if (i == L - 1)
                g.dfac[i] = 2. / g.dx[L - 2];
            else
                g.dfac[i] = 2. / (g.dx[i] + g.dx[i - 1]);
        }
        __syncthreads();
        const int j0 = (g.x[0] == 0.0) ? 0 : -1;
        const int j1 = (g.x[L - 1] == 1.0) ? L - 1 : -1;
        const int nsw = 2 * I.nsteps; // sweep m: axis m & 1 of step m >> 1

        // Phase m: the solve warps run sweep m and then form the vectors of
        // sweep m + 2 (the same axis; the scalars of K2W_STEPS steps when
        // they run out); the factor warps run sweep m + 1.
        auto prepare = [&](int m) {
            const int a = m & 1, n = m >> 1;
            if (m >= nsw)
                return;
            if (a == 0 && n % K2W_STEPS == 0) {
                const int st = n + (q >> 1);
                const double *row = I.rows + (size_t)st * K2_ROW;
                if (q < 2 * K2W_STEPS && st < I.nsteps)
                    axis_scalars_2d(S.ax[st % (2 * K2W_STEPS)][q & 1], q & 1, row, g, L);
                if (q < 2 * K2W_STEPS && st < I.nsteps && !(q & 1))
                    S.inj[st % (2 * K2W_STEPS)] =
                        inject_value(2, row[0], row[1], g.x[0], g.x[1], g.x[2]);
                bar_group(2, ng);
            }
            if (I.frozen >> a & 1)
                return;
            AxisVecs v = vecs(a);
            for (int i = q; i < L; i += ng)
                build_axis_entry(i, L, g, S.ax[n % (2 * K2W_STEPS)][a], 1.0, false, v);
        };
        const bool prep = group == (P ? 2 : 0);
        if (prep) {
            prepare(0);
            prepare(1);
        }
        __syncthreads();
        for (int m = -1; m < nsw; m++) {
            if (group == 1) {
                const int a = (m + 1) & 1;
                if (m + 1 < nsw && !(I.frozen >> a & 1) && q < L) {
                    const AxisScalars &s = S.ax[(m + 1) / 2 % (2 * K2W_STEPS)][a];
                    k2w_factor<KEEP_A>(vecs(a), s, L, s.mig[1 - a] * g.x[q],
                                       (q == j0) ? s.bcs : 0.0, (q == j1) ? s.bce : 0.0,
                                       slice + a * (KEEP_A ? 3 : 2) * stride + q, stride, LP);
                }
            } else if (P && group == 2) {
                prepare(m + 2);
            } else if (m >= 0) {
                const int a = m & 1, k = m >> 1;
                if (a == 0) {
                    if (A.ckpt && k % A.ckpt_every == 0) {
                        // checkpoint for the adjoint: phi before this step, row-major
                        double *c = A.ckpt + A.ckpt_off[I.wid] + (size_t)(k / A.ckpt_every) * L * L;
                        for (int idx = q; idx < L * L; idx += ng) {
                            int r = idx / L, cc = idx - r * L;
                            c[idx] = phi[r * pitch + cc];
                        }
                        bar_group(1, ng);
                    }
                    if (q == 0) {
                        const double inj = S.inj[k % (2 * K2W_STEPS)];
                        if (!(I.frozen & 1) && !(I.nomut & 1))
                            phi[1 * pitch + 0] += inj;
                        if (!(I.frozen & 2) && !(I.nomut & 2))
                            phi[0 * pitch + 1] += inj;
                    }
                    bar_group(1, ng);
                }
                if (!(I.frozen >> a & 1) && q < L)
                    k2w_solve<KEEP_A>(phi + (size_t)q * ((a == 0) ? 1 : pitch),
                                      phi + (size_t)q * ((a == 0) ? 1 : pitch),
                                      (a == 0) ? pitch : 1, L, vecs(a),
                                      S.ax[k % (2 * K2W_STEPS)][a].mig[1 - a] * g.x[q],
                                      slice + a * (KEEP_A ? 3 : 2) * stride + q, stride, LP);
                if (!P) {
                    if (!KEEP_A)
                        bar_group(1, ng); // the solves still read the axis's vectors
                    prepare(m + 2);
                }
            }
            __syncthreads();
        }
        for (int idx = tid; idx < L * L; idx += blockDim.x) {
            int r = idx / L, c = idx - r * L;
            I.out[idx] = phi[r * pitch + c];
        }
        __syncthreads();
    }
}

// ------------------------------- the delj trick's coefficients ahead of the sweep

// k_integrate2d<true> with delta_j and the intervals' coefficients (at, ct of
// solve_line_delj: an exponential, two divisions and some 15 further FP64
// instructions per interval and line, none of which depends on the row before
// or on the density) formed one sweep ahead by k2d_groups(W) W further warps,
// interval i by group i mod k2d_groups(W), and handed over through the
// workspace.  What is left to the solve warps is the recurrence.  With the
// divisions and the products that no chain waits for on the integer pipes
// (div_wide, mul_full) some 40 FP64 instructions remain per point; from three
// warps of lines on they fill the FP64 pipe, whatever the groups.  Every
// operation is solve_line_delj's, so the results are bitwise the same.
// Measured, microseconds per step of one grid with one warp for both / with
// this kernel: L = 31 135 / 41, 60 256 / 95, 90 384 / 194, 128 544 / 361.
//
// Milliseconds of 100 steps of one grid with 2, 3, 4, 5, 6 groups: L = 31 5.78
// 4.11 4.35 4.33 4.33 (8: 4.49), 60 11.8 9.80 9.52 9.68 10.4, 90 22.0 19.7 19.5
// 21.1 22.6, 128 36.8 36.2 36.5 38.0 41.2, 150 53.5 52.7 59.3 66.2; of 40 steps
// of 400 sets at 60 points 14.0 11.9 11.9 12.1 12.8, of 200 at 90 16.9 15.4 15.4
// 17.0 18.3.
constexpr __host__ __device__ int k2d_groups(int W) { return W == 2 || W == 3 ? 4 : 3; }

__host__ __device__ inline size_t k2d_smem_doubles(int L)
{
    return (size_t)L * odd_pitch(L) + 6 * (size_t)L + 8 * (size_t)L;
}

// Workspace of one CTA: [axis][the four arrays of k2d_solve][row][line], then
// the couplings of the sweep being solved.
__host__ __device__ inline size_t k2d_slice_doubles(int L) { return (size_t)9 * L * k2w_pitch(L); }

// solve_line_delj from the products of its intervals' at and ct with dfactor,
// arrays f + k * stride, row i at i * LP: k = 0 a_i = -DF_i at_{i-1}, 1 1/dt +
// DF_i ct_{i-1}, 2 DF_i at_i, 3 c_i = -DF_i ct_i; row 0 has the last two.
__device__ __forceinline__ void k2d_solve(double *__restrict__ ph, int sp,
                                          double *__restrict__ gm,
                                          const double *__restrict__ f, size_t stride, int LP,
                                          int L, double mo, double o, bool c0, bool c1,
                                          const GridVecs &gv, const AxisScalars &s)
{
    constexpr int B = 3;
    auto mfun = [&](double x, double sel) { return xa(xm(mo, xs(o, x)), sel); };
    const double dt = s.dt;
    unsigned rdt[3], rb[3];
    rcp_wide(dt, rdt);
    double fn[4][B]; // the next rows'
    auto load = [&](int i) {
#pragma unroll
        for (int k = 0; k < B; k++)
#pragma unroll
            for (int n = 0; n < 4; n++)
                fn[n][k] = __ldcg(f + n * stride + min(i + k, n < 2 ? L - 1 : L - 2) * LP);
    };
    double cprev = __ldcg(f + 3 * stride);
    double bet = xa(xd(1.0, dt), __ldcg(f + 2 * stride));
    load(1);
    if (c0) {
        const double mf = mfun(gv.x[0], msel_ref(gv.x[0], s.gamma, s.h));
        if (mf <= 0)
            bet = xa(bet, xd(xm(xs(xd(0.5, s.nu), mf), 2.0), gv.dx[0]));
    }
    rcp_wide(bet, rb);
    double u = div_wide(div_wide(ph[0], dt, rdt), bet, rb);
    ph[0] = u;
    for (int i0 = 1; i0 < L; i0 += B) {
        double fv[4][B], pv[B];
#pragma unroll
        for (int k = 0; k < B; k++) {
#pragma unroll
            for (int n = 0; n < 4; n++)
                fv[n][k] = fn[n][k];
            pv[k] = ph[min(i0 + k, L - 1) * sp];
        }
        load(i0 + B);
#pragma unroll
        for (int k = 0; k < B; k++) {
            const int i = i0 + k;
            if (i >= L)
                break;
            const double a = fv[0][k];
            double bb = fv[1][k];
            if (i < L - 1) {
                bb = xa(bb, fv[2][k]);
            } else if (c1) {
                const double ml = mfun(gv.x[L - 1], msel_ref(gv.x[L - 1], s.gamma, s.h));
                if (ml >= 0)
                    bb = xa(bb, xd(xm(-xs(-xd(0.5, s.nu), ml), 2.0), gv.dx[L - 2]));
            }
            const double g = div_wide(cprev, bet, rb);
            gm[i * LP] = g;
            bet = xs(bb, xm(a, g));
            rcp_wide(bet, rb);
            u = div_wide(xs(div_wide(pv[k], dt, rdt), xm(a, u)), bet, rb);
            ph[i * sp] = u;
            cprev = fv[3][k];
        }
    }
    constexpr int C = 8;
    int i = L - 2;
    for (; i >= C - 1; i -= C) {
        double g[C], p[C];
#pragma unroll
        for (int k = 0; k < C; k++) {
            g[k] = __ldcg(gm + (i - k + 1) * LP);
            p[k] = ph[(i - k) * sp];
        }
#pragma unroll
        for (int k = 0; k < C; k++) {
            u = xs(p[k], xm(g[k], u));
            ph[(i - k) * sp] = u;
        }
    }
    for (; i >= 0; i--) {
        u = xs(ph[i * sp], xm(__ldcg(gm + (i + 1) * LP), u));
        ph[i * sp] = u;
    }
}

template <int W>
__global__ void __launch_bounds__(32 * W * (1 + k2d_groups(W)), 1) k_integrate2d_delj(K2Args A)
{
    extern __shared__ __align__(16) double smem[];
    __shared__ K2WShared S;
    constexpr int ng = 32 * W, NG = k2d_groups(W), nc = NG * ng;
    const int tid = threadIdx.x;
    const int group = tid / ng, q = tid - group * ng; // group 0 solves
    const int pitch = odd_pitch(A.Lmax);
    double *phi = smem;
    GridVecs g;
    double *p = smem + (size_t)A.Lmax * pitch;
    g.x = p; p += A.Lmax;
    g.xv = p; p += A.Lmax;
    g.dfac = p; p += A.Lmax;
    g.xInt = p; p += A.Lmax;
    g.ih = p; p += A.Lmax;
    g.dx = p; p += A.Lmax;
    double *vec = p; // G, Pv, Qv, VI of the sweep being prepared
    double *slice = A.gam_glob + (size_t)blockIdx.x * k2d_slice_doubles(A.Lmax);

    for (int iter = 0;; iter++) {
        if (tid == 0)
            S.item = A.counter ? atomicAdd(A.counter, 1) : (iter == 0 ? (int)blockIdx.x : A.nwork);
        __syncthreads();
        const int w = S.item;
        if (w >= A.nwork)
            break;
        const K2Item I = k2_item(A, A.order ? A.order[w] : w);
        const int L = I.L, LP = k2w_pitch(L);
        const size_t stride = (size_t)L * LP;
        for (int i = tid; i < L; i += blockDim.x) {
            double x = I.xx[i];
            g.x[i] = x;
            g.xv[i] = x * (1. - x);
            if (i < L - 1) {
                double d = I.xx[i + 1] - x;
                g.dx[i] = d;
                g.ih[i] = 1.0 / (2 * d);
                g.xInt[i] = 0.5 * (I.xx[i + 1] + x);
            }
        }
        for (int idx = tid; idx < L * L; idx += blockDim.x) {
            int r = idx / L, c = idx - r * L;
            phi[r * pitch + c] = I.src[idx];
        }
        __syncthreads();
        for (int i = tid; i < L; i += blockDim.x) {
            if (i == 0)
                g.dfac[i] = 2. / g.dx[0];
            else if (i == L - 1)
                g.dfac[i] = 2. / g.dx[L - 2];
            else
                g.dfac[i] = 2. / (g.dx[i] + g.dx[i - 1]);
        }
        __syncthreads();
        const int j0 = (g.x[0] == 0.0) ? 0 : -1;
        const int j1 = (g.x[L - 1] == 1.0) ? L - 1 : -1;
        const int nsw = 2 * I.nsteps; // sweep m: axis m & 1 of step m >> 1
        for (int m = -1; m < nsw; m++) {
            if (group) {
                // the coefficients of sweep m + 1
                const int r = tid - ng, a = (m + 1) & 1, n = (m + 1) >> 1;
                if (m + 1 < nsw) {
                    if (a == 0 && n % K2W_STEPS == 0) {
                        const int st = n + (r >> 1);
                        const double *row = I.rows + (size_t)st * K2_ROW;
                        if (r < 2 * K2W_STEPS && st < I.nsteps) {
                            axis_scalars_2d(S.ax[st % (2 * K2W_STEPS)][r & 1], r & 1, row, g, L);
                            if (!(r & 1))
                                S.inj[st % (2 * K2W_STEPS)] =
                                    inject_value(2, row[0], row[1], g.x[0], g.x[1], g.x[2]);
                        }
                        bar_group(2, nc);
                    }
                    if (!(I.frozen >> a & 1)) {
                        const AxisScalars &s = S.ax[n % (2 * K2W_STEPS)][a];
                        for (int t = r; t < 4 * (L - 1); t += nc) {
                            const int k = t / (L - 1), i = t - k * (L - 1);
                            const double d2 = xm(2.0, g.dx[i]);
                            vec[k * L + i] =
                                k == 0   ? msel_ref(g.xInt[i], s.gamma, s.h)
                                : k == 1 ? xd(vfunc_ref(g.x[i], s.nu, 0.0), d2)
                                : k == 2 ? xd(vfunc_ref(g.x[i + 1], s.nu, 0.0), d2)
                                         : vfunc_ref(g.xInt[i], s.nu, 0.0);
                        }
                        bar_group(2, nc);
                        double *f = slice + (size_t)a * 4 * stride + q;
                        if (q < L) {
                            const double mo = s.mig[1 - a], o = g.x[q], idt = xd(1.0, s.dt);
                            for (int i = group - 1; i < L - 1; i += NG) {
                                const double Mk = xa(xmi(xs(o, g.xInt[i]), mo), vec[i]);
                                const double d = delj_of(Mk, vec[3 * L + i], g.dx[i]);
                                const double at = xa(xmi(Mk, d), vec[L + i]);
                                const double ct = xa(xmi(-Mk, xs(1.0, d)), vec[2 * L + i]);
                                const double d0 = g.dfac[i], d1 = g.dfac[i + 1];
                                f[(i + 1) * LP] = -xmi(at, d1);
                                f[stride + (i + 1) * LP] = xa(idt, xmi(ct, d1));
                                f[2 * stride + i * LP] = xmi(at, d0);
                                f[3 * stride + i * LP] = -xmi(ct, d0);
                            }
                        }
                    }
                }
            } else if (m >= 0) {
                const int a = m & 1, k = m >> 1;
                const AxisScalars &s = S.ax[k % (2 * K2W_STEPS)][a];
                if (a == 0) {
                    if (A.ckpt && k % A.ckpt_every == 0) {
                        double *c = A.ckpt + A.ckpt_off[I.wid] + (size_t)(k / A.ckpt_every) * L * L;
                        for (int idx = q; idx < L * L; idx += ng) {
                            int r = idx / L, cl = idx - r * L;
                            c[idx] = phi[r * pitch + cl];
                        }
                        bar_group(1, ng);
                    }
                    if (q == 0) {
                        const double inj = S.inj[k % (2 * K2W_STEPS)];
                        if (!(I.frozen & 1) && !(I.nomut & 1))
                            phi[1 * pitch + 0] += inj;
                        if (!(I.frozen & 2) && !(I.nomut & 2))
                            phi[0 * pitch + 1] += inj;
                    }
                    bar_group(1, ng);
                }
                if (!(I.frozen >> a & 1) && q < L) {
                    k2d_solve(phi + (size_t)q * ((a == 0) ? 1 : pitch), (a == 0) ? pitch : 1,
                              slice + 8 * stride + q, slice + (size_t)a * 4 * stride + q, stride,
                              LP, L, s.mig[1 - a], g.x[q], q == j0, q == j1, g, s);
                }
            }
            __syncthreads();
        }
        for (int idx = tid; idx < L * L; idx += blockDim.x) {
            int r = idx / L, c = idx - r * L;
            I.out[idx] = phi[r * pitch + c];
        }
        __syncthreads();
    }
}

// ------------------------------------------------------- schedule pass

// Walk the reference time loop of two_pops (dadi/Integration.py:346-386) for
// one instance with parametric parameters.  Emits one row per step (when
// rows != null) and returns the number of rows; *status gets DGB_ST_* bits.
// dx0 is the grid's first spacing (only used with use_old_timestep).
__host__ __device__ inline long sched2d_walk(const dgb_inst2d &I, const dgb_settings &st,
                                             double dx0, long max_steps, double *rows,
                                             int *status)
{
    double cur = I.initial_t;
    double nu0 = pform_eval(I.nu[0], cur), nu1 = pform_eval(I.nu[1], cur);
    double m0 = pform_eval(I.m12, cur), m1 = pform_eval(I.m21, cur);
    double g0 = pform_eval(I.gamma[0], cur), g1 = pform_eval(I.gamma[1], cur);
    double h0 = pform_eval(I.h[0], cur), h1 = pform_eval(I.h[1], cur);
    long n = 0;
    int err = 0;
    while (cur < I.T) {
        if (n >= max_steps) {
            err |= DGB_ST_STEPCAP;
            break;
        }
        double d0 = compute_dt(nu0, m0, g0, h0, st, dx0);
        double d1 = compute_dt(nu1, m1, g1, h1, st, dx0);
        double dtm = pymin(d0, d1);
        if (dtm == 0) {
            err |= DGB_ST_ZERODT;
            break;
        }
        double dt = pymin(dtm, I.T - cur);
        double next = cur + dt;
        if (!(dt > 0) || !isfinite(next)) {
            err |= DGB_ST_NONFINITE;
            break;
        }
        nu0 = pform_eval(I.nu[0], next);
        nu1 = pform_eval(I.nu[1], next);
        m0 = pform_eval(I.m12, next);
        m1 = pform_eval(I.m21, next);
        g0 = pform_eval(I.gamma[0], next);
        g1 = pform_eval(I.gamma[1], next);
        h0 = pform_eval(I.h[0], next);
        h1 = pform_eval(I.h[1], next);
        double theta0 = pform_eval(I.theta0, next);
        if (I.T < 0 || nu0 < 0 || nu1 < 0 || m0 < 0 || m1 < 0 || theta0 < 0 || nu0 == 0 ||
            nu1 == 0) {
            err |= DGB_ST_BADPARAM;
            break;
        }
        if (rows) {
            double *r = rows + n * K2_ROW;
            r[0] = dt;
            r[1] = theta0;
            r[2] = nu0;
            r[3] = nu1;
            r[4] = g0;
            r[5] = g1;
            r[6] = h0;
            r[7] = h1;
            r[8] = 1.0;
            r[9] = m0;  // into pop 1 from pop 2 (m12)
            r[10] = m1; // into pop 2 from pop 1 (m21)
        }
        n++;
        cur = next;
    }
    if (status)
        *status |= err;
    return n;
}

// sched2d_walk on two lanes of a warp: lane p evaluates population p's
// forms and timestep (lane 0 also theta0), the two exchange their timesteps
// by shuffle and so take the same steps, and each writes its population's
// entries of the rows.  The FP64 pipe takes a warp instruction in the same
// time whatever the number of active lanes, so the per-step chain (one
// pow and one timestep per population) issues half the FP64 instructions of
// one lane doing both.  The same functions give the same rows and status as
// sched2d_walk.
//
// Per step the chain holds one pow, three divisions and a few comparisons; the
// divisions run on the integer pipes (div_full), the ratio b / a of a growth
// form, constant forms and what the timestep takes from them are evaluated
// once.  4,570 steps: 26.7 ms with everything evaluated at every step, 20.9
// here.
struct FormWalk {
    const dgb_pform *f;
    double q;  // b / a of DGB_PF_EXPGROW
    __device__ explicit FormWalk(const dgb_pform &g)
        : f(&g), q(g.kind == DGB_PF_EXPGROW ? g.b / g.a : 0.0)
    {
    }
    __device__ bool constant() const
    {
        return f->kind != DGB_PF_EXPGROW && f->kind != DGB_PF_EXPLOG && f->kind != DGB_PF_LINEAR;
    }
    // pform_eval(*f, t)
    __device__ double at(double t) const
    {
        if (f->kind == DGB_PF_EXPGROW)
            return f->a * pow(q, div_full(t, f->c));
        return pform_eval(*f, t);
    }
};

__device__ long sched2d_walk_pair(const dgb_inst2d &I, const dgb_settings &st, double dx0,
                                  long max_steps, double *rows, int *status, int p)
{
    const unsigned pair = 3u << (threadIdx.x & 30);
    const FormWalk fnu(I.nu[p]), fm(p ? I.m21 : I.m12), fg(I.gamma[p]), fh(I.h[p]), fth(I.theta0);
    const bool cm = fm.constant(), cg = fg.constant(), ch = fh.constant(), ct = fth.constant();
    double cur = I.initial_t;
    double nu = fnu.at(cur), m = fm.at(cur), g = fg.at(cur), h = fh.at(cur);
    double theta0 = p ? 0.0 : fth.at(cur);
    // what compute_dt takes the largest of, besides 0.25 / nu, when constant
    const bool cdt = cm && cg && ch && !st.use_old_timestep;
    double vm = 0;
    if (cdt) {
        const double t1 = fabs(h + (1 - 2 * h) * 0.5) * 0.5 * (1 - 0.5);
        const double t2 = fabs(h + (1 - 2 * h) * 0.25) * 0.25 * (1 - 0.25);
        const double v3 = fabs(g) * 2 * (t2 > t1 ? t2 : t1);
        vm = (m == m) ? m : -INFINITY; // (a NaN is never the larger)
        if (v3 > vm)
            vm = v3;
    }
    long n = 0;
    int err = 0;
    while (cur < I.T) {
        if (n >= max_steps) {
            err |= DGB_ST_STEPCAP;
            break;
        }
        double mine;
        if (cdt) {
            double mx = div_full(0.25, nu);
            if (vm > mx)
                mx = vm;
            mine = mx > 0 ? div_full(st.timescale_factor, mx) : INFINITY;
        } else {
            mine = compute_dt(nu, m, g, h, st, dx0);
        }
        const double other = __shfl_xor_sync(pair, mine, 1);
        const double dtm = p ? pymin(other, mine) : pymin(mine, other);
        if (dtm == 0) {
            err |= DGB_ST_ZERODT;
            break;
        }
        const double dt = pymin(dtm, I.T - cur);
        const double next = cur + dt;
        if (!(dt > 0) || !isfinite(next)) {
            err |= DGB_ST_NONFINITE;
            break;
        }
        nu = fnu.at(next);
        if (!cm)
            m = fm.at(next);
        if (!cg)
            g = fg.at(next);
        if (!ch)
            h = fh.at(next);
        if (!ct && !p)
            theta0 = fth.at(next);
        const bool bad = nu <= 0 || m < 0 || theta0 < 0;
        if (I.T < 0 || __any_sync(pair, bad)) {
            err |= DGB_ST_BADPARAM;
            break;
        }
        if (rows) {
            double *r = rows + n * K2_ROW;
            if (p == 0) {
                r[0] = dt;
                r[1] = theta0;
                r[2] = nu;
                r[4] = g;
                r[6] = h;
                r[8] = 1.0;
                r[9] = m; // into pop 1 from pop 2 (m12)
            } else {
                r[3] = nu;
                r[5] = g;
                r[7] = h;
                r[10] = m; // into pop 2 from pop 1 (m21)
            }
        }
        n++;
        cur = next;
    }
    *status |= err;
    return n;
}

// Two lanes per schedule (instance, or instance x grid with
// use_old_timestep; sched2d_walk_pair).  fill == 0: count rows; fill == 1:
// write rows at row_off[s] and the status bits.
__global__ void k_sched2d(const dgb_inst2d *insts, int nsched, int ngrids, int per_grid,
                          const double *dx0s, dgb_settings st, long max_steps, int fill,
                          int *row_cnt, const long *row_off, double *table, int *status)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = t >> 1, p = t & 1;
    if (s >= nsched)
        return; // both lanes of the pair
    int inst = per_grid ? s / ngrids : s;
    double dx0 = dx0s[per_grid ? s % ngrids : 0];
    int err = 0;
    // fill == 2: row_cnt holds the room reserved at row_off (an upper bound
    // on the rows); a walk that would exceed it stops with DGB_ST_STEPCAP
    const long cap = (fill == 2) ? std::min<long>(max_steps, row_cnt[s]) : max_steps;
    long n = sched2d_walk_pair(insts[inst], st, dx0, cap,
                               fill ? table + row_off[s] * K2_ROW : nullptr, &err, p);
    if (p)
        return;
    if (fill != 1)
        row_cnt[s] = (int)n;
    if (fill && err)
        atomicOr(status + inst, err);
}

// ------------------------------------------------------------ host side

int k2_smem_fits(int Lmax, bool gam_smem, bool delj, size_t *bytes)
{
    K2Layout l = k2_layout(Lmax, gam_smem, delj);
    if (bytes)
        *bytes = l.total;
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess)
        return 0;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return 0;
    return l.total + sizeof(K2Shared) + 1024 <= (size_t)optin;
}

static int k2_launch(K2Args &A, int nblocks, size_t smem, cudaStream_t st,
                     int threads = K2_THREADS)
{
    if (A.use_delj) {
        if (raise_smem_limit(k_integrate2d<true>))
            return DGB_ERR_CUDA;
        k_integrate2d<true><<<nblocks, threads, smem, st>>>(A);
    } else {
        if (raise_smem_limit(k_integrate2d<false>))
            return DGB_ERR_CUDA;
        k_integrate2d<false><<<nblocks, threads, smem, st>>>(A);
    }
    return cudaGetLastError() == cudaSuccess ? DGB_OK : DGB_ERR_CUDA;
}

// Resident CTAs per SM for a dynamic shared-memory size.  The kernel's
// dynamic-smem limit is raised to the opt-in maximum first: the occupancy
// query honours the current limit, so without this its answer would depend on
// the previous launch.
static int k2_occupancy(bool delj, size_t smem, int threads = K2_THREADS)
{
    int nb = 0;
    cudaError_t e;
    if (delj) {
        raise_smem_limit(k_integrate2d<true>);
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_integrate2d<true>, threads,
                                                          smem);
    } else {
        raise_smem_limit(k_integrate2d<false>);
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_integrate2d<false>, threads,
                                                          smem);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return nb > 0 ? nb : 1;
}

static int k2_num_sms()
{
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm > 0 ? nsm : 1;
}

// Threads per CTA of a batched launch whose grids are at most Lmax points:
// the fewest warps (two to four) that give every line of the largest grid
// its own lane.  A sweep of one line is one lane's dependency chain and the
// FP64 pipe charges a warp instruction whatever its active lanes, so lines
// packed into fewer warps cost fewer pipe cycles per step.  Measured on the
// 4096-instance IM batch at pts 80/90/100, one launch per grid: three warps
// at L = 80 and 90 (27 and 30 of 32 lanes busy, instead of 20 and 23 with
// four) 11.72 s, four warps for every grid 13.39 s, bitwise the same
// densities.  settings->threads = 64, 96 or 128 asks for that size where it
// holds the lines (else the automatic choice applies); 0 is automatic.
// occ gets the CTAs per SM.  Returns 0 for an unsupported setting.
static int k2_pick_threads(const dgb_settings *settings, bool delj, size_t smem, int Lmax,
                           int &occ)
{
    const int want = (settings->threads == K2_AUTO_SHARED) ? 0 : settings->threads;
    if (want != 0 && want != 64 && want != 96 && want != 128)
        return 0;
    int warps = std::min(4, std::max(2, (Lmax + 31) / 32));
    if (want != 0 && Lmax <= want)
        warps = want / 32;
    occ = k2_occupancy(delj, smem + sizeof(K2Shared), 32 * warps);
    return 32 * warps;
}

template <int W> static void (*k2w_kernel(bool keep_a))(K2Args)
{
    // (with a third group the vectors of an axis are rebuilt beside its
    // solves, which then take a from the workspace)
    return keep_a || k2w_groups(W) == 3 ? k_integrate2d_ws<W, true>
                                        : k_integrate2d_ws<W, k2w_groups(W) == 3>;
}

// Whether the caller leaves the shape of a batched launch to the rules here.
static bool k2w_auto(const dgb_settings *s)
{
    return (s->threads == 0 || s->threads == K2_AUTO_SHARED) && s->gam_placement != 1;
}

// CTAs of k_integrate2d_ws per SM for nwork items on sms SMs.  One CTA uses
// half to three quarters of the FP64 pipe (an SM's cycles per grid point and
// warp of lines, one CTA / as many as fit: L = 45 220 / 98, 64 181 / 99, 80
// 136 / 95, 90 151 / 108, 100 110 / 103), but a second one slows the first,
// and a batch of few items per SM ends when its longest item does: 257 IM sets
// on three grids of 31-45 points (5 items per SM) took 88 ms with one CTA and
// 101 with two, 1000 sets at pts 80/90/100 652 with one and 519 with two.
static int k2w_per_sm(long nwork, int sms)
{
    return (int)std::max<long>(1, std::min<long>(5, nwork / (3L * sms)));
}

// Whether the split kernels take grids of up to L points: five warps of lines,
// and the density in shared memory (159 points).
static bool k2w_fits(int L, bool delj)
{
    const size_t smem = (delj ? k2d_smem_doubles(L) : k2w_smem_doubles(L)) * sizeof(double);
    return (L + 31) / 32 <= K2W_MAXWARPS && smem + sizeof(K2WShared) + 1024 <= cta_smem_bytes();
}

constexpr size_t K2W_LIVE_BYTES = (1 + K2W_SMIDS) * sizeof(int);

// The launch of a split kernel.
struct K2WPlan {
    void (*kernel)(K2Args);
    int threads, keep_a;
    int most;       // CTAs per SM of which k2w_live chooses (0: all run)
    size_t live_at; // K2W_LIVE_BYTES of the workspace for it
    size_t smem;
    long nblocks;
};

// Bytes of slices that k_integrate2d_ws keeps within L2.
static size_t k2w_l2_budget()
{
    int dev = 0, l2 = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return (size_t)l2 / 10 * 8;
}

// CTAs per SM of which k2w_live chooses, of `fit` that an SM holds: at most one
// per item, and slices within L2; or k2w_per_sm's if those are more.  0 where
// it does not choose.
static int k2w_most_per_sm(int Lmax, long nwork, int sms, int fit)
{
    if (k2w_groups((Lmax + 31) / 32) != 3 || nwork <= sms || nwork >= (long)(K2W_HEADS - 1) * sms)
        return 0;
    const size_t all = (size_t)sms * k2w_slice_doubles(Lmax, true) * sizeof(double);
    const long most = std::min<long>((nwork + sms - 1) / sms, (long)(k2w_l2_budget() / all));
    return (int)std::min<long>(fit, std::max<long>(most, k2w_per_sm(nwork, sms)));
}

// Plan a split kernel over nwork items on `sms` SMs with `bytes` of workspace
// for the slices; false where none applies: grids beyond five warps of lines
// or shared memory, or too little workspace.  The solves take a from the
// workspace where this launch's slices are within 0.8 of the L2 cache, and
// form it again (one more FP64 instruction a point, a third less traffic)
// where not, whether or not the smaller slices are then within it: 152 grids
// of 128 points 90 us a step with a, 62 without; of 100 points 46 and 51.  The
// rule looks at one launch; 1000 IM sets at pts 80/90/100 in one launch per
// grid, side by side, take 628 ms by it, 660 if all keep their a and 634 if
// none does.
// choose: k2w_live may choose the CTAs per SM.
static bool k2w_plan(int Lmax, bool delj_rows, long nwork, size_t bytes, int sms, bool choose,
                     K2WPlan &p)
{
    if (!k2w_fits(Lmax, delj_rows))
        return false;
    const int warps = (Lmax + 31) / 32;
    p.threads = 32 * warps * (delj_rows ? 1 + k2d_groups(warps) : k2w_groups(warps));
    p.smem = (delj_rows ? k2d_smem_doubles(Lmax) : k2w_smem_doubles(Lmax)) * sizeof(double);
    p.most = 0;
    int occ = 0;
    const size_t budget = k2w_l2_budget();
    void (*(*const kernels[])(bool))(K2Args) = {k2w_kernel<1>, k2w_kernel<2>, k2w_kernel<3>,
                                                k2w_kernel<4>, k2w_kernel<5>};
    void (*const delj[])(K2Args) = {k_integrate2d_delj<1>, k_integrate2d_delj<2>,
                                    k_integrate2d_delj<3>, k_integrate2d_delj<4>,
                                    k_integrate2d_delj<5>};
    const int last = (delj_rows || k2w_groups(warps) == 3) ? 1 : 0;
    for (p.keep_a = 1;; p.keep_a--) {
        const size_t slice =
            (delj_rows ? k2d_slice_doubles(Lmax) : k2w_slice_doubles(Lmax, p.keep_a)) *
            sizeof(double);
        p.kernel = delj_rows ? delj[warps - 1] : kernels[warps - 1](p.keep_a);
        if (raise_smem_limit(p.kernel))
            return false;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, p.kernel, p.threads, p.smem) !=
            cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        const long want = std::min<long>((long)sms * std::min(occ, k2w_per_sm(nwork, sms)),
                                         nwork);
        p.nblocks = std::min<long>((long)(bytes / slice), want);
        if (p.keep_a == last ||
            (p.nblocks == want && (size_t)p.nblocks * slice <= budget)) {
            const int most =
                (delj_rows || !choose) ? 0 : k2w_most_per_sm(Lmax, nwork, sms, occ);
            if (most > 1 && (size_t)sms * most * slice + K2W_LIVE_BYTES <= bytes) {
                p.most = most;
                p.kernel = warps == 1 ? k_integrate2d_ws<1, true, true>
                                      : k_integrate2d_ws<2, true, true>;
                if (raise_smem_limit(p.kernel))
                    return false;
                p.nblocks = (long)sms * most;
                p.live_at = (size_t)p.nblocks * slice;
            }
            break;
        }
    }
    return p.nblocks >= std::min<long>(sms, nwork);
}

// Launch a split kernel over A's work (queue counter already cleared, or null:
// one item per CTA) on `sms` SMs with slices from `slices` on; -1 where none
// applies.  alone: no other launch is meant to run beside this one (the CTAs
// that k2w_live sends home would take places from another's, and other CTAs on
// the SMs upset its estimate: launches per grid, 257 IM sets at 31/38/45
// points, 95.4 ms without it and 101 with it).
static int k2w_launch(K2Args &A, void *slices, size_t bytes, int sms, bool alone,
                      cudaStream_t st)
{
    K2WPlan p;
    if (!k2w_plan(A.Lmax, A.use_delj, A.nwork, bytes, sms, alone && A.order, p))
        return -1;
    A.gam_smem = 0;
    A.gam_glob = (double *)slices;
    if (p.most) {
        int *live = (int *)((char *)slices + p.live_at);
        k2w_live<<<1, K2W_LIVE_THREADS, 0, st>>>(A, (A.Lmax + 31) / 32, sms, p.most, live);
        if (cudaGetLastError() != cudaSuccess)
            return DGB_ERR_CUDA;
        A.live = live;
    }
    p.kernel<<<(unsigned)p.nblocks, p.threads, p.smem, st>>>(A);
    return cudaGetLastError() == cudaSuccess ? DGB_OK : DGB_ERR_CUDA;
}

int k2_integrate_table(double *phi, int L, const double *xx, const double *table, int nsteps,
                       int frozen_mask, int nomut_mask, int use_delj, void *ws, size_t ws_bytes,
                       cudaStream_t st)
{
    // one schedule: rows 0 .. nsteps-1 of the table
    K2Args A = {};
    A.ngrids = 1;
    A.L[0] = L;
    A.xx_all = xx;
    A.phi_out = phi;
    A.table = table;
    A.fixed_cnt = nsteps;
    A.frozen_mask = frozen_mask;
    A.nomut_mask = nomut_mask;
    A.nwork = 1;
    A.Lmax = L;
    A.use_delj = use_delj;
    size_t bytes;
    if (ws) {
        const int rc = k2w_launch(A, ws, ws_bytes, 1, true, st);
        if (rc != -1)
            return rc;
    }
    A.gam_smem = k2_smem_fits(L, true, use_delj, &bytes);
    if (!A.gam_smem) {
        if (!k2_smem_fits(L, false, use_delj, &bytes))
            return DGB_ERR_UNSUPPORTED;
        if (!ws || ws_bytes < (size_t)L * L * sizeof(double))
            return DGB_ERR_WORKSPACE;
        A.gam_glob = (double *)ws;
    }
    return k2_launch(A, 1, bytes, st);
}

// Doubles of a split kernel's slice for grids of up to L points, 0 where none
// runs: what a workspace has to hold beyond k_integrate2d's Thomas scratch.
static size_t k2w_slice(int L, bool delj)
{
    return !k2w_fits(L, delj) ? 0 : delj ? k2d_slice_doubles(L) : k2w_slice_doubles(L, true);
}

size_t k2_table_ws_bytes(int L)
{
    return std::max({(size_t)L * L, k2w_slice(L, false), k2w_slice(L, true)}) * sizeof(double);
}

size_t k2_batch_ws_bytes(int Lmax, long nwork)
{
    const int sms = k2_num_sms(), fit = Lmax <= 64 ? 5 : 2;
    const size_t scratch = (size_t)sms * 4 * Lmax * Lmax; // k_integrate2d, up to four CTAs per SM
    const size_t slice = k2w_slice(Lmax, false);
    const long n = std::max<long>(nwork, 1);
    size_t doubles = std::max(
        {scratch, slice * std::min<long>((long)sms * std::min(k2w_per_sm(n, sms), fit), n),
         k2w_slice(Lmax, true) * std::min<long>(sms, n)});
    const int most = slice ? k2w_most_per_sm(Lmax, n, sms, fit) : 0;
    if (most > 1)
        doubles = std::max(doubles, slice * sms * most + K2W_LIVE_BYTES / sizeof(double));
    return 256 + doubles * sizeof(double);
}

// norder: integrate only the work items order[0 .. norder) (<= 0: all);
// reserve_sms: SMs to leave to launches running at the same time (the CTAs
// are capped at (SMs - reserve_sms) x CTAs per SM).
int k2_batch(int ninst, const int *masks, const int *Ls, int ngrids, const double *xx_all,
             const double *phi0_all, double *phi_out, const double *table, const long *row_off,
             const int *row_cnt, int sched_per_grid, const int *order,
             const dgb_settings *settings, void *ws, size_t ws_bytes, cudaStream_t st,
             double *ckpt = nullptr, const long *ckpt_off = nullptr, int ckpt_every = 0,
             int norder = 0, int reserve_sms = 0)
{
    if (ngrids < 1 || ngrids > K2_MAXG || ninst < 1)
        return DGB_ERR_ARG;
    K2Args A = {};
    A.ngrids = ngrids;
    long xo = 0, po = 0, oo = 0;
    int Lmax = 0;
    for (int gi = 0; gi < ngrids; gi++) {
        if (Ls[gi] < 3)
            return DGB_ERR_ARG;
        A.L[gi] = Ls[gi];
        A.xx_off[gi] = xo;
        A.phi0_off[gi] = po;
        A.out_off[gi] = oo;
        xo += Ls[gi];
        po += (long)Ls[gi] * Ls[gi];
        oo += (long)ninst * Ls[gi] * Ls[gi];
        Lmax = std::max(Lmax, Ls[gi]);
    }
    A.xx_all = xx_all;
    A.phi0_all = phi0_all;
    A.phi_out = phi_out;
    A.table = table;
    A.row_off = row_off;
    A.row_cnt = row_cnt;
    A.sched_per_grid = sched_per_grid;
    A.masks = masks;
    A.order = order;
    A.nwork = (norder > 0 && norder < ninst * ngrids) ? norder : ninst * ngrids;
    A.Lmax = Lmax;
    A.use_delj = settings->use_delj_trick;
    A.ckpt = ckpt;
    A.ckpt_off = ckpt_off;
    A.ckpt_every = ckpt_every > 0 ? ckpt_every : 1;
    if (!ws || ws_bytes < 256)
        return DGB_ERR_WORKSPACE;
    A.counter = (int *)ws;
    size_t bytes_s = 0, bytes_g = 0;
    bool fit_s = k2_smem_fits(Lmax, true, A.use_delj, &bytes_s);
    bool fit_g = k2_smem_fits(Lmax, false, A.use_delj, &bytes_g);
    if (!fit_g)
        return DGB_ERR_UNSUPPORTED;
    int nsm = k2_num_sms();
    int occ_s = fit_s ? k2_occupancy(A.use_delj, bytes_s + sizeof(K2Shared)) : 0;
    int occ_g = k2_occupancy(A.use_delj, bytes_g + sizeof(K2Shared));
    size_t slice = (size_t)Lmax * Lmax * sizeof(double);
    // auto: gam in shared memory only when that does not cost CTAs per SM.
    // Measured on the 4096-instance IM batch at pts 80/90/100: gam in the
    // workspace (two CTAs per SM at L = 100, two warps per SMSP) 13.44 s,
    // gam in shared memory (one CTA per SM) 17.11 s; the back substitution
    // prefetches its L2 operands, and the second warp per SMSP fills the FP64
    // pipe's dependency gaps.
    bool use_s = fit_s && occ_s >= occ_g;
    if (settings->gam_placement == 1) {
        if (!fit_s)
            return DGB_ERR_UNSUPPORTED;
        use_s = true;
    } else if (settings->gam_placement == 2) {
        use_s = false;
    }
    int nblocks;
    size_t smem;
    int threads;
    if (use_s) {
        A.gam_smem = 1;
        smem = bytes_s;
        threads = k2_pick_threads(settings, A.use_delj, smem, A.Lmax, occ_s);
        nblocks = nsm * occ_s;
    } else {
        A.gam_smem = 0;
        A.gam_glob = (double *)((char *)ws + 256);
        smem = bytes_g;
        threads = k2_pick_threads(settings, A.use_delj, smem, A.Lmax, occ_g);
        nblocks = (int)std::min<size_t>((ws_bytes - 256) / slice, (size_t)nsm * occ_g);
    }
    if (threads == 0)
        return DGB_ERR_ARG;
    // automatic shape: factors and solves on their own warps
    if (k2w_auto(settings)) {
        if (cudaMemsetAsync(A.counter, 0, sizeof(int), st) != cudaSuccess)
            return DGB_ERR_CUDA;
        const int rc = k2w_launch(A, (char *)ws + 256, ws_bytes - 256,
                                  reserve_sms > 0 ? std::max(1, nsm - reserve_sms) : nsm,
                                  reserve_sms <= 0 && settings->threads != K2_AUTO_SHARED, st);
        if (rc != -1)
            return rc;
    }
    if (nblocks < 1)
        return DGB_ERR_WORKSPACE;
    nblocks = std::min(nblocks, A.nwork);
    if (reserve_sms > 0) {
        const int occ = use_s ? occ_s : occ_g;
        nblocks = std::min(nblocks, std::max(1, (nsm - reserve_sms) * occ));
    }
    if (cudaMemsetAsync(A.counter, 0, sizeof(int), st) != cudaSuccess)
        return DGB_ERR_CUDA;
    return k2_launch(A, nblocks, smem, st, threads);
}

// ------------------------------------------- allocation-free entry point

// Thomas scratch of dgb_integrate2d_noalloc: one L x L array for L up to
// DGB_NOALLOC_MAX_L (128 KB), resident on every GPU that loads the library.
static __device__ __align__(256) double g_noalloc_gam[DGB_NOALLOC_MAX_L * DGB_NOALLOC_MAX_L];

// Device address of g_noalloc_gam per device, looked up with that device
// current (host code must not use the symbol itself).  Only a successful
// lookup is kept: a failed one (e.g. made during stream capture) is retried
// by the next call.
constexpr int NOALLOC_MAXDEV = 64;
static std::mutex g_noalloc_mu;
static double *g_noalloc_ptr[NOALLOC_MAXDEV];

static int noalloc_scratch(double **ptr)
{
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0)
        return DGB_ERR_CUDA;
    if (dev >= NOALLOC_MAXDEV)
        return DGB_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> g(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_gam) != cudaSuccess || !p) {
            cudaGetLastError();
            return DGB_ERR_CUDA;
        }
        g_noalloc_ptr[dev] = (double *)p;
    }
    *ptr = g_noalloc_ptr[dev];
    return DGB_OK;
}

} // namespace dgb

// ------------------------------------------------------------------ C ABI

extern "C" int dgb_sched2d(const dgb_inst2d *insts, int ninst, int ngrids, const double *dx0s,
                           const dgb_settings *settings, long max_steps, int fill, int *row_cnt,
                           const long *row_off, double *table, int *status, void *stream)
{
    if (!insts || ninst < 1 || ngrids < 1 || !dx0s || !settings || max_steps < 1 ||
        fill < 0 || fill > 2 || (fill != 1 && !row_cnt) ||
        (fill && (!row_off || !table || !status)))
        return DGB_ERR_ARG;
    int per_grid = settings->use_old_timestep ? 1 : 0;
    int nsched = per_grid ? ninst * ngrids : ninst;
    // one warp per block (16 schedules, two lanes each): schedules are long
    // serial chains, spread over the SMs
    const long nthreads = 2L * nsched;
    const int nt = 32;
    dgb::k_sched2d<<<(unsigned)((nthreads + nt - 1) / nt), nt, 0, (cudaStream_t)stream>>>(
        insts, nsched, ngrids, per_grid, dx0s, *settings, max_steps, fill, row_cnt, row_off,
        table, status);
    return cudaGetLastError() == cudaSuccess ? DGB_OK : DGB_ERR_CUDA;
}

extern "C" int dgb_batch2d_integrate(const int *masks, int ninst, const int *Ls, int ngrids,
                                     const double *xx_all, const double *phi0_all,
                                     double *phi_out, const double *table, const long *row_off,
                                     const int *row_cnt, const int *order,
                                     const dgb_settings *settings, void *ws, size_t ws_bytes,
                                     void *stream)
{
    if (!Ls || !xx_all || !phi0_all || !phi_out || !table || !row_off || !row_cnt || !order ||
        !settings)
        return DGB_ERR_ARG;
    return dgb::k2_batch(ninst, masks, Ls, ngrids, xx_all, phi0_all, phi_out, table, row_off,
                         row_cnt, settings->use_old_timestep ? 1 : 0, order, settings, ws,
                         ws_bytes, (cudaStream_t)stream);
}

extern "C" int dgb_batch2d_count_steps(const dgb_inst2d *insts, int ninst,
                                       const dgb_settings *settings, long max_steps,
                                       long *steps_out)
{
    if (!insts || !settings || !steps_out || ninst < 0)
        return DGB_ERR_ARG;
    for (int n = 0; n < ninst; n++)
        steps_out[n] = dgb::sched2d_walk(insts[n], *settings, 1e-3, max_steps, nullptr, nullptr);
    return DGB_OK;
}

extern "C" int dgb_integrate2d_noalloc(double *phi, int L, const double *xx, const double *table,
                                       int nsteps, int frozen_mask, int nomut_mask,
                                       int use_delj_trick, void *stream)
{
    if (!phi || !xx || !table || nsteps < 0 || L < 3)
        return DGB_ERR_ARG;
    if (L > DGB_NOALLOC_MAX_L)
        return DGB_ERR_TOO_LARGE;
    if (nsteps == 0)
        return DGB_OK;
    dgb::K2Args A = {};
    size_t bytes = 0;
    // the Thomas scratch in shared memory where it fits beside phi (as
    // dgb_integrate_table does); only larger grids use the static array
    A.gam_smem = dgb::k2_smem_fits(L, true, use_delj_trick != 0, &bytes);
    if (!A.gam_smem) {
        if (!dgb::k2_smem_fits(L, false, use_delj_trick != 0, &bytes))
            return DGB_ERR_UNSUPPORTED;
        int rc = dgb::noalloc_scratch(&A.gam_glob);
        if (rc)
            return rc;
    }
    A.ngrids = 1;
    A.L[0] = L;
    A.xx_all = xx;
    A.phi_out = phi;
    A.table = table;
    A.fixed_cnt = nsteps;
    A.frozen_mask = frozen_mask;
    A.nomut_mask = nomut_mask;
    A.nwork = 1;
    A.Lmax = L;
    A.use_delj = use_delj_trick;
    return dgb::k2_launch(A, 1, bytes, (cudaStream_t)stream);
}

extern "C" int dgb_batch2d_integrate_ckpt(const int *masks, int ninst, const int *Ls, int ngrids,
                                          const double *xx_all, const double *phi0_all,
                                          double *phi_out, const double *table,
                                          const long *row_off, const int *row_cnt,
                                          const int *order, const dgb_settings *settings,
                                          double *ckpt, const long *ckpt_off, int ckpt_every,
                                          void *ws, size_t ws_bytes, void *stream)
{
    if (!Ls || !xx_all || !phi0_all || !phi_out || !table || !row_off || !row_cnt || !order ||
        !settings || !ckpt || !ckpt_off || ckpt_every < 1)
        return DGB_ERR_ARG;
    return dgb::k2_batch(ninst, masks, Ls, ngrids, xx_all, phi0_all, phi_out, table, row_off,
                         row_cnt, settings->use_old_timestep ? 1 : 0, order, settings, ws,
                         ws_bytes, (cudaStream_t)stream, ckpt, ckpt_off, ckpt_every);
}

extern "C" int dgb_batch2d_integrate_ckpt_part(
    const int *masks, int ninst, const int *Ls, int ngrids, const double *xx_all,
    const double *phi0_all, double *phi_out, const double *table, const long *row_off,
    const int *row_cnt, const int *order, int norder, int reserve_sms,
    const dgb_settings *settings, double *ckpt, const long *ckpt_off, int ckpt_every, void *ws,
    size_t ws_bytes, void *stream)
{
    if (!Ls || !xx_all || !phi0_all || !phi_out || !table || !row_off || !row_cnt || !order ||
        !settings || !ckpt || !ckpt_off || ckpt_every < 1 || norder < 1 ||
        norder > ninst * ngrids)
        return DGB_ERR_ARG;
    return dgb::k2_batch(ninst, masks, Ls, ngrids, xx_all, phi0_all, phi_out, table, row_off,
                         row_cnt, settings->use_old_timestep ? 1 : 0, order, settings, ws,
                         ws_bytes, (cudaStream_t)stream, ckpt, ckpt_off, ckpt_every, norder,
                         reserve_sms);
}

extern "C" int dgb_items2d_integrate(const dgb_item2d *items, int nitems, int Lmax,
                                     const double *xx_all, double *phi_out, const double *table,
                                     const long *row_off, const int *row_cnt, const int *order,
                                     const dgb_settings *settings, int one_per_cta, void *ws,
                                     size_t ws_bytes, void *stream)
{
    using namespace dgb;
    if (!items || nitems < 1 || Lmax < 3 || !xx_all || !phi_out || !table || !row_off ||
        !row_cnt || !settings)
        return DGB_ERR_ARG;
    K2Args A = {};
    A.ngrids = 1;
    A.L[0] = Lmax;
    A.xx_all = xx_all;
    A.phi_out = phi_out;
    A.table = table;
    A.row_off = row_off;
    A.row_cnt = row_cnt;
    A.order = order;
    A.nwork = nitems;
    A.Lmax = Lmax;
    A.use_delj = settings->use_delj_trick;
    A.items = items;
    if (!ws || ws_bytes < 256)
        return DGB_ERR_WORKSPACE;
    A.counter = (int *)ws;
    size_t bytes_s = 0, bytes_g = 0;
    bool fit_s = k2_smem_fits(Lmax, true, A.use_delj, &bytes_s);
    if (!k2_smem_fits(Lmax, false, A.use_delj, &bytes_g))
        return DGB_ERR_UNSUPPORTED;
    // gam placement: 0 shared memory when it fits, 1 shared (must fit),
    // 2 the workspace
    if (settings->gam_placement == 1 && !fit_s)
        return DGB_ERR_UNSUPPORTED;
    if (settings->gam_placement == 2)
        fit_s = false;
    else if (settings->gam_placement == 0 && fit_s &&
             k2_occupancy(A.use_delj, bytes_s + sizeof(K2Shared)) <
                 k2_occupancy(A.use_delj, bytes_g + sizeof(K2Shared)))
        fit_s = false; // as in k2_batch: shared memory only if it costs no CTAs per SM
    int nsm = k2_num_sms();
    int nblocks;
    size_t smem = fit_s ? bytes_s : bytes_g;
    size_t slice = (size_t)Lmax * Lmax * sizeof(double);
    int occ = 1;
    const int threads = k2_pick_threads(settings, A.use_delj, smem, Lmax, occ);
    if (threads == 0)
        return DGB_ERR_ARG;
    if (!one_per_cta && k2w_auto(settings)) {
        if (cudaMemsetAsync(A.counter, 0, sizeof(int), (cudaStream_t)stream) != cudaSuccess)
            return DGB_ERR_CUDA;
        const int rc = k2w_launch(A, (char *)ws + 256, ws_bytes - 256, k2_num_sms(),
                                  settings->threads != K2_AUTO_SHARED, (cudaStream_t)stream);
        if (rc != -1)
            return rc;
    }
    if (one_per_cta) {
        // CTA b integrates item order[b] (or b) and retires: no queue
        A.counter = nullptr;
        nblocks = nitems;
        A.gam_smem = fit_s ? 1 : 0;
        if (!fit_s) {
            if ((ws_bytes - 256) / slice < (size_t)nitems)
                return DGB_ERR_WORKSPACE;
            A.gam_glob = (double *)((char *)ws + 256);
        }
        return k2_launch(A, nblocks, smem, (cudaStream_t)stream, threads);
    }
    if (fit_s) {
        A.gam_smem = 1;
        nblocks = nsm * occ;
    } else {
        A.gam_smem = 0;
        nblocks = (int)std::min<size_t>((ws_bytes - 256) / slice, (size_t)nsm * occ);
        A.gam_glob = (double *)((char *)ws + 256);
    }
    if (nblocks < 1)
        return DGB_ERR_WORKSPACE;
    nblocks = std::min(nblocks, nitems);
    if (cudaMemsetAsync(A.counter, 0, sizeof(int), (cudaStream_t)stream) != cudaSuccess)
        return DGB_ERR_CUDA;
    return k2_launch(A, nblocks, smem, (cudaStream_t)stream, threads);
}

extern "C" int dgb_probe_split2d(int Lmax, long nwork, int use_delj_trick, size_t ws_bytes,
                                 int *ctas, int *keep_a)
{
    using namespace dgb;
    if (Lmax < 3 || nwork < 1 || !ctas || !keep_a)
        return DGB_ERR_ARG;
    K2WPlan p;
    if (ws_bytes < 256 ||
        !k2w_plan(Lmax, use_delj_trick != 0, nwork, ws_bytes - 256, k2_num_sms(), true, p))
        return DGB_ERR_UNSUPPORTED;
    *ctas = (int)p.nblocks;
    *keep_a = p.keep_a;
    return DGB_OK;
}

extern "C" int dgb_sched2d_host(const dgb_inst2d *insts, int ninst,
                                const dgb_settings *settings, long max_steps, double dx0,
                                int *row_cnt, const long *row_off, double *table, int *status)
{
    if (!insts || ninst < 0 || !settings || max_steps < 1 || (!table && !row_cnt) ||
        (table && (!row_off || !status)))
        return DGB_ERR_ARG;
    for (int n = 0; n < ninst; n++) {
        int err = 0;
        long c = dgb::sched2d_walk(insts[n], *settings, dx0, max_steps,
                                   table ? table + row_off[n] * dgb::K2_ROW : nullptr, &err);
        if (!table)
            row_cnt[n] = (int)c;
        else
            status[n] |= err;
    }
    return DGB_OK;
}

namespace dgb {
int preload_integrate2d()
{
    return preload(k_integrate2d<false>) + preload(k_integrate2d<true>) +
           preload(k2w_live) + preload(k_integrate2d_ws<1, true, true>) +
           preload(k_integrate2d_ws<2, true, true>) + preload(k2w_kernel<1>(true)) +
           preload(k2w_kernel<2>(true)) + preload(k2w_kernel<3>(true)) +
           preload(k2w_kernel<4>(true)) + preload(k2w_kernel<5>(true)) +
           preload(k2w_kernel<1>(false)) + preload(k2w_kernel<2>(false)) +
           preload(k2w_kernel<3>(false)) + preload(k2w_kernel<4>(false)) +
           preload(k2w_kernel<5>(false)) + preload(k_integrate2d_delj<1>) +
           preload(k_integrate2d_delj<2>) + preload(k_integrate2d_delj<3>) +
           preload(k_integrate2d_delj<4>) + preload(k_integrate2d_delj<5>) + preload(k_sched2d);
}
} // namespace dgb
