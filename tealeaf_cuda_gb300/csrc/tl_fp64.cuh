// tl_fp64.cuh -- device code shared by the FP64 kernels that run one piece of
// an iteration each (tl_kernels.cu) and those that run whole iterations
// (tl_loop.cu): what the last step of a reduction does with the sums, the
// order of the sums, the 5-point operator.
//
// Order of a grid-wide sum.  A run is 32 columns, one a lane, by some 4-row
// strips, taken from the top down by one warp; the field is cut into bands of
// strips, as few as the device's warps take in one go, so runs side by
// side are at the same rows at the same time and find their neighbours' values
// in the caches.  Bands of more than kLoopRun strips are as many as there are
// warps for, of two lengths that differ by one: with ceil(nstrips / bands) in all of
// them 7 % of the warps had nothing at 2600^2 cells (CG with block-Jacobi 268 us
// an iteration, now 238).  Four runs side by side are a set, a group's 4 warps.  Group q
// of G takes the sets q, q + G, ...; a lane adds up its cells in that order,
// row by row.  The group adds its warps lane by lane, (w0 + w1) + (w2 + w3), then its lanes in
// an xor butterfly.  The groups q, q + S, q + 2S, ... are slot q of S = one a
// multiprocessor, added in that order; then one warp adds the slots: lane l
// takes l, l + 32, ... in order, and a butterfly ends it.  Every kernel keeps
// this order, whether its groups are CTAs of their own or parts of a larger
// one, so all of them give the same bits.
//
// Why 4 warps and lane-wise sums: a multiprocessor finishes two FP64 lanes a
// clock, so an FP64 instruction of a warp costs it 16 clocks.  This order takes
// 8 of them a group of 128 columns' strips (a butterfly in each warp and a
// serial sum over the warps took 48 for twice the cells).
#pragma once

#include "tl_internal.cuh"
#include "tl_device.cuh"

namespace tl {

// ------------------------------------------------------------ epilogues

static __device__ void finish_iteration(DevScalars *s, bool allow_switch) {
    // tea_solve.f90:400-417: error = sqrt|error|; exit when below eps*||r0||
    double e = sqrt(fabs(s->error));
    s->error = e;
    if (fabs(e) < s->eps * s->initial_residual) {
        s->done = kConverged;
        s->n_exit = s->n;
        return;
    }
    if (isnan(e)) {  // breakdown: the reference would carry NaN to max_iters
        s->done = kBreakdown;
        s->n_exit = s->n;
        return;
    }
    s->old_error = e;
    s->n += 1;
    if (s->n > s->max_iters) {
        s->done = kMaxIters;
        s->n_exit = s->n;
        return;
    }
    if (allow_switch && (s->solver == TL_SOLVER_CHEBYSHEV || s->solver == TL_SOLVER_PPCG)) {
        // tea_solve.f90:157-171, evaluated at the top of the next iteration
        bool sw = (!s->first && s->solver == TL_SOLVER_PPCG && s->n > 1) ||
                  (fabs(s->old_error) <= s->epslim && s->n >= s->presteps);
        if (sw) s->done = kSwitch;
    }
}

// tea_solve.f90:266-283: the residual is read every 10th iteration after the
// estimated count
__device__ __forceinline__ bool cheby_reads_norm(const DevScalars *s) { return s->n >= s->est_itc && s->n % 10 == 0; }

static __device__ void run_epilogue(const RedCtx &red, const double *tot, int nv) {
    DevScalars *s = red.sc;
    switch (red.epi) {
    case kEpiStore:
        for (int v = 0; v < nv; ++v) s->sum[v] = tot[v];
        break;
    case kEpiResid:
        s->sum[0] = tot[0];
        s->old_error = tot[0];
        s->initial_residual = sqrt(fabs(tot[0]));
        break;
    case kEpiRro:
        s->sum[0] = tot[0];
        s->rro = tot[0];
        break;
    case kEpiCgW:
        s->pw = tot[0];
        s->alpha = s->rro / s->pw;
        red.cg_alphas[s->n] = s->alpha;
        break;
    case kEpiCgPw:
        s->pw = tot[0];
        s->alpha = s->rro / s->pw;
        red.cg_alphas[s->n] = s->alpha;
        s->p_sel ^= 1;
        break;
    case kEpiCgUr:
        s->rrn = tot[0];
        s->beta = s->rrn / s->rro;
        red.cg_betas[s->n] = s->beta;
        s->error = s->rrn;
        s->rro = s->rrn;
        break;
    case kEpiCgUrFinish:
        s->rrn = tot[0];
        s->beta = s->rrn / s->rro;
        red.cg_betas[s->n] = s->beta;
        s->error = s->rrn;
        s->rro = s->rrn;
        {
            // sqrt|error| < eps r0 needs no square root (600 clocks) while
            // |error| is well above its square
            const double lim = s->eps * s->initial_residual, lim2 = lim * lim;
            if (s->solver == TL_SOLVER_CG && lim2 > 1e-280 && fabs(s->rrn) > lim2 * (1.0 + 1e-9) &&
                s->n < s->max_iters)
                s->n += 1;
            else
                finish_iteration(s, true);
        }
        break;
    case kEpiFinish:
        finish_iteration(s, true);
        break;
    case kEpiFinishNoSwitch:
        finish_iteration(s, false);
        break;
    case kEpiPw:
        s->pw = tot[0];
        break;
    case kEpiPpcgZr:
        s->rro = tot[0];
        s->alpha = s->rro / s->pw;
        break;
    case kEpiPwZr:
        s->pw = tot[0];
        s->rro = tot[1];
        s->alpha = s->rro / s->pw;
        break;
    case kEpiPpcgRrn:
        s->rrn = tot[0];
        s->beta = s->rrn / s->rro;
        s->error = s->rrn;
        s->rro = s->rrn;
        s->ppcg_iters += 1;
        break;
    case kEpiPpcgPw:
        s->pw = tot[0];
        s->alpha = s->rro / s->pw;
        s->p_sel ^= 1;
        break;
    case kEpiPpcgZrFinish:
        s->rrn = tot[0];
        s->beta = s->rrn / s->rro;
        s->error = s->rrn;
        s->rro = tot[1];
        s->ppcg_iters += 1;
        finish_iteration(s, false);
        break;
    case kEpiWzZrFinish:
        s->rrn = -s->alpha * tot[0];
        s->beta = s->rrn / s->rro;
        s->error = s->rrn;
        s->rro = tot[1];
        s->ppcg_iters += 1;
        finish_iteration(s, false);
        break;
    case kEpiZrFinish:
        s->rro = tot[0];
        finish_iteration(s, false);
        break;
    case kEpiCheby:
        if (cheby_reads_norm(s)) s->error = s->rr = tot[0];
        s->cheby_calc_steps += 1;
        s->p_sel ^= 1;
        finish_iteration(s, false);
        break;
    case kEpiChebyNorm:
        s->rr = tot[0];
        break;
    case kEpiChebyFinish:
        if (cheby_reads_norm(s)) s->error = s->rr;  // cheby_calc_steps += 1 at :284
        s->cheby_calc_steps += 1;
        finish_iteration(s, false);
        break;
    case kEpiJacobiStep:
        s->p_sel ^= 1;
        s->error = tot[0];
        finish_iteration(s, false);
        break;
    case kEpiJacobi:
        s->error = tot[0];
        finish_iteration(s, false);
        break;
    default:
        break;
    }
}

// the strips of this warp of a group, in order: f(first column, first row of
// the run, row after its last)
template <class F>
__device__ __forceinline__ void for_runs(const Geo &g, int group, int warp, F f) {
    for (int t = group; t < g.sets; t += g.groups) {
        const int r = t * kGroupWarps + warp;
        if (r >= g.runs) break;
        const int b = r / g.tiles_x, tx = r - b * g.tiles_x;
        const int s0 = b * g.band + min(b, g.longer), s1 = min(s0 + g.band + (b < g.longer), g.nstrips);
        f(tx * kWarpCols, s0 * kStrip, min(s1 * kStrip, g.ny));
    }
}

// xor butterfly over the warp's lanes
__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
    return x;
}

// the sum over a group's 4 warps; sh: [4][32] of the group; every thread of
// the group's CTA has stored its value and passed a barrier.  Called by one
// whole warp, and the same in all its lanes.
__device__ __forceinline__ double group_sum(const double (*sh)[32], int lane) {
    return warp_sum((sh[0][lane] + sh[1][lane]) + (sh[2][lane] + sh[3][lane]));
}

// grid-wide sums of one-group CTAs; the last CTA (a ticket, nobody waits)
// adds the partials, a warp a sum if there are several, and runs the epilogue
template <int NV>
__device__ __forceinline__ void grid_reduce(double (&acc)[NV > 0 ? NV : 1], const RedCtx &red, int sms) {
    constexpr int N = NV > 0 ? NV : 1;
    __shared__ double sh[N][kGroupWarps][32];
    __shared__ double slot[kMaxSlots];
    __shared__ int is_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int v = 0; v < NV; ++v) sh[v][warp][lane] = acc[v];
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const double t = group_sum(sh[v], lane);
            if (lane == 0) red.partials[v * kMaxRedBlocks + blockIdx.x] = t;
        }
        if (lane == 0) {
            __threadfence();
            is_last = atomicAdd(red.counter, 1u) == gridDim.x - 1;
        }
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    const int groups = gridDim.x, slots = groups < sms ? groups : sms;
    double tot[N];
    if (NV > 1) {
        // a warp a sum
        static_assert(NV <= kGroupWarps, "a warp a sum");
        __shared__ double all[N];
        if (warp < NV) {
            const double *part = red.partials + warp * kMaxRedBlocks;
            double t = 0.0;
            for (int c = lane; c < slots; c += 32) {
                double s = __ldcg(&part[c]);
                for (int q = c + slots; q < groups; q += slots) s += __ldcg(&part[q]);
                t = c == lane ? s : t + s;
            }
            t = warp_sum(t);
            if (lane == 0) all[warp] = t;
        }
        __syncthreads();
#pragma unroll
        for (int v = 0; v < NV; ++v) tot[v] = all[v];
    } else if (NV == 1) {
        for (int c = threadIdx.x; c < slots; c += kGroupThreads) {
            double t = __ldcg(&red.partials[c]);
            for (int q = c + slots; q < groups; q += slots) t += __ldcg(&red.partials[q]);
            slot[c] = t;
        }
        __syncthreads();
        if (warp == 0) {
            double t = lane < slots ? slot[lane] : 0.0;
            for (int c = lane + 32; c < slots; c += 32) t += slot[c];
            tot[0] = warp_sum(t);
        }
    }
    if (threadIdx.x == 0) {
        run_epilogue(red, tot, NV);
        __threadfence();
        *red.counter = 0u;
    }
}

// ------------------------------------------------------------- helpers

// diag(A) of tea_leaf_common.cuknl:137-139: (1 + (Ky_n + Ky_c)) + (Kx_e + Kx_c)
__device__ __forceinline__ double diag_at(const double *__restrict__ kx,
                                          const double *__restrict__ ky, int64_t i, int pitch) {
    return (1.0 + (ky[i + pitch] + ky[i])) + (kx[i + 1] + kx[i]);
}

// A x on the m rows of a strip (tea_leaf_common.cuknl:28-34).  xc receives
// the centre values.  Rows beyond m are neither read nor written.
template <class X>
__device__ __forceinline__ void strip_apply(const double *__restrict__ kx,
                                            const double *__restrict__ ky,
                                            const double *__restrict__ dg, int pitch,
                                            int64_t base, int m, X x, double (&xc)[4],
                                            double (&ax)[4]) {
    double xr[6];   // rows -1..4
    double kyr[5];  // faces of rows 0..4
#pragma unroll
    for (int k = -1; k <= 4; ++k)
        if (k <= m) xr[k + 1] = x(base + (int64_t)k * pitch);
#pragma unroll
    for (int k = 0; k <= 4; ++k)
        if (k <= m) kyr[k] = ky[base + (int64_t)k * pitch];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (k < m) {
            const int64_t i = base + (int64_t)k * pitch;
            const double kxc = kx[i], kxe = kx[i + 1];
            const double xw = x(i - 1), xe = x(i + 1);
            const double diag = dg[i];
            const double a = fma(kyr[k + 1], xr[k + 2], kyr[k] * xr[k]);
            const double b = fma(kxe, xe, kxc * xw);
            ax[k] = fma(diag, xr[k + 1], -a) - b;
            xc[k] = xr[k + 1];
        }
    }
}

struct LoadX {
    const double *__restrict__ f;
    __device__ __forceinline__ double operator()(int64_t i) const { return f[i]; }
};

__device__ __forceinline__ double coef(const double *p, double v) { return p ? *p : v; }

}  // namespace tl
