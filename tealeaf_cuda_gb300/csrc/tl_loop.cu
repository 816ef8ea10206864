// tl_loop.cu -- whole FP64 iterations: the fused passes of the device-resident
// solves, and the kernels that run many iterations in one launch.
//
// CG in two passes an iteration instead of three (tea_leaf_cg.cuknl:43-161):
//   pass 1  u += alpha p, p' = z + beta p, w = A p', sum p'.w
//   pass 2  r -= alpha w, z = M^-1 r, sum r.z, the exit test
// alpha and beta of pass 1 are those of the iteration before (0 in the
// first), so the u and p updates read the old p once and p' is never read
// back: 12 FP64 instructions and 112 bytes a cell and iteration (jac_diag)
// instead of 12 and 128.  The neighbours' p' are computed again from z and p
// (p' goes to the other of two buffers); a last pass brings u and p up to
// date.  Every value is that of the one-piece kernels, bit for bit.
#include "tl_loop.cuh"

namespace tl {

namespace {

// pass 2 on a run (BodyCgUr without u).  HBM-bound (24 bytes a cell, 40 with
// jac_diag); a row's registers are loaded again, for the row four further
// down, as soon as they are used.
template <int PC, class Ready>
__device__ __forceinline__ void cg_pass2(const Geo &g, const CgArgs &a, int i0, int jb, int je, AlphaBeta &ab,
                                         Ready ready, double &acc) {
    constexpr bool DIAG = PC == TL_PREC_JAC_DIAG, BLOCK = PC == TL_PREC_JAC_BLOCK;
    const int i = i0 + (threadIdx.x & 31);
    const bool own = i < g.nx;
    const int64_t P = g.pitch;
    int64_t c = (int64_t)(i + g.h) + (int64_t)(jb + g.h) * P;
    // per row w, r and Mi; the strip's factors
    double w[4], r[4], mi[4];
    StripFactors fac;
    auto load_row = [&](int k, int row, int64_t at) {
        if (own && row < je) {
            w[k] = __ldcg(a.w + at);
            r[k] = __ldcg(a.r + at);
            if (DIAG) mi[k] = a.mi[at];
        }
    };
#pragma unroll
    for (int k = 0; k < 4; ++k) load_row(k, jb + k, c + k * P);
    if (BLOCK && own) load_factors(a, g, c, jb, je, fac);
    if (!ready() || !own) return;
    for (int j0 = jb; j0 < je; j0 += kStrip) {
        const int m = min(kStrip, je - j0);
        double rv[4], zv[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            rv[k] = k < m ? fma(-ab.alpha, w[k], r[k]) : 0.0;
            if (k < m) a.r[c + k * P] = rv[k];
            if (DIAG) zv[k] = rv[k] * mi[k];
        }
        if (BLOCK) {
            strip_solve(fac, rv, zv);
            if (j0 + kStrip < je) load_factors(a, g, c + kStrip * P, j0 + kStrip, je, fac);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k < m) {
                if (PC != TL_PREC_NONE) a.z[c + k * P] = zv[k];
                acc = fma(rv[k], PC == TL_PREC_NONE ? rv[k] : zv[k], acc);
            }
            load_row(k, j0 + kStrip + k, c + (kStrip + k) * P);
        }
        c += kStrip * P;
    }
}

// the passes as kernels of their own
template <bool FIVE>
__global__ void __launch_bounds__(kGroupThreads, 4) k_cg_pass1(Geo g, CgArgs a, RedCtx red) {
    if (*(volatile const int *)red.done) return;
    const bool sel = red.sc->p_sel != 0;
    const double *pin = sel ? a.p1 : a.p0;
    double *pout = sel ? a.p0 : a.p1;
    AlphaBeta ab{red.sc->alpha, red.sc->beta};
    double acc[1] = {0.0};
    for_runs(g, blockIdx.x, threadIdx.x >> 5, [&](int i0, int jb, int je) {
        cg_pass1<4, FIVE>(g, a, pin, pout, i0, jb, je, ab, [] { return true; }, acc[0]);
    });
    grid_reduce<1>(acc, red, g.sms);
}

// (block-Jacobi: 4 CTAs a multiprocessor, in two even goes.  At the 80 registers
// that let six in the other two had it to themselves: 101.2 and 215.7 us at 2600^2
// and 4096^2 cells, 101.8 and 204.8 with four, 103.7 and 209.7 with eight of 64.)
template <int PC>
__global__ void __launch_bounds__(kGroupThreads, PC == TL_PREC_JAC_BLOCK ? 4 : 8) k_cg_pass2(Geo g, CgArgs a, RedCtx red) {
    if (*(volatile const int *)red.done) return;
    AlphaBeta ab{red.sc->alpha, 0.0};
    double acc[1] = {0.0};
    for_runs(g, blockIdx.x, threadIdx.x >> 5, [&](int i0, int jb, int je) {
        cg_pass2<PC>(g, a, i0, jb, je, ab, [] { return true; }, acc[0]);
    });
    grid_reduce<1>(acc, red, g.sms);
}

template <int PC, class Shape>
__global__ void __launch_bounds__(Shape::kThreads, 1) k_cg_loop(LoopArgs L, CgArgs a) {
    if (*(volatile const int *)&L.sc->done) return;
    __shared__ LoopShared S;
    if (!loop_begin(L, S)) return;
    if (threadIdx.x >= blockDim.x - 32) {
        for (int it = 0; it < L.iters; ++it) {
            loop_meet<1>(L, S, kEpiCgPw);
            if (S.stalled) break;
            loop_meet<1>(L, S, kEpiCgUrFinish);
            if (S.stalled || S.sc.done) break;
        }
    } else {
        for (int it = 0;; ++it) {
            AlphaBeta ab{0.0, 0.0};
            if (it > 0) loop_met();
            const bool sel = S.sc.p_sel != 0;
            const double *pin = sel ? a.p1 : a.p0;
            double *pout = sel ? a.p0 : a.p1;
            bool asked = false, go = false;
            // the scalars of the iteration before: beta and the exit test
            auto ready1 = [&] {
                if (!asked) {
                    asked = true;
                    if (it > 0) loop_scalars();
                    go = !S.sc.done && !S.stalled && it < L.iters;
                    ab.alpha = S.sc.alpha;
                    ab.beta = S.sc.beta;
                }
                return go;
            };
            loop_pass<1>(L, S, [&](int i0, int jb, int je, double (&acc)[1]) {
                cg_pass1<Shape::kAhead, false>(L.g, a, pin, pout, i0, jb, je, ab, ready1, acc[0]);
            });
            if (!ready1()) break;
            loop_arrive<1>(L, S);
            loop_met();
            asked = false;
            auto ready2 = [&] {
                if (!asked) {
                    asked = true;
                    loop_scalars();
                    go = !S.stalled;
                    ab.alpha = S.sc.alpha;
                }
                return go;
            };
            loop_pass<1>(L, S, [&](int i0, int jb, int je, double (&acc)[1]) {
                cg_pass2<PC>(L.g, a, i0, jb, je, ab, ready2, acc[0]);
            });
            if (!ready2()) break;
            loop_arrive<1>(L, S);
        }
    }
    loop_end(L, S);
}

// u += alpha p, p = src + beta p with the last iteration's alpha and beta,
// from whichever buffer holds p into the first
__global__ void __launch_bounds__(kGroupThreads) k_cg_finish(Geo g, CgArgs a, const DevScalars *__restrict__ sc) {
    const double *pin = sc->p_sel ? a.p1 : a.p0;
    const double alpha = sc->alpha, beta = sc->beta;
    const bool swapped = a.rs && sc->p_sel;  // mixed PPCG: r and r_store take turns as p's buffers do
    const int lane = threadIdx.x & 31;
    for_runs(g, blockIdx.x, threadIdx.x >> 5, [&](int i0, int jb, int je) {
        const int i = i0 + lane;
        if (i >= g.nx) return;
        for (int j0 = jb; j0 < je; j0 += kStrip) {
            const int m = min(kStrip, je - j0);
            const int64_t base = (int64_t)(i + g.h) + (int64_t)(j0 + g.h) * g.pitch;
            double pv[4], uv[4], sv[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < m) {
                    const int64_t c = base + (int64_t)k * g.pitch;
                    pv[k] = pin[c];
                    uv[k] = a.u[c];
                    sv[k] = a.src[c];
                }
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < m) {
                    const int64_t c = base + (int64_t)k * g.pitch;
                    a.u[c] = fma(alpha, pv[k], uv[k]);
                    a.p0[c] = fma(beta, pv[k], sv[k]);
                    if (swapped) {
                        const double r = a.rs[c];
                        a.rs[c] = a.r[c];
                        a.r[c] = r;
                    }
                }
        }
    });
}

// ------------------------------------------- Chebyshev and PPCG inner steps

// One step of either polynomial method (tea_leaf_cheby.cuknl:71-152,
// tea_leaf_ppcg.cuknl:154-244) in one pass instead of two: with x the field
// the operator acts on,
//   Chebyshev  r = u0 - A u, p = al p + be M^-1 r, u' = u + p       (x = u)
//   PPCG       rtemp -= A sd, sd' = al sd + be M^-1 rtemp, utemp += sd'  (x = sd)
// x' goes to the other of two buffers, so that the neighbours still read x.
// The residual r = u0 - A u (+ r.r) is the same walk without an update.
// FP64-bound: 10 (none), 11 (diag) or 14 (block) instructions a cell; a pass
// of its own for u += p or the sd update read and wrote 24 to 48 bytes a cell
// more and waited once more for the grid.
enum StepMode { kStepCheby, kStepPpcg, kStepPpcgLast, kStepResidual };

struct StepArgs {
    double *x0, *x1;   // u or sd: the two buffers
    double *f;         // u0 or rtemp
    double *q;         // p or utemp
    double *r, *rs, *z, *w;
    const double *kx, *ky, *dg, *mi, *cp, *bfp, *rd;
    const double *alphas, *betas;
    int inner;
};

struct StepCoef {
    double al, be;
    bool norm;  // Chebyshev: the sum r.r is wanted
};

// one step on a run; ready(): waits for the coefficients
template <int PC, StepMode MODE, int D, class Ready>
__device__ __forceinline__ void step_pass(const Geo &g, const StepArgs &a, const double *__restrict__ xin,
                                          double *__restrict__ xout, int i0, int jb, int je, StepCoef &co, Ready ready,
                                          double (&acc)[MODE == kStepPpcgLast ? 2 : 1]) {
    constexpr bool BLOCK = PC == TL_PREC_JAC_BLOCK, DIAG = PC == TL_PREC_JAC_DIAG;
    constexpr bool CHEBY = MODE == kStepCheby, LAST = MODE == kStepPpcgLast;
    // cells around the field that x is read from: the residual's u has its halo, which
    // reflective boundaries couple in
    constexpr int H = MODE == kStepResidual ? 1 : 0;
    const int lane = threadIdx.x & 31, i = i0 + lane;
    const bool own = i < g.nx, ownx = i < g.nx + H;
    const int64_t P = g.pitch;
    int64_t c = (int64_t)(i + g.h) + (int64_t)(jb + g.h) * P;
    const int ek = (lane >> 1) & 3, ecol = (lane & 1) ? i0 + kWarpCols : i0 - 1;
    const bool eon = lane < 8 && ecol >= -H && ecol < g.nx + H, fon = lane < 8 && (lane & 1) && ecol <= g.nx;
    int64_t e = (int64_t)(ecol + g.h) + (int64_t)(jb + ek + g.h) * P;
    // a row's Kx, diag, f and q (and Mi), the next row's x and Ky; x and Kx beside
    double xl[D], ky[D], kx[D], dg[D], f[D], q[D], mi[D], ex, ef;
    auto load_row = [&](int k, int row, int64_t at) {
        const bool in = own && row < je;
        xl[k] = ownx && row < je && row + 1 < g.ny + H ? __ldcg(xin + at + P) : 0.0;
        ky[k] = in ? a.ky[at + P] : 0.0;
        kx[k] = in ? a.kx[at] : 0.0;
        dg[k] = in ? a.dg[at] : 0.0;
        f[k] = in ? __ldcg(a.f + at) : 0.0;
        if (!BLOCK && MODE != kStepResidual) q[k] = in ? __ldcg(a.q + at) : 0.0;
        if (DIAG) mi[k] = in ? a.mi[at] : 0.0;
    };
    auto load_edge = [&](int j0) {
        const bool v = j0 + ek < je;
        ex = v && eon ? __ldcg(xin + e) : 0.0;
        ef = v && fon ? a.kx[e] : 0.0;
    };
    double xm = ownx && jb > -H ? __ldcg(xin + c - P) : 0.0, x0 = ownx ? __ldcg(xin + c) : 0.0;
    double kyv = own ? a.ky[c] : 0.0;
#pragma unroll
    for (int k = 0; k < D; ++k) load_row(k, jb + k, c + k * P);
    load_edge(jb);
    if (!ready()) return;
    for (int j0 = jb; j0 < je; j0 += kStrip) {
        const double edge = ex, face = ef;
        e += kStrip * P;
        load_edge(j0 + kStrip);
        double rv[4], xc[4] = {}, qv[4] = {};
        // the row's new values from its r and z
        auto finish = [&](int k, double r, double z, double m) {
            const int64_t at = c + k * P;
            if (MODE == kStepResidual) {
                a.r[at] = r;
                acc[0] = fma(r, r, acc[0]);
                return;
            }
            double be_z;
            if (PC == TL_PREC_NONE || BLOCK) be_z = co.be * z;
            else if (CHEBY) be_z = (co.be * m) * r;
            else be_z = (co.be * r) * m;
            if (CHEBY) {
                const double p = fma(co.al, qv[k], be_z);
                a.q[at] = p;
                xout[at] = xc[k] + p;
                if (co.norm) acc[0] = fma(r, r, acc[0]);
            } else {
                const double sd = fma(co.al, xc[k], be_z), ut = qv[k] + sd;
                a.f[at] = r;
                xout[at] = sd;
                a.q[at] = ut;
                if (LAST) {
                    const double rr = __ldcg(a.r + at);
                    a.z[at] = ut;
                    acc[0] = fma(rr - __ldcg(a.rs + at), ut, acc[0]);
                    acc[LAST ? 1 : 0] = fma(rr, ut, acc[LAST ? 1 : 0]);
                }
            }
        };
#pragma unroll
        for (int kb = 0; kb < 4; kb += D) {
            double x[D + 2], t[D], b[D];
            x[0] = xm;
            x[1] = x0;
#pragma unroll
            for (int d = 0; d < D; ++d) x[d + 2] = xl[d];
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const int k = kb + d;
                double xw = __shfl_up_sync(0xffffffffu, x[d + 1], 1), xe = __shfl_down_sync(0xffffffffu, x[d + 1], 1);
                double kxe = __shfl_down_sync(0xffffffffu, kx[d], 1);
                const double ew = __shfl_sync(0xffffffffu, edge, 2 * k), ee = __shfl_sync(0xffffffffu, edge, 2 * k + 1);
                const double fe = __shfl_sync(0xffffffffu, face, 2 * k + 1);
                if (lane == 0) xw = ew;
                if (lane == 31) {
                    xe = ee;
                    kxe = fe;
                }
                // the face east of the last column
                if (i == g.nx - 1 && lane < 31 && j0 + k < je) kxe = a.kx[c + k * P + 1];
                t[d] = (d == 0 ? kyv : ky[d > 0 ? d - 1 : 0]) * x[d];
                b[d] = fma(kxe, xe, kx[d] * xw);
            }
#pragma unroll
            for (int d = 0; d < D; ++d) t[d] = fma(ky[d], x[d + 2], t[d]);
#pragma unroll
            for (int d = 0; d < D; ++d) t[d] = fma(dg[d], x[d + 1], -t[d]);
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const int k = kb + d;
                rv[k] = f[d] - (t[d] - b[d]);
                xc[k] = x[d + 1];
                if (!BLOCK && MODE != kStepResidual) qv[k] = q[d];
            }
            if (!BLOCK) {
#pragma unroll
                for (int d = 0; d < D; ++d)
                    if (own && j0 + kb + d < je) finish(kb + d, rv[kb + d], rv[kb + d], DIAG ? mi[d] : 0.0);
            }
            xm = x[D];
            x0 = x[D + 1];
            kyv = ky[D - 1];
#pragma unroll
            for (int d = 0; d < D; ++d) load_row(d, j0 + kb + d + D, c + (kb + d + D) * P);
        }
        if (BLOCK && own) {
            // the factors and q are loaded only now: 30 registers that the
            // stencil has no room for
            double zv[4];
            const int m = min(kStrip, je - j0);
            StripFactors fac;
            asm volatile("" ::: "memory");
            load_factors(a, g, c, j0, je, fac);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                qv[k] = k < m ? __ldcg(a.q + c + k * P) : 0.0;
                if (k >= m) rv[k] = 0.0;
            }
            strip_solve(fac, rv, zv);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < m) finish(k, rv[k], zv[k], 0.0);
        }
        c += kStrip * P;
    }
}

// PPCG, after p.w: r_store = r, r -= alpha w, and the start of the inner steps,
// rtemp = r, sd = utemp = M^-1 r / theta (tea_leaf_ppcg.cuknl:58-89; M^-1 r
// itself is never read).  HBM-bound: 56 to 88 bytes a cell.
template <int PC, class Ready>
__device__ __forceinline__ void ppcg_pass2(const Geo &g, const StepArgs &a, int i0, int jb, int je, double theta_r,
                                           double &alpha, Ready ready) {
    constexpr bool BLOCK = PC == TL_PREC_JAC_BLOCK, DIAG = PC == TL_PREC_JAC_DIAG;
    const int i = i0 + (threadIdx.x & 31);
    const bool own = i < g.nx;
    const int64_t P = g.pitch;
    int64_t c = (int64_t)(i + g.h) + (int64_t)(jb + g.h) * P;
    double w[4], r[4], mi[4];
    StripFactors fac;
    auto load_row = [&](int k, int row, int64_t at) {
        if (own && row < je) {
            w[k] = __ldcg(a.w + at);
            r[k] = __ldcg(a.r + at);
            if (DIAG) mi[k] = a.mi[at];
        }
    };
#pragma unroll
    for (int k = 0; k < 4; ++k) load_row(k, jb + k, c + k * P);
    if (BLOCK && own) load_factors(a, g, c, jb, je, fac);
    if (!ready() || !own) return;
    for (int j0 = jb; j0 < je; j0 += kStrip) {
        const int m = min(kStrip, je - j0);
        double rv[4], zv[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            rv[k] = k < m ? fma(-alpha, w[k], r[k]) : 0.0;
            zv[k] = DIAG ? rv[k] * mi[k] : rv[k];
        }
        if (BLOCK) {
            strip_solve(fac, rv, zv);
            if (j0 + kStrip < je) load_factors(a, g, c + kStrip * P, j0 + kStrip, je, fac);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k < m) {
                const int64_t at = c + k * P;
                const double sd = zv[k] * theta_r;
                a.rs[at] = r[k];
                a.r[at] = rv[k];
                a.f[at] = rv[k];
                a.x0[at] = sd;
                a.q[at] = sd;
            }
            load_row(k, j0 + kStrip + k, c + (kStrip + k) * P);
        }
        c += kStrip * P;
    }
}

// (all 8 CTAs of a multiprocessor at once: block-Jacobi at 4096^2 cells 260 -> 220 us)
template <int PC>
__global__ void __launch_bounds__(kGroupThreads, 8) k_ppcg_pass2(Geo g, StepArgs a, const DevScalars *sc) {
    if (*(volatile const int *)&sc->done) return;
    const double theta_r = 1.0 / sc->theta;
    double alpha = sc->alpha;
    for_runs(g, blockIdx.x, threadIdx.x >> 5, [&](int i0, int jb, int je) {
        ppcg_pass2<PC>(g, a, i0, jb, je, theta_r, alpha, [] { return true; });
    });
}

// step 1..inner of PPCG (x starts in the first buffer), or a Chebyshev step
template <int PC, StepMode MODE>
__global__ void __launch_bounds__(kGroupThreads, 4) k_step(Geo g, StepArgs a, int step, RedCtx red) {
    if (*(volatile const int *)red.done) return;
    constexpr int NV = MODE == kStepCheby ? 1 : MODE == kStepPpcgLast ? 2 : 0;
    constexpr bool CHEBY = MODE == kStepCheby;
    const int st = CHEBY ? red.sc->cheby_calc_steps : step;
    const bool odd = CHEBY ? red.sc->p_sel != 0 : (step - 1) & 1;
    StepCoef co{a.alphas[st - 1], a.betas[st - 1], CHEBY && cheby_reads_norm(red.sc)};
    double acc[NV > 0 ? NV : 1];
#pragma unroll
    for (int v = 0; v < (NV > 0 ? NV : 1); ++v) acc[v] = 0.0;
    for_runs(g, blockIdx.x, threadIdx.x >> 5, [&](int i0, int jb, int je) {
        step_pass<PC, MODE, 4>(g, a, odd ? a.x1 : a.x0, odd ? a.x0 : a.x1, i0, jb, je, co, [] { return true; }, acc);
    });
    if (NV > 0) grid_reduce<NV>(acc, red, g.sms);
}

__global__ void __launch_bounds__(kGroupThreads, 4) k_residual(Geo g, StepArgs a, RedCtx red) {
    StepCoef co{};
    double acc[1] = {0.0};
    for_runs(g, blockIdx.x, threadIdx.x >> 5, [&](int i0, int jb, int je) {
        step_pass<TL_PREC_NONE, kStepResidual, 4>(g, a, a.x0, nullptr, i0, jb, je, co, [] { return true; }, acc);
    });
    if (red.epi != kEpiNone) grid_reduce<1>(acc, red, g.sms);
}

template <int PC, class Shape>
__global__ void __launch_bounds__(Shape::kThreads, 1) k_cheby_loop(LoopArgs L, StepArgs a) {
    if (*(volatile const int *)&L.sc->done) return;
    __shared__ LoopShared S;
    __shared__ struct {
        StepCoef co;
        bool sel, go;
    } T[2];  // what step `it` needs, in T[it & 1]
    if (!loop_begin(L, S)) return;
    const bool control = threadIdx.x >= blockDim.x - 32;
    // the next step's coefficients (the control warp's first lane)
    auto next = [&](int it) {
        const DevScalars *sc = &S.sc;
        auto &t = T[it & 1];
        t.go = !sc->done && !S.stalled && it < L.iters;
        t.sel = sc->p_sel != 0;
        t.co.norm = cheby_reads_norm(sc);
        if (t.go) {
            t.co.al = a.alphas[sc->cheby_calc_steps - 1];
            t.co.be = a.betas[sc->cheby_calc_steps - 1];
        }
    };
    if (control && (threadIdx.x & 31) == 0) next(0);
    __syncthreads();
    if (control) {
        for (int it = 0; T[it & 1].go; ++it) {
            if (T[it & 1].co.norm) {
                loop_meet<1>(L, S, kEpiCheby, [&] { next(it + 1); });
            } else {
                // no sum to wait for: the epilogue runs beside the pass
                if ((threadIdx.x & 31) == 0) {
                    RedCtx red{};
                    red.sc = &S.sc;
                    red.epi = kEpiCheby;
                    double none[1] = {0.0};
                    run_epilogue(red, none, 1);
                    next(it + 1);
                }
                __syncwarp();
                loop_meet<0>(L, S, kEpiNone);
                if (S.stalled) break;
            }
        }
    } else {
        bool norm = false;  // of the step before: its successor's scalars come with the sum
        for (int it = 0;; ++it) {
            if (it > 0) loop_met();
            if (norm) loop_scalars();
            const bool sel = T[it & 1].sel, go = T[it & 1].go;
            if (!go || S.stalled) break;
            StepCoef co = T[it & 1].co;
            norm = co.norm;
            loop_pass<1>(L, S, [&](int i0, int jb, int je, double (&acc)[1]) {
                step_pass<PC, kStepCheby, Shape::kAhead>(L.g, a, sel ? a.x1 : a.x0, sel ? a.x0 : a.x1, i0, jb, je, co,
                                                         [] { return true; }, acc);
            });
            if (norm) loop_arrive<1>(L, S);
            else loop_arrive<0>(L, S);
        }
    }
    loop_end(L, S);
}

template <int PC, class Shape>
__global__ void __launch_bounds__(Shape::kThreads, 1) k_ppcg_loop(LoopArgs L, StepArgs a, CgArgs cg) {
    if (*(volatile const int *)&L.sc->done) return;
    __shared__ LoopShared S;
    if (!loop_begin(L, S)) return;
    const double theta_r = 1.0 / S.sc.theta;
    if (threadIdx.x >= blockDim.x - 32) {
        for (int it = 0; it < L.iters; ++it) {
            loop_meet<1>(L, S, kEpiPpcgPw);
            if (S.stalled) break;
            for (int st = 0; st < a.inner && !S.stalled; ++st) loop_meet<0>(L, S, kEpiNone);
            if (S.stalled) break;
            loop_meet<2>(L, S, kEpiPpcgZrFinish);
            if (S.stalled || S.sc.done) break;
        }
    } else {
        auto yes = [] { return true; };
        for (int it = 0;; ++it) {
            AlphaBeta ab{0.0, 0.0};
            if (it > 0) loop_met();
            const bool sel = S.sc.p_sel != 0;
            const double *pin = sel ? cg.p1 : cg.p0;
            double *pout = sel ? cg.p0 : cg.p1;
            bool asked = false, go = false;
            auto ready1 = [&] {
                if (!asked) {
                    asked = true;
                    if (it > 0) loop_scalars();
                    go = !S.sc.done && !S.stalled && it < L.iters;
                    ab.alpha = S.sc.alpha;
                    ab.beta = S.sc.beta;
                }
                return go;
            };
            loop_pass<1>(L, S, [&](int i0, int jb, int je, double (&acc)[1]) {
                cg_pass1<Shape::kAhead, false>(L.g, cg, pin, pout, i0, jb, je, ab, ready1, acc[0]);
            });
            if (!ready1()) break;
            loop_arrive<1>(L, S);
            loop_met();
            asked = false;
            auto ready2 = [&] {
                if (!asked) {
                    asked = true;
                    loop_scalars();
                    go = !S.stalled;
                    ab.alpha = S.sc.alpha;
                }
                return go;
            };
            loop_pass<0>(L, S, [&](int i0, int jb, int je, double (&)[1]) {
                ppcg_pass2<PC>(L.g, a, i0, jb, je, theta_r, ab.alpha, ready2);
            });
            if (!ready2()) break;
            for (int st = 1; st <= a.inner; ++st) {
                loop_arrive<0>(L, S);
                StepCoef co{a.alphas[st - 1], a.betas[st - 1], false};
                loop_met();
                if (S.stalled) break;
                const double *xin = st & 1 ? a.x0 : a.x1;
                double *xout = st & 1 ? a.x1 : a.x0;
                if (st < a.inner)
                    loop_pass<0>(L, S, [&](int i0, int jb, int je, double (&acc)[1]) {
                        step_pass<PC, kStepPpcg, Shape::kAhead>(L.g, a, xin, xout, i0, jb, je, co, yes, acc);
                    });
                else
                    loop_pass<2>(L, S, [&](int i0, int jb, int je, double (&acc)[2]) {
                        step_pass<PC, kStepPpcgLast, Shape::kAhead>(L.g, a, xin, xout, i0, jb, je, co, yes, acc);
                    });
            }
            if (S.stalled) break;
            loop_arrive<2>(L, S);
        }
    }
    loop_end(L, S);
}

// what the loops leave to do: u (Chebyshev) from whichever buffer holds it into
// the first, and w = A u, r = u0 - w of the last step, whose u is in the
// other buffer; (PPCG) an odd number of inner steps leaves sd in the second
__global__ void __launch_bounds__(kGroupThreads) k_cheby_finish(Geo g, StepArgs a, const DevScalars *__restrict__ sc,
                                                                 bool copy) {
    const bool sel = sc->p_sel != 0;
    const double *now = sel ? a.x1 : a.x0, *old = sel ? a.x0 : a.x1;
    const int lane = threadIdx.x & 31;
    for_runs(g, blockIdx.x, threadIdx.x >> 5, [&](int i0, int jb, int je) {
        const int i = i0 + lane;
        if (i >= g.nx) return;
        for (int j = jb; j < je; ++j) {
            const int64_t c = (int64_t)(i + g.h) + (int64_t)(j + g.h) * g.pitch;
            if (copy) {
                a.x0[c] = now[c];
            } else {
                // the halo of the second buffer is not set: 0 there, as the faces
                const double n = j + 1 < g.ny ? old[c + g.pitch] : 0.0, s = j > 0 ? old[c - g.pitch] : 0.0;
                const double e = i + 1 < g.nx ? old[c + 1] : 0.0, w = i > 0 ? old[c - 1] : 0.0;
                const double t = fma(a.ky[c + g.pitch], n, a.ky[c] * s);
                const double b = fma(a.kx[c + 1], e, a.kx[c] * w);
                const double ax = fma(a.dg[c], old[c], -t) - b;
                a.w[c] = ax;
                a.r[c] = a.f[c] - ax;
            }
        }
    });
}

// ----------------------------------------------------------------- Jacobi

// u' = (u0 + sum K u_nb) / (1 + sum K), sum |u' - u| (BodyJacobi, from one
// buffer to the other instead of with a copy of u first)
__device__ __forceinline__ void jacobi_pass(const Geo &g, const StepArgs &a, const double *__restrict__ xin,
                                            double *__restrict__ xout, int i0, int jb, int je, double &acc) {
    const int i = i0 + (threadIdx.x & 31);
    if (i >= g.nx) return;
    const int64_t P = g.pitch;
    auto at = [&](int64_t c, bool in) { return in ? __ldcg(xin + c) : 0.0; };
    for (int j0 = jb; j0 < je; j0 += kStrip) {
        const int64_t c0 = (int64_t)(i + g.h) + (int64_t)(j0 + g.h) * P;
        double x[6], e[4], w[4], f[4], kx[4], kxe[4], ky[5];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const int row = j0 + k - 1;
            x[k] = at(c0 + (k - 1) * P, row >= 0 && row < g.ny && row <= je);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (j0 + k < je) {
                const int64_t c = c0 + k * P;
                e[k] = at(c + 1, i + 1 < g.nx);
                w[k] = at(c - 1, i > 0);
                f[k] = a.f[c];
                kx[k] = a.kx[c];
                kxe[k] = a.kx[c + 1];
                if (k == 0) ky[0] = a.ky[c];
                ky[k + 1] = a.ky[c + P];
            }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (j0 + k < je) {
                double num = fma(kxe[k], e[k], f[k]);
                num = fma(kx[k], w[k], num);
                num = fma(ky[k + 1], x[k + 2], num);
                num = fma(ky[k], x[k], num);
                const double den = (1.0 + (kx[k] + kxe[k])) + (ky[k] + ky[k + 1]);
                const double v = num / den;
                xout[c0 + k * P] = v;
                acc += fabs(v - x[k + 1]);
            }
    }
}

__global__ void __launch_bounds__(kGroupThreads) k_jacobi(Geo g, StepArgs a, RedCtx red) {
    if (*(volatile const int *)red.done) return;
    const bool sel = red.sc->p_sel != 0;
    double acc[1] = {0.0};
    for_runs(g, blockIdx.x, threadIdx.x >> 5, [&](int i0, int jb, int je) {
        jacobi_pass(g, a, sel ? a.x1 : a.x0, sel ? a.x0 : a.x1, i0, jb, je, acc[0]);
    });
    grid_reduce<1>(acc, red, g.sms);
}

template <class Shape>
__global__ void __launch_bounds__(Shape::kThreads, 1) k_jacobi_loop(LoopArgs L, StepArgs a) {
    if (*(volatile const int *)&L.sc->done) return;
    __shared__ LoopShared S;
    if (!loop_begin(L, S)) return;
    if (threadIdx.x >= blockDim.x - 32) {
        for (int it = 0; it < L.iters; ++it) {
            loop_meet<1>(L, S, kEpiJacobiStep);
            if (S.stalled || S.sc.done) break;
        }
    } else {
        for (int it = 0;; ++it) {
            if (it > 0) {
                loop_met();
                loop_scalars();
            }
            if (S.sc.done || S.stalled || it >= L.iters) break;
            const bool sel = S.sc.p_sel != 0;
            loop_pass<1>(L, S, [&](int i0, int jb, int je, double (&acc)[1]) {
                jacobi_pass(L.g, a, sel ? a.x1 : a.x0, sel ? a.x0 : a.x1, i0, jb, je, acc[0]);
            });
            loop_arrive<1>(L, S);
        }
    }
    loop_end(L, S);
}

StepArgs step_args(Chunk *c) {
    StepArgs a;
    const bool pp = c->cfg.solver == TL_SOLVER_PPCG;
    a.x0 = pp ? c->sd : c->u;
    a.x1 = pp ? c->sd_alt : c->un;
    a.f = pp ? c->rtemp : c->u0;
    a.q = pp ? c->utemp : c->p;
    a.r = c->r;
    a.rs = c->r_store;
    a.z = c->z;
    a.w = c->w;
    a.kx = c->kx;
    a.ky = c->ky;
    a.dg = c->diag;
    a.mi = c->mi;
    a.cp = c->cp;
    a.bfp = c->bfp;
    a.rd = c->rdiag;
    a.alphas = c->ch_alphas;
    a.betas = c->ch_betas;
    a.inner = c->cfg.ppcg_inner_steps;
    return a;
}

}  // namespace

int launch_residual(Chunk *c, int epi) {
    StepArgs a = step_args(c);
    a.x0 = c->u;
    a.f = c->u0;
    return launch_named(c, "residual", [&] {
        k_residual<<<c->g.groups, kGroupThreads, 0, c->stream>>>(c->g, a, red_ctx(c, epi, false));
    });
}

int launch_cg_pass1(Chunk *c, bool ppcg) {
    const bool five = ppcg && c->cfg.precision == TL_PRECISION_MIXED;
    return launch_named(c, ppcg ? "ppcg_pw" : "cg_pw", [&] {
        const RedCtx red = red_ctx(c, ppcg ? kEpiPpcgPw : kEpiCgPw, true);
        if (five) k_cg_pass1<true><<<c->g.groups, kGroupThreads, 0, c->stream>>>(c->g, cg_args(c, ppcg), red);
        else k_cg_pass1<false><<<c->g.groups, kGroupThreads, 0, c->stream>>>(c->g, cg_args(c, ppcg), red);
    });
}

int launch_cg_pass2(Chunk *c) {
    return by_precond(c, [&](auto pc) {
        return launch_named(c, "cg_rz", [&] {
            k_cg_pass2<pc()><<<c->g.groups, kGroupThreads, 0, c->stream>>>(c->g, cg_args(c),
                                                                          red_ctx(c, kEpiCgUrFinish, true));
        });
    });
}

int launch_cg_finish(Chunk *c, bool ppcg) {
    return launch_named(c, ppcg ? "ppcg_up" : "cg_up", [&] {
        k_cg_finish<<<c->g.groups, kGroupThreads, 0, c->stream>>>(c->g, cg_args(c, ppcg), c->sc);
    });
}

int launch_cg_loop(Chunk *c) {
    return by_precond(c, [&](auto pc) {
        return launch_loop(c, k_cg_loop<pc(), ShapeSmall>, k_cg_loop<pc(), ShapeLarge>, cg_args(c));
    });
}

int launch_cheby_step(Chunk *c) {
    return by_precond(c, [&](auto pc) {
        return launch_named(c, "cheby_step", [&] {
            k_step<pc(), kStepCheby><<<c->g.groups, kGroupThreads, 0, c->stream>>>(c->g, step_args(c), 0,
                                                                                  red_ctx(c, kEpiCheby, true));
        });
    });
}

int launch_cheby_loop(Chunk *c) {
    return by_precond(c, [&](auto pc) {
        return launch_loop(c, k_cheby_loop<pc(), ShapeSmall>, k_cheby_loop<pc(), ShapeLarge>, step_args(c));
    });
}

int launch_cheby_finish(Chunk *c) {
    int rc = TL_OK;
    for (int copy = 0; copy < 2 && !rc; ++copy)
        rc = launch_named(c, "cheby_finish", [&] {
            k_cheby_finish<<<c->g.groups, kGroupThreads, 0, c->stream>>>(c->g, step_args(c), c->sc, copy != 0);
        });
    return rc;
}

int ppcg_alloc(Chunk *c) {
    if (c->sd_alt) return TL_OK;
    void *p;
    const int rc = dalloc(c, &p, c->alloc_elems * sizeof(double));
    if (rc == TL_ERR_ALLOC) {
        // the single pieces need no second buffer; the chunk keeps to them, as
        // its graph of iterations holds them from now on
        cudaGetLastError();
        set_error("%s", "");
        c->no_sd_alt = true;
        return TL_OK;
    }
    if (rc) return rc;
    c->sd_alt = (double *)p + c->lead;
    return TL_OK;
}

int launch_ppcg_pass2(Chunk *c) {
    return by_precond(c, [&](auto pc) {
        return launch_named(c, "ppcg_r", [&] {
            k_ppcg_pass2<pc()><<<c->g.groups, kGroupThreads, 0, c->stream>>>(c->g, step_args(c), c->sc);
        });
    });
}

int launch_ppcg_step(Chunk *c, int step) {
    return by_precond(c, [&](auto pc) {
        return launch_named(c, "ppcg_step", [&] {
            if (step < c->cfg.ppcg_inner_steps)
                k_step<pc(), kStepPpcg><<<c->g.groups, kGroupThreads, 0, c->stream>>>(c->g, step_args(c), step,
                                                                                     red_ctx(c, kEpiNone, true));
            else
                k_step<pc(), kStepPpcgLast><<<c->g.groups, kGroupThreads, 0, c->stream>>>(
                    c->g, step_args(c), step, red_ctx(c, kEpiPpcgZrFinish, true));
        });
    });
}

int launch_ppcg_loop(Chunk *c) {
    return by_precond(c, [&](auto pc) {
        return launch_loop(c, k_ppcg_loop<pc(), ShapeSmall>, k_ppcg_loop<pc(), ShapeLarge>, step_args(c),
                           cg_args(c, true));
    });
}

int launch_ppcg_finish(Chunk *c) {
    const int rc = launch_cg_finish(c, true);
    if (rc || c->cfg.precision == TL_PRECISION_MIXED || c->cfg.ppcg_inner_steps % 2 == 0) return rc;
    return launch_copy(c, c->sd, c->sd_alt, false);
}

int launch_jacobi_step(Chunk *c) {
    return launch_named(c, "jacobi", [&] {
        k_jacobi<<<c->g.groups, kGroupThreads, 0, c->stream>>>(c->g, step_args(c), red_ctx(c, kEpiJacobiStep, true));
    });
}

int launch_jacobi_loop(Chunk *c) {
    return launch_loop(c, k_jacobi_loop<ShapeSmall>, k_jacobi_loop<ShapeLarge>, step_args(c));
}

int launch_jacobi_finish(Chunk *c) {
    return launch_named(c, "jacobi_finish", [&] {
        k_cheby_finish<<<c->g.groups, kGroupThreads, 0, c->stream>>>(c->g, step_args(c), c->sc, true);
    });
}

// Short runs: the loop saves the launches (2 to 13 an iteration) and their
// waits; in long ones 16 warps a multiprocessor do not keep HBM as busy as the
// passes' own kernels, and those of 96 registers spill (tl_loop.cuh).
// Microseconds an iteration, loop / graph of passes (PPCG with 10 inner steps):
//                      500^2 (run 1)  1080^2 (2)   1540^2 (4)   2060^2 (7)    2200^2 (8)
//   CG, none           14.1 / 24.8    35 / 50      65 / 82      106 / 126     122 / 137
//   CG, jac_diag       15.1 / 25.4    41 / 55      78 / 88      128 / 136     148 / 148
//   CG, block          17.2 / 28.2    49 / 68      94 / 110     154 / 173     173 / 191
//   Chebyshev, none    10.9 / 18.8    31 / 44      60 / 73      100 / 116     114 / 127
//   Chebyshev, diag    11.6 / 19.4    34 / 47      67 / 79      111 / 125     126 / 137
//   Chebyshev, block   13.1 / 21.6    40 / 53      80 / 92      133 / 145     150 / 161
//   PPCG, none         105 / 129      317 / 354    629 / 660    1052 / 1089   1200 / 1228
//   PPCG, jac_diag     113 / 136      347 / 386    685 / 733    1146 / 1202   1303 / 1350
//   Jacobi             15.1 / 19.8    46 / 53      88 / 95      152 / 158     173 / 176
// (PPCG with block-Jacobi: ppcg_loop_pays)
bool loop_pays(const Chunk *c) {
    return c->loop_ok && !c->profiling && !c->cfg.reflective_boundary && c->g.run <= kLoopRun;
}

}  // namespace tl
