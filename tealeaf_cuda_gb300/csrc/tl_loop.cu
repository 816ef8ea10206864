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
//
// One launch runs `iters` iterations: one CTA a multiprocessor (co-resident:
// a cooperative launch), a tile group always on the same CTA, the grid's CTAs
// meeting at each sum.  A CTA stores its partial sum, counts itself in (one
// atomic on one word) and polls that word; then every CTA adds the same
// partials in the same order and runs the scalar epilogue on its own copy of
// the scalars.  A wait that runs out (about two seconds) stops the solve with
// an error.  Measured on GB300, in clocks: one meeting 2450 to 3200 at any
// number of CTAs (an FP64 dependency is 64, a trip to L2 400); letting
// every CTA poll every other's flag took 7000 with 152 of them, the last
// arriver's adding and publishing for all 6900, clusters with a leader each
// 10000.
#include <math.h>
#include <string.h>

#include <type_traits>

#include "tl_fp64.cuh"

namespace tl {

namespace {

constexpr long long kLoopWaitCycles = 4000000000LL;  // ~2 s
// A CTA has its multiprocessor's groups (up to 8) in rounds of L.per_round at a
// time.  One more warp, the control warp, runs the meetings and the scalar
// code, so that the others' registers hold nothing but their passes.
constexpr int kLoopWarps = kGroupsPerSm * kGroupWarps;
struct LoopArgs {
    Geo g;
    DevScalars *sc;
    double *partials;        // [2][kMaxSlots][kLoopSums]
    unsigned int *arrived;   // CTAs that have come to a meeting, over all launches of a solve
    unsigned int *base;      // the value of `arrived` when the launch began
    double *cg_alphas, *cg_betas;
    int depth;      // groups of the busiest CTA
    int per_round;  // groups a CTA takes at a time
    int iters;
};

constexpr int kLoopSums = 2;  // sums a meeting carries at most

struct LoopShared {
    DevScalars sc;
    double sh[kLoopSums][kLoopWarps][32];
    double part[kLoopSums][kGroupsPerSm];
    unsigned int target;  // `arrived` when every CTA has come to the meeting
    int parity;
    int stalled;
};

// named barriers (0 is __syncthreads) of the CTA's warps
enum LoopBarrier {
    kBarSums = 1,  // passing warps only: their sums are in shared memory
    kBarIn,        // the groups' sums are there: the control warp goes to the meeting
    kBarMet,       // every CTA has come: what they stored may be read
    kBarScalars    // the epilogue has run: the scalars may be read
};
__device__ __forceinline__ void bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// A meeting of all CTAs that carries NV sums in the order of tl_fp64.cuh.  The
// passing warps put their lanes' sums into S.sh, go on to the next pass with
// met() before its first loads and wait for the scalars once those are on
// their way, so that the loads' trip to L2 and the serial scalar code overlap.
template <int NV>
__device__ __forceinline__ void loop_arrive(const LoopArgs &L, LoopShared &S) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, passing = blockDim.x - 32;
    if (NV > 0) {
        bar_sync(kBarSums, passing);
        if (warp < L.depth) {  // one warp a group
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const double t = group_sum(&S.sh[v][warp * kGroupWarps], lane);
                if (lane == 0) S.part[v][warp] = t;
            }
        }
    }
    bar_arrive(kBarIn, blockDim.x);
}
__device__ __forceinline__ void loop_met() { bar_sync(kBarMet, blockDim.x); }
__device__ __forceinline__ void loop_scalars() { bar_sync(kBarScalars, blockDim.x); }

// the control warp's part (NV = 0: no sums, no epilogue, and nobody waits for
// scalars)
struct Nothing {
    __device__ __forceinline__ void operator()() const {}
};
template <int NV, class Then = Nothing>
__device__ __forceinline__ void loop_meet(const LoopArgs &L, LoopShared &S, int epi, Then then = Then()) {
    const int lane = threadIdx.x & 31, slots = gridDim.x, cta = blockIdx.x;
    bar_sync(kBarIn, blockDim.x);
    if (lane == 0) {
        double *mine = L.partials + ((size_t)S.parity * kMaxSlots + cta) * kLoopSums;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            double t = S.part[v][0];
            for (int q = 1; q * slots + cta < L.g.groups; ++q) t += S.part[v][q];
            __stcg(mine + v, t);
        }
        if (slots > 1) {
            // release: what the CTA stored before (the barrier above) and the partials
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(L.arrived) : "memory");
            const long long t0 = clock64();
            for (;;) {
                unsigned int v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(L.arrived) : "memory");
                if ((int)(v - S.target) >= 0) break;
                if (clock64() - t0 > kLoopWaitCycles) {
                    S.stalled = 1;
                    break;
                }
            }
        }
    }
    __syncwarp();
    bar_arrive(kBarMet, blockDim.x);
    if (NV == 0) {
        if (lane == 0) S.target += slots;
        __syncwarp();
        return;
    }
    const double *p = L.partials + (size_t)S.parity * kMaxSlots * kLoopSums;
    double tot[NV > 0 ? NV : 1];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        double t = 0.0;
#pragma unroll 1
        for (int c0 = lane; c0 < slots; c0 += 5 * 32) {  // 152 slots: one trip
            double x[5];
#pragma unroll
            for (int k = 0; k < 5; ++k)
                if (c0 + 32 * k < slots) x[k] = __ldcg(p + (c0 + 32 * k) * kLoopSums + v);
#pragma unroll
            for (int k = 0; k < 5; ++k)
                if (c0 + 32 * k < slots) t = c0 + 32 * k == lane ? x[k] : t + x[k];
        }
        tot[v] = warp_sum(t);
    }
    if (lane == 0) {
        RedCtx red{};
        red.sc = &S.sc;
        red.epi = epi;
        red.cg_alphas = L.cg_alphas;
        red.cg_betas = L.cg_betas;
        run_epilogue(red, tot, NV);
        S.target += slots;
        S.parity ^= 1;
        then();
    }
    __syncwarp();
    bar_arrive(kBarScalars, blockDim.x);
}

__device__ __forceinline__ void loop_begin(const LoopArgs &L, LoopShared &S) {
    static_assert(sizeof(DevScalars) % sizeof(int) == 0, "copied by words");
    for (int k = threadIdx.x; k < (int)(sizeof(DevScalars) / sizeof(int)); k += blockDim.x)
        ((int *)&S.sc)[k] = ((const int *)L.sc)[k];
    if (threadIdx.x == 0) {
        S.target = *L.base + gridDim.x;
        S.parity = 0;
        S.stalled = 0;
    }
    __syncthreads();
}

// CTA 0 hands the scalars on, and the arrivals counted so far (every CTA has
// read both: it has come to the same last meeting)
__device__ __forceinline__ void loop_end(const LoopArgs &L, LoopShared &S) {
    __syncthreads();
    if (S.stalled) {
        if (threadIdx.x == 0) *(volatile int *)&L.sc->done = kStalled;
        return;
    }
    if (blockIdx.x != 0) return;
    for (int k = threadIdx.x; k < (int)(sizeof(DevScalars) / sizeof(int)); k += blockDim.x)
        ((int *)L.sc)[k] = ((const int *)&S.sc)[k];
    if (threadIdx.x == 0 && gridDim.x > 1) *L.base = S.target - gridDim.x;
}

// a pass over the runs of this (passing) warp of a loop kernel's CTA, round by
// round: f(first column, first row, row after the last, sums)
template <int NV, class F>
__device__ __forceinline__ void loop_pass(const LoopArgs &L, LoopShared &S, F f) {
    const int lane = threadIdx.x & 31, warp = (int)(threadIdx.x >> 5);
#pragma unroll 1
    for (int q = warp / kGroupWarps; q < L.depth; q += L.per_round) {
        const int group = q * (int)gridDim.x + (int)blockIdx.x;
        double acc[NV > 0 ? NV : 1];
#pragma unroll
        for (int v = 0; v < (NV > 0 ? NV : 1); ++v) acc[v] = 0.0;
        if (group < L.g.groups)
            for_runs(L.g, group, warp & (kGroupWarps - 1), [&](int i0, int jb, int je) { f(i0, jb, je, acc); });
#pragma unroll
        for (int v = 0; v < NV; ++v) S.sh[v][q * kGroupWarps + (warp & (kGroupWarps - 1))][lane] = acc[v];
    }
}

// ------------------------------------------------------------------- CG

struct CgArgs {
    double *u, *r, *z, *w;
    double *p0, *p1;    // p's two buffers (DevScalars::p_sel)
    const double *src;  // z, or r without a preconditioner
    const double *kx, *ky, *dg, *mi, *cp, *bfp, *rd;
    double *rs;         // r_store, where the last pass sets it
};

// the block-Jacobi factors of the strip whose first row is at c (row j0)
template <class A>
__device__ __forceinline__ void load_factors(const A &a, const Geo &g, int64_t c, int j0, int je, StripFactors &f) {
    const int64_t P = g.pitch;
    f.b0 = a.dg[c];
    f.y0 = a.rd[c - (int64_t)(j0 + g.h) * P + (int64_t)(j0 / kStrip) * P];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const bool in = j0 + k + 1 < je;
        f.ky[k] = in ? a.ky[c + (k + 1) * P] : 0.0;
        f.bf[k] = in ? a.bfp[c + (k + 1) * P] : 0.0;
        f.cp[k] = in ? a.cp[c + k * P] : 0.0;
    }
}

struct AlphaBeta {
    double alpha, beta;
};

// pass 1 on a run.  FP64-bound: 37 instructions a strip (9 a cell and the
// column beside the warp's).  A row's registers are loaded again, for the row
// D further down, as soon as they are used.  D = 4: a strip's loads all leave
// at once and its rows are computed side by side, for the few warps of a small
// grid (a warp alone has an FP64 result every 64 clocks if it does not wait
// for the one before); D = 2 where 16 warps share the registers.  Arrays that
// other CTAs write during the launch are read past L1 (__ldcg).  ready():
// waits for alpha and beta, false if the solve has ended; called once the
// first loads are on their way.
// FIVE: the operator as one product and four fused subtractions (5 FP64
// instructions instead of 6; another rounding, so only for the mixed-precision
// solve, which has no reference bits to keep)
template <int D, bool FIVE, class Ready>
__device__ __forceinline__ void cg_pass1(const Geo &g, const CgArgs &a, const double *__restrict__ pin,
                                         double *__restrict__ pout, int i0, int jb, int je, AlphaBeta &ab, Ready ready,
                                         double &acc) {
    const int lane = threadIdx.x & 31, i = i0 + lane;
    const bool own = i < g.nx;
    const int64_t P = g.pitch;
    int64_t c = (int64_t)(i + g.h) + (int64_t)(jb + g.h) * P;  // row 0 of the strip
    // beside the warp's columns: lane 2k has the west column of row k, lane
    // 2k + 1 the east one (and its face)
    const int ek = (lane >> 1) & 3, ecol = (lane & 1) ? i0 + kWarpCols : i0 - 1;
    const bool eon = lane < 8 && ecol >= 0 && ecol < g.nx, fon = lane < 8 && (lane & 1) && ecol <= g.nx;
    int64_t e = (int64_t)(ecol + g.h) + (int64_t)(jb + ek + g.h) * P;
    // a row's u, Kx and diag, the next row's z, p and Ky; z, p and Kx beside
    double z[D], p[D], ky[D], u[D], kx[D], dg[D], ez, ep, ef;
    auto load_row = [&](int k, int row, int64_t at) {
        const bool in = own && row < je, next = in && row + 1 < g.ny;
        z[k] = next ? __ldcg(a.src + at + P) : 0.0;
        p[k] = next ? __ldcg(pin + at + P) : 0.0;
        ky[k] = in ? a.ky[at + P] : 0.0;
        kx[k] = in ? a.kx[at] : 0.0;
        dg[k] = in ? a.dg[at] : 0.0;
        u[k] = in ? __ldcg(a.u + at) : 0.0;
    };
    auto load_edge = [&](int j0) {
        const bool v = j0 + ek < je;
        ez = v && eon ? __ldcg(a.src + e) : 0.0;
        ep = v && eon ? __ldcg(pin + e) : 0.0;
        ef = v && fon ? a.kx[e] : 0.0;
    };
    // rows -1 and 0 (0 outside the field, where the faces are 0)
    const bool up = own && jb > 0;
    double xm = up ? __ldcg(a.src + c - P) : 0.0, x0 = own ? __ldcg(a.src + c) : 0.0;
    double pm = up ? __ldcg(pin + c - P) : 0.0, p0 = own ? __ldcg(pin + c) : 0.0;
    double kyv = own ? a.ky[c] : 0.0;
#pragma unroll
    for (int k = 0; k < D; ++k) load_row(k, jb + k, c + k * P);
    load_edge(jb);
    if (!ready()) return;
    xm = fma(ab.beta, pm, xm);
    x0 = fma(ab.beta, p0, x0);
    for (int j0 = jb; j0 < je; j0 += kStrip) {
        const double edge = fma(ab.beta, ep, ez), face = ef;
        e += kStrip * P;
        load_edge(j0 + kStrip);
#pragma unroll
        for (int kb = 0; kb < 4; kb += D) {
            // D rows side by side: x of rows kb - 1 .. kb + D
            double x[D + 2], po[D], t[D], b[D];
            x[0] = xm;
            x[1] = x0;
            po[0] = p0;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                x[d + 2] = fma(ab.beta, p[d], z[d]);
                if (d + 1 < D) po[d + 1] = p[d];
            }
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
                const double kyc = d == 0 ? kyv : ky[d > 0 ? d - 1 : 0];
                if (FIVE) {
                    t[d] = fma(-kyc, x[d], dg[d] * x[d + 1]);
                    t[d] = fma(-kxe, xe, t[d]);
                    t[d] = fma(-kx[d], xw, t[d]);
                } else {
                    t[d] = kyc * x[d];
                    b[d] = fma(kxe, xe, kx[d] * xw);
                }
            }
#pragma unroll
            for (int d = 0; d < D; ++d) t[d] = fma(FIVE ? -ky[d] : ky[d], x[d + 2], t[d]);
            if (!FIVE) {
#pragma unroll
                for (int d = 0; d < D; ++d) t[d] = fma(dg[d], x[d + 1], -t[d]);
#pragma unroll
                for (int d = 0; d < D; ++d) t[d] = t[d] - b[d];
            }
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const int64_t at = c + (kb + d) * P;
                if (own && j0 + kb + d < je) {
                    pout[at] = x[d + 1];
                    a.w[at] = t[d];
                    a.u[at] = fma(ab.alpha, po[d], u[d]);
                    acc = fma(x[d + 1], t[d], acc);
                }
            }
            xm = x[D];
            x0 = x[D + 1];
            p0 = p[D - 1];
            kyv = ky[D - 1];
#pragma unroll
            for (int d = 0; d < D; ++d) load_row(d, j0 + kb + d + D, c + (kb + d + D) * P);
        }
        c += kStrip * P;
    }
}

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

template <int PC>
__global__ void __launch_bounds__(kGroupThreads, PC == TL_PREC_JAC_BLOCK ? 6 : 8) k_cg_pass2(Geo g, CgArgs a, RedCtx red) {
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
    loop_begin(L, S);
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

// ppcg: the outer iteration of PPCG, whose z is never r itself
CgArgs cg_args(Chunk *c, bool ppcg = false) {
    CgArgs a;
    a.u = c->u;
    a.r = c->r;
    a.z = c->z;
    a.w = c->w;
    a.p0 = c->p;
    a.p1 = c->un;
    a.src = ppcg || c->cfg.precond != TL_PREC_NONE ? c->z : c->r;
    a.kx = c->kx;
    a.ky = c->ky;
    a.dg = c->diag;
    a.mi = c->mi;
    a.cp = c->cp;
    a.bfp = c->bfp;
    a.rd = c->rdiag;
    a.rs = ppcg && c->cfg.precision == TL_PRECISION_MIXED ? c->r_store : nullptr;
    return a;
}

template <class F>
int launch_named(Chunk *c, const char *name, F &&launch) {
    int slot = -1;
    if (c->profiling && !c->capturing) prof_begin(c, name, &slot);
    launch();
    if (slot >= 0) prof_end(c, slot);
    c->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, name);
    return TL_OK;
}

// u += alpha p, p = src + beta p with the last iteration's alpha and beta,
// from whichever buffer holds p into the first
__global__ void __launch_bounds__(kGroupThreads) k_cg_finish(Geo g, CgArgs a, const DevScalars *__restrict__ sc) {
    const double *pin = sc->p_sel ? a.p1 : a.p0;
    const double alpha = sc->alpha, beta = sc->beta;
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
                    // mixed PPCG does without r_store: the r before the last update
                    if (a.rs) a.rs[c] = fma(alpha, a.w[c], a.r[c]);
                }
        }
    });
}

LoopArgs loop_args(Chunk *c) {
    LoopArgs L;
    L.g = c->g;
    L.sc = c->sc;
    L.partials = c->loop_partials;
    L.arrived = c->loop_arrived;
    L.base = c->loop_arrived + 1;
    L.cg_alphas = c->cg_alphas;
    L.cg_betas = c->cg_betas;
    // a launch of some tens of milliseconds at most
    const long long cells = (long long)c->nx * c->ny;
    const long long it = (1LL << 30) / (cells > 0 ? cells : 1);
    L.iters = it < 16 ? 16 : it > 1024 ? 1024 : (int)it;
    return L;
}

// ------------------------------------------- Chebyshev and PPCG inner steps

// One step of either polynomial method (tea_leaf_cheby.cuknl:71-152,
// tea_leaf_ppcg.cuknl:154-244) in one pass instead of two: with x the field
// the operator acts on,
//   Chebyshev  r = u0 - A u, p = al p + be M^-1 r, u' = u + p       (x = u)
//   PPCG       rtemp -= A sd, sd' = al sd + be M^-1 rtemp, utemp += sd'  (x = sd)
// x' goes to the other of two buffers, so that the neighbours still read x.
// FP64-bound: 10 (none), 11 (diag) or 14 (block) instructions a cell; a pass
// of its own for u += p or the sd update read and wrote 24 to 48 bytes a cell
// more and waited once more for the grid.
enum StepMode { kStepCheby, kStepPpcg, kStepPpcgLast };

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
    const int lane = threadIdx.x & 31, i = i0 + lane;
    const bool own = i < g.nx;
    const int64_t P = g.pitch;
    int64_t c = (int64_t)(i + g.h) + (int64_t)(jb + g.h) * P;
    const int ek = (lane >> 1) & 3, ecol = (lane & 1) ? i0 + kWarpCols : i0 - 1;
    const bool eon = lane < 8 && ecol >= 0 && ecol < g.nx, fon = lane < 8 && (lane & 1) && ecol <= g.nx;
    int64_t e = (int64_t)(ecol + g.h) + (int64_t)(jb + ek + g.h) * P;
    // a row's Kx, diag, f and q (and Mi), the next row's x and Ky; x and Kx beside
    double xl[D], ky[D], kx[D], dg[D], f[D], q[D], mi[D], ex, ef;
    auto load_row = [&](int k, int row, int64_t at) {
        const bool in = own && row < je;
        xl[k] = in && row + 1 < g.ny ? __ldcg(xin + at + P) : 0.0;
        ky[k] = in ? a.ky[at + P] : 0.0;
        kx[k] = in ? a.kx[at] : 0.0;
        dg[k] = in ? a.dg[at] : 0.0;
        f[k] = in ? __ldcg(a.f + at) : 0.0;
        if (!BLOCK) q[k] = in ? __ldcg(a.q + at) : 0.0;
        if (DIAG) mi[k] = in ? a.mi[at] : 0.0;
    };
    auto load_edge = [&](int j0) {
        const bool v = j0 + ek < je;
        ex = v && eon ? __ldcg(xin + e) : 0.0;
        ef = v && fon ? a.kx[e] : 0.0;
    };
    double xm = own && jb > 0 ? __ldcg(xin + c - P) : 0.0, x0 = own ? __ldcg(xin + c) : 0.0;
    double kyv = own ? a.ky[c] : 0.0;
#pragma unroll
    for (int k = 0; k < D; ++k) load_row(k, jb + k, c + k * P);
    load_edge(jb);
    if (!ready()) return;
    for (int j0 = jb; j0 < je; j0 += kStrip) {
        const double edge = ex, face = ef;
        e += kStrip * P;
        load_edge(j0 + kStrip);
        double rv[4], xc[4], qv[4];
        // the row's new values from its r and z
        auto finish = [&](int k, double r, double z, double m) {
            const int64_t at = c + k * P;
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
                if (!BLOCK) qv[k] = q[d];
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

template <int PC>
__global__ void __launch_bounds__(kGroupThreads) k_ppcg_pass2(Geo g, StepArgs a, const DevScalars *sc) {
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

template <int PC, class Shape>
__global__ void __launch_bounds__(Shape::kThreads, 1) k_cheby_loop(LoopArgs L, StepArgs a) {
    if (*(volatile const int *)&L.sc->done) return;
    __shared__ LoopShared S;
    __shared__ struct {
        StepCoef co;
        bool sel, go;
    } T[2];  // what step `it` needs, in T[it & 1]
    loop_begin(L, S);
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
    loop_begin(L, S);
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
    loop_begin(L, S);
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

// The shapes of a loop kernel's CTA: groups at a time and the rows that pass 1
// loads ahead.  Registers are shared by four quarters of the multiprocessor,
// so 9 warps (with the control warp) can have 168 each, 17 have 96.
//   depth 1, 2: 2 groups of 168 registers, the four rows of a strip at once;
//   more:       4 groups of 96 registers, 2 rows ahead, in 1 or 2 rounds.
// (3 groups of 128 registers, 4 rows ahead, in up to 3 rounds: 519 us an
// iteration at 4096^2 against 442.)
template <int GROUPS, int AHEAD>
struct LoopShape {
    static constexpr int kGroups = GROUPS, kAhead = AHEAD, kThreads = GROUPS * kGroupThreads + 32;
};
using ShapeSmall = LoopShape<2, 4>;
using ShapeLarge = LoopShape<4, 2>;

// one cooperative launch of a loop kernel; TL_ERR_STATE if the device cannot
// hold its CTAs at once (the caller then runs the passes one by one)
template <class K, class... A>
int launch_shape(Chunk *c, K kernel, int groups, A... a) {
    const long long cells = (long long)c->nx * c->ny;
    const int slots = c->g.groups < c->g.sms ? c->g.groups : c->g.sms;
    LoopArgs L;
    L.g = c->g;
    L.sc = c->sc;
    L.partials = c->loop_partials;
    L.arrived = c->loop_arrived;
    L.base = c->loop_arrived + 1;
    L.cg_alphas = c->cg_alphas;
    L.cg_betas = c->cg_betas;
    L.depth = (c->g.groups + slots - 1) / slots;
    L.per_round = L.depth < groups ? L.depth : groups;
    // a launch of some tens of milliseconds at most
    const long long it = (1LL << 30) / cells;
    L.iters = it < 16 ? 16 : it > 1024 ? 1024 : (int)it;
    void *args[] = {&L, &a...};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void *)kernel, dim3(slots),
                                                      dim3(L.per_round * kGroupThreads + 32), args, 0, c->stream);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
        cudaGetLastError();
        c->loop_ok = false;
        return TL_ERR_STATE;
    }
    if (e != cudaSuccess) return cuda_fail(e, "cudaLaunchCooperativeKernel");
    c->launches++;
    return TL_OK;
}

template <class K1, class K2, class... A>
int launch_loop(Chunk *c, K1 small, K2 large, A... a) {
    return c->g.groups <= 2 * c->g.sms ? launch_shape(c, small, ShapeSmall::kGroups, a...)
                                       : launch_shape(c, large, ShapeLarge::kGroups, a...);
}

// f(preconditioner as a type)
template <int PC>
using Pc = std::integral_constant<int, PC>;
template <class F>
int by_precond(const Chunk *c, F f) {
    switch (c->cfg.precond) {
    case TL_PREC_JAC_BLOCK: return f(Pc<TL_PREC_JAC_BLOCK>());
    case TL_PREC_JAC_DIAG: return f(Pc<TL_PREC_JAC_DIAG>());
    default: return f(Pc<TL_PREC_NONE>());
    }
}

}  // namespace

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
// passes' own kernels.  Microseconds an iteration of CG + jac_diag, loop and
// graph of passes: 14.5 and 24.5 at 512^2 (run 1), 37 and 51 at 1024^2 (2), 71
// and 82 at 1400^2 (4), 127 and 133 at 2048^2 (7), 223 and 215 at 2816^2 (13).
bool loop_pays(const Chunk *c) {
    return c->loop_ok && !c->profiling && !c->cfg.reflective_boundary && c->g.run <= 8;
}

}  // namespace tl
