// tl_loop.cuh -- what the kernels that run many iterations in one launch share
// (tl_loop.cu: FP64; tl_mixed_loop.cu: mixed-precision PPCG; tl_mixed.cu: FP32 CG): the meetings of
// their thread blocks, the walk over the runs, pass 1 of a CG iteration, the
// launch.
//
// One launch runs `iters` iterations: one CTA a multiprocessor (co-resident:
// a cooperative launch), a tile group always on the same CTA, the grid's CTAs
// meeting at each sum.  A CTA stores its partial sum, counts itself in (one
// atomic on one word) and polls that word; then every CTA adds the same
// partials in the same order and runs the scalar epilogue on its own copy of
// the scalars.  Before anything else the CTAs gather (loop_gather): one that
// other streams' kernels keep from starting for about two seconds makes the
// launch return with nothing done, and the passes go on one by one.  Once
// gathered, a wait of two seconds means that the device does not go on: it stops
// the solve with an error.  Measured on GB300, in clocks: one meeting 2450 to 3200 at any
// number of CTAs (an FP64 dependency is 64, a trip to L2 400); letting
// every CTA poll every other's flag took 7000 with 152 of them, the last
// arriver's adding and publishing for all 6900, clusters with a leader each
// 10000.
#pragma once

#include <type_traits>

#include "tl_fp64.cuh"

namespace tl {

namespace {

constexpr long long kLoopWaitCycles = 4000000000LL;  // ~2 s: the default of both limits
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
    unsigned int *gate;      // 2 round + 1: the launch of that round goes on, 2 round: it does not
    unsigned int round;      // this launch's number
    long long start_wait;    // clocks to wait for the CTAs to start (below 0: as if one had not),
    long long wait;          // and for them to come to a meeting
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
    int gathered;
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
                if (clock64() - t0 > L.wait) {
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

// whether every CTA of the launch is there, the same answer in all of them (one
// thread a CTA).  The last to arrive says yes, the first whose wait runs out no;
// the word that either sets first stands, also for a CTA that starts later.  After
// a no the last CTA to arrive counts the launch's arrivals off and tells the host.
__device__ __forceinline__ bool loop_gather(const LoopArgs &L, unsigned int target) {
    const unsigned int yes = 2 * L.round + 1, no = 2 * L.round;
    // an earlier launch's word until this one's answer
    unsigned int word = *(volatile unsigned int *)L.gate;
    auto answer = [&](unsigned int mine) {
        if (word >> 1 == L.round) return word;
        const unsigned int was = atomicCAS(L.gate, word, mine);
        return was == word ? mine : was;
    };
    unsigned int before;
    // (release: what was read so far, the base among it, was read before)
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(L.arrived) : "memory");
    if (before + 1 == target) {
        const bool go = answer(L.start_wait < 0 ? no : yes) == yes;
        if (!go) {
            *L.base = target;
            *(volatile int *)&L.sc->done = kNotStarted;
        }
        return go;
    }
    const long long t0 = clock64();
    for (;;) {
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(L.gate) : "memory");
        if (v >> 1 == L.round) return v == yes;
        if (clock64() - t0 > L.start_wait) return answer(no) == yes;
    }
}

// false: the launch does nothing
__device__ __forceinline__ bool loop_begin(const LoopArgs &L, LoopShared &S) {
    static_assert(sizeof(DevScalars) % sizeof(int) == 0, "copied by words");
    for (int k = threadIdx.x; k < (int)(sizeof(DevScalars) / sizeof(int)); k += blockDim.x)
        ((int *)&S.sc)[k] = ((const int *)L.sc)[k];
    if (threadIdx.x == 0) {
        S.target = *L.base + gridDim.x;
        S.parity = 0;
        S.stalled = 0;
        S.gathered = 1;
        if (gridDim.x > 1) {
            S.gathered = loop_gather(L, S.target);
            S.target += gridDim.x;
        }
    }
    __syncthreads();
    return S.gathered != 0;
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
    double *rs;         // r_store, where r takes turns with it (mixed PPCG), else null
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

// ppcg: the outer iteration of PPCG, whose z is never r itself
[[maybe_unused]] CgArgs cg_args(Chunk *c, bool ppcg = false) {
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

// The shapes of a loop kernel's CTA: groups at a time and the rows that pass 1
// loads ahead.  Registers are shared by four quarters of the multiprocessor,
// so 9 warps (with the control warp) can have 168 each, 17 have 96.
//   depth 1, 2: 2 groups of 168 registers, the four rows of a strip at once;
//   more:       4 groups of 96 registers, 2 rows ahead, in 1 or 2 rounds.
// The second spills: bytes stored and loaded a thread 54 / 116 (none), 146 / 208
// (jac_diag) and 242 / 284 (block) in CG, 106 / 124, 156 / 172 and 568 / 452 in PPCG, 32 /
// 80 to 148 / 172 in Chebyshev, 60 / 92 in Jacobi, 22 / 32 to 52 / 68 in mixed PPCG; the
// first only in PPCG with block-Jacobi (124 / 156) and jac_diag (4 / 8).
// (3 groups of 128 registers, 4 rows ahead, in up to 3 rounds: 519 us an
// iteration at 4096^2 against 442.)
template <int GROUPS, int AHEAD>
struct LoopShape {
    static constexpr int kGroups = GROUPS, kAhead = AHEAD, kThreads = GROUPS * kGroupThreads + 32;
};
using ShapeSmall = LoopShape<2, 4>;
using ShapeLarge = LoopShape<4, 2>;

// groups of the busiest CTA of a loop kernel
[[maybe_unused]] int loop_depth(const Chunk *c) {
    const int slots = c->g.groups < c->g.sms ? c->g.groups : c->g.sms;
    return (c->g.groups + slots - 1) / slots;
}

// one cooperative launch of a loop kernel of `slots` CTAs; TL_ERR_STATE if the
// device cannot hold them at once (the caller then runs the passes one by one).
// L has the groups and their depth; the rest is filled in.
template <class K, class... A>
int launch_coop(Chunk *c, K kernel, LoopArgs &L, int slots, int threads, size_t smem, A... a) {
    const long long cells = (long long)c->nx * c->ny;
    L.sc = c->sc;
    L.partials = c->loop_partials;
    L.arrived = c->loop_arrived;
    L.base = c->loop_arrived + 1;
    L.gate = c->loop_arrived + 32;
    L.round = ++c->loop_round & 0x7FFFFFFFu;
    L.start_wait = c->loop_start_wait == -1 ? kLoopWaitCycles : c->loop_start_wait;
    L.wait = c->loop_wait >= 0 ? c->loop_wait : kLoopWaitCycles;
    L.cg_alphas = c->cg_alphas;
    L.cg_betas = c->cg_betas;
    // a launch of some tens of milliseconds at most
    const long long it = (1LL << 30) / cells;
    L.iters = c->loop_iters > 0 ? c->loop_iters : it < 16 ? 16 : it > 1024 ? 1024 : (int)it;
    void *args[] = {&L, &a...};
    cudaError_t e = cudaSuccess;
    if (smem) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
        e = cudaLaunchCooperativeKernel((const void *)kernel, dim3(slots), dim3(threads), args, smem, c->stream);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
        cudaGetLastError();
        c->loop_ok = false;
        return TL_ERR_STATE;
    }
    if (e != cudaSuccess) return cuda_fail(e, "cudaLaunchCooperativeKernel");
    c->launches++;
    return TL_OK;
}
template <class K, class... A>
int launch_shape(Chunk *c, K kernel, int groups, size_t smem, A... a) {
    LoopArgs L;
    L.g = c->g;
    L.depth = loop_depth(c);
    L.per_round = L.depth < groups ? L.depth : groups;
    return launch_coop(c, kernel, L, c->g.groups < c->g.sms ? c->g.groups : c->g.sms,
                       L.per_round * kGroupThreads + 32, smem, a...);
}

[[maybe_unused]] int loop_groups(const Chunk *c) {
    return c->g.groups <= ShapeSmall::kGroups * c->g.sms ? ShapeSmall::kGroups : ShapeLarge::kGroups;
}
// (smem: dynamic shared memory beside the kernel's own)
template <class K1, class K2, class... A>
int launch_loop_smem(Chunk *c, K1 small, K2 large, size_t smem, A... a) {
    return loop_groups(c) == ShapeSmall::kGroups ? launch_shape(c, small, ShapeSmall::kGroups, smem, a...)
                                                 : launch_shape(c, large, ShapeLarge::kGroups, smem, a...);
}
template <class K1, class K2, class... A>
int launch_loop(Chunk *c, K1 small, K2 large, A... a) {
    return launch_loop_smem(c, small, large, 0, a...);
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

}  // namespace tl
