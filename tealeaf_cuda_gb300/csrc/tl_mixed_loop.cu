// tl_mixed_loop.cu -- mixed-precision PPCG, many outer iterations in one launch
// (tl_loop.cuh): FP64 outer iteration, FP32 inner steps.
//
// An outer iteration is inner + 2 passes over the field, each ended by a meeting
// of the grid:
//   u += alpha p, p' = z + beta p, w = A p', sum p'.w               (FP64)
//   r -= alpha w; rtemp = r, sd = utemp = M^-1 rtemp / theta        (FP64, FP32)
//   inner - 1 steps of the polynomial preconditioner                (FP32)
//   the last step; z = utemp, sums w.z and r.z, the exit test       (FP32, FP64)
// The inner steps are those of k_pp_step operation for operation, so a solve has
// the bits of the one-pass-a-step and the fused forms.  For grids whose FP32
// fields stay in L2 and whose fused passes (k_pp_fused) would leave the
// multiprocessors half empty: a pass of five steps there goes through 2 T + 4
// strips at least, one after the other, whatever the size.
//
// The inner steps read and write 40 bytes a cell each, 36 of them values that
// only the cell's own thread uses: rtemp, utemp, Kx, Ky and the
// preconditioner.  As many of those arrays as fit are kept in shared memory for
// the whole launch (a warp's strips in slots of 4 rows by 32 columns, 16-byte
// loads); only sd goes through L2.  At 1024^2 with block-Jacobi an outer
// iteration takes 89 us (123 with every array in L2, loaded row by row): the
// nine plain steps 3.6 us each, their meetings 1.4 each, the FP64 passes 20
// and 9.5 us.  (The new r in the other of two buffers, which keeps the old one for
// r_store, costs 0.5 % at 512^2, 2.9 % at 1024^2 and 1.2 % at 1400^2; r, r_store and
// p's two buffers rotating through three, and the iteration once in the code for
// each place of r, cost as much or more.)
#include <type_traits>

#include "tl_loop.cuh"
#include "tl_mixed.cuh"

namespace tl {

namespace {

struct MixedArgs {
    float *sd0, *sd1, *rtemp, *utemp;
    const float *kx, *ky, *mi, *cp, *bfp;  // bfp: 1/diag in each strip's first row
    double *r0, *r1, *z;  // r and r_store take turns (DevScalars::p_sel)
    const double *w;
    const double *alphas, *betas;
    int inner;
    int shared_arrays, slots;  // private arrays in shared memory, strips a CTA has there
};

// The private arrays, those first that shared memory takes first: what a step
// writes, then the preconditioner and the faces.  A strip's slot holds a
// float4 a lane, its column's four rows, so a strip's values of an array are one
// 16-byte load; missing rows and columns are 0.
enum PrivateArray {
    kRt = 0,
    kUt,
    kPre,        // bfp or Mi
    kKyn,        // the face above the row
    kKx,
    kCp,
    kKxe         // the face east of the column
};
// (an array's place depends on which there are)
template <int PC>
__host__ __device__ constexpr int private_place(int q) {
    return q - (PC == TL_PREC_NONE && q > kPre ? 1 : 0) - (PC != TL_PREC_JAC_BLOCK && q > kCp ? 1 : 0);
}
template <int PC>
__host__ __device__ constexpr bool private_has(int q) {
    return !(PC == TL_PREC_NONE && q == kPre) && !(PC != TL_PREC_JAC_BLOCK && q == kCp);
}
template <int PC>
__host__ __device__ constexpr int private_arrays() {
    return private_place<PC>(kKxe) + 1;
}

// a strip of a CTA's run: its slot, its first cell, its rows.  32-bit offsets: a
// loop's fields are far below 2^31 elements.
struct Strip {
    int slot;
    int c, P;
    int m;  // 0 for lanes beyond the field
};

template <int PC, int Q>
__device__ __forceinline__ float4 *private_slot(const MixedArgs &a, float4 *smem, int slot) {
    return smem + (private_place<PC>(Q) * a.slots + slot) * kWarpCols + (int)(threadIdx.x & 31);
}
// (ALL: they are all there, known when the kernel is compiled)
template <int PC, bool ALL, int Q>
__device__ __forceinline__ bool private_shared(const MixedArgs &a) {
    return ALL || private_place<PC>(Q) < a.shared_arrays;
}
template <int PC, int Q>
__device__ __forceinline__ float *private_global(const MixedArgs &a) {
    return Q == kRt    ? a.rtemp
           : Q == kUt  ? a.utemp
           : Q == kPre ? const_cast<float *>(PC == TL_PREC_JAC_BLOCK ? a.bfp : a.mi)
           : Q == kKyn ? const_cast<float *>(a.ky)
           : Q == kCp  ? const_cast<float *>(a.cp)
                       : const_cast<float *>(a.kx);
}
// a strip's rows of an array that is in L2 (Kyn: the row above, Kxe: the column beside)
template <int PC, int Q>
__device__ __forceinline__ void global_rows(const MixedArgs &a, const Strip &s, float (&v)[4]) {
    const float *f = private_global<PC, Q>(a);
    const int c = s.c + (Q == kKyn ? s.P : Q == kKxe ? 1 : 0);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = k < s.m ? f[c + k * s.P] : 0.f;
}
template <int PC, bool ALL, int Q>
__device__ __forceinline__ void private_load(const MixedArgs &a, float4 *smem, const Strip &s, float (&v)[4]) {
    if (private_shared<PC, ALL, Q>(a)) {
        const float4 t = *private_slot<PC, Q>(a, smem, s.slot);
        v[0] = t.x;
        v[1] = t.y;
        v[2] = t.z;
        v[3] = t.w;
    } else {
        global_rows<PC, Q>(a, s, v);
    }
}
template <int PC, bool ALL, int Q>
__device__ __forceinline__ void private_store(const MixedArgs &a, float4 *smem, const Strip &s, const float (&v)[4]) {
    if (private_shared<PC, ALL, Q>(a)) {
        *private_slot<PC, Q>(a, smem, s.slot) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
        float *f = private_global<PC, Q>(a);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < s.m) f[s.c + k * s.P] = v[k];
    }
}
template <int PC, bool ALL, int Q>
__device__ __forceinline__ void private_fill(const MixedArgs &a, float4 *smem, const Strip &s) {
    if (private_has<PC>(Q) && private_shared<PC, ALL, Q>(a)) {
        float v[4];
        global_rows<PC, Q>(a, s, v);
        *private_slot<PC, Q>(a, smem, s.slot) = make_float4(v[0], v[1], v[2], v[3]);
    }
}
// loads after this line are not moved before it (they would be held in registers that there are none of)
__device__ __forceinline__ void load_later() { asm volatile("" ::: "memory"); }

// z = M^-1 x of a strip: the block solve of k_pp_step (zeros in the factors of
// missing rows leave zeros there), Mi, or nothing.  kyn: the faces above rows 0..3
template <int PC>
__device__ __forceinline__ void precondition(const float (&x)[4], const float (&pre)[4], const float (&kyn)[4],
                                             const float (&cp)[4], float (&z)[4]) {
    if (PC == TL_PREC_JAC_BLOCK) {
        z[0] = x[0] * pre[0];
#pragma unroll
        for (int k = 1; k < 4; ++k) z[k] = fmaf(kyn[k - 1], z[k - 1], x[k]) * pre[k];
#pragma unroll
        for (int k = 2; k >= 0; --k) z[k] = fmaf(-cp[k], z[k + 1], z[k]);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) z[k] = PC == TL_PREC_JAC_DIAG ? x[k] * pre[k] : x[k];
    }
}

// r_new = r_old - alpha w and the start of the inner steps on a run: rtemp = r_new, sd = utemp
// = M^-1 rtemp / theta
template <int PC, bool ALL, class Ready>
__device__ __forceinline__ void mixed_start(const Geo &g, const MixedArgs &a, float4 *smem, int slot,
                                            const double *__restrict__ r_old, double *__restrict__ r_new, int i0,
                                            int jb, int je, float theta_r, double &alpha, Ready ready) {
    const int i = i0 + (threadIdx.x & 31);
    Strip s{slot, (i + g.h) + (jb + g.h) * g.pitch, g.pitch, 0};
    for (int j0 = jb; j0 < je; j0 += kStrip, s.c += kStrip * s.P, ++s.slot) {
        s.m = i < g.nx ? min(kStrip, je - j0) : 0;
        double w[4], r[4];
        float pre[4], kyn[4], cp[4], x[4], z[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            w[k] = k < s.m ? __ldcg(a.w + s.c + k * s.P) : 0.0;
            r[k] = k < s.m ? __ldcg(r_old + s.c + k * s.P) : 0.0;
        }
        if (PC != TL_PREC_NONE) private_load<PC, ALL, kPre>(a, smem, s, pre);
        if (PC == TL_PREC_JAC_BLOCK) {
            private_load<PC, ALL, kKyn>(a, smem, s, kyn);
            private_load<PC, ALL, kCp>(a, smem, s, cp);
        }
        if (!ready()) return;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const double rv = fma(-alpha, w[k], r[k]);
            if (k < s.m) r_new[s.c + k * s.P] = rv;
            x[k] = (float)rv;
        }
        precondition<PC>(x, pre, kyn, cp, z);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            z[k] *= theta_r;
            if (k < s.m) a.sd0[s.c + k * s.P] = z[k];
        }
        private_store<PC, ALL, kRt>(a, smem, s, x);
        private_store<PC, ALL, kUt>(a, smem, s, z);
    }
}

// one inner step on a run; LAST: z = utemp (FP64) and the sums w.z and r.z
// instead of sd and rtemp.  A strip's sd and the columns beside it are loaded
// while the strip before is computed; what waits for L2 is the run's first load.
template <int PC, bool ALL, bool LAST>
__device__ __forceinline__ void mixed_step(const Geo &g, const MixedArgs &a, float4 *smem, int slot,
                                           const float *__restrict__ xin, float *__restrict__ xout, const double *r,
                                           int i0, int jb, int je, float al, float be, double (&acc)[LAST ? 2 : 1]) {
    const int lane = threadIdx.x & 31, i = i0 + lane;
    const bool own = i < g.nx;
    Strip s{slot, (i + g.h) + (jb + g.h) * g.pitch, g.pitch, 0};
    // the first and last lane load the column beside the warp's
    const bool beside = lane == 0 ? i0 > 0 : lane == 31 && i + 1 < g.nx;
    const float *xb = xin + (lane == 0 ? -1 : 1);
    float xm = own && jb > 0 ? __ldcg(xin + s.c - s.P) : 0.f;
    float kyc = own ? a.ky[s.c] : 0.f;
    // sd of the next strip and of the row above it, and beside it
    float xn[5], en[4];
    xn[4] = own ? __ldcg(xin + s.c) : 0.f;
    // FULL: a strip of four rows in 32 columns of the field
    const bool wide = i0 + kWarpCols <= g.nx;
    auto load_next = [&](auto full, const float *px, const float *pb, int j0) {
        constexpr bool FULL = decltype(full)::value;
        xn[0] = xn[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool in = FULL || j0 + k < je;
            // (the row above the field's last: 0)
            xn[k + 1] = (FULL && k < 3) || (in && own && j0 + k + 1 < g.ny) ? __ldcg(px + (k + 1) * s.P) : 0.f;
            en[k] = in && beside ? __ldcg(pb + k * s.P) : 0.f;
        }
    };
    auto next = [&](int c, int j0) {
        if (wide && j0 + kStrip <= je) load_next(std::true_type{}, xin + c, xb + c, j0);
        else load_next(std::false_type{}, xin + c, xb + c, j0);
    };
    next(s.c, jb);
    auto strip = [&](auto full, int j0) {
        constexpr bool FULL = decltype(full)::value;
        s.m = FULL ? kStrip : own ? min(kStrip, je - j0) : 0;
        float x[6], e[4], kyn[4], f[4], rv[4], z[4];
        x[0] = xm;
#pragma unroll
        for (int k = 0; k < 4; ++k) e[k] = en[k];
#pragma unroll
        for (int k = 0; k < 5; ++k) x[k + 1] = xn[k];
        if (j0 + kStrip < je) next(s.c + kStrip * s.P, j0 + kStrip);
        {
            float kx[4], kxe[4];
            private_load<PC, ALL, kKyn>(a, smem, s, kyn);
            private_load<PC, ALL, kKx>(a, smem, s, kx);
            private_load<PC, ALL, kKxe>(a, smem, s, kxe);
            private_load<PC, ALL, kRt>(a, smem, s, f);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float xw = __shfl_up_sync(0xffffffffu, x[k + 1], 1), xe = __shfl_down_sync(0xffffffffu, x[k + 1], 1);
                if (lane == 0) xw = e[k];
                if (lane == 31) xe = e[k];
                rv[k] = f[k] - cell_apply(x[k + 1], x[k + 2], x[k], xw, xe, kyn[k],
                                          k == 0 ? kyc : kyn[k > 0 ? k - 1 : 0], kxe[k], kx[k]);
                if (!FULL && PC == TL_PREC_JAC_BLOCK && k >= s.m) rv[k] = 0.f;
            }
        }
        load_later();
        {
            float pre[4], cp[4];
            if (PC != TL_PREC_NONE) private_load<PC, ALL, kPre>(a, smem, s, pre);
            if (PC == TL_PREC_JAC_BLOCK) private_load<PC, ALL, kCp>(a, smem, s, cp);
            precondition<PC>(rv, pre, kyn, cp, z);
        }
        xm = x[4];
        kyc = kyn[3];
        load_later();
        private_load<PC, ALL, kUt>(a, smem, s, f);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            z[k] = fmaf(al, x[k + 1], be * z[k]);
            f[k] = f[k] + z[k];
        }
        if (LAST) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < s.m) {
                    const int at = s.c + k * s.P;
                    const double zv = (double)f[k];
                    a.z[at] = zv;
                    acc[0] = fma(__ldcg(a.w + at), zv, acc[0]);
                    acc[LAST ? 1 : 0] = fma(__ldcg(r + at), zv, acc[LAST ? 1 : 0]);
                }
        } else {
            float *po = xout + s.c;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < s.m) po[k * s.P] = z[k];
            private_store<PC, ALL, kRt>(a, smem, s, rv);
            private_store<PC, ALL, kUt>(a, smem, s, f);
        }
        s.c += kStrip * s.P;
        ++s.slot;
    };
    for (int j0 = jb; j0 < je; j0 += kStrip) {
        if (wide && j0 + kStrip <= je) strip(std::true_type{}, j0);
        else strip(std::false_type{}, j0);
    }
}

// a pass of this (passing) warp over its runs with their slots: f(first column,
// first row, row after the last, first slot, sums)
template <int NV, class F>
__device__ __forceinline__ void slot_pass(const LoopArgs &L, LoopShared &S, F f) {
    // the warp's run of the group it takes next: group after group, its 4 warps' runs
    int slot = (int)(threadIdx.x >> 5) * L.g.run;
    loop_pass<NV>(L, S, [&](int i0, int jb, int je, double (&acc)[NV > 0 ? NV : 1]) {
        f(i0, jb, je, slot, acc);
        slot += L.per_round * kGroupWarps * L.g.run;
    });
}

template <int PC, bool ALL, class Shape>
__global__ void __launch_bounds__(Shape::kThreads, 1) k_mixed_ppcg_loop(LoopArgs L, MixedArgs a, CgArgs cg) {
    if (*(volatile const int *)&L.sc->done) return;
    __shared__ LoopShared S;
    extern __shared__ float4 smem[];
    if (!loop_begin(L, S)) return;
    const float theta_r = (float)(1.0 / S.sc.theta);
    if (threadIdx.x >= blockDim.x - 32) {
        for (int it = 0; it < L.iters; ++it) {
            loop_meet<1>(L, S, kEpiPpcgPw);
            if (S.stalled) break;
            for (int st = 0; st < a.inner && !S.stalled; ++st) loop_meet<0>(L, S, kEpiNone);
            if (S.stalled) break;
            loop_meet<2>(L, S, kEpiWzZrFinish);
            if (S.stalled || S.sc.done) break;
        }
    } else {
        slot_pass<0>(L, S, [&](int i0, int jb, int je, int slot, double (&)[1]) {
            const int i = i0 + (threadIdx.x & 31);
            Strip s{slot, (i + L.g.h) + (jb + L.g.h) * L.g.pitch, L.g.pitch, 0};
            for (int j0 = jb; j0 < je; j0 += kStrip, s.c += kStrip * s.P, ++s.slot) {
                s.m = i < L.g.nx ? min(kStrip, je - j0) : 0;
                private_fill<PC, ALL, kPre>(a, smem, s);
                private_fill<PC, ALL, kKyn>(a, smem, s);
                private_fill<PC, ALL, kKx>(a, smem, s);
                private_fill<PC, ALL, kCp>(a, smem, s);
                private_fill<PC, ALL, kKxe>(a, smem, s);
            }
        });
        for (int it = 0;; ++it) {
            AlphaBeta ab{0.0, 0.0};
            if (it > 0) loop_met();
            const bool sel = S.sc.p_sel != 0;
            const double *pin = sel ? cg.p1 : cg.p0;
            double *pout = sel ? cg.p0 : cg.p1, *r_new = sel ? a.r0 : a.r1;
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
                cg_pass1<Shape::kAhead, true>(L.g, cg, pin, pout, i0, jb, je, ab, ready1, acc[0]);
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
            slot_pass<0>(L, S, [&](int i0, int jb, int je, int slot, double (&)[1]) {
                mixed_start<PC, ALL>(L.g, a, smem, slot, sel ? a.r1 : a.r0, r_new, i0, jb, je, theta_r, ab.alpha,
                                     ready2);
            });
            if (!ready2()) break;
            for (int st = 1; st <= a.inner; ++st) {
                loop_arrive<0>(L, S);
                const float al = (float)a.alphas[st - 1], be = (float)a.betas[st - 1];
                loop_met();
                if (S.stalled) break;
                const float *xin = st & 1 ? a.sd0 : a.sd1;
                float *xout = st & 1 ? a.sd1 : a.sd0;
                if (st < a.inner)
                    slot_pass<0>(L, S, [&](int i0, int jb, int je, int slot, double (&acc)[1]) {
                        mixed_step<PC, ALL, false>(L.g, a, smem, slot, xin, xout, r_new, i0, jb, je, al, be, acc);
                    });
                else
                    slot_pass<2>(L, S, [&](int i0, int jb, int je, int slot, double (&acc)[2]) {
                        mixed_step<PC, ALL, true>(L.g, a, smem, slot, xin, xout, r_new, i0, jb, je, al, be, acc);
                    });
            }
            if (S.stalled) break;
            loop_arrive<2>(L, S);
        }
    }
    loop_end(L, S);
}

}  // namespace

int launch_mixed_ppcg_loop(Chunk *c) {
    Mixed *mx = mixed_of(c);
    MixedArgs a;
    a.sd0 = mx->sd[0];
    a.sd1 = mx->sd[1];
    a.rtemp = mx->rtemp;
    a.utemp = mx->utemp;
    a.kx = mx->kx;
    a.ky = mx->ky;
    a.mi = mx->mi;
    a.cp = mx->cp;
    a.bfp = mx->bfp;
    a.r0 = c->r;
    a.r1 = c->r_store;
    a.z = c->z;
    a.w = c->w;
    a.alphas = c->ch_alphas;
    a.betas = c->ch_betas;
    a.inner = c->cfg.ppcg_inner_steps;
    a.slots = loop_depth(c) * kGroupWarps * c->g.run;
    return by_precond(c, [&](auto pc) {
        // what a multiprocessor has left beside the kernel's own 17 KB and the reserved 1 KB
        const size_t room = 208 * 1024, array = (size_t)a.slots * kWarpCols * sizeof(float4);
        a.shared_arrays = (int)(room / array);
        if (a.shared_arrays > private_arrays<pc()>()) a.shared_arrays = private_arrays<pc()>();
        if (a.shared_arrays == private_arrays<pc()>())
            return launch_loop_smem(c, k_mixed_ppcg_loop<pc(), true, ShapeSmall>,
                                    k_mixed_ppcg_loop<pc(), true, ShapeLarge>, a.shared_arrays * array, a,
                                    cg_args(c, true));
        return launch_loop_smem(c, k_mixed_ppcg_loop<pc(), false, ShapeSmall>,
                                k_mixed_ppcg_loop<pc(), false, ShapeLarge>, a.shared_arrays * array, a,
                                cg_args(c, true));
    });
}

}  // namespace tl
