// tl_device.cuh -- device helpers shared by the FP64 kernels (tl_kernels.cu)
// and the mixed-precision ones (tl_mixed.cu).
#pragma once

#include <stdint.h>

namespace tl {

// x / b, bit for bit, from the correctly rounded reciprocal y of b: two residual
// corrections of x y.  The first leaves an error below an ulp, and from there, y
// being correctly rounded, the second rounds correctly (Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", 1990, theorem
// on division; no quotient of 2^-863 or more underflows while |b| < 2^150).  5
// fused multiply-adds where the division operator takes about twice as many
// FP64 instructions.  Divided instead: an x so small that the residuals would
// underflow, and whatever gives no finite q (the corrections turn an infinite
// quotient, or one by an infinite b, into NaN).  A zero x gives its sign to q.
static __device__ __noinline__ double div_slow(double x, double b) { return x / b; }
__device__ __forceinline__ double div_by(double x, double b, double y) {
    double q = x * y;
    q = fma(fma(-b, q, x), y, q);
    q = fma(fma(-b, q, x), y, q);
    const unsigned int ex = ((unsigned int)__double2hiint(x) >> 20) & 0x7FFu;  // biased exponents
    const unsigned int eq = ((unsigned int)__double2hiint(q) >> 20) & 0x7FFu;
    if (ex < 160u || eq == 0x7FFu) q = x == 0.0 ? x * y : div_slow(x, b);
    return q;
}

// block-Jacobi strip solve z = M^-1 x (tea_block_jacobi.cuknl:11-46); y0: 1 / diag
// of the strip's first row
__device__ __forceinline__ void strip_block_solve(const double *__restrict__ dg, double y0,
                                                  const double *__restrict__ ky,
                                                  const double *__restrict__ cp,
                                                  const double *__restrict__ bfp, int pitch,
                                                  int64_t base, int m, const double (&x)[4],
                                                  double (&z)[4]) {
    double dp[4];
    dp[0] = div_by(x[0], dg[base], y0);
#pragma unroll
    for (int k = 1; k < 4; ++k)
        if (k < m) {
            const int64_t i = base + (int64_t)k * pitch;
            dp[k] = fma(ky[i], dp[k - 1], x[k]) * bfp[i];
        }
#pragma unroll
    for (int k = 3; k >= 0; --k) {
        if (k == m - 1) {
            z[k] = dp[k];
        } else if (k < m - 1) {
            const int64_t i = base + (int64_t)k * pitch;
            z[k] = fma(-cp[i], z[k + 1], dp[k]);
        }
    }
}

// strip_block_solve on values that are in registers: the first row's diagonal
// and its reciprocal, Ky and bfp of rows 1..3, cp of rows 0..2.  A strip cut
// short by the field's top has zeros in the missing rows (of x too): the
// same operations then leave z = 0 there and dp in the last row.
struct StripFactors {
    double b0, y0, ky[3], bf[3], cp[3];
};
__device__ __forceinline__ void strip_solve(const StripFactors &f, const double (&x)[4], double (&z)[4]) {
    const double d0 = div_by(x[0], f.b0, f.y0);
    const double d1 = fma(f.ky[0], d0, x[1]) * f.bf[0];
    const double d2 = fma(f.ky[1], d1, x[2]) * f.bf[1];
    z[3] = fma(f.ky[2], d2, x[3]) * f.bf[2];
    z[2] = fma(-f.cp[2], z[3], d2);
    z[1] = fma(-f.cp[1], z[2], d1);
    z[0] = fma(-f.cp[0], z[1], d0);
}

}  // namespace tl
