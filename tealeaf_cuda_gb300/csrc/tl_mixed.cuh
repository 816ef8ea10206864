// tl_mixed.cuh -- the FP32 state of the mixed-precision solves (tl_mixed.cu,
// tl_mixed_loop.cu) and the arithmetic they share.
#pragma once

#include "tl_internal.cuh"

namespace tl {

struct Mixed {
    float *kx, *ky, *mi, *d, *r, *p, *w, *z;
    float *sd[2], *rtemp, *utemp, *cp, *bfp;   // PPCG inner steps
    float *rtemp2;                             // second rtemp of the fused inner passes
    double *fpartials;                         // one per CTA of a fused inner pass
    double *partials;            // one per CTA of the vectorised kernels
    unsigned int *counter;
    int vtiles_x, vtiles;        // tiles of the vectorised kernels
    std::vector<void *> allocs;
};

inline Mixed *mixed_of(Chunk *c) { return (Mixed *)c->mixed; }

// A x of one cell in the difference form (four fused steps)
__device__ __forceinline__ float cell_apply(float c, float n, float s, float w, float e, float kyn,
                                            float kyc, float kxe, float kxc) {
    float v = fmaf(kyn, c - n, c);
    v = fmaf(kyc, c - s, v);
    v = fmaf(kxe, c - e, v);
    return fmaf(kxc, c - w, v);
}

}  // namespace tl
