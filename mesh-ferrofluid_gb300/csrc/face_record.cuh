// face_record.cuh -- per-face records of the MoM pair kernels (mom_tiers.cu writes them) and the test that
// divides the EFIE's separated pairs between sym_pairs_kernel and mom_sym_regular_rows_kernel.
#pragma once
#include <cuda_runtime.h>

namespace mb {

constexpr int kRec = 32;
enum {
    kC = 0,      // centroid (hi)
    kRho2 = 3,   // max |corner - centroid|^2; NaN: the face takes part in tier 4 only
    kCl = 4,     // centroid (lo): hi + lo carries ~48 bits
    kEdge = 7,   // RWG edge id of local edge e at 7 + 4 e (int bits)
    kA = 8,      // corner a - centroid at 8 + 4 a
    kHalf = 19,  // +-l / 2 of local edge e at 19 + 4 e (RWG sign of the reference)
    kN = 20,     // normal
    kAA = 24,    // |A_0|^2, |A_1|^2, |A_2|^2
    kAB = 28     // A_0.A_1, A_1.A_2, A_2.A_0
};

__device__ __forceinline__ float centre_dist2(float dx, float dy, float dz) {
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

// Whether sym_pairs_kernel takes the pair (the same arithmetic in mom_sym.cu's kernel of the others).
__device__ __forceinline__ bool sym_pair_far(float r2, float rho2p, float rho2q, float k) {
    const float r = __fadd_rn(__fsqrt_rn(rho2p), __fsqrt_rn(rho2q)), lim = __fmul_rn(2.f, r);
    return r2 >= __fmul_rn(lim, lim) && __fmul_rn(k, r) <= 0.6f;
}

}  // namespace mb
