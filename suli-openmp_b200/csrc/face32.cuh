// face32.cuh — the FP32 face conductance of the multigrid's level-0 operator, formed by the
// pressure set-up (k_fp64.cu) and by the level-0 kernels of the inner solve (k_mixed.cu).
#pragma once

namespace suli {

// c2/(rho_a + rho_b) with the hardware reciprocal (2 ulp): the preconditioner's operator only
// has to be the same everywhere it is formed, and this is the one formula used for it.  The .ftz
// form, the same value for normal numbers: __fdividef also rescales subnormal divisors, several
// instructions for each of the 17 faces a quad forms, and the level-0 kernels are half bound by
// instruction issue (inner solves of a 256x128x128 step 8.62 -> 8.38 ms).
__device__ __forceinline__ float face_div(float c2, float rsum) {
    float q;
    asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(q) : "f"(c2), "f"(rsum));
    return q;
}

// face conductance of the level-0 operator between two cells (FP32, the formula OpRho uses)
__device__ __forceinline__ float face_rho(float c2, double ra, double rb) {
    return face_div(c2, (float)ra + (float)rb);
}

}  // namespace suli
