// The face velocity of Mom2Face (fields.F90:235-285) from one line of cells; host code too, for its accuracy test.
#pragma once
#include "gam_common.cuh"

namespace gam {

// Vf at one face (explicit fused multiply-adds): the Central8 sums along dT1 of volume * velocity over that of the
// volumes (clamped at TINY), each weight applied to its volume once for the four sums. A is the accumulation type:
// double on the FP64 path, float on the FP32-flux path, whose velocities and volumes are float copies and whose Vf
// is stored as float.
//
// In single precision the sums run over the velocities' differences from the cell below the face, which are exact or
// small where the flow is smooth: the result is off by little more than that cell's own rounding. Against 64 bits (root
// mean square over the velocity's) 3.6e-8 on smooth flows and 9.1e-8 on random ones, where float sums of the products
// volume * velocity, themselves rounded once from double, are off by 0.9-1.5e-7 and 9.4e-8.
template <typename A>
__host__ __device__ __forceinline__ void mom2face_sum(const A* wV, const A* w0, const A* w1, const A* w2, A& f0, A& f1,
                                                      A& f2) {
    constexpr bool single = sizeof(A) == 4;
    const A c0 = single ? w0[3] : A(0), c1 = single ? w1[3] : A(0), c2 = single ? w2[3] : A(0);
    A sV = A(0), s0 = A(0), s1 = A(0), s2 = A(0);
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        A w = A(wC8(n)) * wV[n];
        sV = sV + w;
        s0 = fma(w, single ? w0[n] - c0 : w0[n], s0);
        s1 = fma(w, single ? w1[n] - c1 : w1[n], s1);
        s2 = fma(w, single ? w2[n] - c2 : w2[n], s2);
    }
    const bool ok = sV > A(TINY);
    const A idV = A(1) / (ok ? sV : A(TINY));   // one reciprocal for the three quotients
    if (single) {
        const A q = ok ? A(1) : sV * idV;
        f0 = fma(s0, idV, c0 * q); f1 = fma(s1, idV, c1 * q); f2 = fma(s2, idV, c2 * q);
    } else {
        f0 = s0 * idV; f1 = s1 * idV; f2 = s2 * idV;
    }
}

}  // namespace gam
