// Correctly rounded division by a divisor fixed for a whole launch.
//
// The snapshot store divides every cell by dt ((p_3 - p_1)*0.5/dt,
// solver_acoustic_SS.f90:447).  A full IEEE division per cell costs the
// forward snapshot passes about a third of their time, so the quotient is
// formed from y = RN(1/b), computed once on the host, with two refinement
// steps q <- q + (a - b*q)*y in fused multiply-adds (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Develop. 34(1), 1990).  q0 = RN(a*y) is within two
// units in the last place of a/b; the first step makes q faithful (within one
// unit); for a faithful q the remainder a - b*q is exactly representable and
// the second step returns RN(a/b), the round-to-nearest-even quotient.  The
// argument assumes that neither the remainder nor the quotient leaves the
// normal range, so it serves 2^-100 <= |a| <= 2^100.  Smaller nonzero
// dividends (the numerical precursor of the finite-difference stencil fills
// the wavefield ahead of the wave with them) take div_tiny below; a zero
// dividend (b > 0) is its own quotient; Inf, NaN, huge values and a missing
// reciprocal (y = 0) take the division itself.  The refinement runs for every
// lane and the exceptions are selected afterwards, so that the zeros of a
// wavefield not yet reached by the wave cost no branch.
// tests/test_gpu_division.py compares the result bit for bit with the
// division of CUDA over all 2^32 values of a for the time steps of the
// benchmark workloads and a set of seeded random ones.
#pragma once

namespace fwi {

__device__ __forceinline__ float div_main(float a, float b, float y) {
    float q = __fmul_rn(a, y);
    float r = __fmaf_rn(-q, b, a);
    q = __fmaf_rn(r, y, q);
    r = __fmaf_rn(-q, b, a);
    return __fmaf_rn(r, y, q);
}

// RN(a/b) for 0 < |a| < 2^-100: the quotient q of a*2^64 (a normal dividend)
// scaled back by 2^-64, exactly if it is normal.  A quotient below 2^-126 is
// rounded a second time, to a multiple t of 2^-149; that is RN(a/b) as long as
// q is not half-way between two of them, or is the quotient itself.  Else
// a/b lies on the side of the exact remainder: where t is on the other one,
// the neighbour across q is the result.
__device__ __forceinline__ float div_tiny(float a, float b, float y) {
    const float s = __fmul_rn(a, 0x1p64f), q = div_main(s, b, y), r = __fmaf_rn(-q, b, s);
    const float t = __fmul_rn(q, 0x1p-64f), d = __fmaf_rn(t, -0x1p64f, q);
    const bool across = fabsf(d) == 0x1p-86f && r != 0.f && (r > 0.f) == (d > 0.f);
    return across ? __fadd_rn(t, copysignf(0x1p-149f, d)) : t;
}

__device__ __forceinline__ float div_by_const(float a, float b, float y) {
    const float m = fabsf(a);
    float q = div_main(a, b, y);
    if (m == 0.f) q = a;
    else if (m < 0x1p-100f && y != 0.f) q = div_tiny(a, b, y);
    else if (!(m <= 0x1p100f) || y == 0.f) q = __fdiv_rn(a, b);
    return q;
}

// Four of them in place: the quotients of all four at once, then one branch for
// the tiny dividends and one for the other exceptions.  The precursor is tiny
// almost everywhere, and its quotients go through the longest chain: with a
// branch per cell and the double-rounded quotients formed from integers, a
// snapshot step of three 400 x 2000 shots took 7.0 us more than another one,
// now 2.8.
__device__ __forceinline__ void div4_by_const(float* a, float b, float y) {
    float q[4];
    bool tiny = false, other = y == 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float m = fabsf(a[e]);
        q[e] = m == 0.f ? a[e] : div_main(a[e], b, y);
        tiny |= m < 0x1p-100f && m != 0.f;
        other |= !(m <= 0x1p100f);
    }
    if (tiny) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float t = div_tiny(a[e], b, y), m = fabsf(a[e]);
            if (m < 0x1p-100f && m != 0.f) q[e] = t;
        }
    }
    if (other) {
#pragma unroll
        for (int e = 0; e < 4; ++e) q[e] = div_by_const(a[e], b, y);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) a[e] = q[e];
}

}  // namespace fwi
