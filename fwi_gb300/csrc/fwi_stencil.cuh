// Device helpers shared by the step kernels (fwi_step.cu) and the resident
// kernel (fwi_resident.cu): packed FP32 arithmetic and the interior update.
// Both files are compiled with --fmad=false.
#pragma once
#include <cuda_runtime.h>

namespace fwi {

namespace {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ float4 ldg4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

__device__ __forceinline__ void to_arr(float4 v, float* a) { a[0] = v.x; a[1] = v.y; a[2] = v.z; a[3] = v.w; }
__device__ __forceinline__ float4 from_arr(const float* a) { return make_float4(a[0], a[1], a[2], a[3]); }
// Four FP64 values (32-byte aligned) in one access: two 16-byte halves leave
// half-written sectors on their way to L2 (three 400 x 2000 shots resident, an
// imaging step: 12.9 -> 11.8 us more than another one).
__device__ __forceinline__ void ld_d4(const double* p, double2& a, double2& b) {
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_d4(double* p, double2 a, double2 b) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a.x), "d"(a.y), "d"(b.x), "d"(b.y) : "memory");
}
// Packed FP32 pairs (Blackwell f32x2 add/fma: two independently rounded FP32
// operations per instruction), used by the interior and bottom updates.
// Products are formed as fma(a, b, +0): ptxas contracts a packed multiply
// feeding a packed add into a fused multiply-add (even with --fmad=false),
// which would change the rounding.  fma with a +0 addend is the correctly
// rounded product and is not contracted; it differs from a*b only in the
// sign of a zero product, which changes no nonzero value downstream (these
// updates only add and multiply).  An addend of -0 would keep the sign too,
// but then fma(a, b, -0) is a plain product to ptxas and is contracted
// again.  Lane columns (0,1) and (2,3) form the two pairs; x-neighbour pairs
// at odd offsets are re-paired.
__device__ __forceinline__ float2 pr(const float4& v, int k) { return k == 0 ? make_float2(v.x, v.y) : make_float2(v.z, v.w); }
__device__ __forceinline__ float2 mul0(float2 a, float2 b) { return __ffma2_rn(a, b, make_float2(0.f, 0.f)); }

// The interior update (solver_acoustic_SS.f90:433-434) of four columns, with
// the 2R+1 rows given by an accessor: q(i) is row y-R+i.
// The centre terms of both derivatives and the 2p term are the same rounded
// sum p + p; each derivative sum starts from its centre product (the
// reference adds it to 0, which changes nothing but the sign of a zero).
// x-neighbour pairs at odd offsets straddle two register pairs: their sums
// are formed with two scalar adds straight into a pair.
// SRC: whether source values may be injected, `src` whether they are (without them the reference adds 0).
template <int R, bool SRC = true, typename QF>
__device__ __forceinline__ void interior_update2f(QF q, float4 L, float4 Rt, float4 pm1, float4 cc, const float* sv,
                                                  const float2* cp, float* p3, bool src = true) {
    const float4 C = q(R);
    const float w[12] = {L.x, L.y, L.z, L.w, C.x, C.y, C.z, C.w, Rt.x, Rt.y, Rt.z, Rt.w};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float2 pc = pr(C, k);
        const float2 p2 = __fadd2_rn(pc, pc);  // p(j) + p(j)
        const float2 c0 = mul0(cp[0], p2);     // centre term, x and y alike
        // space_deriv2x: s = s + coef(i)*(p(j+i) + p(j-i))
        float2 ax = c0;
#pragma unroll
        for (int i = 1; i <= R; ++i) {
            const int a = 4 + 2 * k + i, b = 4 + 2 * k - i;
            const float2 sx = (i & 1) ? make_float2(w[a] + w[b], w[a + 1] + w[b + 1])
                                      : __fadd2_rn(make_float2(w[a], w[a + 1]), make_float2(w[b], w[b + 1]));
            ax = __fadd2_rn(ax, mul0(cp[i], sx));
        }
        // space_deriv2y: s = s + (p(j+i) + p(j-i))*coef(i)
        float2 ay = c0;
#pragma unroll
        for (int i = 1; i <= R; ++i) ay = __fadd2_rn(ay, mul0(__fadd2_rn(pr(q(R + i), k), pr(q(R - i), k)), cp[i]));
        // p_3 = -p_1 + 2p + (d2x + d2y + source)*c2
        const float2 pm = pr(pm1, k);
        const float2 t = __fadd2_rn(make_float2(-pm.x, -pm.y), p2);
        float2 d = __fadd2_rn(ax, ay);
        if (SRC && src) d = __fadd2_rn(d, make_float2(sv[2 * k], sv[2 * k + 1]));
        const float2 u = mul0(d, pr(cc, k));
        const float2 r = __fadd2_rn(t, u);
        p3[2 * k] = r.x;
        p3[2 * k + 1] = r.y;
    }
}

template <int R>
__device__ __forceinline__ void interior_update2(const float4* q, float4 L, float4 Rt, float4 pm1, float4 cc,
                                                 const float* sv, const float2* cp, float* p3) {
    interior_update2f<R>([&](int i) { return q[i]; }, L, Rt, pm1, cc, sv, cp, p3);
}

}  // namespace

}  // namespace fwi
