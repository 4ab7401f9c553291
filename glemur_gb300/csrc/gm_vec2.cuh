// gm_vec2.cuh -- two x-neighbouring points as one operand.
//
// The stage kernel works on pairs of points.  In FP32 a pair is one packed
// f32x2 register pair: an add, multiply or FMA of both points is one
// instruction (add/mul/fma.rn.f32x2), so the floating-point part of the issue
// stream is half as long; the FMA pipe itself runs at the same rate (measured
// on a GB300: 39 T scalar and 40 T packed FMA/s, 4.2 and 2.1 warp instructions
// per clock and SM).  In FP64 a pair is two doubles.  The same templates run
// on single points, with the same operations in the same order, so a point's
// result does not depend on where in a tile it lies.
#pragma once

#include <stdint.h>

namespace gmk {

struct F2 { unsigned long long v; };
struct D2 { double x, y; };

template <typename T> struct PairOf;
template <> struct PairOf<float> { using type = F2; };
template <> struct PairOf<double> { using type = D2; };

__device__ __forceinline__ F2 mk2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ D2 mk2(double a, double b) { return D2{a, b}; }
__device__ __forceinline__ float lo(F2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return x;
}
__device__ __forceinline__ float hi(F2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return y;
}
__device__ __forceinline__ double lo(D2 a) { return a.x; }
__device__ __forceinline__ double hi(D2 a) { return a.y; }

// splat<V>(x): x in every lane of V
template <typename V, typename T> __device__ __forceinline__ V splat(T x);
template <> __device__ __forceinline__ F2 splat<F2, float>(float x) { return mk2(x, x); }
template <> __device__ __forceinline__ D2 splat<D2, double>(double x) { return D2{x, x}; }
template <> __device__ __forceinline__ float splat<float, float>(float x) { return x; }
template <> __device__ __forceinline__ double splat<double, double>(double x) { return x; }

__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float vsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float vneg(float a) { return -a; }
__device__ __forceinline__ double vadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double vsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double vmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double vfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double vneg(double a) { return -a; }

__device__ __forceinline__ F2 vadd(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 vsub(F2 a, F2 b) {
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 vmul(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
// folds into the consuming instruction (measured: fma.rn.f32x2 with a negated
// operand runs as fast as without)
__device__ __forceinline__ F2 vneg(F2 a) { return mk2(-lo(a), -hi(a)); }
__device__ __forceinline__ D2 vadd(D2 a, D2 b) { return D2{vadd(a.x, b.x), vadd(a.y, b.y)}; }
__device__ __forceinline__ D2 vsub(D2 a, D2 b) { return D2{vsub(a.x, b.x), vsub(a.y, b.y)}; }
__device__ __forceinline__ D2 vmul(D2 a, D2 b) { return D2{vmul(a.x, b.x), vmul(a.y, b.y)}; }
__device__ __forceinline__ D2 vfma(D2 a, D2 b, D2 c) { return D2{vfma(a.x, b.x, c.x), vfma(a.y, b.y, c.y)}; }
__device__ __forceinline__ D2 vneg(D2 a) { return D2{-a.x, -a.y}; }

// a b - c
template <typename V>
__device__ __forceinline__ V vfms(V a, V b, V c) { return vfma(a, b, vneg(c)); }

// Shared memory by 32-bit address: LD(a) a point, LD2(a) a pair (aligned to the
// pair).  An address held as a number stays in its register; addresses derived
// from the shared array's symbol were recomputed at every use (25 of 515
// instructions per pair and plane).
template <typename T> struct Sh;
template <> struct Sh<float> {
    static __device__ __forceinline__ float ld(uint32_t a) {
        float r;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(r) : "r"(a));
        return r;
    }
    static __device__ __forceinline__ F2 ld2(uint32_t a) {
        F2 r;
        asm volatile("ld.shared.b64 %0, [%1];" : "=l"(r.v) : "r"(a));
        return r;
    }
    static __device__ __forceinline__ void st(uint32_t a, float v) {
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
    }
    static __device__ __forceinline__ void st2(uint32_t a, F2 v) {
        asm volatile("st.shared.b64 [%0], %1;" ::"r"(a), "l"(v.v) : "memory");
    }
    // ... where `on` (one predicated instruction, no branch)
    static __device__ __forceinline__ void st2_if(bool on, uint32_t a, F2 v) {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared.b64 [%0], %1;\n\t}" ::"r"(a), "l"(v.v),
                     "r"((uint32_t)on)
                     : "memory");
    }
};
template <> struct Sh<double> {
    static __device__ __forceinline__ double ld(uint32_t a) {
        double r;
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(r) : "r"(a));
        return r;
    }
    static __device__ __forceinline__ D2 ld2(uint32_t a) {
        D2 r;
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(r.x), "=d"(r.y) : "r"(a));
        return r;
    }
    static __device__ __forceinline__ void st(uint32_t a, double v) {
        asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
    }
    static __device__ __forceinline__ void st2(uint32_t a, D2 v) {
        asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
    }
    static __device__ __forceinline__ void st2_if(bool on, uint32_t a, D2 v) {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p st.shared.v2.f64 [%0], {%1, %2};\n\t}" ::"r"(a),
                     "d"(v.x), "d"(v.y), "r"((uint32_t)on)
                     : "memory");
    }
};

// pairs and points in global memory (pairs aligned)
__device__ __forceinline__ void stv(float* p, F2 a) { *reinterpret_cast<unsigned long long*>(p) = a.v; }
__device__ __forceinline__ void stv(double* p, D2 a) { *reinterpret_cast<double2*>(p) = make_double2(a.x, a.y); }
__device__ __forceinline__ void stv(float* p, float a) { *p = a; }
__device__ __forceinline__ void stv(double* p, double a) { *p = a; }

__device__ __forceinline__ F2 ldv2(const float* p) { return F2{*reinterpret_cast<const unsigned long long*>(p)}; }
__device__ __forceinline__ D2 ldv2(const double* p) {
    const double2 q = *reinterpret_cast<const double2*>(p);
    return D2{q.x, q.y};
}

template <typename V>
__device__ __forceinline__ void vcross(const V a[3], const V b[3], V c[3]) {
    c[0] = vfms(a[1], b[2], vmul(a[2], b[1]));
    c[1] = vfms(a[2], b[0], vmul(a[0], b[2]));
    c[2] = vfms(a[0], b[1], vmul(a[1], b[0]));
}

}  // namespace gmk
