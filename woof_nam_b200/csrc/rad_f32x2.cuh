// rad_f32x2.cuh -- two floats side by side in one 64-bit register pair: the packed single-precision operations of
// sm_100 (add / sub / mul / fma .f32x2).  Each acts on both halves with the rounding of its scalar form, so a pair
// of independent g-points costs one issue slot per operation instead of two: with one g-point per lane the column kernels
// issued on 55-62 % of their cycles with the FMA pipe at 18-28 %, so issue slots, not FMA lanes, were what they ran out of
// (in pairs: 52-68 % and 14-31 % at half the time or less in the R/T and the LW sweeps).
#pragma once
#include <cuda_runtime.h>

namespace rad {

struct F2 {
    float x, y;
};
__device__ __forceinline__ F2 f2(float a) { return F2{a, a}; }
#define RAD_F32X2_OP2(name, op)                                                                                        \
    __device__ __forceinline__ F2 name(F2 a, F2 b)                                                                     \
    {                                                                                                                  \
        F2 d;                                                                                                          \
        asm("{\n .reg .b64 a, b, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n " op                               \
            " d, a, b;\n mov.b64 {%0, %1}, d;\n}"                                                                      \
            : "=f"(d.x), "=f"(d.y)                                                                                     \
            : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                                                 \
        return d;                                                                                                      \
    }
RAD_F32X2_OP2(operator+, "add.rn.ftz.f32x2")
RAD_F32X2_OP2(operator-, "sub.rn.ftz.f32x2")
RAD_F32X2_OP2(operator*, "mul.rn.ftz.f32x2")
RAD_F32X2_OP2(f2_add_rm, "add.rm.ftz.f32x2")   // rounded down
#undef RAD_F32X2_OP2
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)   // a b + c
{
    F2 d;
    asm("{\n .reg .b64 a, b, c, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n mov.b64 c, {%6, %7};\n"
        " fma.rn.ftz.f32x2 d, a, b, c;\n mov.b64 {%0, %1}, d;\n}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ F2 operator*(F2 a, float b) { return a * f2(b); }
__device__ __forceinline__ F2 operator+(F2 a, float b) { return a + f2(b); }
__device__ __forceinline__ F2 operator-(float a, F2 b) { return f2(a) - b; }
__device__ __forceinline__ F2 operator-(F2 a, float b) { return a - f2(b); }
__device__ __forceinline__ F2 neg2(F2 a) { return F2{-a.x, -a.y}; }
__device__ __forceinline__ F2 nma2(F2 a, F2 b, F2 c) { return fma2(neg2(a), b, c); }   // c - a b
__device__ __forceinline__ F2 max2(F2 a, float b) { return F2{fmaxf(a.x, b), fmaxf(a.y, b)}; }
__device__ __forceinline__ F2 min2(F2 a, float b) { return F2{fminf(a.x, b), fminf(a.y, b)}; }
__device__ __forceinline__ F2 clamp01(F2 a) { return F2{__saturatef(a.x), __saturatef(a.y)}; }
__device__ __forceinline__ F2 sqrt2(F2 a) { return F2{sqrtf(a.x), sqrtf(a.y)}; }
// a / b within 2 ulp for 2^-126 <= |b| <= 2^126 (div.approx: the same bound as the compiler's non-IEEE division,
// without its rescaling of the operands).  Above 2^126 the reciprocal, and with it the quotient, is flushed to zero; so
// a divisor that may be larger (an optical depth the caller gives) is divided by as F2_DOWN times it, a power of two
// that changes no rounding, and F2_DOWN goes into the quotient's next factor.
constexpr float F2_DOWN = 0.0625f;
__device__ __forceinline__ F2 div2(F2 a, F2 b) { return F2{__fdividef(a.x, b.x), __fdividef(a.y, b.y)}; }
__device__ __forceinline__ F2 rcp2(F2 a) { return F2{__fdividef(1.0f, a.x), __fdividef(1.0f, a.y)}; }
// a / b from r = rcp2(b) with one Newton step on the quotient (q + r (a - q b)): within an ulp of the quotient.
__device__ __forceinline__ F2 quot2(F2 a, F2 b, F2 r)
{
    const F2 q = a * r;
    return fma2(nma2(q, b, a), r, q);
}
__device__ __forceinline__ float ex2a(float x)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The same names on one float, for code that runs a pair or a single g-point (V = F2 or float).
template <class V> __device__ __forceinline__ V vset(float a);
template <> __device__ __forceinline__ F2 vset<F2>(float a) { return f2(a); }
template <> __device__ __forceinline__ float vset<float>(float a) { return a; }
__device__ __forceinline__ float fma2(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ float nma2(float a, float b, float c) { return fmaf(-a, b, c); }
__device__ __forceinline__ float f2_add_rm(float a, float b) { return __fadd_rd(a, b); }
__device__ __forceinline__ float max2(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ float div2(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ float rcp2(float a) { return __fdividef(1.0f, a); }
__device__ __forceinline__ float quot2(float a, float b, float r)
{
    const float q = a * r;
    return fmaf(nma2(q, b, a), r, q);
}
// a <= b, a < b per component
struct B2 {
    bool x, y;
};
__device__ __forceinline__ B2 le2(F2 a, float b) { return B2{a.x <= b, a.y <= b}; }
__device__ __forceinline__ bool le2(float a, float b) { return a <= b; }
__device__ __forceinline__ B2 lt2(F2 a, float b) { return B2{a.x < b, a.y < b}; }
__device__ __forceinline__ bool lt2(float a, float b) { return a < b; }
__device__ __forceinline__ F2 sel2(B2 c, F2 a, F2 b) { return F2{c.x ? a.x : b.x, c.y ? a.y : b.y}; }
__device__ __forceinline__ float sel2(bool c, float a, float b) { return c ? a : b; }

}  // namespace rad
