// Arithmetic that the kernels write out operation by operation: reciprocal roots,
// packed float pairs, and a square root and a quotient in place of the library's
// (tests/cuda/arith_check.cu runs them against those).
#pragma once

#include <cuda_runtime.h>

#include <cfloat>

namespace fpb {

template <class T>
__device__ __forceinline__ T rsqrt_t(T v);
// float: the hardware reciprocal square root (rsqrtf's result on normal
// numbers) with arguments below the smallest normal float taken as that
// smallest normal (no rescaling of subnormal arguments; at a zero radius the
// projection's scale stays rp times a finite number, 0)
template <>
__device__ __forceinline__ float rsqrt_t<float>(float v) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fmaxf(v, FLT_MIN)));
    return r;
}
template <>
__device__ __forceinline__ double rsqrt_t<double>(double v) { return rsqrt(v); }

// Packed float pairs (a lane's two columns) in 64-bit registers: sm_100's f32x2
// arithmetic, each half one IEEE float32 operation rounded to nearest, with one
// exception: the assembler fuses a packed product into the packed difference that
// is its only use (one rounding less; on 131072 pairs all of the fused form), while
// a product with another use, and scalar differences of a packed product, stay
// apart. A difference of a product used nowhere else is written in scalar
// operations (sub_apart). Held as 64-bit values throughout: pairs packed from float2
// around every operation cost 84 register moves of 436 instructions per step.
typedef unsigned long long F2;
__device__ __forceinline__ F2 pk(float x, float y) {
    F2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
    return d;
}
__device__ __forceinline__ float lo(F2 a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float hi(F2 a) { return __uint_as_float((unsigned)(a >> 32)); }
__device__ __forceinline__ F2 sub2(F2 a, F2 b) {  // a - b
    F2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {  // a b
    F2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {  // a b + c, one rounding
    F2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// sqrt of both halves (>= 0): s = x y from the hardware's reciprocal root y,
// then one Newton step on s with its residual x - s^2 formed exactly by a fused
// operation (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000", 1990): the error before the last rounding is about 2^-44 of s,
// below sqrtf's half unit in all but about four cases in 10^6. Without the
// library call's branches (two per row and lane). Arguments below 2^-100, whose
// residual would fall among the subnormals (and below 2^-126 their reciprocal
// root at its clamp), are taken 2^96 times larger and their roots 2^-48; the
// residual of an infinite one is NaN, and the larger of that and x 2^-66 (below
// the root of every finite x) is infinite. The gradients of an image at 2^-46 of
// one square to such arguments, and a gap without them stops its solve early.
// Measured against the same without the two, and against sqrtf, on a
// solve of 64 x 512^2 with pixel weights: 36.84 to 37.14 ms, 35.70 to 36.50;
// 8 x 128^3: 88.6 to 89.1, 83.1 to 84.8 ms.
__device__ __forceinline__ F2 sqrt2(F2 x) {
    const bool a = lo(x) < 0x1p-100f, b = hi(x) < 0x1p-100f;
    const F2 xs = mul2(x, pk(a ? 0x1p96f : 1.f, b ? 0x1p96f : 1.f));
    const F2 y = pk(rsqrt_t(lo(xs)), rsqrt_t(hi(xs)));
    const F2 s = mul2(xs, y);
    const F2 e = pk(fmaf(-lo(s), lo(s), lo(xs)), fmaf(-hi(s), hi(s), hi(xs)));
    const F2 r = mul2(fma2(mul2(e, pk(0.5f, 0.5f)), y, s), pk(a ? 0x1p-48f : 1.f, b ? 0x1p-48f : 1.f));
    const F2 low = mul2(x, pk(0x1p-66f, 0x1p-66f));
    return pk(fmaxf(lo(r), lo(low)), fmaxf(hi(r), hi(low)));
}

// x / nr from yr = 1 / nr rounded: the quotient of the reciprocal corrected twice
// by its residual, formed exactly by a fused operation (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000", 1990): the rounded quotient,
// as the division gives it, while nothing underflows or overflows (equal to it on
// 4 M operands of 2^-300 to 2^300).
__device__ __forceinline__ double div_by(double x, double nr, double yr) {
    double q = __dmul_rn(x, yr);
    q = __fma_rn(__fma_rn(-q, nr, x), yr, q);
    return __fma_rn(__fma_rn(-q, nr, x), yr, q);
}

}  // namespace fpb
