// sfwi_d2.cuh — sums and products of 48 bits on the FP32 pipe, for what was
// FP64: the GB300's FP64 rate is 1/64 of its FP32 rate.
#pragma once

namespace sfwi {

// float pairs: the unevaluated sum h + l of two floats, |l| <= ulp(h)/2
// (Dekker 1971, Knuth's two-sum; the product's error term by FMA)
struct D2 {
    float h, l;
};
__device__ __forceinline__ D2 quick2(float a, float b) {  // |a| >= |b| or a = 0
    const float s = __fadd_rn(a, b);
    return D2{s, __fadd_rn(b, -__fadd_rn(s, -a))};
}
__device__ __forceinline__ D2 sum2(float a, float b) {
    const float s = __fadd_rn(a, b), t = __fadd_rn(s, -a);
    return D2{s, __fadd_rn(__fadd_rn(a, -__fadd_rn(s, -t)), __fadd_rn(b, -t))};
}
__device__ __forceinline__ D2 operator+(D2 a, D2 b) {  // to 2^-47 (|a| + |b|)
    const D2 s = sum2(a.h, b.h);
    return quick2(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ D2 operator-(D2 a) { return D2{-a.h, -a.l}; }
__device__ __forceinline__ D2 operator*(D2 a, D2 b) {
    const float p = __fmul_rn(a.h, b.h);
    float e = __fmaf_rn(a.h, b.h, -p);
    e = __fmaf_rn(a.h, b.l, e);
    e = __fmaf_rn(a.l, b.h, e);
    return quick2(p, e);
}
// acc + a b, the product exact
__device__ __forceinline__ D2 add_product(D2 acc, float a, float b) {
    const float p = __fmul_rn(a, b), e = __fmaf_rn(a, b, -p);
    const D2 s = sum2(acc.h, p);
    return quick2(s.h, __fadd_rn(s.l, __fadd_rn(acc.l, e)));
}

}  // namespace sfwi
