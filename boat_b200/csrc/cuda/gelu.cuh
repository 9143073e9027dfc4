// gelu.cuh - GELU in its exact erf form and its derivative, shared by the element-wise kernels and the
// GEMM epilogues.
#pragma once
#include <stdint.h>

namespace boatcu {

// Phi(x) = (1 + erf(x/sqrt 2))/2 and e = exp(-x^2/2) from one exponential: erf by Abramowitz &
// Stegun 7.1.26, erf(z) = 1 - (a1 t + ... + a5 t^5) exp(-z^2), t = 1/(1 + p z), |error| <= 1.5e-7,
// whose exponential at z = |x|/sqrt 2 is the exp(-x^2/2) that the derivative needs anyway.
// erff + expf cost ~40 instructions per element and made the element-wise kernels instruction-bound
// (55 % of HBM bandwidth); this form needs one ex2, one rcp and a dozen FMAs.
// The halves below (1 - erf = 2 half_erfc) are folded into the coefficients, 1/sqrt 2 into p.
constexpr float kGeluP = 0.3275911f * 0.70710678118654752f, kGeluLog2 = -0.72134752044448170f, kGeluNorm = 0.3989422804014327f;
constexpr float kGeluA0 = 0.5f * 0.254829592f, kGeluA1 = 0.5f * -0.284496736f, kGeluA2 = 0.5f * 1.421413741f, kGeluA3 = 0.5f * -1.453152027f,
                kGeluA4 = 0.5f * 1.061405429f;

// one MUFU instruction each (relative error ~2^-22, far inside the 1.5e-7 of the formula)
__device__ __forceinline__ float gelu_ex2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float gelu_rcp(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ void gelu_parts(float x, float& phi, float& e) {
    e = gelu_ex2(x * x * kGeluLog2);                               // exp(-x^2/2)
    const float t = gelu_rcp(fmaf(fabsf(x), kGeluP, 1.0f));
    float poly = fmaf(kGeluA4, t, kGeluA3);
    poly = fmaf(poly, t, kGeluA2);
    poly = fmaf(poly, t, kGeluA1);
    poly = fmaf(poly, t, kGeluA0);
    const float half_erfc = poly * t * e;                          // (1 - erf(z)) / 2
    phi = x >= 0.f ? 1.0f - half_erfc : half_erfc;
}
__device__ __forceinline__ float gelu_f(float x) {
    float phi, e;
    gelu_parts(x, phi, e);
    return x * phi;
}
__device__ __forceinline__ float gelu_grad_f(float x) {
    float phi, e;
    gelu_parts(x, phi, e);
    return fmaf(x * kGeluNorm, e, phi);
}

// The same for two elements, the same bits, two to an instruction where the FMA pipe has such ones: beside a GEMM's main
// loop every instruction of the epilogue takes an issue slot from the warps that feed the tensor core.
struct GeluPair {
    uint64_t x, phi, e;
    static __device__ __forceinline__ uint64_t pack(float a, float b) {
        uint64_t r;
        asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
        return r;
    }
    static __device__ __forceinline__ void unpack(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
    static __device__ __forceinline__ uint64_t mul(uint64_t a, uint64_t b) {
        uint64_t r;
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
        return r;
    }
    static __device__ __forceinline__ uint64_t fma(uint64_t a, uint64_t b, uint64_t c) {
        uint64_t r;
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
        return r;
    }
    static __device__ __forceinline__ uint64_t both(float v) { return pack(v, v); }

    __device__ __forceinline__ GeluPair(float x0, float x1) {
        x = pack(x0, x1);
        float e0, e1, t0, t1, h0, h1, c0, c1;
        unpack(mul(mul(x, x), both(kGeluLog2)), e0, e1);
        e = pack(gelu_ex2(e0), gelu_ex2(e1));
        unpack(fma(pack(fabsf(x0), fabsf(x1)), both(kGeluP), both(1.0f)), t0, t1);
        const uint64_t t = pack(gelu_rcp(t0), gelu_rcp(t1));
        uint64_t poly = fma(both(kGeluA4), t, both(kGeluA3));
        poly = fma(poly, t, both(kGeluA2));
        poly = fma(poly, t, both(kGeluA1));
        poly = fma(poly, t, both(kGeluA0));
        const uint64_t half = mul(mul(poly, t), e);
        unpack(half, h0, h1);
        unpack(fma(half, both(-1.0f), both(1.0f)), c0, c1);
        phi = pack(x0 >= 0.f ? c0 : h0, x1 >= 0.f ? c1 : h1);
    }
    __device__ __forceinline__ void value(float& a, float& b) const { unpack(mul(x, phi), a, b); }
    __device__ __forceinline__ uint64_t grad() const { return fma(mul(x, both(kGeluNorm)), e, phi); }
};

}  // namespace boatcu
