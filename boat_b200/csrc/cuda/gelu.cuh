// gelu.cuh - GELU in its exact erf form and its derivative, shared by the element-wise kernels and the
// GEMM epilogues.
#pragma once

namespace boatcu {

// Phi(x) = (1 + erf(x/sqrt 2))/2 and e = exp(-x^2/2) from one exponential: erf by Abramowitz &
// Stegun 7.1.26, erf(z) = 1 - (a1 t + ... + a5 t^5) exp(-z^2), t = 1/(1 + p z), |error| <= 1.5e-7,
// whose exponential at z = |x|/sqrt 2 is the exp(-x^2/2) that the derivative needs anyway.
// erff + expf cost ~40 instructions per element and made the element-wise kernels instruction-bound
// (55 % of HBM bandwidth); this form needs one ex2, one rcp and a dozen FMAs.
__device__ __forceinline__ void gelu_parts(float x, float& phi, float& e) {
    const float z = fabsf(x) * 0.70710678118654752f;
    // one MUFU instruction each (relative error ~2^-22, far inside the 1.5e-7 of the formula)
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-0.72134752044448170f * x * x));   // exp(-x^2/2)
    float t;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fmaf(0.3275911f, z, 1.0f)));
    float poly = fmaf(1.061405429f, t, -1.453152027f);
    poly = fmaf(poly, t, 1.421413741f);
    poly = fmaf(poly, t, -0.284496736f);
    poly = fmaf(poly, t, 0.254829592f);
    const float half_erfc = 0.5f * poly * t * e;                   // (1 - erf(z)) / 2
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
    return fmaf(x * 0.3989422804014327f, e, phi);
}

}  // namespace boatcu
