// The exact GELU of the correctors, gelu(z) = z Phi(z), and its derivative
// Phi(z) + z phi(z), from one polynomial and one hardware exp2.
//
// With t = |z| the Gaussian tail Q(t) = (1 - erf(t / sqrt 2)) / 2 is 2^(p(t) - 1), where p
// is smooth and nearly quadratic with p(0) = 0: t times a degree-9 polynomial (weighted
// least squares on [0, 5.4], iterated to a minimax fit of Q; 4.8e-10 of absolute error with the
// coefficients rounded to FP32) serves every t, since beyond it p keeps falling (p(14) =
// -2689).  Leaving out the constant keeps its rounding away from small z.  The hardware's
// exp2 is low by 2e-8 to 5e-8 on average, which sums over many cells would not average
// out: p is raised by 2^-25 (1 + t^2), in its last step and by one unit in the last place of
// its second coefficient.  The mean errors over 1/4 of z are then below 4e-9 for gelu and
// 5e-9 for its derivative (8e-9 and 1.1e-8 without; 5e-8 and 1.2e-8 with erff).  Phi(z) is 1 - Q
// for z > 0 and Q for z <= 0, without the cancellation of
// 1 + erf for negative z: gelu(z) = max(z, 0) - |z| Q.  Two values share the packed FP32
// multiply-adds: about 12 instructions a value, against about 30 with erff.  NaN gives NaN;
// gelu is infinite at +infinity and NaN at -infinity, its derivative NaN at both, as erff's.
#pragma once
#include "common.cuh"

namespace inc {
namespace act {

INC_DEV float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Q(|z|) of two values
INC_DEV float2 gauss_tail2(float2 z) {
    const float2 t = make_float2(fabsf(z.x), fabsf(z.y));
    constexpr float c[10] = {-1.1511040925979614f,    -0.4592241644859314f,   -0.05242001637816429f,
                             0.00689349789172411f,    6.756559741916135e-05f, -0.0003273837792221457f,
                             9.60516044870019e-05f,   -1.5609344700351357e-05f, 1.4468790823229938e-06f,
                             -5.966594329720465e-08f};
    float2 p = make_float2(c[9], c[9]);
#pragma unroll
    for (int i = 8; i >= 0; --i) p = __ffma2_rn(p, t, make_float2(c[i], c[i]));
    p = __ffma2_rn(p, t, make_float2(2.9802322387695312e-08f, 2.9802322387695312e-08f));
    return __fmul2_rn(make_float2(ex2_approx(p.x), ex2_approx(p.y)), make_float2(0.5f, 0.5f));
}

// z Q(|z|) of two values (Q is 0 from z = 14 on: the bound keeps it from meeting infinity)
INC_DEV float2 tail_product2(float2 z, float2 q) {
    return __fmul2_rn(make_float2(fminf(z.x, 64.f), fminf(z.y, 64.f)), q);
}

// gelu of two values: max(z, 0) - |z Q(|z|)|
INC_DEV float2 gelu2(float2 z) {
    const float2 w = tail_product2(z, gauss_tail2(z));
    return make_float2(fmaxf(z.x, 0.f) - fabsf(w.x), fmaxf(z.y, 0.f) - fabsf(w.y));
}

// the derivative of gelu at two values: Phi(z) + z phi(z), phi(z) = exp(-z^2 / 2) / sqrt(2 pi)
INC_DEV float2 gelu_grad2(float2 z) {
    const float2 q = gauss_tail2(z);
    constexpr float k = -0.72134752044448170f, d = 0.39894228040143268f;  // -log2(e) / 2, 1 / sqrt(2 pi)
    const float2 zk = __fmul2_rn(__fmul2_rn(z, z), make_float2(k, k));
    const float2 zd = __fmul2_rn(z, make_float2(d, d));
    return make_float2(fmaf(zd.x, ex2_approx(zk.x), z.x > 0.f ? 1.f - q.x : q.x),
                       fmaf(zd.y, ex2_approx(zk.y), z.y > 0.f ? 1.f - q.y : q.y));
}

// gelu and its derivative of two values
INC_DEV void gelu_both2(float2 z, float2& g, float2& gp) {
    const float2 q = gauss_tail2(z), w = tail_product2(z, q);
    constexpr float k = -0.72134752044448170f, d = 0.39894228040143268f;  // -log2(e) / 2, 1 / sqrt(2 pi)
    g = make_float2(fmaxf(z.x, 0.f) - fabsf(w.x), fmaxf(z.y, 0.f) - fabsf(w.y));
    const float2 zk = __fmul2_rn(__fmul2_rn(z, z), make_float2(k, k));
    const float2 zd = __fmul2_rn(z, make_float2(d, d));
    gp = make_float2(fmaf(zd.x, ex2_approx(zk.x), z.x > 0.f ? 1.f - q.x : q.x),
                     fmaf(zd.y, ex2_approx(zk.y), z.y > 0.f ? 1.f - q.y : q.y));
}

}  // namespace act
}  // namespace inc
