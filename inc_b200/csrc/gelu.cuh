// The exact GELU of the correctors, gelu(z) = z Phi(z), and its derivative
// Phi(z) + z phi(z), from one polynomial and one hardware exp2.
//
// With t = |z| the Gaussian tail Q(t) = (1 - erf(t / sqrt 2)) / 2 is 2^p(t), where
// p = log2 Q is smooth and nearly quadratic: a degree-10 polynomial on [0, 6.5]
// (weighted least squares iterated to a minimax fit of Q's absolute error, 1.2e-8)
// serves every t, since beyond it p keeps falling (p(14) = -424, where exp2 is 0).
// Phi(z) is 1 - Q for z > 0 and Q for z <= 0, without the cancellation of 1 + erf for
// negative z: gelu(z) = max(z, 0) - |z| Q.  Two values share the packed FP32
// multiply-adds: about 10 instructions a value, against about 30 with erff.  NaN and
// infinite arguments give NaN.
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
    constexpr float c[11] = {-0.9999999403953552f,    -1.151106357574463f,    -0.459200918674469f,
                             -0.052508581429719925f,  0.00705707585439086f,   -9.881718142423779e-05f,
                             -0.00022807865752838552f, 6.0456019127741456e-05f, -8.072857781371567e-06f,
                             5.776356601927546e-07f,  -1.751712552788831e-08f};
    float2 p = make_float2(c[10], c[10]);
#pragma unroll
    for (int i = 9; i >= 0; --i) p = __ffma2_rn(p, t, make_float2(c[i], c[i]));
    return make_float2(ex2_approx(p.x), ex2_approx(p.y));
}

// gelu of two values: max(z, 0) - |z Q(|z|)|
INC_DEV float2 gelu2(float2 z) {
    const float2 w = __fmul2_rn(z, gauss_tail2(z));
    return make_float2(fmaxf(z.x, 0.f) - fabsf(w.x), fmaxf(z.y, 0.f) - fabsf(w.y));
}

// gelu and its derivative of two values
INC_DEV void gelu_both2(float2 z, float2& g, float2& gp) {
    const float2 q = gauss_tail2(z), w = __fmul2_rn(z, q);
    constexpr float k = -0.72134752044448170f, d = 0.39894228040143268f;  // -log2(e) / 2, 1 / sqrt(2 pi)
    g = make_float2(fmaxf(z.x, 0.f) - fabsf(w.x), fmaxf(z.y, 0.f) - fabsf(w.y));
    const float2 zk = __fmul2_rn(__fmul2_rn(z, z), make_float2(k, k));
    const float2 zd = __fmul2_rn(z, make_float2(d, d));
    gp = make_float2(fmaf(zd.x, ex2_approx(zk.x), z.x > 0.f ? 1.f - q.x : q.x),
                     fmaf(zd.y, ex2_approx(zk.y), z.y > 0.f ? 1.f - q.y : q.y));
}

}  // namespace act
}  // namespace inc
