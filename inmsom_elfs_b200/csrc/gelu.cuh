// GELU of the closure network in the tanh form of Hendrycks & Gimpel
// (2016), x * g(x) with the gate g(x) = 0.5 (1 + tanh(sqrt(2/pi)(x +
// 0.044715 x^3))), the gate through the hardware tanh (tanh.approx.f32,
// relative error about 2^-11: below the BF16 rounding, 2^-9, of the
// activations).  Two forms of the one definition, so that the network the
// training kernel (closure_tc.cu) trains is the one that inference
// (closure.cu) runs: gelu_both, the value with its derivative g + x g',
// g' = 0.5 (1 - t^2) (sqrt(2/pi) + 3 * 0.044715 sqrt(2/pi) x^2), t the tanh,
// for training, and gelu2_pair, twice the value of two numbers, for
// inference.
#pragma once

namespace inmsom {
namespace closure {

constexpr float GELU_C0 = 0.7978845608028654f, GELU_C1 = 0.7978845608028654f * 0.044715f;

__device__ __forceinline__ float tanh_hw(float x)
{
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// 2 GELU = x (1 + t) of two values at once, in the two-wide FP32
// instructions: one multiplication fewer than GELU itself and bit for bit
// twice its value (a power-of-two scale commutes with the rounding).  The
// inference kernel feeds it to the next layer with that layer's weights
// halved, which leaves every product a * w unchanged
__device__ __forceinline__ void gelu2_pair(float &x, float &y)
{
    asm("{\n\t.reg .b64 v, q, c0, c1;\n\t.reg .f32 a, b;\n\t"
        "mov.b64 v, {%0, %1};\n\tmov.b64 c0, {%2, %2};\n\tmov.b64 c1, {%3, %3};\n\t"
        "mul.rn.f32x2 q, v, v;\n\tfma.rn.f32x2 q, c1, q, c0;\n\tmul.rn.f32x2 q, v, q;\n\t"
        "mov.b64 {a, b}, q;\n\ttanh.approx.f32 a, a;\n\ttanh.approx.f32 b, b;\n\tmov.b64 q, {a, b};\n\t"
        "fma.rn.f32x2 v, v, q, v;\n\tmov.b64 {%0, %1}, v;\n\t}"
        : "+f"(x), "+f"(y)
        : "f"(GELU_C0), "f"(GELU_C1));
}

// GELU and its derivative with one hyperbolic tangent (the training kernel)
__device__ __forceinline__ void gelu_both(float x, float &y, float &d)
{
    const float x2 = x * x, t = tanh_hw(x * fmaf(GELU_C1, x2, GELU_C0)), h = 0.5f * x;
    y = fmaf(h, t, h);
    d = fmaf(0.5f, 1.0f + t, h * (1.0f - t * t) * fmaf(3.0f * GELU_C1, x2, GELU_C0));
}

}  // namespace closure
}  // namespace inmsom
