// Gated activations of feed-forwards (g = gate, u = up):
//   0 silu:   g / (1 + exp(-g)) * u
//   1 relu:   max(g, 0) * u
//   2 clamped sigmoid gate: g' = min(g, limit), u' = clamp(u, -limit, limit); g' * sigmoid(alpha g') * (u' + shift)
//   3 the tanh form of GELU on g, times u
//   4 relu2:  max(g, 0)^2 * u
// Without a gate the same functions of the one sum, with nothing to multiply (all but 2).
#pragma once

#define ACT_SILU 0
#define ACT_RELU 1
#define ACT_CLAMPED 2
#define ACT_GELU_TANH 3
#define ACT_RELU2 4

__device__ __forceinline__ float gated_activation(float g, float u, int act, float limit, float alpha, float shift) {
    if (act == ACT_RELU) return fmaxf(g, 0.f) * u;
    if (act == ACT_RELU2) { const float r = fmaxf(g, 0.f); return r * r * u; }
    if (act == ACT_GELU_TANH)        // 0.5 g (1 + tanh(sqrt(2/pi) (g + 0.044715 g^3))) u
        return 0.5f * g * (1.0f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) * u;
    if (act == ACT_CLAMPED) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
        return g / (1.0f + expf(-alpha * g)) * (u + shift);
    }
    return g / (1.0f + expf(-g)) * u;
}
