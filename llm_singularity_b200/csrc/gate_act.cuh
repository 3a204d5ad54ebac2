// The activations of gated feed-forwards in 32-bit with CUDA's own functions, by id: act(g) * u.  silu(g) =
// g / (1 + exp(-g)); gelu in its tanh form, 0.5 g (1 + tanh(sqrt(2 / pi) (g + 0.044715 g^3))); none (gate * up);
// or the capped form with a limit L: g' = min(g, L), u' = clamp(u, -L, L), g' sigmoid(1.702 g') (u' + 1).
#pragma once

enum : int { LSB_ACT_SILU = 1, LSB_ACT_GELU_TANH = 2, LSB_ACT_NONE = 3, LSB_ACT_CAPPED_GLU = 5 };

__device__ __forceinline__ float lsb_gated(float g, float u, int act, float limit) {
    float a;
    if (act == LSB_ACT_CAPPED_GLU) {
        const float gc = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit) + 1.f;
        a = gc / (1.f + expf(-1.702f * gc));
    } else if (act == LSB_ACT_SILU) a = g / (1.f + expf(-g));
    else if (act == LSB_ACT_GELU_TANH)
        a = 0.5f * g * (1.f + tanhf(0.7978845608f * (g + 0.044715f * g * g * g)));
    else a = g;
    return a * u;
}
