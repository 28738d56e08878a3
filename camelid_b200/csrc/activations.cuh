// The activations of the dense feed-forwards, shared by the kernels that apply them to finished sums.
#pragma once

__device__ __forceinline__ float gelu_tanh_f(float z) {
    return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}

// The activations of the dense feed-forwards: 0 none, 1 GELU (tanh form), 2 the square of ReLU, 3 GELU (exact,
// 0.5 z (1 + erf(z / sqrt 2))).
__device__ __forceinline__ float apply_act(float v, int act) {
    if (act == 1) return gelu_tanh_f(v);
    if (act == 2) { const float p = fmaxf(v, 0.f); return p * p; }
    if (act == 3) return 0.5f * v * (1.0f + erff(v * 0.7071067811865476f));
    return v;
}
