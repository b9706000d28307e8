// What the kernels of a mixture of small feed-forward layers share: the activations without a gate and a token's weight of an expert.
#pragma once

#include "common.cuh"

namespace experts {

__device__ __forceinline__ float activate(float v, int kind) {
    if (kind == 0) { const float r = fmaxf(v, 0.f); return r * r; }                                    // relu^2
    if (kind == 1) return 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));  // gelu (tanh)
    if (kind == 3) return v / (1.f + expf(-v));                                                        // silu
    return v;
}

// Where the weights stand: w [tokens, ld], or null: 1 / listed for the entries of table[ids[token]] (an id outside the table reads its first
// row), 1 for the shared expert, whose number is E.
struct Weights {
    const float* w;
    int ld;
    const int *ids, *table;
    int listed, vocab, E;

    __device__ __forceinline__ float of(int token, int e) const {
        if (w) return __ldcg(w + (size_t)token * ld + e);
        if (e == E) return 1.f;
        int id = ids[token];
        if (id < 0 || id >= vocab) id = 0;
        float share = 0.f;
        for (int c = 0; c < listed; ++c) share = table[(size_t)id * listed + c] == e ? 1.f / (float)listed : share;
        return share;
    }
};

}  // namespace experts
