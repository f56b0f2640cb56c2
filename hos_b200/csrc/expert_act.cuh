// The routed experts' activations.
#pragma once
#include "common.cuh"

namespace hos {

enum ExpertAct : int { kGatedSwish = 0, kReluSquare = 1 };

// y of an expert's inner number from its 32-bit gate and up products (kReluSquare: from the up product, given as g)
template <int ACT>
__device__ __forceinline__ float expert_act(float g, float u, float limit, float alpha, float up_shift) {
    if (ACT == kReluSquare) {
        const float r = fmaxf(g, 0.f);
        return r * r;
    }
    if (limit > 0.f) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
    }
    return g / (1.f + expf(-alpha * g)) * (u + up_shift);
}

}  // namespace hos
