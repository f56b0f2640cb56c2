// The rotation of the latent attention's query and key parts.
#pragma once
#include "common.cuh"

namespace hos {

// ---- rotary pairs ----------------------------------------------------------------------------
// The first rot_dims of P numbers are rotated, angle = position * inv_freq[i]; style 0 pairs (i, i + rot_dims / 2), style 1
// pairs (2i, 2i + 1).
struct LatentRot {
    const float* inv_freq;
    int rot_dims, style;
};

// number j of the rotated part `src`; tab: (sin, cos) per pair
template <typename T>
__device__ __forceinline__ float rotated(const T* __restrict__ src, int j, const float2* tab, const LatentRot& r) {
    if (j >= r.rot_dims) return to_float(src[j]);
    const int half = r.rot_dims >> 1;
    const bool second = r.style == 0 ? j >= half : (j & 1) != 0;
    const int i = r.style == 0 ? (second ? j - half : j) : j >> 1;
    const float2 sc = tab[i];
    const float u = to_float(src[r.style == 0 ? i : 2 * i]), v = to_float(src[r.style == 0 ? i + half : 2 * i + 1]);
    return second ? v * sc.y + u * sc.x : u * sc.y - v * sc.x;
}

}  // namespace hos
