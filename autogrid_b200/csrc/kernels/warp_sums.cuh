// Sums of several values over a warp.
#pragma once
#include <cuda_runtime.h>

namespace agb {

// Sums of V (a power of two, at most 16) values over the warp.  Each halving
// step hands half of the values to the other half of the lanes, so that V
// values take V - 1 + 5 - log2(V) shuffles instead of 5 V.  Lane l returns the
// sum of value l / (32 / V).
template <int V> __device__ __forceinline__ float warp_sums(float (&v)[V], int lane)
{
    int o = 16;
#pragma unroll
    for (int n = V / 2; n >= 1; n >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n; i++) {
            const float keep = up ? v[n + i] : v[i], give = up ? v[i] : v[n + i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
        o >>= 1;
    }
#pragma unroll
    for (int p = 16 / V; p >= 1; p >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], p);
    return v[0];
}

}  // namespace agb
