// Sums of several values over the lanes of a warp, in a fixed order.
#pragma once

namespace plx {
namespace {

// Adds v[0..V) over the lanes: every lane ends with the sums of the values whose
// index bits it owns, V / 32 of them (at least one); returns the first one's index.
template <int V>
__device__ __forceinline__ int lane_sums(double (&v)[V], int lane) {
    int base = 0;
    int len = V;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (len > 1) {
            const bool up = lane & o;
            len >>= 1;
#pragma unroll
            for (int k = 0; k < V / 2; ++k)
                if (k < len) {
                    const double send = up ? v[k] : v[k + len], keep = up ? v[k + len] : v[k];
                    v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            if (up) base += len;
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
    return base;
}

}  // namespace
}  // namespace plx
