// Pulse edges of comparison words, shared by the demodulator and the pulse scans.
#pragma once

namespace vhsd {

// Edge bits of 32 consecutive samples given the state before the first one.
// NaN samples (and samples past the end) keep the state.
__device__ __forceinline__ unsigned edge_bits(unsigned cond, unsigned hold, unsigned& st) {
    if (hold == 0u) {
        unsigned prev = (cond << 1) | st;
        st = cond >> 31;
        return cond ^ prev;
    }
    unsigned s = st, edges = 0u;
    for (int b = 0; b < 32; b++) {
        if ((hold >> b) & 1u) continue;
        unsigned c = (cond >> b) & 1u;
        if (c != s) edges |= 1u << b;
        s = c;
    }
    st = s;
    return edges;
}

}  // namespace vhsd
