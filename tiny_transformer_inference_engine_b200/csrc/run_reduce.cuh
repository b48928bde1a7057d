// Sums of several values per lane over a power-of-two number of adjacent lanes at once.
#pragma once

namespace ttie {

// Sums over 2 * O adjacent lanes (`slice` is the lane's index among them) of CNT values per lane at once: at
// every step a lane hands half of its values to the partner and adds the partner's other half to the half it keeps, so the
// run costs CNT - 1 shuffles instead of CNT * log2(lanes); once a lane is down to one value the remaining steps are plain
// butterfly additions.  Afterwards a lane holds, in v[0 ..], the totals of the values base, base + 1, ... (max(1, CNT / lanes) of them).
template <int O, int CNT>
struct RunReduce {
    static __device__ __forceinline__ void run(float* v, int slice, int& base) {
        if constexpr (O >= 1) {
            if constexpr (CNT > 1) {
                constexpr int HALF = CNT / 2;
                const bool up = (slice & O) != 0;
#pragma unroll
                for (int i = 0; i < HALF; ++i) {
                    const float send = up ? v[i] : v[i + HALF];
                    const float keep = up ? v[i + HALF] : v[i];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, O);
                }
                if (up) base += HALF;
                RunReduce<O / 2, HALF>::run(v, slice, base);
            } else {
                v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
                RunReduce<O / 2, 1>::run(v, slice, base);
            }
        }
    }
};

}  // namespace ttie
