// Many sums over a warp's lanes at once, shared by the adjoint kernels.
#pragma once

#include "fmb_common.cuh"

namespace fmb {

// Sums of N values over a warp's lanes: every step exchanges half of what is left, a value without a partner is added in
// both lanes; one value remains per lane. `fold_ids` does to their numbers what `fold` does to the values.
template <int N, int BIT, int SIZE>
__device__ __forceinline__ void fold_step(float (&v)[SIZE], int lane) {
    constexpr int H = N / 2, M = N - H;
    const bool upper = (lane & BIT) != 0;
#pragma unroll
    for (int i = 0; i < H; ++i) {
        const float keep = upper ? v[i + M] : v[i], send = upper ? v[i] : v[i + M];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, BIT);
    }
    if (N & 1) v[M - 1] += __shfl_xor_sync(0xffffffffu, v[M - 1], BIT);
}
template <int N, int BIT, int SIZE>
__device__ __forceinline__ void fold(float (&v)[SIZE], int lane) {
    if constexpr (BIT > 0) {
        fold_step<N, BIT>(v, lane);
        fold<N - N / 2, BIT / 2>(v, lane);
    }
}
template <int N, int BIT, int SIZE>
__device__ __forceinline__ void fold_ids(int (&id)[SIZE], int lane) {
    if constexpr (BIT > 0) {
        constexpr int H = N / 2, M = N - H;
#pragma unroll
        for (int i = 0; i < H; ++i) id[i] = (lane & BIT) ? id[i + M] : id[i];
        fold_ids<M, BIT / 2>(id, lane);
    }
}

}  // namespace fmb
