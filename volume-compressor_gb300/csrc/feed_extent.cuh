// What the feeding warps of the tensor-core inverse transform (idct_mma.cuh) find
// out about an atom between them: the norm of its coefficients and how far along
// kz they go.
#pragma once
#include <stdint.h>

namespace vcg {

// Every warp puts its part for atom i, the warps meet, and one thread takes the
// atom's. Nothing keeps the other warps from putting theirs for atom i + 1
// meanwhile, so the parts of an odd and an even atom lie apart; those of atom
// i + 2 come after the meeting for i + 1, which that thread reaches after it has
// taken atom i's.
template <int WARPS>
struct FeedExtent {
    float norm[2][WARPS];
    uint32_t far[2][WARPS];

    __device__ __forceinline__ void put(uint32_t i, int warp, float n, uint32_t f) {
        norm[i & 1u][warp] = n;
        far[i & 1u][warp] = f;
    }
    __device__ __forceinline__ void take(uint32_t i, float &n, uint32_t &f) const {
        n = norm[i & 1u][0];
        f = far[i & 1u][0];
        for (int w = 1; w < WARPS; ++w) {
            n += norm[i & 1u][w];
            f = far[i & 1u][w] > f ? far[i & 1u][w] : f;
        }
    }
};

}  // namespace vcg
