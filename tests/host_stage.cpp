// Whether a stream is staged in shared memory (volume-compressor_gb300/csrc/
// rangecoder.cuh, stage_fits), built for the host with stand-ins for the CUDA
// intrinsics that the header names. Test infrastructure (tests/test_host_stage.py).
// Prints the lengths and rooms for which the answer is not that of 64-bit sums.
#include <stdint.h>
#include <stdio.h>

#define __device__
#define __host__
#define __forceinline__ inline
#define __global__
#define __constant__

static inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
template <class T> static inline T __ldg(const T *p) { return *p; }
static inline uint32_t __byte_perm(uint32_t, uint32_t, uint32_t) { return 0; }
static inline uint32_t __funnelshift_l(uint32_t, uint32_t, uint32_t) { return 0; }
static inline int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
static inline bool __any_sync(uint32_t, bool v) { return v; }
static inline uint32_t __reduce_max_sync(uint32_t, uint32_t v) { return v; }
struct uint2 { uint32_t x, y; };
struct uint4 { uint32_t x, y, z, w; };
static inline uint4 make_uint4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) { return uint4{a, b, c, d}; }

#include "rangecoder.cuh"

int main() {
    const uint32_t rooms[] = {0, 1, 15, 16, 17, 128, 22 * 1024, 40 * 1024, 226 * 1024};
    int tried = 0;
    auto check = [&](uint32_t len, uint32_t room) {
        ++tried;
        if (vcg::stage_fits(len, room) != ((uint64_t)len + vcg::kStagePad <= room)) printf("%u in %u\n", len, room);
    };
    for (uint32_t room : rooms) {
        for (uint32_t d = 0; d < 300; ++d) {
            check(d, room);
            check(0xFFFFFFFFu - d, room);
            check(0x80000000u - 150u + d, room);
            check(room - 150u + d, room);
        }
    }
    printf("%d tried\n", tried);
    return 0;
}
