// Placement of the per-lane decoder's warps and the loop they run (device),
// shared by the plain and the batched decode.
#pragma once
#include <stdint.h>

#include "rangecoder.cuh"

namespace vcg {

// A CTA is two warps per SM sub-partition, and one CTA per SM takes 8 x SMs
// warps' worth of atoms (32 consecutive ones of the payload-length order per
// warp). The first four warps of the CTAs hold the longer half, the longest on
// different SMs; each of the other four shares a sub-partition with one of
// them, the shortest with the longest, so that the sub-partitions carry about
// the same work and the longest atoms, which end last, run with the shortest
// ones or alone (warp w of a CTA runs on sub-partition w mod 4). Measured on the
// 32,768 atoms of the 1024^3 benchmark volume against the hardware's own placement
// of one-warp CTAs: 5.99 -> 5.57 ms at target 10, 3.94 -> 3.55 at 20, 0.72 -> 0.65
// at 100.
constexpr uint32_t kLaneWarps = 8;
constexpr int kLaneThreads = 32 * kLaneWarps;

// Four more warps, one per sub-partition, take the longest atoms alone where the
// others fill at most one warp of lanes a sub-partition: a lane's decision takes
// two to three times as long as a lone atom's, so the longest atoms set the time.
// Beside two warps of lanes they slow those down by more than they save: 32,768
// atoms take 6.40 ms with them and 5.57 without, 10,846 at target 50 1.46 and 1.83,
// 16,969 of four LODs at target 20 4.9 and 6.73.
constexpr uint32_t kSoloWarps = 4;
constexpr int kLaneCta = kLaneThreads + 32 * kSoloWarps;
constexpr uint32_t kSoloStage = 22u * 1024u;                 // stream bytes such a warp stages in shared memory
constexpr uint32_t kSoloSmem = kSoloWarps * kSoloStage;      // two CTAs of it fit an SM

// how many of n atoms run alone
__host__ __device__ inline uint32_t lane_solo(uint32_t n, uint32_t sms) {
    const uint32_t k = kSoloWarps * sms;
    return n > 32u * 4u * sms ? 0u : n < k ? n : k;
}

// the place in the payload-length order of the calling warp's atom, one of the
// solo warps of the first `sms` CTAs (else past every atom)
__device__ __forceinline__ uint32_t lane_solo_rank(uint32_t sms) {
    return blockIdx.x < sms ? ((threadIdx.x >> 5) - kLaneWarps) * sms + blockIdx.x : 0xFFFFFFFFu;
}

// The whole warp calls this: lane 0 decodes the stream and returns 1 for a
// malformed one; the others return at once.
template <class Sink>
__device__ __forceinline__ int solo_decode(uint8_t *stage, const uint8_t *src, uint32_t len, const uint32_t *bstart,
                                           Sink &&sink) {
    const uint32_t lane = threadIdx.x & 31u;
    const bool fits = stage_fits(len, kSoloStage);
    if (fits) stage_stream(stage, src, len, lane);
    __syncwarp();
    if (lane) return 0;
    return fits ? rc_decode_levels_sm(stage, len, bstart, sink) : rc_decode_levels_lat(src, len, bstart, sink);
}

inline unsigned lane_grid(uint64_t n_atoms, uint32_t sms) {
    const uint64_t warps = (n_atoms + 31) / 32, per = (uint64_t)kLaneWarps * sms;
    return (unsigned)((warps + per - 1) / per * sms);
}

// place of the calling thread's warp in the payload-length order of warps
__device__ __forceinline__ uint32_t lane_warp_rank(uint32_t sms) {
    const uint32_t w = threadIdx.x >> 5, pass = blockIdx.x / sms, slots = 4u * sms;
    const uint32_t slot = (w & 3u) * sms + blockIdx.x % sms;
    return w < 4u ? 2u * pass * slots + slot : (2u * pass + 2u) * slots - 1u - slot;
}

// Payload bytes (of a warp's longest atom) from which a round takes no zeros at
// once: longer payloads mean denser coefficients, whose runs of zeros are shorter.
// The line comes from 1,024 atoms replicated to 32,768, six zeros at once against
// none: 4.64 against 4.50 ms at a mean of 3,220 bytes (target 10), 2.85 against
// 3.34 at 1,624 (target 20), 0.56 against 0.76 at 323 (target 100). The 32,768
// different atoms of the 1024^3 benchmark volume, whose longest set the time, don't
// bear it out: six at once for every warp 5.40, 3.19 and 0.65 ms, none 5.60, 4.13
// and 0.91, by this line 5.57, 3.55 and 0.65.
constexpr uint32_t kLaneDenseBytes = 2560;

// The whole warp decodes its lanes' atoms (len: payload bytes, longest in lane 0).
__device__ __forceinline__ void decode_lanes(RcLane &L, uint32_t len, const uint32_t *bstart) {
    if (__shfl_sync(0xFFFFFFFFu, len, 0) >= kLaneDenseBytes)
        while (__any_sync(0xFFFFFFFFu, L.c != kLaneDone)) L.rounds<0>(bstart);
    else
        while (__any_sync(0xFFFFFFFFu, L.c != kLaneDone)) L.rounds<6>(bstart);
}

}  // namespace vcg
