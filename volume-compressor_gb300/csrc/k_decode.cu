// Decode kernels: per-atom list capacities + scan, range decoders, and the
// dequantise + inverse DCT-32 + crop.
//
//   k_caps       one thread per box atom: coefficient-list capacity
//   k_scan_u64   one CTA: exclusive scan of the capacities (list placement)
//   k_rc_decode  one thread per PRESENT atom: serial range decode of its
//                payload into (scan position, level) pairs (src/vc/vc.c:545-560);
//                one atom per warp for small decodes
//   k_rc_lanes   the same for large ones: one atom per lane, the longest of
//                a middling one alone in a warp
//   k_idct       persistent, one CTA per SM: levels dequantised
//                (src/vc/vc.c:327-338), inverse passes along x, y, z on the tensor
//                cores (idct_mma.cuh), dc added, clamped, cropped into the box
//                (src/vc/vc.c:219-229, 1535-1555); atoms that cannot go there,
//                and small decodes (k_idct_bf), take the butterfly on a 32x32x32
//                i32 tile in shared memory (idct_tile.cuh)
#include <cuda_runtime.h>
#include <stdint.h>

#include "dct32.cuh"
#include "kernels.cuh"
#include "idct_mma.cuh"
#include "idct_tile.cuh"
#include "rangecoder.cuh"
#include "rc_lanes.cuh"

namespace vcg {


__global__ void k_caps(DecodeJob J) {
    uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= J.n_atoms) return;
    uint32_t az, ay, ax;
    box_atom(J, t, az, ay, ax);
    vcd_atom e = J.atoms[job_atom(J, t, az, ay, ax)];
    uint64_t cap = 0;
    if (e.kind == VCD_PRESENT) {   // slots of the list, a multiple of 32 (the host's entry_cap)
        cap = 8ull * (e.len - 1) + 64ull;
        if (cap > VCD_MAX_ENTRIES) cap = VCD_MAX_ENTRIES;
        cap = (cap + 31) & ~31ull;
    }
    J.ent_off[t] = cap;
}

// Exclusive scan of v[0..n) in place (+ base), total -> *total. One CTA of 1024
// threads walks the array in tiles of 4096 carrying the running sum.
__global__ void __launch_bounds__(1024) k_scan_u64(uint64_t *v, uint64_t n, uint64_t base, uint64_t *total) {
    __shared__ uint64_t warp_sum[32];
    __shared__ uint64_t carry_s;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) carry_s = base;
    __syncthreads();
    for (uint64_t tile = 0; tile < n; tile += 4096) {
        uint64_t i0 = tile + (uint64_t)tid * 4;
        uint64_t a[4];
        uint64_t s = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            a[j] = (i0 + j < n) ? v[i0 + j] : 0;
            uint64_t x = a[j];
            a[j] = s;
            s += x;
        }
        uint64_t incl = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint64_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) warp_sum[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            uint64_t w = warp_sum[lane], wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                uint64_t y = __shfl_up_sync(0xFFFFFFFFu, wi, o);
                if (lane >= o) wi += y;
            }
            warp_sum[lane] = wi - w;   // exclusive prefix of warp totals
        }
        __syncthreads();
        uint64_t excl = carry_s + warp_sum[wid] + (incl - s);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i0 + j < n) v[i0 + j] = excl + a[j];
        __syncthreads();
        if (tid == 1023) carry_s = excl + s;
        __syncthreads();
    }
    if (tid == 0 && total) *total = carry_s;
}

// One warp per CTA, G atoms per warp (rc_lanes_for): G = 1 runs a one-atom
// decoder on lane 0, G > 1 the lockstep decoder on lanes 0..G-1. With J.order
// (G = 1 only), CTA i decodes the i-th atom of the payload-length order. With
// `stage` bytes of dynamic shared memory (G = 1) the whole warp first copies the
// atom's stream there, for rc_decode_levels_sm; streams that do not fit are read
// from global memory (rc_decode_levels_lat; without staging the compact
// rc_decode_levels_lane).
__global__ void __launch_bounds__(32) k_rc_decode(DecodeJob J, uint32_t G, uint32_t stage_bytes) {
    extern __shared__ __align__(16) uint8_t stage[];
    __shared__ uint32_t bstart[9];
    if (threadIdx.x < 9) bstart[threadIdx.x] = J.band_start[threadIdx.x];
    __syncthreads();
    const uint32_t lane = threadIdx.x;
    const bool staged = G == 1 && stage_bytes;
    if (G == 1 && !staged && lane != 0) return;
    const uint32_t slot = G == 1 ? 0u : lane;   // (G = 1: every lane of a staging warp takes lane 0's atom)
    uint64_t t = (uint64_t)blockIdx.x * G + slot;
    if (J.order) {
        if (t >= J.sort_ctl[kSortBuckets]) return;
        t = J.order[t];
    }
    bool active = false;
    vcd_atom e = {};
    if (slot < G && t < J.n_atoms) {
        uint32_t az, ay, ax;
        box_atom(J, t, az, ay, ax);
        e = J.atoms[job_atom(J, t, az, ay, ax)];
        active = e.kind == VCD_PRESENT;
        if (!active && lane == 0) J.cnt[t] = 0;
    }
    bool in_smem = false;
    if (staged) {
        const uint32_t len = active ? e.len - 1u : 0u;
        in_smem = active && stage_fits(len, stage_bytes);
        if (in_smem) {
            stage_stream(stage, J.arc + e.off + 1, len, lane);
            __syncwarp();
        }
        if (lane != 0) return;
    }
    uint32_t cap = 0, n = 0;
    uint32_t *dst = J.ent;
    if (active) {
        cap = 8u * (e.len - 1u) + 64u;
        if (e.len - 1u > VCD_MAX_ENTRIES / 8u || cap > VCD_MAX_ENTRIES) cap = VCD_MAX_ENTRIES;
        dst = J.ent + J.ent_off[t];
    }
    // entries carry the scan position; the transform kernel maps it to raster
    auto sink = [&](uint32_t p, uint32_t lv) {
        if (n < cap) dst[n] = p | (lv << 16);
        ++n;
    };
    int bad = 0;
    if (G == 1) {
        if (in_smem) bad = rc_decode_levels_sm(stage, e.len - 1, bstart, sink);
        else if (active && stage_bytes) bad = rc_decode_levels_lat(J.arc + e.off + 1, e.len - 1, bstart, sink);
        else if (active) bad = rc_decode_levels_lane(J.arc + e.off + 1, e.len - 1, bstart, sink);
    } else {
        bad = rc_decode_levels_warp(J.arc + e.off + 1, active ? e.len - 1 : 0u, active, bstart, sink);
    }
    if (!active) return;
    uint32_t flags = (n > cap ? kEntOverflow : 0u) | (bad ? kEntBad : 0u);
    J.cnt[t] = (n > cap ? cap : n) | flags;
    atomicAdd(J.nnz_total, (unsigned long long)(n > cap ? cap : n));
    if (bad) atomicMin(J.err, (uint32_t)(t < 0xFFFFFFFFull ? t : 0xFFFFFFFEull));
}

// ---- per-lane decoder (RcLane) for large decodes. The atoms are first put in
// order of payload length, longest first (a counting sort on length / 32), so
// that the 32 atoms of a warp need about the same number of steps: a warp
// runs until its slowest lane is done.
__device__ __forceinline__ uint32_t len_bucket(uint32_t len) {
    const uint32_t k = len >> 5;
    return kSortBuckets - 1u - (k < kSortBuckets - 1u ? k : kSortBuckets - 1u);
}

__global__ void k_len_hist(DecodeJob J) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= J.n_atoms) return;
    uint32_t az, ay, ax;
    box_atom(J, t, az, ay, ax);
    const vcd_atom e = J.atoms[job_atom(J, t, az, ay, ax)];
    if (e.kind == VCD_PRESENT) atomicAdd(&J.sort_ctl[len_bucket(e.len)], 1u);
}

// exclusive scan of the kSortBuckets counters in place; their sum -> ctl[kSortBuckets]
__global__ void __launch_bounds__(1024) k_len_scan(uint32_t *ctl) {
    __shared__ uint32_t warp_sum[32];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
    uint32_t a[4], s = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        a[j] = s;
        s += ctl[tid * 4 + j];
    }
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31) warp_sum[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        const uint32_t w = warp_sum[lane];
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, wi, o);
            if (lane >= (uint32_t)o) wi += y;
        }
        warp_sum[lane] = wi - w;
        if (lane == 31) ctl[kSortBuckets] = wi;
    }
    __syncthreads();
    const uint32_t base = warp_sum[wid] + incl - s;
#pragma unroll
    for (int j = 0; j < 4; ++j) ctl[tid * 4 + j] = base + a[j];
}

__global__ void k_len_scatter(DecodeJob J) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= J.n_atoms) return;
    uint32_t az, ay, ax;
    box_atom(J, t, az, ay, ax);
    const vcd_atom e = J.atoms[job_atom(J, t, az, ay, ax)];
    if (e.kind == VCD_PRESENT) J.order[atomicAdd(&J.sort_ctl[len_bucket(e.len)], 1u)] = (uint32_t)t;
    else J.order[J.sort_ctl[kSortBuckets] + atomicAdd(&J.sort_ctl[kSortBuckets + 1], 1u)] = (uint32_t)t;   // after them
}

static_assert(kSortBuckets == 4 * 1024, "k_len_scan: 1024 threads x 4 counters");

template <bool SOLO>
__global__ void __launch_bounds__(SOLO ? kLaneCta : kLaneThreads) k_rc_lanes(DecodeJob J, uint32_t sms) {
    extern __shared__ __align__(16) uint8_t stage[];
    __shared__ uint32_t bstart[10];   // the band table and a copy of its end (RcLane)
    __shared__ uint32_t S[kLaneWarps][kLaneRows * 32];
    if (threadIdx.x < 10) bstart[threadIdx.x] = J.band_start[threadIdx.x < 9 ? threadIdx.x : 8];
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t n_present = J.sort_ctl[kSortBuckets], alone = SOLO ? lane_solo(n_present, sms) : 0u;
    if constexpr (SOLO) if (threadIdx.x >= kLaneThreads) {
        const uint32_t s = lane_solo_rank(sms);
        if (s >= alone) return;
        const uint64_t t = J.order[s];
        uint32_t az, ay, ax;
        box_atom(J, t, az, ay, ax);
        const vcd_atom e = J.atoms[job_atom(J, t, az, ay, ax)];
        uint32_t cap = 8u * (e.len - 1u) + 64u, n = 0;
        if (e.len - 1u > VCD_MAX_ENTRIES / 8u || cap > VCD_MAX_ENTRIES) cap = VCD_MAX_ENTRIES;
        uint32_t *dst = J.ent + J.ent_off[t];
        const int bad = solo_decode(stage + ((threadIdx.x >> 5) - kLaneWarps) * kSoloStage, J.arc + e.off + 1, e.len - 1u,
                                    bstart, [&](uint32_t p, uint32_t lv) {
                                        if (n < cap) dst[n] = p | (lv << 16);
                                        ++n;
                                    });
        if (lane) return;
        J.cnt[t] = (n > cap ? cap : n) | (n > cap ? kEntOverflow : 0u) | (bad ? kEntBad : 0u);
        atomicAdd(J.nnz_total, (unsigned long long)(n > cap ? cap : n));
        if (bad) atomicMin(J.err, (uint32_t)(t < 0xFFFFFFFFull ? t : 0xFFFFFFFEull));
        return;
    }
    const uint64_t i = alone + 32ull * lane_warp_rank(sms) + lane;
    const bool active = i < n_present;
    uint64_t t = 0;
    vcd_atom e = {};
    uint32_t cap = 0;
    uint32_t *dst = J.ent;
    if (active) {
        t = J.order[i];
        uint32_t az, ay, ax;
        box_atom(J, t, az, ay, ax);
        e = J.atoms[job_atom(J, t, az, ay, ax)];
        cap = 8u * (e.len - 1u) + 64u;
        if (e.len - 1u > VCD_MAX_ENTRIES / 8u || cap > VCD_MAX_ENTRIES) cap = VCD_MAX_ENTRIES;
        dst = J.ent + J.ent_off[t];
    }
    RcLane L;
    L.init(J.arc + e.off + 1, e.len - 1u, active, bstart, &S[threadIdx.x >> 5][lane], 32, dst, cap);
    decode_lanes(L, e.len, bstart);
    if (!active) return;
    const uint32_t n = L.n > cap ? cap : L.n;
    J.cnt[t] = n | (L.n > cap ? kEntOverflow : 0u) | (L.bad ? kEntBad : 0u);
    atomicAdd(J.nnz_total, (unsigned long long)n);
    if (L.bad) atomicMin(J.err, (uint32_t)(t < 0xFFFFFFFFull ? t : 0xFFFFFFFEull));
}

// Solo atoms: the first n atoms of the length order (the longest payloads)
// each get a warp of their own whose lane 0 runs the latency decoder, on a
// second stream beside k_rc_lanes, which takes the atoms after them. The
// longest atoms set the per-lane decoder's time (every lane steps at about the
// same pace, whatever its atom, bound by its own dependency chain). Off by
// default (vcg_set_rc_solo): where the solo warps land is the hardware's choice,
// and a second kernel may run after the first instead of beside it. Where it
// pays, k_rc_lanes has solo warps of its own (lane_solo).
__global__ void __launch_bounds__(32) k_rc_solo(DecodeJob J, uint32_t n) {
    __shared__ uint32_t bstart[9];
    if (threadIdx.x < 9) bstart[threadIdx.x] = J.band_start[threadIdx.x];
    __syncthreads();
    const uint32_t k = blockIdx.x;
    if (threadIdx.x != 0 || k >= n || k >= J.sort_ctl[kSortBuckets]) return;
    const uint64_t t = J.order[k];
    uint32_t az, ay, ax;
    box_atom(J, t, az, ay, ax);
    const vcd_atom e = J.atoms[job_atom(J, t, az, ay, ax)];   // PRESENT: the order puts those first
    uint32_t cap = 8u * (e.len - 1u) + 64u;
    if (e.len - 1u > VCD_MAX_ENTRIES / 8u || cap > VCD_MAX_ENTRIES) cap = VCD_MAX_ENTRIES;
    uint32_t *dst = J.ent + J.ent_off[t];
    uint32_t m = 0;
    auto sink = [&](uint32_t p, uint32_t lv) {
        if (m < cap) dst[m] = p | (lv << 16);
        ++m;
    };
    const int bad = rc_decode_levels_lat(J.arc + e.off + 1, e.len - 1u, bstart, sink);
    J.cnt[t] = (m > cap ? cap : m) | (m > cap ? kEntOverflow : 0u) | (bad ? kEntBad : 0u);
    atomicAdd(J.nnz_total, (unsigned long long)(m > cap ? cap : m));
    if (bad) atomicMin(J.err, (uint32_t)(t < 0xFFFFFFFFull ? t : 0xFFFFFFFEull));
}

// ctl[kSortBuckets + 2] = the PRESENT atoms left to the per-lane warps after n solo atoms
__global__ void k_solo_split(uint32_t *ctl, uint32_t n) {
    const uint32_t np = ctl[kSortBuckets];
    ctl[kSortBuckets + 2] = np - (n < np ? n : np);
}

void launch_len_scan(uint32_t *sort_ctl, cudaStream_t s) { k_len_scan<<<1, 1024, 0, s>>>(sort_ctl); }

static void launch_len_sort(const DecodeJob &J, cudaStream_t s) {
    const unsigned nb = (unsigned)((J.n_atoms + 255) / 256);
    cudaMemsetAsync(J.sort_ctl, 0, sort_ctl_words() * 4, s);
    k_len_hist<<<nb, 256, 0, s>>>(J);
    k_len_scan<<<1, 1024, 0, s>>>(J.sort_ctl);
    k_len_scatter<<<nb, 256, 0, s>>>(J);
}

// Shared memory per CTA that stages a stream of a decode of n one-atom warps,
// the longest payload max_len bytes: enough for every stream if the CTAs that
// one SM gets then fit it (228 KiB, 1 KiB of it reserved per CTA); with at most
// one atom per sub-partition as much as fits (a longer stream is read from
// global memory), above that all or none (0). Measured, range decode of 2,048
// and 3,072 atoms: staged 3.35 / 3.91 ms at target 10, 1.84 / 2.17 at 20, 0.33 /
// 0.39 at 100; the compact decoder from global memory 4.40 ms for 2,048 at 10;
// the per-lane decoder 4.58 / 4.58 at 10.
constexpr uint32_t kStageMax = 226u * 1024u;
static uint32_t stage_bytes_for(uint64_t n, uint32_t max_len, uint32_t sms) {
    const uint64_t per_sm = (n + sms - 1) / sms;
    const uint64_t room = 228ull * 1024u / per_sm;
    const uint32_t fit = room > 1280u ? (uint32_t)(room - 1152u < kStageMax ? room - 1152u : kStageMax) & ~127u : 0u;
    if (stage_fits(max_len, fit)) return (max_len + kStagePad + 127u) & ~127u;
    return n <= 4ull * sms ? fit : 0u;
}

constexpr uint32_t kUnstagedPerSm = 28;

// The range decode of every PRESENT box atom:
//   up to rc_scalar_warps() atoms per SM sub-partition: one atom per warp,
//     longest payload first above one per sub-partition (the tail is the
//     shortest atoms), the stream staged in shared memory if all streams fit
//     (at the default policy up to kUnstagedPerSm atoms per SM if not: 4,320
//     atoms at target 10 take 5.75 ms so and 4.39 a lane each, 4,000, which fit,
//     4.74 and 4.43; of 10 KB streams 4,160 take 9.1 and 8.8, 3,200 8.6 and 8.7);
//   above: the per-lane decoder over atoms sorted by payload length, the
//     rc_solo_for() longest on the latency decoder (k_rc_solo, a warp each,
//     on the second stream of ev, between its fork and join events).
// Without an order buffer (no-alloc path) the unsorted forms are used.
static void launch_rc(const DecodeJob &J, int num_sms, cudaStream_t s, const StageEvents *ev) {
    uint32_t G = rc_lanes_for(J.n_atoms, (uint32_t)num_sms, rc_scalar_warps());
    const bool sorted = J.order && J.sort_ctl && rc_sorts(J.n_atoms, (uint32_t)num_sms);
    const uint32_t stage = G == 1 ? stage_bytes_for(J.n_atoms, J.max_len, (uint32_t)num_sms) : 0u;
    if (sorted && G == 1 && !stage && rc_scalar_warps() == kRcScalarWarpsDefault &&
        J.n_atoms > (uint64_t)kUnstagedPerSm * (uint32_t)num_sms)
        G = 32;
    if (sorted) launch_len_sort(J, s);
    if (G > 1 && sorted) {
        const uint32_t ns = ev && ev->side && ev->fork && ev->join ? rc_solo_for(J.n_atoms, (uint32_t)num_sms) : 0u;
        DecodeJob Jl = J;
        if (ns) {
            // (fewer PRESENT atoms than ns: k_solo_split's count is 0 and the
            // shifted order is not read)
            k_solo_split<<<1, 1, 0, s>>>(J.sort_ctl, ns);
            cudaEventRecord(ev->fork, s);
            cudaStreamWaitEvent(ev->side, ev->fork, 0);
            k_rc_solo<<<ns, 32, 0, ev->side>>>(J, ns);
            cudaEventRecord(ev->join, ev->side);
            Jl.order = J.order + ns;
            Jl.sort_ctl = J.sort_ctl + 2;   // Jl.sort_ctl[kSortBuckets]: the per-lane count
        }
        const unsigned lane_blocks = lane_grid(J.n_atoms - ns, (uint32_t)num_sms);
        smem_attr((const void *)k_rc_lanes<true>, (int)kSoloSmem);
        if (!lane_blocks) {   // every atom solo on the second stream
        } else if (lane_solo((uint32_t)(J.n_atoms < 0xFFFFFFFFull ? J.n_atoms : 0xFFFFFFFFull), (uint32_t)num_sms)) {
            k_rc_lanes<true><<<lane_blocks, kLaneCta, kSoloSmem, s>>>(Jl, (uint32_t)num_sms);
        } else {
            k_rc_lanes<false><<<lane_blocks, kLaneThreads, 0, s>>>(Jl, (uint32_t)num_sms);
        }
        if (ns) cudaStreamWaitEvent(s, ev->join, 0);
        return;
    }
    DecodeJob Jr = J;
    if (!sorted) {
        Jr.order = nullptr;
        Jr.sort_ctl = nullptr;
    }
    if (stage) smem_attr((const void *)k_rc_decode, (int)kStageMax);
    k_rc_decode<<<(unsigned)((J.n_atoms + G - 1) / G), 32, stage, s>>>(Jr, G, stage);
}

// Box atom t without the tensor cores: zeros (ABSENT, KNOWN_ZERO, malformed), or
// dequantise + butterfly + crop into the box raster, by NT threads (tid =
// 0..NT-1) that meet at barrier BAR (tile_sync); ends with one.
template <int NT, int BAR>
__device__ __forceinline__ void idct_atom(const DecodeJob &J, uint64_t t, int32_t *T, const int32_t *dqs,
                                          const int32_t *dqb, const uint32_t *alt, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
    uint32_t az, ay, ax;
    box_atom(J, t, az, ay, ax);
    const vcd_atom e = J.atoms[job_atom(J, t, az, ay, ax)];
    Crop k;
    const uint32_t gx = ax * 32, gy = ay * 32, gz = az * 32;
    k.set(gx, gy, gz, J.x0, J.y0, J.z0, J.x1, J.y1, J.z1);
    uint8_t *obase = J.out + ((uint64_t)(gz + k.lz0 - J.z0) * J.oy + (gy + k.ly0 - J.y0)) * J.ox + (gx + k.lx0 - J.x0);
    const uint32_t c = e.kind == VCD_PRESENT ? J.cnt[t] : kEntBad;
    if (e.kind != VCD_PRESENT || (c & kEntBad)) {   // ABSENT / KNOWN_ZERO -> zeros
        zero_window<NT>(obase, J.ox, J.oy, k, (uint32_t)tid);
        return;
    }
    const int32_t dc = J.arc[e.off];
    idct_tile_xy<NT, BAR>(T, J.arc, e, c, J.ent + J.ent_off[t], J.scan, J.band_start, dqs, dqb, alt, tid);
    const bool full = k.lz0 == 0 && k.lz1 == 32;
    for (int y = warp; y < 32; y += NT / 32) {
        int32_t o[32];
        idct_col_z(T, y, lane, o);
        if (full) store_col_full(obase, J.ox, J.oy, k, y, lane, o, dc);
        else store_col(obase, J.ox, J.oy, k, y, lane, o, dc);
    }
    tile_sync<NT, BAR>();
}
__device__ __noinline__ void idct_atom_other(const DecodeJob &J, uint64_t t, int32_t *T, int tid) {   // in k_idct
    idct_atom<kMmaThreads, kMmaBar>(J, t, T, J.dq->step, J.dq->bias, J.alt_mask, tid);
}

// Few atoms: the butterfly on the CUDA cores. With one to three atoms per SM the
// tensor-core kernel's start (TMEM, matrix pieces, first lists) and the chain of
// its passes are not hidden: one atom 33 us against 20, 576 atoms 68 against 66,
// 4,096 atoms 0.36 ms against 0.58.
constexpr int kBfThreads = 512;   // 16 warps per atom (measured faster than 8 on GB300)
constexpr uint64_t kMmaAtomsPerSm = 4;
__global__ void __launch_bounds__(kBfThreads, 1) k_idct_bf(DecodeJob J) {
    extern __shared__ int32_t T[];   // 32 slabs x padded 32x32 (idct_tile.cuh)
    __shared__ int32_t dqs[VCD_NCLASS], dqb[VCD_NCLASS];
    __shared__ uint32_t alt[1024];
    const int tid = threadIdx.x;
    for (int i = tid; i < VCD_NCLASS; i += kBfThreads) { dqs[i] = J.dq->step[i]; dqb[i] = J.dq->bias[i]; }
    for (int i = tid; i < 1024; i += kBfThreads) alt[i] = J.alt_mask[i];
    __syncthreads();
    for (uint64_t t = J.t_lo + blockIdx.x; t < J.t_hi; t += gridDim.x) idct_atom<kBfThreads, 0>(J, t, T, dqs, dqb, alt, tid);
}

// Dynamic shared memory of k_idct from a 1024-byte boundary on: the operand of
// the tensor-core passes, or the butterfly's tile in its place; the matrix
// pieces; the feeders' ring.
constexpr uint32_t kIdctB = (uint32_t)((kIdctTileBytes + 1023) & ~(size_t)1023);
constexpr size_t kIdctSmem = 1024 + kIdctB + kMmaB + kMmaRing;
static_assert(kMmaA <= kIdctB, "the matrix pieces lie behind the operand and the tile");

// Persistent: one CTA per SM, atoms blockIdx.x, blockIdx.x + grid, ...
__global__ void __launch_bounds__(kMmaCta, 1) k_idct(DecodeJob J) {
    extern __shared__ uint8_t dyn[];
    __shared__ __align__(16) MmaShared M;
    uint8_t *A = dyn + ((1024u - (smem_u32(dyn) & 1023u)) & 1023u), *B = A + kIdctB, *ring = B + kMmaB;
    const int tid = threadIdx.x;
    mma_setup(M, B);
    if (tid >= kMmaFeed) {
        mma_feed(M, ring, J.dq, J.place, [&](uint32_t i, MmaAtom &a) {
            const uint64_t t = J.t_lo + blockIdx.x + (uint64_t)i * gridDim.x;
            if (t >= J.t_hi) return false;
            uint32_t az, ay, ax;
            box_atom(J, t, az, ay, ax);
            const vcd_atom e = J.atoms[job_atom(J, t, az, ay, ax)];
            a.id = t;
            a.src = J.ent + J.ent_off[t];
            const uint32_t c = e.kind == VCD_PRESENT ? J.cnt[t] : kEntBad;
            a.n = c & kEntMask;
            a.tensor = !(c & (kEntBad | kEntOverflow));
            a.dc = a.tensor ? (int32_t)J.arc[e.off] : 0;
            const uint32_t gx = ax * 32, gy = ay * 32, gz = az * 32;
            a.crop.set(gx, gy, gz, J.x0, J.y0, J.z0, J.x1, J.y1, J.z1);
            a.out = J.out + ((uint64_t)(gz + a.crop.lz0 - J.z0) * J.oy + (gy + a.crop.ly0 - J.y0)) * J.ox +
                    (gx + a.crop.lx0 - J.x0);
            return true;
        });
    } else if (tid >= kMmaIssuer) {
        if (tid == kMmaIssuer) mma_issue(M, umma_lo(smem_u32(A)), umma_lo(smem_u32(B)));
    } else {
        const bool ok = mma_atoms(
            A, M, ring,
            [&](const MmaAtom &a, int y, int x, int z, uint32_t (&o)[16]) {
                store_magic(a.out, J.ox, J.oy, a.crop, y, x, z, o, a.dc);
            },
            [&](const MmaAtom &a, uint8_t *T) {   // zeros, a list that overflowed, coefficients too large
                idct_atom_other(J, a.id, reinterpret_cast<int32_t *>(T), tid);
            });
        if (!ok) atomicExch(J.fail, 1u);   // a wait ran out: the call fails
    }
    mma_release(M);
    if (tid == 0 && M.starved) atomicExch(J.fail, 1u);
}

void launch_scan_u64(uint64_t *v, uint64_t n, uint64_t base, uint64_t *total, cudaStream_t s) {
    k_scan_u64<<<1, 1024, 0, s>>>(v, n, base, total);
}

void launch_idct(const DecodeJob &J, int num_sms, cudaStream_t s, uint64_t t_lo, uint64_t t_hi) {
    if (t_hi <= t_lo) return;
    DecodeJob Jr = J;
    Jr.t_lo = t_lo;
    Jr.t_hi = t_hi;
    const uint64_t n = t_hi - t_lo;
    const uint64_t grid = n < (uint64_t)num_sms ? n : (uint64_t)num_sms;
    if (!J.place || n < kMmaAtomsPerSm * (uint64_t)num_sms) {   // (the no-alloc path: at most 64 atoms, no places)
        smem_attr((const void *)k_idct_bf, (int)kIdctTileBytes);
        k_idct_bf<<<(unsigned)grid, kBfThreads, kIdctTileBytes, s>>>(Jr);
    } else {
        smem_attr((const void *)k_idct, (int)kIdctSmem);
        k_idct<<<(unsigned)grid, kMmaCta, kIdctSmem, s>>>(Jr);
    }
}

void launch_decode_lists(const DecodeJob &J, int num_sms, cudaStream_t s) {
    if (!J.n_atoms) return;
    launch_rc(J, num_sms, s, nullptr);
    launch_idct(J, num_sms, s, 0, J.n_atoms);
}

void launch_decode_front(const DecodeJob &J, int num_sms, cudaStream_t s, const StageEvents *ev) {
    if (ev) cudaEventRecord(ev->ev[0], s);
    unsigned nb = (unsigned)((J.n_atoms + 127) / 128);
    if (J.n_atoms) {
        k_caps<<<nb, 128, 0, s>>>(J);
        launch_scan_u64(J.ent_off, J.n_atoms, 0, nullptr, s);
    }
    if (ev) cudaEventRecord(ev->ev[1], s);
    if (J.n_atoms) launch_rc(J, num_sms, s, ev);
    if (ev) cudaEventRecord(ev->ev[2], s);
}

}  // namespace vcg
