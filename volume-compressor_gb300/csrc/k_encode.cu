// Encode kernels.
//
//   k_fwd         one CTA per atom: gather (zero padding outside the volume),
//                 sum -> zero flag + dc (src/vc/vc.c:599-604), forward DCT-32
//                 passes x, y per z-slab then z per column (src/vc/vc.c:212-218),
//                 dead-zone quantiser as the release build evaluates it
//                 (src/vc/vc.c:293-306), levels scattered to scan order in
//                 shared memory and compacted to (scan position, level) lists
//   k_rc_encode_groups / k_rc_encode_lanes   range coder (src/vc/vc.c:528-544):
//                 lengths, and the sums that k_resolve makes payloads
//                 [dc][bytes] of at their archive offsets (src/vc/vc.c:595-622)
//   k_long / k_rc_encode_long   atoms too long for their sums: the bytes, which
//                 k_resolve copies; k_rc_encode_rest: without room for sums
//   k_rc_sizes    lengths alone, from the decisions' costs
//   k_consume / k_slots   canonical layout: bytes consumed per atom in append
//                 order (an L2 block of 512 KiB at a region's first atom, then the
//                 payload) and the 16-byte L2 slots (src/vc/vc.c:1082-1159)
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "dct32.cuh"
#include "k_encode.cuh"
#include "kernels.cuh"
#include "rc_encode.cuh"

namespace vcg {

// k_fwd holds an atom's tile and levels, so an SM runs one CTA: 16 warps of it,
// two rows or lines a thread, hide each other's latency (the 37,451 atoms of a
// 1024^3 pyramid in 6.3 ms; 8 warps and the transform kept for later passes, 8.7).
// The integer pipes bound it: multiplies of the passes, then the quantiser's
// arithmetic, which groups without a level skip.
constexpr int kFwdThreads = 512;
constexpr int kQuantThreads = 256;
constexpr size_t kFwdSmem = kTileBytes + 32768 * sizeof(int16_t);

// 32 voxels of row (z, y) of atom (az, ay, ax), zero outside the volume, packed
// little-endian into 8 words.
__device__ __forceinline__ void load_row(const uint8_t *vol, uint32_t nx, uint32_t ny, uint32_t nz, uint32_t gx,
                                         uint32_t gy, uint32_t gz, uint32_t (&w)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = 0;
    if (gy >= ny || gz >= nz || gx >= nx) return;
    const uint8_t *p = vol + ((uint64_t)gz * ny + gy) * nx + gx;
    if (gx + 32 <= nx && ((uintptr_t)p & 15u) == 0) {
        uint4 a = __ldg(reinterpret_cast<const uint4 *>(p));
        uint4 b = __ldg(reinterpret_cast<const uint4 *>(p + 16));
        w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
        return;
    }
    uint32_t cnt = nx - gx < 32 ? nx - gx : 32;
    for (uint32_t i = 0; i < cnt; ++i) w[i >> 2] |= (uint32_t)__ldg(p + i) << (8 * (i & 3));
}

// A coefficient with its class, as the quantiser needs it: |cf| in bits 0-16
// (the transform of 8-bit voxels about a centre in [0, 255] reaches at most
// 46,132, the DC of a block 255 away from its centre), the class in bits 17-24,
// the sign in bit 31. Quantising it needs no scan order or class lookup.
__device__ __forceinline__ uint32_t coef_pack(int32_t cf, uint32_t cls) {
    const uint32_t mag = cf < 0 ? 0u - (uint32_t)cf : (uint32_t)cf;
    return mag | (cls << 17) | ((uint32_t)cf & 0x80000000u);
}

// Quantiser constants of an atom's q by class. A magnitude of at least `least`
// has a level: the smallest whole number not below the dead zone dz.
struct QuantShared {
    uint32_t least[VCD_NCLASS];
    float dz[VCD_NCLASS], rr[VCD_NCLASS];
    __device__ __forceinline__ void load(const vcd_quant &q) {
        for (int i = threadIdx.x; i < VCD_NCLASS; i += blockDim.x) {
            dz[i] = q.dz[i];
            rr[i] = q.rr[i];
            least[i] = (uint32_t)__float2int_ru(fminf(fmaxf(q.dz[i], 0.0f), 1e9f));
        }
    }
    __device__ __forceinline__ bool has(uint32_t w) const { return (w & 0x1FFFFu) >= least[(w >> 17) & 0xFFu]; }
};

// Dead-zone quantiser of a packed coefficient, as the release build evaluates
// it (src/vc/vc.c:293-306): level = trunc((|cf| - dz) r' + 1) for |cf| >= dz,
// clamped, with the coefficient's sign.
__device__ __forceinline__ int32_t quant_packed(uint32_t w, const QuantShared &q) {
    const uint32_t cls = (w >> 17) & 0xFFu;
    const float fa = __int2float_rn((int32_t)(w & 0x1FFFFu));
    int32_t level = __float2int_rz(__fadd_rn(__fmul_rn(__fsub_rn(fa, q.dz[cls]), q.rr[cls]), 1.0f));
    if (level > 32767) level = 32767;
    level = q.has(w) ? level : 0;
    return (w >> 31) ? -level : level;
}

// Quantise one atom in scan order and compact its nonzero levels into the list
// dst (scan position | level << 16, in scan order); returns the count (every
// thread). Warp w owns kPer scan positions from kPer w on, 128 at a time,
// each lane 4 consecutive ones (pk4(p) gives the packed coefficients of scan
// positions p..p+3): pass 1 quantises, keeps the levels in lv and counts them;
// pass 2 places each lane's entries after a warp prefix sum of the per-lane
// counts, skipping groups without a nonzero level.
template <int NT, class Pk4>
__device__ __forceinline__ uint32_t quant_compact(Pk4 &&pk4, const QuantShared &q, int16_t *lv, uint32_t *wcnt,
                                                  uint32_t *dst) {
    constexpr uint32_t kPer = 32768 / (NT / 32);
    static_assert(kPer % 512 == 0, "whole groups of loads");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t p0 = (uint32_t)warp * kPer + 4u * (uint32_t)lane;
    uint32_t cnt = 0;
    // groups of kG x 128 positions: every load of a group is issued before the
    // first level is stored
    constexpr uint32_t kG = 4;
#pragma unroll 1
    for (uint32_t i = 0; i < kPer; i += 128 * kG) {
        uint4 w[kG];
#pragma unroll
        for (uint32_t g = 0; g < kG; ++g) w[g] = pk4(p0 + i + 128 * g);
#pragma unroll
        for (uint32_t g = 0; g < kG; ++g) {
            uint2 out = make_uint2(0u, 0u);
            // most groups of the upper bands have no level at all
            if (__any_sync(0xFFFFFFFFu, q.has(w[g].x) || q.has(w[g].y) || q.has(w[g].z) || q.has(w[g].w))) {
                const int32_t l0 = quant_packed(w[g].x, q), l1 = quant_packed(w[g].y, q);
                const int32_t l2 = quant_packed(w[g].z, q), l3 = quant_packed(w[g].w, q);
                out = make_uint2((uint32_t)(uint16_t)l0 | ((uint32_t)l1 << 16),
                                 (uint32_t)(uint16_t)l2 | ((uint32_t)l3 << 16));
                cnt += (uint32_t)(l0 != 0) + (uint32_t)(l1 != 0) + (uint32_t)(l2 != 0) + (uint32_t)(l3 != 0);
            }
            *reinterpret_cast<uint2 *>(lv + p0 + i + 128 * g) = out;
        }
    }
    cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
    if (lane == 0) wcnt[warp] = cnt;
    __syncthreads();
    uint32_t base = 0, total = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) {
        const uint32_t v = wcnt[w];
        base += w < warp ? v : 0u;
        total += v;
    }
#pragma unroll 4
    for (uint32_t i = 0; i < kPer; i += 128) {
        const uint32_t p = p0 + i;
        const uint2 pk = *reinterpret_cast<const uint2 *>(lv + p);
        if (!__any_sync(0xFFFFFFFFu, (pk.x | pk.y) != 0u)) continue;
        const uint32_t lw[4] = {pk.x & 0xFFFFu, pk.x >> 16, pk.y & 0xFFFFu, pk.y >> 16};
        const uint32_t k = (uint32_t)(lw[0] != 0) + (uint32_t)(lw[1] != 0) + (uint32_t)(lw[2] != 0) +
                           (uint32_t)(lw[3] != 0);
        uint32_t incl = k;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += y;
        }
        uint32_t *d = dst + base + (incl - k);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (lw[j]) *d++ = (p + (uint32_t)j) | (lw[j] << 16);
        base += __shfl_sync(0xFFFFFFFFu, incl, 31);
    }
    __syncthreads();   // lv and wcnt are reused by the next atom
    return total;
}

__global__ void __launch_bounds__(kFwdThreads, 1) k_fwd(FwdJob J) {
    extern __shared__ int32_t smem[];
    int32_t *T = smem;                                          // the padded atom tile (dct32.cuh)
    int16_t *L = reinterpret_cast<int16_t *>(smem + kTileInts); // levels in scan order
    __shared__ QuantShared q;
    __shared__ uint32_t red[32];
    __shared__ uint32_t wcnt[kFwdThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int cur_lod = -1;

    for (uint64_t t = blockIdx.x; t < J.n_atoms; t += gridDim.x) {
        int lod;
        uint32_t az, ay, ax;
        const uint64_t ca = J.first + t;   // canonical index
        J.lay.coords(ca, lod, az, ay, ax);
        const int qi = J.qsel ? (int)J.qsel[t] : lod;
        if (qi != cur_lod) {   // uniform across the CTA: quantiser constants of this atom
            __syncthreads();   // every thread is done with the previous constants
            q.load(J.q[qi]);
            cur_lod = qi;
            __syncthreads();
        }
        const bool cached = J.coef && ca < J.coef_n;
        uint32_t *cptr = cached ? J.coef + ca * 32768ull : nullptr;
        uint32_t *dst = J.ent + t * (uint64_t)VCD_MAX_ENTRIES;
        int32_t dc;
        uint32_t total;
        if (cached && !J.coef_store) {
            // the transform of this atom was kept: quantise straight from it
            const uint32_t dcz = J.coef_dc[ca];
            if (dcz & kMetaZero) {
                if (tid == 0) J.meta[t] = kMetaZero;
                continue;
            }
            dc = (int32_t)(dcz & 0xFFu);
            total = quant_compact<kFwdThreads>(
                [&](uint32_t p) { return __ldcs(reinterpret_cast<const uint4 *>(cptr + p)); }, q, L, wcnt, dst);
        } else {
            const uint8_t *vol = J.vol[lod];
            const uint32_t nx = J.dims[lod][0], ny = J.dims[lod][1], nz = J.dims[lod][2];
            // rows r = tid + kFwdThreads j: z = r >> 5, y = r & 31 (lane)
            constexpr int kRows = 1024 / kFwdThreads;
            uint32_t w[kRows][8];
            uint32_t s = 0;
#pragma unroll
            for (int j = 0; j < kRows; ++j) {
                int r = tid + kFwdThreads * j;
                load_row(vol, nx, ny, nz, ax * 32, ay * 32 + (r & 31), az * 32 + (r >> 5), w[j]);
#pragma unroll
                for (int i = 0; i < 8; ++i) s = __dp4a(w[j][i], 0x01010101u, s);
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
            if (lane == 0) red[warp] = s;
            __syncthreads();
            uint32_t sum = 0;
#pragma unroll
            for (int i = 0; i < kFwdThreads / 32; ++i) sum += red[i];
            if (sum == 0) {   // all-zero atom: no payload (src/vc/vc.c:601)
                if (tid == 0) {
                    J.meta[t] = kMetaZero;
                    if (cached) J.coef_dc[ca] = kMetaZero;
                }
                __syncthreads();
                continue;
            }
            dc = (int32_t)((sum + 16384u) / 32768u);
            if (cached && tid == 0) J.coef_dc[ca] = (uint32_t)dc;
            // pass along x for the thread's rows, straight from registers
#pragma unroll
            for (int j = 0; j < kRows; ++j) {
                int r = tid + kFwdThreads * j;
                int32_t v[32], o[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = (int32_t)((w[j][i >> 2] >> (8 * (i & 3))) & 0xFFu) - dc;
                fdct32_line(v, o);
                int32_t *S = T + (r >> 5) * kSlabPitch + (r & 31) * kRowPitch;
#pragma unroll
                for (int k = 0; k < 32; ++k) S[k] = o[k];
            }
            __syncthreads();
            // pass along y, warp per z-slab, lane per column kx
            for (int z = warp; z < 32; z += kFwdThreads / 32) {
                int32_t *S = T + z * kSlabPitch + lane;
                int32_t v[32], o[32];
#pragma unroll
                for (int y = 0; y < 32; ++y) v[y] = S[y * kRowPitch];
                fdct32_line(v, o);
#pragma unroll
                for (int k = 0; k < 32; ++k) S[k * kRowPitch] = o[k];
            }
            __syncthreads();
            // pass along z per column (ky, kx = lane), coefficients back in place
            for (int ky = warp; ky < 32; ky += kFwdThreads / 32) {
                int32_t *C = T + ky * kRowPitch + lane;
                int32_t v[32], o[32];
#pragma unroll
                for (int z = 0; z < 32; ++z) v[z] = C[z * kSlabPitch];
                fdct32_line(v, o);
#pragma unroll
                for (int kz = 0; kz < 32; ++kz) C[kz * kSlabPitch] = o[kz];
            }
            __syncthreads();
            auto tile = [&](uint32_t p) {
                const uint4 at = __ldg(reinterpret_cast<const uint4 *>(J.place + p));
                auto get = [&](uint32_t a) { return coef_pack(T[a & 0xFFFFu], a >> 16); };
                const uint4 w = make_uint4(get(at.x), get(at.y), get(at.z), get(at.w));
                if (cached) *reinterpret_cast<uint4 *>(cptr + p) = w;   // kept in scan order
                return w;
            };
            total = quant_compact<kFwdThreads>(tile, q, L, wcnt, dst);
        }
        if (tid == 0) J.meta[t] = total | ((uint32_t)dc << 16);
    }
}

// LOD0 atoms whose transform was kept: quantise in scan order and compact, with
// a quarter of the shared memory of k_fwd (three CTAs per SM).
constexpr size_t kQuantSmem = 32768 * sizeof(int16_t);

__global__ void __launch_bounds__(kQuantThreads) k_quant_cached(FwdJob J) {
    extern __shared__ int16_t lv[];
    __shared__ QuantShared q;
    __shared__ uint32_t wcnt[kQuantThreads / 32];
    const int tid = threadIdx.x;
    uint64_t have = ~0ull;
    for (uint64_t t = blockIdx.x; t < J.n_atoms * J.sets; t += gridDim.x) {
        const uint64_t set = t / J.n_atoms, ca = J.first + t % J.n_atoms;
        if (set != have) {   // uniform across the CTA, which is past the previous set's last atom
            q.load(J.q[set]);
            have = set;
            __syncthreads();
        }
        const uint32_t dcz = J.coef_dc[ca];
        if (dcz & kMetaZero) {
            if (tid == 0) J.meta[t] = kMetaZero;
            continue;
        }
        const uint32_t *cptr = J.coef + ca * 32768ull;
        const uint32_t total = quant_compact<kQuantThreads>(
            [&](uint32_t p) { return __ldcs(reinterpret_cast<const uint4 *>(cptr + p)); }, q, lv, wcnt,
            J.ent + t * (uint64_t)VCD_MAX_ENTRIES);
        if (tid == 0) J.meta[t] = total | ((dcz & 0xFFu) << 16);
    }
}

constexpr size_t size_smem(int A) { return sizeof(EncCosts) + 8 * (size_t)A * kRingPitch * 4; }

// Atom t's list, or none; whether it is present (its dc is coded) and not among
// those marked `without`.
__device__ __forceinline__ bool enc_atom(const RcJob &J, uint64_t t, const uint32_t *&ent, uint32_t &nnz,
                                         uint32_t without = 0u) {
    const uint32_t meta = t < J.n_atoms ? J.meta[t] : kMetaZero;
    const bool on = !(meta & (kMetaZero | without));
    nnz = on ? meta & 0xFFFFu : 0u;
    ent = J.ent + (on ? t : 0) * (uint64_t)VCD_MAX_ENTRIES;
    return on;
}

// Atom t is left to k_rc_encode_long.
__device__ __forceinline__ void mark_long(const RcJob &J, uint64_t t) {
    J.meta[t] |= kMetaLong;
    J.longs[1u + atomicAdd(J.longs, 1u)] = (uint32_t)t;
}

// Few atoms: kEncGroups groups of G atoms per CTA. Warps 0..3 code, the warps
// after them produce, warp w for group w % 4 (the same SM sub-partition). Without
// SUMS: the lengths of the atoms in doubt, G = 1.
template <bool SUMS>
__global__ void __launch_bounds__(32 * kEncGroups * enc_group_warps(kGroupMax)) k_rc_encode_groups(RcJob J, uint32_t G) {
    extern __shared__ __align__(16) uint8_t gmem[];
    __shared__ uint32_t bstart[9];
    if (threadIdx.x < 9) bstart[threadIdx.x] = J.band_start[threadIdx.x];
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, c = warp % kEncGroups, w = warp / kEncGroups;
    EncGroup g;
    g.init(gmem + c * enc_group_bytes(G), G, 1u + c);
    const uint64_t n = SUMS ? J.n_atoms : J.doubt[0];
    for (uint64_t b = blockIdx.x; b * kEncGroups * G < n; b += gridDim.x) {
        const uint64_t t0 = (b * kEncGroups + c) * G;
        const uint32_t slot = w == 0u ? lane : (enc_group_split(G) ? 0u : 2u * (w - 1u)) + (lane >> 4);
        uint64_t t = slot < G ? t0 + slot : n;
        t = t >= n ? J.n_atoms : SUMS ? t : J.doubt[1u + t];
        const uint32_t *ent;
        uint32_t nnz;
        const bool on = enc_atom(J, t, ent, nnz, SUMS ? kMetaLong : 0u);
        if (w == 0u) {
            const uint32_t eob = nnz ? (ent[nnz - 1u] & 0xFFFFu) + 1u : 0u;
            const uint32_t k = enc_consume<SUMS>(g, on, eob, SUMS ? J.sums + (on ? t : 0) * kSums : nullptr, lane);
            if (t < J.n_atoms) {
                if (!SUMS && on) atomicAdd(J.totals + 3 * (t / J.per), (unsigned long long)(k + 1u - J.len[t]));
                J.len[t] = on ? k + 1u : 0u;
                if (SUMS && on && k >= kSumsMax + 5u) mark_long(J, t);
            }
        } else {
            const bool split = enc_group_split(G);
            enc_produce(g, slot, ent, nnz, bstart, lane, !split || w == 1u, !split || w == 2u);
        }
        g.sync();   // the counts are the next atoms'
    }
}

// Lengths alone: A atoms at a time, A / 4 warps their bands (as many atoms a warp
// as A, so with 32 of them a warp's bands are alike), A / 2 warps the unary
// contexts of two each; those that the costs leave in doubt are collected for
// the coder. A pass over 540 atoms of 30,000 decisions takes 0.25 ms (A 4; the
// coder 1.14 ms), one over 32,768 of 48,700 takes 4.3 ms (A 32; a coder's lane each 5.7, the lockstep coder 9.3).
template <int A>
__global__ void __launch_bounds__(24 * A) k_rc_sizes(RcJob J) {
    extern __shared__ __align__(16) uint8_t gmem[];
    EncCosts &T = *reinterpret_cast<EncCosts *>(gmem);
    uint32_t *ring = reinterpret_cast<uint32_t *>(gmem + sizeof(EncCosts));
    __shared__ uint32_t bstart[9];
    __shared__ unsigned long long cost[A];
    __shared__ uint32_t lo[A], hi[A];
    const uint32_t tid = threadIdx.x;
    if (tid < 9) bstart[tid] = J.band_start[tid];
    for (uint32_t i = tid; i < sizeof(EncCosts) / 16; i += blockDim.x)
        reinterpret_cast<uint4 *>(gmem)[i] = __ldg(reinterpret_cast<const uint4 *>(J.costs) + i);
    const uint32_t lane = tid & 31u, warp = tid >> 5;
    const bool bands = warp < A / 4;
    const uint32_t b = A == 4 ? lane & 7u : warp;   // the lane's band
    const uint32_t a = !bands ? 2u * (warp - A / 4) + (lane >> 4) : A == 4 ? lane >> 3 : lane;
    for (uint64_t t0 = (uint64_t)blockIdx.x * A; t0 < J.n_atoms; t0 += (uint64_t)gridDim.x * A) {
        if (tid < A) cost[tid] = 0, lo[tid] = 0, hi[tid] = 0;
        __syncthreads();
        const uint32_t *ent;
        uint32_t nnz;
        enc_atom(J, t0 + a, ent, nnz);
        const EncSize r = bands ? enc_size_bands<A == 4>(T, ent, nnz, b, bstart, ring + tid * kRingPitch)
                                : enc_size_rest(T, ent, nnz, lane);
        atomicAdd(&cost[a], (unsigned long long)r.cost);
        atomicAdd(&lo[a], r.lo);
        atomicAdd(&hi[a], r.hi);
        __syncthreads();
        if (tid < 32u) {
            const uint64_t t = tid < A ? t0 + tid : J.n_atoms;
            const uint32_t m = t < J.n_atoms ? J.meta[t] : kMetaZero;
            const bool on = !(m & kMetaZero);
            const uint32_t i = tid % A;
            // the end of the list is 16 bypass decisions; an interval of 2^32 - 1
            // to start with costs less than one unit
            const uint64_t least = 16ull * kCostOne + cost[i] - lo[i];
            const uint64_t most = 16ull * kCostOne + cost[i] + hi[i] + 16u * kCostBypass + 1u;
            uint32_t n = (uint32_t)((least - 1u) / (8ull * kCostOne));
            bool sure = most < (n + 1ull) * 8ull * kCostOne;
            if (!(m & 0xFFFFu)) n = 2u, sure = true;   // 16 halvings of 2^32 - 1
            if (t < J.n_atoms) J.len[t] = on ? n + 6u : 0u;
            if (on && !sure) J.doubt[1u + atomicAdd(J.doubt, 1u)] = (uint32_t)t;
            if (A == 4) {   // its atoms may be of two sets
                if (on) {
                    unsigned long long *tot = J.totals + 3 * (t / J.per);
                    atomicAdd(tot, n + 6ull);
                    atomicAdd(tot + 1, 1ull);
                    if (!sure) atomicAdd(tot + 2, 1ull);
                }
                continue;
            }
            const uint32_t bytes = __reduce_add_sync(0xFFFFFFFFu, on ? n + 6u : 0u);
            const uint32_t present = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, on));
            const uint32_t doubt = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, on && !sure));
            if (tid == 0u && present) {
                atomicAdd(J.totals, (unsigned long long)bytes);
                atomicAdd(J.totals + 1, (unsigned long long)present);
                if (doubt) atomicAdd(J.totals + 2, (unsigned long long)doubt);
            }
        }
    }
}

// Many atoms: a lane each, G per warp.
constexpr uint32_t kLanesWarps = 4;

__global__ void __launch_bounds__(32 * kLanesWarps) k_rc_encode_lanes(RcJob J, uint32_t G) {
    __shared__ uint32_t bstart[9];
    __shared__ __align__(16) uint32_t mem[kLanesWarps][kEncWarpWords];
    if (threadIdx.x < 9) bstart[threadIdx.x] = J.band_start[threadIdx.x];
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint64_t t = lane < G ? ((uint64_t)blockIdx.x * kLanesWarps + warp) * G + lane : J.n_atoms;
    const uint32_t *ent;
    uint32_t nnz;
    const bool on = enc_atom(J, t, ent, nnz, kMetaLong);
    const uint32_t n = enc_lanes<4, 3, 2>(on, ent, nnz, bstart, J.sums + (on ? t : 0) * kSums, mem[warp], lane);
    if (t < J.n_atoms) J.len[t] = on ? n + 1u : 0u;
    if (on && n >= kSumsMax + 5u) mark_long(J, t);
}

// Where the payload of atom t goes.
__device__ __forceinline__ uint8_t *resolve_dst(const ResolveJob &J, uint64_t t) {
    if (J.dst_off) return J.arc + J.dst_off[t];
    const uint64_t a = J.canon_first + t;   // canonical index
    return J.arc + J.pos[a] + (J.lay.first_in_region(a) ? kL2Bytes : 0ull);
}

// Bytes that a slot of sums holds.
constexpr uint32_t kSlotBytes = kSums * 4u;

// A warp per atom: [dc] and the coder bytes, from its sums or, if it is marked
// long, from its slot; without slots, or past one, it is collected for
// k_rc_encode_rest.
__global__ void __launch_bounds__(256) k_resolve(ResolveJob J) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= J.n_atoms) return;
    const uint32_t meta = J.meta[t];
    if (meta & kMetaZero) return;
    uint8_t *dst = resolve_dst(J, t);
    if (lane == 0) dst[0] = (uint8_t)((meta >> 16) & 0xFFu);
    const uint32_t n = J.len[t] - 6u;   // sums less one
    if (J.sums && !(meta & kMetaLong)) {
        enc_resolve(J.sums + t * kSums, n, dst + 1, lane);
    } else if (J.sums && n + 5u <= kSlotBytes) {
        for (uint32_t i = lane; i < (n + 8u) / 4u; i += 32u) {
            const uint32_t w = J.sums[t * kSums + i];
            for (uint32_t k = 0; k < 4u && 4u * i + k < n + 5u; ++k) dst[1u + 4u * i + k] = (uint8_t)(w >> (8u * k));
        }
    } else if (lane == 0) {
        J.rest[1u + atomicAdd(J.rest, 1u)] = (uint32_t)t;
    }
}

// The calling warp's atoms of a list (how many, which) coded in lockstep from
// their lists, the atoms spread evenly over the SM sub-partitions (slots) at up to
// 32 a warp; every atom has its warp, a loop over them would spill. dst(t): where
// its bytes go; done(t, n): called with their count.
template <class Dst, class Done>
__device__ __forceinline__ void code_listed(const uint32_t *list, uint32_t slots, const uint32_t *ent,
                                            const uint32_t *meta, const uint32_t *bstart, uint32_t cap, Dst &&dst,
                                            Done &&done) {
    const uint32_t lane = threadIdx.x & 31u, n = list[0];
    const uint32_t k = (n + 32u * slots - 1u) / (32u * slots), G = k ? (n + k * slots - 1u) / (k * slots) : 1u;
    const uint64_t i0 = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * G;
    if (i0 >= n) return;
    const uint32_t i = (uint32_t)i0 + lane;
    const bool on = lane < G && i < n;
    const uint64_t t = on ? list[1u + i] : 0u;
    const uint32_t bytes = rc_encode_levels_warp<true>(ent + t * (uint64_t)VCD_MAX_ENTRIES, on ? meta[t] & 0xFFFFu : 0u,
                                                       on, bstart, on ? dst(t) : nullptr, cap);
    if (on) done(t, bytes);
}

// the CTAs of 128 threads that code a list of up to n_atoms
static unsigned listed_ctas(uint64_t n_atoms, uint64_t slots) {
    const uint64_t k = (n_atoms + 32 * slots - 1) / (32 * slots), warps = n_atoms < k * slots ? n_atoms : k * slots;
    return (unsigned)((warps + 3) / 4);
}

__global__ void __launch_bounds__(128) k_rc_encode_rest(ResolveJob J, uint32_t slots) {
    __shared__ uint32_t bstart[9];
    if (threadIdx.x < 9) bstart[threadIdx.x] = J.band_start[threadIdx.x];
    __syncthreads();
    code_listed(J.rest, slots, J.ent, J.meta, bstart, 0xFFFFFFFFu, [&](uint64_t t) { return resolve_dst(J, t) + 1; },
                [](uint64_t, uint32_t) {});
}

void launch_resolve(const ResolveJob &J, int num_sms, cudaStream_t s) {
    if (!J.n_atoms) return;
    cudaMemsetAsync(J.rest, 0, 4, s);
    k_resolve<<<(unsigned)((J.n_atoms + 7) / 8), 256, 0, s>>>(J);
    const uint32_t slots = 4u * (uint32_t)num_sms;
    k_rc_encode_rest<<<listed_ctas(J.n_atoms, slots), 128, 0, s>>>(J, slots);
}

// Atoms with more sums than their slot holds (white noise at the finest
// quantisers) are coded from their lists after the others, their bytes into the
// slot. The coder marks them when it is done. Where there are more than its groups
// take, its own pass would cost nearly as much, so an atom is marked before it, and
// left out, if the bypass decisions of its list's escapes and signs alone, a bit
// each, tell it: a warp per atom; only a list that can be long is read. White noise
// at q 0.05, 640^3 / 1024^3: 122 / 154 ms, where the coder took every atom first
// and its list again after it 219 / 284.
constexpr uint32_t kLongBits = 8u * kSumsMax;
__global__ void __launch_bounds__(256) k_long(RcJob J) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= J.n_atoms) return;
    const uint32_t meta = J.meta[t], nnz = meta & 0xFFFFu;
    if (meta & kMetaZero || nnz < kLongBits / 32u) return;   // an entry has at most 32
    const uint32_t *ent = J.ent + t * (uint64_t)VCD_MAX_ENTRIES;
    uint32_t sum = 0;
    for (uint32_t i = lane; i < nnz; i += 32u) {
        const int32_t lv = (int32_t)__ldg(ent + i) >> 16;
        uint32_t bits;
        sum += enc_tail((uint32_t)(lv < 0 ? -lv : lv), false, &bits);
    }
    sum = __reduce_add_sync(0xFFFFFFFFu, sum);
    if (lane == 0 && sum >= kLongBits) mark_long(J, t);
}

__global__ void __launch_bounds__(128) k_rc_encode_long(RcJob J, uint32_t slots) {
    __shared__ uint32_t bstart[9];
    if (threadIdx.x < 9) bstart[threadIdx.x] = J.band_start[threadIdx.x];
    __syncthreads();
    code_listed(J.longs, slots, J.ent, J.meta, bstart, kSlotBytes,
                [&](uint64_t t) { return reinterpret_cast<uint8_t *>(J.sums + t * kSums); },
                [&](uint64_t t, uint32_t n) { J.len[t] = n + 1u; });
}

void launch_rc_long(const RcJob &J, int num_sms, cudaStream_t s) {
    if (!J.n_atoms) return;
    const uint32_t slots = 4u * (uint32_t)num_sms;
    k_rc_encode_long<<<listed_ctas(J.n_atoms, slots), 128, 0, s>>>(J, slots);
}

// consume[a] = (first atom of its region ? L2 block : 0) + payload length
__global__ void k_consume(PlaceJob J) {
    uint64_t a = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= J.n_total) return;
    J.pos[a] = (J.lay.first_in_region(a) ? kL2Bytes : 0ull) + J.len[a];
}

__global__ void k_slots(PlaceJob J) {
    uint64_t a = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= J.n_total) return;
    int lod;
    uint32_t az, ay, ax;
    J.lay.coords(a, lod, az, ay, ax);
    const uint64_t blk = J.pos[J.lay.region_first(lod, az, ay, ax)];
    uint8_t *slot = J.arc + blk + ((((uint64_t)(az & 31) * 32 + (ay & 31)) * 32 + (ax & 31)) * 16);
    const uint32_t len = J.len[a];
    uint4 v;
    if (len == 0) {   // known-zero atom (src/vc/vc.c:1133-1141)
        v = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 2u);
    } else {
        const uint64_t off = J.pos[a] + (J.lay.first_in_region(a) ? kL2Bytes : 0ull);
        v = make_uint4((uint32_t)off, (uint32_t)(off >> 32), len, 1u | ((J.dc[a] & 0xFFu) << 8));
    }
    // an L2 block starts wherever the cursor was (any byte offset): store bytewise
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 16; ++i) slot[i] = (uint8_t)(w[i >> 2] >> (8 * (i & 3)));
}

__global__ void k_gather_dc(const uint32_t *meta, uint64_t n, uint8_t *dc, uint32_t *zero) {
    uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) *zero = 0;
    if (t < n) dc[t] = (meta[t] & kMetaZero) ? 0 : (uint8_t)(meta[t] >> 16);
}

void enc_set_smem() {
    smem_attr((const void *)k_fwd, (int)kFwdSmem);
    smem_attr((const void *)k_quant_cached, (int)kQuantSmem);
    smem_attr((const void *)k_rc_encode_groups<true>, (int)(kEncGroups * enc_group_bytes(kGroupMax)));
    smem_attr((const void *)k_rc_sizes<4>, (int)size_smem(4));
    smem_attr((const void *)k_rc_sizes<32>, (int)size_smem(32));
}

void launch_quant_cached(const FwdJob &J, int num_sms, cudaStream_t s) {
    enc_set_smem();
    if (!J.n_atoms) return;
    const uint64_t cap = (uint64_t)num_sms * 3, n = J.n_atoms * J.sets;
    k_quant_cached<<<(unsigned)(n < cap ? n : cap), kQuantThreads, kQuantSmem, s>>>(J);
}

void launch_fwd(const FwdJob &J, int num_sms, cudaStream_t s) {
    enc_set_smem();
    if (!J.n_atoms) return;
    uint64_t grid = J.n_atoms < (uint64_t)num_sms ? J.n_atoms : (uint64_t)num_sms;
    k_fwd<<<(unsigned)grid, kFwdThreads, kFwdSmem, s>>>(J);
}

void enc_tables(EncTables *et, const vcd_tables *vt) {
    memset(et, 0, sizeof *et);
    for (uint32_t p = 0; p < 32768; ++p) {
        const uint32_t r = vt->scan[p], f = (r >> 10) + ((r >> 5) & 31u) + (r & 31u);
        // the alternate step's class where it applies (src/vc/vc.c:273-279, 293-306)
        const uint32_t cls = f + 94u * ((vt->alt_mask[r >> 5] >> (r & 31u)) & 1u);
        et->place[p] = (r >> 10) * kSlabPitch + ((r >> 5) & 31u) * kRowPitch + (r & 31u) | cls << 16;
    }
    EncCosts *t = &et->costs;
    const double bit = kCostOne, e = 4096.0 / 16777216.0 * 1.4427 * 1.0001;   // log2(e) and the square term, above
    for (uint32_t c = 1; c < 4096; ++c)
        t->one[c] = make_uint2((uint32_t)llround((12.0 - log2((double)c)) * bit),
                               (uint32_t)ceil(e * bit / c) + kCostSlack);
    for (uint32_t q0 = 1; q0 < 4096; ++q0) {
        uint32_t q = q0;
        double cost = 0.0, err = 0.0;
        for (int j = 0; j < 8; ++j) {
            const double c = 4096.0 - q;
            cost += 12.0 - log2(c);
            err += e * bit / c;
            q -= q >> 5;
        }
        t->eight[q0] = make_uint2((uint32_t)llround(fmin(cost * bit, 4294967295.0)),
                                  (uint32_t)fmin(ceil(err) + kCostSlack, 65535.0) << 16 | q);
    }
}

// Lengths alone come from costs (three CTAs of 4 atoms an SM while that holds
// them all, else two of 32), and where they have to be exact the atoms in doubt,
// one in a thousand, are then coded. With sums, up to kGroupMax atoms per SM
// sub-partition (4,864 on 152 SMs) run as groups, one coder warp per
// sub-partition; more of them a lane each, with the fewest warps per
// sub-partition that hold them at 32 a warp, spread evenly. At the line: 4,681
// atoms of 30,000 decisions in 2.6 ms as groups of 8 and 3.2 ms a lane each, of
// 164,000 decisions in 9.6 and 21.6 ms.
uint64_t size_sets_atoms(int num_sms) { return 12ull * (uint64_t)num_sms; }

uint64_t enc_group_atoms(int num_sms) { return (uint64_t)kGroupMax * kEncGroups * (uint64_t)num_sms; }

void launch_rc_encode(const RcJob &J, int num_sms, cudaStream_t s) {
    if (!J.n_atoms) return;
    const uint64_t slots = (uint64_t)kEncGroups * (uint64_t)num_sms;
    if (!J.sums) {
        if (J.pass != RcJob::kDoubt) {
            cudaMemsetAsync(J.doubt, 0, 4, s);
            const uint64_t sms = (uint64_t)num_sms;
            if (J.n_atoms <= size_sets_atoms(num_sms)) {
                k_rc_sizes<4><<<(unsigned)((J.n_atoms + 3) / 4), 96, size_smem(4), s>>>(J);
            } else {
                const uint64_t nb = (J.n_atoms + 31) / 32;
                k_rc_sizes<32><<<(unsigned)(nb < 2 * sms ? nb : 2 * sms), 768, size_smem(32), s>>>(J);
            }
        }
        if (J.pass == RcJob::kNear) return;
        const uint64_t ng = (J.n_atoms + kEncGroups - 1) / kEncGroups;
        k_rc_encode_groups<false><<<(unsigned)(ng < (uint64_t)num_sms ? ng : (uint64_t)num_sms),
                                    32u * kEncGroups * enc_group_warps(1), kEncGroups * enc_group_bytes(1), s>>>(J, 1);
        return;
    }
    if (J.n_atoms <= enc_group_atoms(num_sms)) {
        const uint32_t G = (uint32_t)((J.n_atoms + slots - 1) / slots);
        const unsigned nb = (unsigned)((J.n_atoms + kEncGroups * G - 1) / (kEncGroups * G));
        const unsigned nt = 32u * kEncGroups * enc_group_warps(G);
        k_rc_encode_groups<true><<<nb, nt, kEncGroups * enc_group_bytes(G), s>>>(J, G);
        return;
    }
    k_long<<<(unsigned)((J.n_atoms + 7) / 8), 256, 0, s>>>(J);
    const uint64_t k = (J.n_atoms + 32 * slots - 1) / (32 * slots);
    const uint32_t G = (uint32_t)((J.n_atoms + k * slots - 1) / (k * slots));
    const uint64_t warps = (J.n_atoms + G - 1) / G;
    k_rc_encode_lanes<<<(unsigned)((warps + kLanesWarps - 1) / kLanesWarps), 32 * kLanesWarps, 0, s>>>(J, G);
}

void launch_consume(const PlaceJob &J, cudaStream_t s) {
    k_consume<<<(unsigned)((J.n_total + 255) / 256), 256, 0, s>>>(J);
}

void launch_slots(const PlaceJob &J, cudaStream_t s) {
    k_slots<<<(unsigned)((J.n_total + 255) / 256), 256, 0, s>>>(J);
}

void launch_gather_dc(const uint32_t *meta, uint64_t n, uint8_t *dc, uint32_t *zero, cudaStream_t s) {
    k_gather_dc<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(meta, n, dc, zero);
}

}  // namespace vcg
