// Inverse DCT-32 of one atom on the fp16 tensor cores, exact (device).
//
// A pass is OUT = V C over the atom's 1024 lines, 128 lines a tile
// (tcgen05.mma, M = lines, N = 64, K = 64). The integers are split into fp16
// pieces, whose products and fp32 sums are exact:
//   v = 256 h + l, 0 <= l < 256     pieces h and l / 128 along K (32 + 32)
//   c = 64 c1 + c0, -32 <= c0 < 32  pieces along N: columns 0-31 sum c1 v,
//                                   32-63 c0 v (coefficient entries 256 c, 128 c)
// With H and L the two sums, the reference's (64 H + L + 8192) >> 14 is
// floor((H + floor((L + 8192) / 64)) / 256): two fused multiply-adds that round
// down onto an integer grid and two additions, for two outputs at once. Adding
// 2^23 + 0x660000 leaves the next pass's pieces in the bytes of the result: bits
// 8-23 are the fp16 number 1536 + h, the low byte under the top byte 0x4B the
// fp16 number 14 + l / 128, so a byte permute and a packed subtraction each make
// two pieces.
//
// Every partial sum stays below 2^24 when the atom's coefficients have a 2-norm
// of at most kMmaNorm: a column of c1 has norm at most 259 and a line's pieces
// exceed the line's norm by at most 2886, and a pass multiplies the norm of the
// atom by at most 1.001 and adds 91 (its rounding), so
// |H| <= 259 (58,300 + 2,886) and |H| + |L| / 64 < 2^24 in all three passes. An
// atom of 8-bit voxels has a norm of at most 46,159. A larger one (large
// quantiser steps, hostile levels) takes the butterfly, so every input gives
// the reference's result.
//
// What bounds it on GB300 is shared memory: an MMA reads 6 KB of it in 50
// cycles (96 MMAs an atom), and clearing, scattering and the two rearrangements
// between passes take about 5,200 wavefronts more.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

#include "dct32.cuh"
#include "feed_extent.cuh"
#include "idct_tile.cuh"

namespace vcg {

constexpr float kMmaNorm = 58000.0f;
constexpr uint32_t kMmaTile = 16384;             // bytes of a tile's operand: 128 lines x 64 fp16
constexpr uint32_t kMmaA = 8 * kMmaTile;         // the atom's operand
constexpr uint32_t kMmaB = 64 * 64 * 2;          // the matrix pieces

// ---- tcgen05, mbarrier
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// Waits until the phase of parity `parity` is complete; false after a quarter of a
// second (a try gives up after 4 us on GB300, whatever the hint; TIMES: so many
// quarters). What the CTA's roles wait for takes some 10 us an atom.
#ifndef VCG_WAIT_TRIES
#define VCG_WAIT_TRIES (1u << 16)
#endif
template <uint32_t TIMES = 1>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < TIMES * VCG_WAIT_TRIES; ++i) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 0x4000;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t dst) {   // all 512 columns; one warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(dst) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t t) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(t));
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// operand descriptors, 128-byte swizzle: low word (start address, a step of 16
// bytes each; between 64-line halves: 8,192 bytes) and high word (1,024 bytes
// between swizzle blocks)
__device__ __forceinline__ uint32_t umma_lo(uint32_t addr) { return (addr >> 4) | ((8192u >> 4) << 16); }
constexpr uint32_t kUmmaHi = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ void umma(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, bool acc) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 A, B;\n\tsetp.ne.u32 p, %4, 0;\n\tmov.b64 A, {%1, %5};\n\t"
                 "mov.b64 B, {%2, %5};\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], A, B, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "r"(b), "r"(idesc), "r"((uint32_t)acc), "r"(kUmmaHi)
                 : "memory");
}
// fp32 sums, fp16 operands, 128 x 64, A along K (lines are rows) or along M
constexpr uint32_t kIdescK = (1u << 4) | ((64u >> 3) << 17) | ((128u >> 4) << 24);
constexpr uint32_t kIdescM = kIdescK | (1u << 15);

#define VC_LD16(v, t)                                                                                                  \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "                                                             \
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"                                     \
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),     \
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),            \
                   "=r"(v[15])                                                                                         \
                 : "r"(t))

// One tile of a pass by one thread: lines of the operand at `a` (descriptor low
// words), B at `b`, sums to TMEM column block d, then bar. Along_m: operand along
// M (the first pass: along K). half: only the first 16 values of a line are used.
template <bool Along_m>
__device__ __forceinline__ void mma_tile(uint32_t d, uint32_t a, uint32_t b, bool half, uint32_t bar) {
    constexpr uint32_t idesc = Along_m ? kIdescM : kIdescK, step = (Along_m ? 2048u : 32u) >> 4;
    umma(d, a, b, idesc, false);
    if (!half) umma(d, a + step, b + 2u, idesc, true);
    umma(d, a + 2u * step, b + 4u, idesc, true);
    if (!half) umma(d, a + 3u * step, b + 6u, idesc, true);
    tc_commit(bar);
}

// Matrix pieces of the inverse pass into B (64 rows n of 64 fp16 k, 128-byte
// swizzle): rows 0-31 c1, 32-63 c0; k < 32 for h (times 256), the rest for l
__device__ __forceinline__ void mma_load_b(uint8_t *B, int tid, int nt) {
    for (int i = tid; i < 64 * 64; i += nt) {
        const int n = i >> 6, k = i & 63;
        const int c = c_cmat[k & 31][n & 31];
        const int c0 = ((c + 32) & 63) - 32, c1 = (c - c0) >> 6;
        const int p = (n < 32 ? c1 : c0) * (k < 32 ? 256 : 128);
        const uint32_t off = (uint32_t)n * 128u + ((((uint32_t)k >> 3) ^ ((uint32_t)n & 7u)) << 4) + ((uint32_t)k & 7u) * 2u;
        *reinterpret_cast<__half *>(B + off) = __int2half_rn(p);
    }
}

// Pieces of a coefficient (magic: kMagicBits + v): h in the low half, l in the high half
__device__ __forceinline__ uint32_t mma_pieces(uint32_t magic) {
    uint32_t w = __byte_perm(magic, 0, 0x3021);
    asm("add.f16x2 %0, %0, %1;" : "+r"(w) : "r"(0xCB00E600u));
    return w;
}
// Constants of the rounding, each twice; opaque so that they stay in registers
struct MmaRound {
    uint64_t c64, c256, b0, b1, b2;
    __device__ __forceinline__ static uint64_t twice(uint32_t bits) {
        uint64_t v;
        asm volatile("mov.b64 %0, {%1, %1};" : "=l"(v) : "r"(bits));
        return v;
    }
    __device__ __forceinline__ void set() {
        c64 = twice(0x3C800000u);    // 1 / 64
        c256 = twice(0x3B800000u);   // 1 / 256
        b0 = twice(0x4B400080u);     // 1.5 * 2^23 + 128: the grid, and 8192 / 64
        b1 = twice(0xCB400000u);     // -1.5 * 2^23
        b2 = twice(kMagicBits);
    }
};
// Half of the thread's line of a tile: 16 rounded outputs as magic numbers
// (kMagicBits + output), from TMEM column t on
__device__ __forceinline__ void mma_outputs(const MmaRound &R, uint32_t t, uint32_t (&o)[16]) {
    uint32_t h[16], l[16];
    VC_LD16(h, t);
    VC_LD16(l, t + 32u);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
        asm("{\n\t.reg .b64 H, L;\n\tmov.b64 H, {%2, %3};\n\tmov.b64 L, {%4, %5};\n\t"
            "fma.rm.f32x2 L, L, %6, %8;\n\tadd.rn.f32x2 L, L, %9;\n\tadd.rn.f32x2 H, H, L;\n\t"
            "fma.rm.f32x2 H, H, %7, %10;\n\tmov.b64 {%0, %1}, H;\n\t}"
            : "=r"(o[i]), "=r"(o[i + 1])
            : "r"(h[i]), "r"(h[i + 1]), "r"(l[i]), "r"(l[i + 1]), "l"(R.c64), "l"(R.c256), "l"(R.b0), "l"(R.b1),
              "l"(R.b2));
    }
}
// pieces of two outputs
__device__ __forceinline__ uint32_t mma_hi(uint32_t o0, uint32_t o1) {
    uint32_t w = __byte_perm(o0, o1, 0x6521);
    asm("add.f16x2 %0, %0, %1;" : "+r"(w) : "r"(0xE600E600u));
    return w;
}
__device__ __forceinline__ uint32_t mma_lo(uint32_t o0, uint32_t o1) {
    uint32_t w = __byte_perm(o0, o1, 0x7430);
    asm("add.f16x2 %0, %0, %1;" : "+r"(w) : "r"(0xCB00CB00u));
    return w;
}

// Operands of the second and third pass lie along M: row k (h of input k; row 32
// + k: l) of 64 lines in 128 bytes, 8 rows a swizzle block of 1,024 bytes, 64
// rows (8,192 bytes) for each half of the tile's lines.

// A CTA that transforms atoms: 16 warps on the atom in hand, in groups of four
// that read a tile's sums (a quarter of the lines each); a warp that issues the
// MMAs (an issuing thread waits for the tensor cores' queue, 50 cycles per MMA);
// three warps that prepare the next atoms: their lists, dequantised, go through a
// ring of chunks of (place, pieces) pairs, from which the 16 warps only scatter.
constexpr int kMmaThreads = 512, kMmaIssuer = kMmaThreads, kMmaFeed = kMmaThreads + 32, kMmaFeeders = 96;
constexpr int kMmaCta = kMmaFeed + kMmaFeeders;
constexpr int kMmaBar = 5;                 // named barrier of the 16 warps; 6: of the feeders
constexpr uint32_t kMmaChunk = 1536, kMmaChunks = 6;
constexpr uint32_t kMmaRing = kMmaChunk * kMmaChunks * 8;   // bytes
constexpr uint32_t kMmaAtoms = 64;         // descriptions kept, made 32 at a time: the feeders are at most
                                           // kMmaChunks atoms ahead of the 16 warps, which look back one

struct MmaAtom {
    const uint32_t *src;       // list (scan position | level << 16)
    uint32_t n;                // its entries
    uint32_t tensor;           // 1: a list for the tensor cores; 0: the caller's other way
    int32_t dc;
    uint64_t id;               // the caller's
    Crop crop;                 // where its voxels go (plain decode)
    uint8_t *out;
    uint32_t fits, tiles;      // small enough for exact sums; tiles of four kz up to the last level
    uint32_t more;             // 0: no such atom
};
struct MmaShared {
    uint64_t bar[24];          // MMAs done: per pass and tile
    uint64_t scattered;        // the first operand is written: per warp of the 16
    uint64_t stored[4];        // a group's last outputs of the atom before are read: per warp
    uint64_t second[8];        // a tile's second operand is written: per warp of its group
    uint64_t third;            // the third operand is written: per warp of the 16
    uint64_t full[kMmaChunks], empty[kMmaChunks];
    uint64_t drained;          // the issuing thread is done with the tensor cores
    MmaAtom atom[kMmaAtoms];
    uint32_t count[kMmaChunks];   // entries of the chunk | kMmaLast
    uint32_t tmem;             // TMEM base
    uint32_t gave_up;          // a wait of the 16 warps ran out: set before an arrival at scattered, read after them all
    uint32_t starved;          // a wait of the feeders did
    FeedExtent<kMmaFeeders / 32> extent;
    int2 dq[VCD_NCLASS];       // step, bias + 128
};
constexpr uint32_t kMmaLast = 1u << 30;

__device__ __forceinline__ void mma_sync16() { asm volatile("bar.sync %0, %1;" ::"n"(kMmaBar), "n"(kMmaThreads) : "memory"); }
__device__ __forceinline__ void mma_sync_feeders() { asm volatile("bar.sync 6, %0;" ::"n"(kMmaFeeders) : "memory"); }
// A barrier of NT threads; true on every thread if v is true on one
template <int BAR, int NT>
__device__ __forceinline__ bool mma_sync_or(bool v) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred p, %2, %3, p;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(r)
                 : "r"((uint32_t)v), "n"(BAR), "n"(NT)
                 : "memory");
    return r != 0;
}
__device__ __forceinline__ bool mma_sync16_or(bool v) { return mma_sync_or<kMmaBar, kMmaThreads>(v); }
__device__ __forceinline__ void mma_arrive(uint64_t &bar, bool on = true) {   // one arrival per warp, if on its first lane
    __syncwarp();
    if ((threadIdx.x & 31) == 0 && on)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&bar)) : "memory");
}

// Barriers, TMEM and the matrix pieces; ends with a barrier. Every warp.
__device__ __forceinline__ void mma_setup(MmaShared &M, uint8_t *B) {
    const int tid = threadIdx.x;
    if (tid == 0) {
        for (int i = 0; i < 24; ++i) mbar_init(smem_u32(&M.bar[i]), 1);
        mbar_init(smem_u32(&M.scattered), kMmaThreads / 32);
        mbar_init(smem_u32(&M.third), kMmaThreads / 32);
        mbar_init(smem_u32(&M.drained), 1);
        M.gave_up = M.starved = 0;
        for (int i = 0; i < 4; ++i) mbar_init(smem_u32(&M.stored[i]), 4);
        for (int i = 0; i < 8; ++i) mbar_init(smem_u32(&M.second[i]), 4);
        for (uint32_t i = 0; i < kMmaChunks; ++i) {
            mbar_init(smem_u32(&M.full[i]), kMmaFeeders / 32);
            mbar_init(smem_u32(&M.empty[i]), kMmaThreads / 32);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < 32) tmem_alloc(smem_u32(&M.tmem));
    mma_load_b(B, tid, kMmaCta);
    fence_async_smem();
    tc_before();
    __syncthreads();
    tc_after();
}
__device__ __forceinline__ void mma_release(MmaShared &M) {
    tc_before();
    __syncthreads();
    tc_after();
    if (threadIdx.x < 32) tmem_free(M.tmem);
}

// The feeding warps: describe(i, a) gives atom i of the CTA or returns false
// after the last one (called by one warp, 32 atoms at once, so that their table
// entries, counts and offsets load together); place: see vcd_tables.
// A thread whose wait for a free chunk ran out writes no chunk any more but meets
// the others at every barrier, until they all return before the next 32 atoms.
template <class Describe>
__device__ __forceinline__ void mma_feed(MmaShared &M, uint8_t *ring, const vcd_dq *dq, const uint32_t *place,
                                         Describe &&describe) {
    const int tid = threadIdx.x - kMmaFeed, lane = tid & 31, warp = tid >> 5;
    constexpr int kB = kMmaChunk / kMmaFeeders;   // a chunk's list loads, then its lookups, in flight together
    uint32_t c = 0;        // chunks handed over
    bool ok = true;
    uint32_t w[kB];        // the list of the chunk in hand: loaded while the one before is worked on
    auto load = [&](const uint32_t *src, uint32_t m) {
#pragma unroll
        for (int j = 0; j < kB; ++j) w[j] = (uint32_t)(j * kMmaFeeders + tid) < m ? __ldg(src + j * kMmaFeeders + tid) : 0u;
    };
    auto entries = [&](const MmaAtom &a) { return a.more && a.tensor ? a.n : 0u; };
    for (uint32_t i = 0;; ++i) {
        if (i % 32u == 0) {
            if (i == 0)   // (in front of the loop it costs two more spilled registers and 45 us of 2 ms)
                for (int k = tid; k < VCD_NCLASS; k += kMmaFeeders) M.dq[k] = make_int2(dq->step[k], dq->bias[k] + 128);
            if (warp == 0) {
                MmaAtom a;
                a.n = a.tensor = 0;
                a.more = describe(i + lane, a);
                M.atom[(i + lane) % kMmaAtoms] = a;
            }
            if (mma_sync_or<6, kMmaFeeders>(!ok)) return;
        }
        MmaAtom &a = M.atom[i % kMmaAtoms];
        const bool more = a.more;
        const uint32_t n = entries(a);
        const uint32_t *src = a.src;
        if (i % 32u == 0) load(src, n);   // (else loaded with the atom before)
        float norm = 0.0f;
        uint32_t far = 0;
        for (uint32_t i0 = 0;; i0 += kMmaChunk) {
            const uint32_t slot = c % kMmaChunks, use = c / kMmaChunks;
            const uint32_t m = n - i0 < kMmaChunk ? n - i0 : kMmaChunk;
            const bool last = i0 + m >= n;
            uint32_t r[kB];
            int32_t l[kB];   // (level 0, from a crafted escape, dequantises to 0)
#pragma unroll
            for (int j = 0; j < kB; ++j) {
                if (j * kMmaFeeders < (int)m) r[j] = __ldg(place + (w[j] & 0xFFFFu));
                l[j] = (int32_t)w[j] >> 16;
            }
            if (!last) {
                load(src + i0 + kMmaChunk, n - i0 - kMmaChunk);
            } else if (more && (i + 1) % 32u) {
                const MmaAtom &b = M.atom[(i + 1) % kMmaAtoms];
                load(b.src, entries(b));
            }
            if (use && ok && !mbar_wait(smem_u32(&M.empty[slot]), (use + 1u) & 1u)) {
                ok = false;
                M.starved = 1;
            }
            uint2 *E = reinterpret_cast<uint2 *>(ring) + slot * kMmaChunk;
#pragma unroll
            for (int j = 0; j < kB; ++j)
                if ((uint32_t)(j * kMmaFeeders + tid) < m) {
                    const int2 d = M.dq[r[j] >> 17];
                    const uint32_t mag = (uint32_t)(l[j] < 0 ? -l[j] : l[j]);
                    int32_t v = (int32_t)(mag * (uint32_t)d.x + (uint32_t)d.y) >> 8;   // src/vc/vc.c:327-338, i32 wrap
                    v = l[j] < 0 ? (int32_t)(0u - (uint32_t)v) : l[j] == 0 ? 0 : v;
                    const float f = (float)v;
                    norm = __fmaf_rn(f, f, norm);
                    const uint32_t at = r[j] & 0x1FFFFu;
                    far = max(far, at);
                    if (ok) E[j * kMmaFeeders + tid] = make_uint2(at, mma_pieces(kMagicBits + (uint32_t)v));
                }
            if (last && more) {   // the atom's norm and extent along kz (4,096 bytes each)
                float s = norm;
#pragma unroll
                for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
                const uint32_t fw = __reduce_max_sync(0xFFFFFFFFu, far);
                if (lane == 0) M.extent.put(i, warp, s, fw);
                mma_sync_feeders();
                if (tid == 0) {
                    uint32_t f;
                    M.extent.take(i, s, f);
                    a.fits = s <= kMmaNorm * kMmaNorm;   // (NaN or infinite: no)
                    a.tiles = f / kMmaTile + 1u;
                }
            }
            if (tid == 0 && ok) M.count[slot] = m | (last ? kMmaLast : 0u);
            mma_arrive(M.full[slot], ok);
            ++c;
            if (last) break;
        }
        if (!more) return;
    }
}

// The issuing thread, up to the last atom or a wait that ran out.
__device__ __forceinline__ void mma_issue_atoms(MmaShared &M, uint32_t a, uint32_t b) {
    const uint32_t bar = smem_u32(M.bar), second = smem_u32(M.second), stored = smem_u32(M.stored);
    constexpr uint32_t tile = kMmaTile >> 4;
    uint32_t parity = 0;
    for (uint32_t i = 0;; ++i) {
        if (!mbar_wait(smem_u32(&M.scattered), i & 1u) || M.gave_up) return;
        const MmaAtom &at = M.atom[i % kMmaAtoms];
        if (!at.more) return;
        const bool tensor = at.tensor && at.fits;
        const uint32_t nt = at.tiles;
        tc_after();
        if (tensor)
            for (uint32_t t = 0; t < 4; ++t) {
                if (t < nt) mma_tile<false>(M.tmem + 64u * t, a + t * tile, b, false, bar + 8u * t);
                else tc_commit(bar + 8u * t);   // a tile left out: its barriers keep step
            }
        for (uint32_t t = 4; t < 8; ++t) {
            if (!mbar_wait(stored + 8u * (t - 4u), i & 1u)) return;
            tc_after();
            if (!tensor) continue;
            if (t >= nt) tc_commit(bar + 8u * t);
            else mma_tile<false>(M.tmem + 64u * t, a + t * tile, b, false, bar + 8u * t);
        }
        if (!tensor) continue;
        for (uint32_t t = 0; t < 8; ++t) {
            if (!mbar_wait(second + 8u * t, parity)) return;
            tc_after();
            if (t >= nt) tc_commit(bar + 64u + 8u * t);
            else mma_tile<true>(M.tmem + 64u * t, a + t * tile, b, false, bar + 64u + 8u * t);
        }
        if (!mbar_wait(smem_u32(&M.third), parity)) return;
        tc_after();
        for (uint32_t t = 0; t < 8; ++t) mma_tile<true>(M.tmem + 64u * t, a + t * tile, b, nt <= 4, bar + 128u + 8u * t);
        parity ^= 1u;
    }
}

// The issuing thread; when it returns, nothing is in flight any more (TMEM may be freed).
__device__ __forceinline__ void mma_issue(MmaShared &M, uint32_t a, uint32_t b) {
    mma_issue_atoms(M, a, b);
    tc_commit(smem_u32(&M.drained));
    mbar_wait(smem_u32(&M.drained), 0u);
}

__device__ __forceinline__ void mma_clear(uint8_t *A) {
    uint4 *A4 = reinterpret_cast<uint4 *>(A) + threadIdx.x;
#pragma unroll
    for (int i = 0; i < (int)(kMmaA / 16) / kMmaThreads; ++i) A4[i * kMmaThreads] = make_uint4(0, 0, 0, 0);
}

// The 16 warps: every atom the feeders describe. out(a, y, x, z, o) receives a
// (y, x) line's outputs z .. z + 15 along z (z = 0, 16) as magic numbers, x =
// the lane; other(a, A) transforms an atom that is not for the tensor cores, with
// A (kMmaA bytes at least; left as it is) at hand. False, on every thread, when a
// wait ran out.
//
// No warp leaves alone, so that none is missed at a barrier: a warp whose wait
// ran out goes on to the next scatter, says so before its arrival there, and all
// of them return once they have all arrived. That last wait cannot run out: each
// warp's scatter is at most 23 waits.
//
// The passes of an atom follow one another through the same operand space and
// sums, so an atom alone leaves the tensor cores idle in between. Its last
// outputs (tiles 4-7 of the third pass) are therefore stored while the next
// atom's first pass runs on tiles 0-3.
template <class Out, class Other>
__device__ __forceinline__ bool mma_atoms(uint8_t *A, MmaShared &M, const uint8_t *ring, Out &&out,
                                          Other &&other) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, group = warp >> 2, quarter = warp & 3;
    const uint32_t bar = smem_u32(M.bar), tq = M.tmem + ((uint32_t)quarter << 21);
    MmaRound R;
    R.set();
    bool ok = true, clean = false, pending = false;   // clean: A is zero; pending: outputs of tile group + 4 are due
    uint32_t c = 0, parity = 0;
    uint32_t o[16];
    auto outputs = [&](const MmaAtom &at, int t) {   // lines (y, x): y = 4 t + quarter, lane = x; outputs along z
#pragma unroll
        for (int z = 0; z < 32; z += 16) {
            mma_outputs(R, tq + 64u * t + z, o);
            out(at, 4 * t + quarter, lane, z, o);
        }
        tc_before();
    };
    for (uint32_t i = 0;; ++i) {
        if (!clean) {
            mma_clear(A);
            clean = true;
        }
        if (mma_sync16_or(!ok)) return false;
        uint32_t flags;
        do {   // scatter
            const uint32_t slot = c % kMmaChunks;
            ok = __all_sync(0xFFFFFFFFu, ok && mbar_wait(smem_u32(&M.full[slot]), (c / kMmaChunks) & 1u));
            flags = ok ? M.count[slot] : kMmaLast;
            const uint32_t m = flags & 0xFFFFu;
            const uint2 *E = reinterpret_cast<const uint2 *>(ring) + slot * kMmaChunk;
#pragma unroll
            for (int j = 0; j < (int)kMmaChunk / kMmaThreads; ++j)
                if ((uint32_t)(j * kMmaThreads + tid) < m) {
                    const uint2 e = E[j * kMmaThreads + tid];
                    *reinterpret_cast<uint16_t *>(A + e.x) = (uint16_t)e.y;
                    *reinterpret_cast<uint16_t *>(A + (e.x ^ 64u)) = (uint16_t)(e.y >> 16);   // l: the row's other half
                }
            mma_arrive(M.empty[slot], ok);
            ++c;
        } while (!(flags & kMmaLast));
        const MmaAtom &at = M.atom[i % kMmaAtoms];
        fence_async_smem();
        if (!ok) M.gave_up = 1;
        mma_arrive(M.scattered);
        if (pending) {   // the atom before: its last outputs
            const MmaAtom &b = M.atom[(i + kMmaAtoms - 1u) % kMmaAtoms];
            tc_after();
            outputs(b, group + 4);
            mma_arrive(M.stored[group]);
            pending = false;
        } else {
            mma_arrive(M.stored[group]);
        }
        if (!mbar_wait<32>(smem_u32(&M.scattered), i & 1u) || M.gave_up) return false;
        if (!at.more) return true;
        if (!(at.tensor && at.fits)) {
            mma_sync16();
            other(at, A);
            clean = false;
            continue;
        }
        const int nt = at.tiles;
#pragma unroll 1
        for (int t = group; t < 8; t += 4) {   // lines (kz, ky): quarter = kz & 3, lane = ky; outputs along x
            if (t < nt) {
                ok &= mbar_wait(bar + 8u * t, parity);
                tc_after();
                // as inputs ky of the lines (kz, x): 32 lines in a row, 64 bytes of rows ky and 32 + ky
                uint8_t *T = A + t * kMmaTile + ((uint32_t)quarter >> 1) * 8192u + ((uint32_t)lane >> 3) * 1024u + ((uint32_t)lane & 7u) * 128u;
                const uint32_t c0 = ((uint32_t)quarter & 1u) * 4u, s = (uint32_t)lane & 7u;
#pragma unroll
                for (int x = 0; x < 32; x += 16) {
                    mma_outputs(R, tq + 64u * t + x, o);
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        uint8_t *d = T + (((c0 + x / 8 + k) ^ s) << 4);
                        *reinterpret_cast<uint4 *>(d) =
                            make_uint4(mma_hi(o[8 * k], o[8 * k + 1]), mma_hi(o[8 * k + 2], o[8 * k + 3]),
                                       mma_hi(o[8 * k + 4], o[8 * k + 5]), mma_hi(o[8 * k + 6], o[8 * k + 7]));
                        *reinterpret_cast<uint4 *>(d + 4096) =
                            make_uint4(mma_lo(o[8 * k], o[8 * k + 1]), mma_lo(o[8 * k + 2], o[8 * k + 3]),
                                       mma_lo(o[8 * k + 4], o[8 * k + 5]), mma_lo(o[8 * k + 6], o[8 * k + 7]));
                    }
                }
                fence_async_smem();
                tc_before();
            }
            mma_arrive(M.second[t]);
        }
        // every tile's second pass is done with its operand before the third's is written
        for (int t = 0; t < nt; ++t) ok &= mbar_wait(bar + 64u + 8u * t, parity);
        tc_after();
        const int np = nt <= 4 ? 4 : 8;   // (the third pass takes 16 or 32 kz)
#pragma unroll 1
        for (int t = group; t < np; t += 4) {   // lines (kz, x): lane = x; outputs along y
            // as input kz of the lines (y, x): tile y >> 2, line (y & 3) * 32 + x, rows kz and 32 + kz (4096 bytes on)
            const uint32_t kz = 4u * t + (uint32_t)quarter, s = kz & 7u, cx = (uint32_t)lane >> 3;
            if (t >= nt) {   // no level at this kz: zero rows, 16 blocks of 64 lines
                uint8_t *Z = A + (uint32_t)(lane >> 3) * 8192u + (kz >> 3) * 1024u + s * 128u + ((uint32_t)lane & 7u) * 16u;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    *reinterpret_cast<uint4 *>(Z + j * 32768) = make_uint4(0, 0, 0, 0);
                    *reinterpret_cast<uint4 *>(Z + j * 32768 + 4096) = make_uint4(0, 0, 0, 0);
                }
                continue;
            }
            uint8_t *T = A + (kz >> 3) * 1024u + s * 128u + ((uint32_t)lane & 7u) * 2u;
            uint8_t *T0 = T + ((cx ^ s) << 4), *T1 = T + (((4u + cx) ^ s) << 4);   // even, odd y
#pragma unroll
            for (int y0 = 0; y0 < 32; y0 += 16) {
                mma_outputs(R, tq + 64u * t + y0, o);
#pragma unroll
                for (int y = y0; y < y0 + 16; y += 2) {
                    const uint32_t hi = mma_hi(o[y - y0], o[y - y0 + 1]), lo = mma_lo(o[y - y0], o[y - y0 + 1]);
                    const int d = (y >> 2) * (int)kMmaTile + ((y >> 1) & 1) * 8192;
                    *reinterpret_cast<uint16_t *>(T0 + d) = (uint16_t)hi;
                    *reinterpret_cast<uint16_t *>(T0 + d + 4096) = (uint16_t)lo;
                    *reinterpret_cast<uint16_t *>(T1 + d) = (uint16_t)(hi >> 16);
                    *reinterpret_cast<uint16_t *>(T1 + d + 4096) = (uint16_t)(lo >> 16);
                }
            }
        }
        fence_async_smem();
        tc_before();
        mma_arrive(M.third);
        ok &= mbar_wait(bar + 128u + 8u * group, parity);
        tc_after();
        outputs(at, group);
        for (int t = 0; t < 8; ++t) ok &= mbar_wait(bar + 128u + 8u * t, parity);   // A is free
        mma_clear(A);
        pending = true;
        parity ^= 1u;
    }
}

}  // namespace vcg
