// Range encoders without a carry.
//
// Between two renormalisations the interval only shrinks, by at least every
// split added to its low end, so the splits of one such stretch add up to less
// than 2^32, a digit. The coder stores the running sum of all splits, modulo
// 2^32, at every renormalisation; digit k is sum k less sum k - 1, and the
// coder's bytes are the n + 5 bytes of sum D[k] 256^(n-k), k = 0..n, most
// significant first. enc_resolve adds the digits up, a warp per atom. So a
// coder keeps no 64-bit low end, no held-back bytes and no byte loop (the
// reference carries into bytes it holds back, src/vc/vc.c:369-380), and its one
// pass gives the length and the bytes, wherever these will go.
#pragma once
#include <stdint.h>

#include "rangecoder.cuh"

namespace vcg {

// Words of an atom's slot of sums. Coders check their count every step or pair of
// rounds (at most 256 decisions of at most 7.05 bits) and at kSumsMax or more go
// on counting over the slot's last words; such an atom is coded by
// k_rc_encode_long instead.
constexpr uint32_t kSums = 32768;
constexpr uint32_t kSumsMax = kSums - 512;

// A decision as one multiplication: the interval becomes the upper 32 bits of
// range * q + c. Below the split, q is the probability << 20 and c = 0. Above
// it, q is 2^32 less that and c = 2^32 - 1: range - floor(range p / 4096)
// exactly. A bypass decision halves the interval whichever bit it codes; its
// one adds the half to the low end, which c = 1 notes (it does not reach the
// upper word). q = c = 2^32 - 1 changes nothing.
struct EncTok { uint32_t q, c; };
constexpr uint32_t kAbove = 0xFFFFFFFFu;

__device__ __forceinline__ EncTok enc_tok(uint32_t ps, bool b) {   // ps: probability << 20
    return {b ? 0u - ps : ps, b ? kAbove : 0u};
}

// The interval and the sum of the splits added to its low end, modulo 2^32 and
// never reset: digit k is sum k less sum k - 1.
template <bool WRITE>
struct EncDigits {
    uint32_t range, sum, n;   // interval width, running sum, digits stored
    uint32_t *out;

    __device__ __forceinline__ void init(uint32_t *o) { range = 0xFFFFFFFFu; sum = 0; n = 0; out = o; }
    // The interval after a decision, r: one byte on where it fell below 2^24.
    // Selects: an instruction under a predicate just computed waits 18 cycles
    // for it, a select 8.
    __device__ __forceinline__ void renorm(uint32_t r) {
        uint32_t k;
#ifdef __CUDA_ARCH__
        asm("{\n\t.reg .pred p;\n\t.reg .b32 s;\n\tsetp.lt.u32 p, %2, 0x1000000;\n\tshl.b32 s, %2, 8;\n\t"
            "selp.b32 %0, s, %2, p;\n\tselp.b32 %1, 1, 0, p;\n\t}"
            : "=r"(range), "=r"(k)
            : "r"(r));
#else
        k = r < kTop ? 1u : 0u;
        range = k ? r << 8 : r;
#endif
        if (WRITE && k) out[n] = sum;
        n += k;
    }
    __device__ __forceinline__ void token(EncTok t) {
        const uint32_t r = (uint32_t)(((uint64_t)range * t.q + t.c) >> 32);
        if (WRITE) {
            const uint32_t a = (int32_t)t.c < 0 ? range - r : r;
            sum += t.c & 1u ? a : 0u;
        }
        renorm(r);
    }
    __device__ __forceinline__ void bypass(bool b) { token({0x80000000u, b ? 1u : 0u}); }
};

// Bypass decisions of a magnitude's end, left-aligned in *bits: the EG0 escape
// of m - 12 where m > 12 (nb ones, a zero, the nb low bits of m - 11), then the
// sign (src/vc/vc.c:471-490). Returns their count, at most 32.
__device__ __forceinline__ uint32_t enc_tail(uint32_t m, bool neg, uint32_t *bits) {
    const bool esc = m > 12u;
    const uint32_t x1 = esc ? m - 11u : 1u;
    const uint32_t nb = 31u - (uint32_t)__clz((int)x1);
    const uint32_t one = 1u << nb;
    const uint32_t v = ((((one - 1u) << (nb + 1u)) | (x1 & (one - 1u))) << 1) | (neg ? 1u : 0u);
    const uint32_t cnt = esc ? 2u * nb + 2u : 1u;
    *bits = v << (32u - cnt);
    return cnt;
}

// ---------------------------------------------------------------- few atoms
// What is coded, and with which probability, depends on the list alone. A group
// is one coder warp and half as many producer warps as it has atoms: a producer
// turns the lists of two atoms into tokens, 16 entries of each at a time (lane k
// of a half steps unary context k through them, lane 12 stores the significance
// decisions, lane j entry j's bypass decisions), and the coder takes the tokens
// of the step before, a lane per atom, in one straight line: the interval's own
// chain (multiply, compare, select: 27 cycles a decision alone, 34 beside the
// producers) is all that is left to wait for. Groups of one or two atoms have
// two producers, one for the significance decisions and one for the rest, which
// then keep ahead of the coder. One pass over 540 atoms of 30,000 decisions each
// (the longest 51,000): 1.14 ms for the sizes and 1.24 ms with the sums, against
// 2.0 and 3.4 ms for rc_encode_levels_warp with an atom per warp.
constexpr uint32_t kTokStep = 256;              // tokens of an atom and step at most (an entry's nonzero part has 43)
constexpr uint32_t kTokPitch = kTokStep + 10;   // lanes on different banks, a look ahead of four pairs
constexpr uint32_t kEncGroups = 4;              // groups of a CTA: a coder warp on each SM sub-partition
constexpr uint32_t kGroupMax = 8;               // atoms of a group at most

// Shared bytes of a group of G atoms, and its threads.
__host__ __device__ constexpr uint32_t enc_group_bytes(uint32_t G) {
    return 2u * G * kTokPitch * 8u + 2u * 32u * 4u;
}
__host__ __device__ constexpr bool enc_group_split(uint32_t G) { return G <= 2u; }
__host__ __device__ constexpr uint32_t enc_group_warps(uint32_t G) {
    return enc_group_split(G) ? 3u : 1u + (G + 1u) / 2u;
}

#ifdef __CUDACC__
struct EncGroup {
    EncTok *tok;        // [2][G][kTokPitch]
    uint32_t *cnt;      // [2][32] tokens of each atom, a multiple of 8; 0: its list has ended
    uint32_t G, bar, threads;

    __device__ __forceinline__ void init(void *mem, uint32_t G_, uint32_t bar_) {
        G = G_;
        tok = static_cast<EncTok *>(mem);
        cnt = reinterpret_cast<uint32_t *>(tok + 2u * G * kTokPitch);
        bar = bar_;
        threads = 32u * enc_group_warps(G);
    }
    __device__ __forceinline__ void sync() const {
        asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(threads) : "memory");
    }
    // any atom with tokens in step s; for the whole group after its sync
    __device__ __forceinline__ bool any(uint32_t s, uint32_t lane) const {
        return __any_sync(0xFFFFFFFFu, lane < G && cnt[(s & 1u) * 32u + (lane < G ? lane : 0u)] != 0u);
    }
};

// A producer warp: the lists of two atoms of the group, one per half of the warp
// (ent[0..nnz), scan position | level << 16; nnz = 0 for none; slot: its atom):
// their significance decisions, the others, or both.
__device__ __forceinline__ void enc_produce(const EncGroup &g, uint32_t slot, const uint32_t *ent, uint32_t nnz,
                                            const uint32_t *band_start, uint32_t lane, bool sig, bool rest) {
    const uint32_t l = lane & 15u, half = lane & 16u;
    const uint32_t clane = l < 12u ? l : 0xFFFFu, clane1 = clane + 1u;
    const bool own = slot < g.G;
    const bool zlane = l == 12u && own && sig;
    uint32_t ctx = 2048u, q = 2048u, bnd = 0, bend = band_start[1];   // q: 4096 - significance probability
    auto run = [&](EncTok *d, uint32_t k) {   // k zeros
        for (; k >= 4u; k -= 4u, d += 4) {
            const uint32_t c1 = q - (q >> 5), c2 = c1 - (c1 >> 5), c3 = c2 - (c2 >> 5);
            if (zlane) {
                d[0] = {q * 0xFFF00000u, 0u};
                d[1] = {c1 * 0xFFF00000u, 0u};
                d[2] = {c2 * 0xFFF00000u, 0u};
                d[3] = {c3 * 0xFFF00000u, 0u};
            }
            q = c3 - (c3 >> 5);
        }
        for (; k; --k, ++d) {
            if (zlane) *d = {q * 0xFFF00000u, 0u};
            q -= q >> 5;
        }
    };
    auto band = [&]() {
        ++bnd;
        bend = band_start[bnd + 1u];
        q = 2048u;
    };
    uint32_t i0 = 0, pos = 0;
    uint32_t cur = l < nnz ? __ldg(ent + l) : 0u, nxt = 16u + l < nnz ? __ldg(ent + 16u + l) : 0u;
    for (uint32_t s = 0;; ++s) {
        EncTok *tok = g.tok + ((s & 1u) * g.G + (own ? slot : 0u)) * kTokPitch;
        const bool on = i0 + l < nnz;
        const uint32_t p = cur & 0xFFFFu;
        const int32_t lv = (int32_t)cur >> 16;
        const uint32_t m = on ? (uint32_t)(lv < 0 ? -lv : lv) : 0u, mm = m < 12u ? m : 12u;
        uint32_t bits;
        const uint32_t tail = enc_tail(m, lv < 0, &bits);
        const uint32_t pl = __shfl_up_sync(0xFFFFFFFFu, p, 1, 16);
        const uint32_t z = on ? p - (l ? pl + 1u : pos) : 0u;   // zeros before the entry
        const uint32_t len = on ? z + 1u + mm + tail : 0u;
        uint32_t end = len;
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, end, o, 16);
            if ((int)l >= o) end += y;
        }
        // the entries that fit this step; none: as many of the first one's zeros as do
        const uint32_t ok = __ballot_sync(0xFFFFFFFFu, on && end <= kTokStep) >> half & 0xFFFFu;
        const uint32_t E = (uint32_t)__popc(ok), Emax = __reduce_max_sync(0xFFFFFFFFu, E);
        const uint32_t z0 = __shfl_sync(0xFFFFFFFFu, z, 0, 16);
        const uint32_t zc = E == 0u && i0 < nnz ? (z0 < kTokStep ? z0 : kTokStep) : 0u;
        const uint32_t last = E ? E - 1u : 0u;
        const uint32_t fit = __shfl_sync(0xFFFFFFFFu, end, (int)last, 16);
        const uint32_t all = E ? fit : zc;
        const uint32_t next = __shfl_sync(0xFFFFFFFFu, p, last, 16) + 1u;
        const uint32_t at = end - tail - mm;   // first unary decision; the nonzero one and its zeros end before it
        // the first entry past this band
        const uint32_t jb = (uint32_t)__ffs((int)(__ballot_sync(0xFFFFFFFFu, on && p >= bend) >> half & 0xFFFFu)) - 1u;
        uint32_t sp = pos;
        if (zc && sig) {   // zeros alone, without the entry that ends them
            uint32_t d = 0;
            while (d < zc) {
                if (sp == bend) band();
                const uint32_t k = bend - sp < zc - d ? bend - sp : zc - d;
                run(tok + d, k);
                d += k;
                sp += k;
            }
        }
        // Four zeros at most before every entry and no band's end: no branch.
        const uint32_t az = at << 16 | z;
        auto four = [&](uint32_t d, uint32_t r) {   // r zeros of 0..4 at token d
            const uint32_t c1 = q - (q >> 5), c2 = c1 - (c1 >> 5), c3 = c2 - (c2 >> 5), c4 = c3 - (c3 >> 5);
            if (zlane && r > 0u) tok[d] = {q * 0xFFF00000u, 0u};
            if (zlane && r > 1u) tok[d + 1u] = {c1 * 0xFFF00000u, 0u};
            if (zlane && r > 2u) tok[d + 2u] = {c2 * 0xFFF00000u, 0u};
            if (zlane && r > 3u) tok[d + 3u] = {c3 * 0xFFF00000u, 0u};
            const uint32_t e1 = r > 0u ? c1 : q, e2 = r > 1u ? c2 : e1, e3 = r > 2u ? c3 : e2;
            q = r > 3u ? c4 : e3;
        };
        auto one = [&](uint32_t d, bool act) {
            const uint32_t pr = 4096u - q;
            if (zlane && act) tok[d] = enc_tok(pr << 20, true);
            q += act ? pr >> 5 : 0u;
        };
        if (!sig) {
        } else if (!__any_sync(0xFFFFFFFFu, l < E && (z > 4u || l >= jb))) {
#pragma unroll 4
            for (uint32_t j = 0; j < Emax; ++j) {
                const uint32_t w = __shfl_sync(0xFFFFFFFFu, az, (int)j, 16);
                const bool act = j < E;
                const uint32_t zr = act ? w & 0xFFFFu : 0u, aj = w >> 16;
                four(aj - 1u - zr, zr);
                one(aj - 1u, act);
            }
        } else {
#pragma unroll 1
            for (uint32_t j = 0; j < Emax; ++j) {
                const uint32_t w = __shfl_sync(0xFFFFFFFFu, az, (int)j, 16);
                const bool act = j < E;
                uint32_t zr = act ? w & 0xFFFFu : 0u;
                const uint32_t aj = w >> 16;
                uint32_t d = aj - 1u - zr;
                if (act && j >= jb) {   // a band may end before this entry
                    while (sp + zr >= bend) {
                        const uint32_t k = bend - sp;
                        run(tok + d, k);
                        d += k;
                        zr -= k;
                        sp = bend;
                        band();
                    }
                }
                sp = act ? sp + zr + 1u : sp;
                const uint32_t k = zr & ~3u;
                run(tok + d, k);
                four(d + k, zr & 3u);
                one(aj - 1u, act);
            }
        }
        if (rest) {
#pragma unroll 8
            for (uint32_t j = 0; j < 16u; ++j) {
                const uint32_t w = __shfl_sync(0xFFFFFFFFu, m | at << 16, (int)j, 16);
                const uint32_t mj = w & 0xFFFFu;
                const bool has = j < E && mj > clane, b = mj > clane1;
                if (has) tok[(w >> 16) + l] = enc_tok(ctx << 20, b);
                const uint32_t nc = ctx + (uint32_t)((int32_t)((b ? 31u : 4096u) - ctx) >> 5);
                ctx = has ? nc : ctx;
            }
            if (l < E) {
                uint32_t d = end - tail;
                for (uint32_t t = tail; t; --t, bits <<= 1) tok[d++] = {0x80000000u, bits >> 31};
            }
        }
        const uint32_t pad = (0u - all) & 7u;
        if (own && sig && l < pad) tok[all + l] = {kAbove, kAbove};
        if (own && sig && l == 0u) g.cnt[(s & 1u) * 32u + slot] = all + pad;
        pos = E ? next : pos + zc;
        i0 += E;
        const uint32_t from = E + l;
        const uint32_t a = __shfl_sync(0xFFFFFFFFu, cur, (int)(from & 15u), 16);
        const uint32_t b = __shfl_sync(0xFFFFFFFFu, nxt, (int)(from & 15u), 16);
        cur = from < 16u ? a : b;
        nxt = i0 + 16u + l < nnz ? __ldg(ent + i0 + 16u + l) : 0u;
        g.sync();
        if (!g.any(s, lane)) break;
    }
}

// The coder warp of a group: lane a, where on, codes the group's atom a (eob: its
// last entry's scan position + 1, or 0) and returns its byte count; its sums go
// to out, kSums words.
template <bool WRITE>
__device__ __forceinline__ uint32_t enc_consume(const EncGroup &g, bool on, uint32_t eob, uint32_t *out,
                                                uint32_t lane) {
    EncDigits<WRITE> e;
    e.init(out);
    uint32_t over = 0;
    if (on)
        for (int i = 15; i >= 0; --i) e.bypass((eob >> i) & 1u);
    const uint32_t a = lane < g.G ? lane : 0u;
    for (uint32_t s = 0;; ++s) {
        g.sync();
        if (!g.any(s, lane)) break;
        const uint32_t cnt = lane < g.G ? g.cnt[(s & 1u) * 32u + a] : 0u;
        const uint32_t n = __reduce_max_sync(0xFFFFFFFFu, cnt);
        const uint4 *tp = reinterpret_cast<const uint4 *>(g.tok + ((s & 1u) * g.G + a) * kTokPitch);
        uint4 v[4];
#pragma unroll
        for (int y = 0; y < 4; ++y) v[y] = tp[y];
#pragma unroll 1
        for (uint32_t t = 0; t < n; t += 8u) {
            const uint32_t off = (uint32_t)((int32_t)(cnt - 1u - t) >> 31);   // all ones past the atom's tokens
            tp += 4;
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                const EncTok t0 = {v[y].x | off, v[y].y | off};
                const EncTok t1 = {v[y].z | off, v[y].w | off};
                v[y] = tp[y];   // at most the row's padding
                e.token(t0);
                e.token(t1);
            }
        }
        if (WRITE && e.n >= kSumsMax) {   // too long for its slot: count on, keep the last sums' place
            over += e.n - (kSumsMax - 512u);
            e.n = kSumsMax - 512u;
        }
    }
    if (WRITE && on) out[e.n] = e.sum;
    return e.n + over + 5u;
}
#endif

// ---------------------------------------------------------------- one atom per lane
// Rounds: up to 2 kZ - 1 zeros, the nonzero that ends them, kU unary and kB
// bypass decisions, each where the lane is at that point of its list; a lane
// goes on with its next entry in its next round, at its own pace. What a lane
// does is known before the round's multiplies, so lanes never part and a round
// is bound by its instructions (about 200). 32,768 atoms of 48,700 decisions each
// take 7.0 ms (kZ 4, kU 3, kB 2), against 7.1 ms for the sizes and then 13.1 ms
// for the bytes in lockstep (rc_encode_levels_warp).
constexpr uint32_t kEncRows = 12;        // unary contexts, a row of 32 lanes each
constexpr uint32_t kRing = 32;           // list entries a lane holds in shared memory
constexpr uint32_t kRingPitch = 36;      // words: 16-byte pieces, lanes on different banks
constexpr uint32_t kRingAhead = 6;       // pieces of four entries in flight or held
constexpr uint32_t kEncWarpWords = (kEncRows + 4) * 32 + 32 * kRingPitch;   // rows past the last are read, not used

__device__ __forceinline__ void ring_copy(uint32_t *dst, const uint32_t *src) {
#ifdef __CUDA_ARCH__
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
#else
    for (int i = 0; i < 4; ++i) dst[i] = src[i];
#endif
}
__device__ __forceinline__ void ring_commit() {
#ifdef __CUDA_ARCH__
    asm volatile("cp.async.commit_group;" ::: "memory");
#endif
}
template <int N>
__device__ __forceinline__ void ring_wait() {
#ifdef __CUDA_ARCH__
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
#endif
}

// Up to N zeros at once: all N if the run z holds them and none but the last
// renormalises (the splits only shrink). c = 4096 - probability loses c >> 5
// with each.
template <int N, bool WRITE>
__device__ __forceinline__ void enc_zeros(EncDigits<WRITE> &e, uint32_t &q, uint32_t &z) {
    uint32_t t = e.range, c = q;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        t = __umulhi(t, c * 0xFFF00000u);   // rc_split(t, 4096 - c)
        c -= c >> 5;
    }
    uint32_t r;
#ifdef __CUDA_ARCH__
    uint32_t k;
    asm("{\n\t.reg .pred p, w;\n\tsetp.ge.u32 w, %4, %8;\n\tsetp.ge.and.u32 p, %5, %9, w;\n\t"
        "selp.b32 %0, %5, %6, p;\n\tselp.b32 %1, %7, %3, p;\n\tselp.b32 %2, %8, 0, p;\n\t}"
        : "=r"(r), "=r"(c), "=r"(k)
        : "r"(q), "r"(z), "r"(t), "r"(e.range), "r"(c), "n"(N), "n"(N == 1 ? 0u : kTop));
    q = c;
    z -= k;
#else
    const bool ok = z >= (uint32_t)N && t >= (N == 1 ? 0u : kTop);
    q = ok ? c : q;
    z = ok ? z - (uint32_t)N : z;
    r = ok ? t : e.range;
#endif
    if (N == 1) e.renorm(r);
    else e.range = r;
}

template <int kZ, int kU, int kB>
struct EncLane {
    EncDigits<true> e;
    const uint32_t *ent;
    uint32_t *row, *ring;   // this lane's unary contexts (32 words apart) and list entries
    uint32_t nnz, i;        // list length, the entry being coded
    uint32_t pos, ep, bend, bnd;   // next position, the entry's, the band's end
    uint32_t q;             // 4096 - significance probability
    uint32_t u;             // 0: before the entry, 1..12: unary decision, 13: bypass, 64: done
    uint32_t m, mm, bits, cnt;   // magnitude, at most 12 of it, bypass decisions left-aligned and their count
    uint32_t over;

    __device__ __forceinline__ void take(uint32_t x) {
        const int32_t lv = (int32_t)x >> 16;
        ep = x & 0xFFFFu;
        m = (uint32_t)(lv < 0 ? -lv : lv);
        mm = m < 12u ? m : 12u;
        cnt = enc_tail(m, lv < 0, &bits);
    }

    // every lane of the warp; lanes without an atom have nnz_ = 0 and on = false
    __device__ __forceinline__ void init(bool on, const uint32_t *ent_, uint32_t nnz_, const uint32_t *band_start,
                                         uint32_t *out, uint32_t *row_, uint32_t *ring_) {
        e.init(out);
        ent = ent_; row = row_; ring = ring_; nnz = nnz_;
        const uint32_t eob = nnz ? (ent[nnz - 1] & 0xFFFFu) + 1u : 0u;
#pragma unroll
        for (uint32_t k = 0; k < kEncRows; ++k) row[k * 32u] = 2048u;
#pragma unroll
        for (uint32_t k = 0; k < kRingAhead; ++k)
            if (4u * k < nnz) ring_copy(ring + 4u * k, ent + 4u * k);
        ring_commit();
        if (on)
            for (int b = 15; b >= 0; --b) e.bypass((eob >> b) & 1u);
        i = 0; pos = 0; bnd = 0; bend = band_start[1]; q = 2048u; over = 0;
        u = on && nnz ? 0u : 64u;
        ring_wait<0>();
        take(nnz ? ring[0] : 0u);
    }

    __device__ __forceinline__ void round(const uint32_t *band_start) {
        // the entry after this one, in case this round ends this one
        const uint32_t nx = ring[(i + 1u) % kRing];
        const bool sigp = u == 0u;
        const uint32_t tgt = ep < bend ? ep : bend;
        uint32_t z = sigp ? tgt - pos : 0u;
        if (kZ >= 8) enc_zeros<8>(e, q, z);
        if (kZ >= 4) enc_zeros<4>(e, q, z);
        if (kZ >= 2) enc_zeros<2>(e, q, z);
        enc_zeros<1>(e, q, z);
        pos = sigp ? tgt - z : pos;
        const bool at = sigp && z == 0u;
        const bool hit = at && ep < bend;
        e.token({hit ? q * 0x100000u : kAbove, kAbove});   // 2^32 less the probability << 20
        q = hit ? q + ((4096u - q) >> 5) : q;
        u = hit ? 1u : u;
        // unary decisions left, ones left (a one while more remains), the row of the next one
        const uint32_t u0 = u - 1u;
        const bool un = u0 < 12u;
        const uint32_t left = un ? mm - u0 : 0u, ones = m - u0;
        uint32_t *c = row + (un ? u0 * 32u : 0u);
#pragma unroll
        for (int s = 0; s < kU; ++s) {
            const bool on = left > (uint32_t)s, b = !(on && ones <= (uint32_t)s + 1u);
            const uint32_t p = c[s * 32];
            e.token({on ? (b ? 0u - (p << 20) : p << 20) : kAbove, b ? kAbove : 0u});
            const uint32_t np = p + (uint32_t)((int32_t)((b ? 31u : 4096u) - p) >> 5);
            if (on) c[s * 32] = np;
        }
        u = un ? (left <= (uint32_t)kU ? 13u : u + (uint32_t)kU) : u;
        const bool by = u == 13u;
        const uint32_t have = by ? cnt : 0u;
#pragma unroll
        for (int s = 0; s < kB; ++s) {
            const bool on = have > (uint32_t)s;
            const uint32_t t = e.range >> 1;
            if (on && (int32_t)(bits << s) < 0) e.sum += t;
            e.renorm(on ? t : e.range);
        }
        const bool end = by && cnt <= (uint32_t)kB;
        bits = by ? bits << kB : bits;
        cnt = by ? cnt - (uint32_t)kB : cnt;
        if (end) {
            ++i;
            pos = ep + 1u;
            u = i < nnz ? 0u : 64u;
            take(nx);
            const uint32_t j = (i & ~3u) + 4u * (kRingAhead - 1u);
            if ((i & 3u) == 0u && j < nnz) ring_copy(ring + j % kRing, ent + j);
        }
        ring_commit();
        if (at && !hit) {   // the band's end
            pos = bend;
            ++bnd;
            bend = band_start[bnd + 1u];
            q = 2048u;
        }
        ring_wait<8>();
    }
};

// Every lane of the warp calls this; lanes with on code their list and return
// the coder's byte count. mem: kEncWarpWords words of the warp.
template <int kZ, int kU, int kB>
__device__ __forceinline__ uint32_t enc_lanes(bool on, const uint32_t *ent, uint32_t nnz, const uint32_t *band_start,
                                              uint32_t *out, uint32_t *mem, uint32_t lane) {
    EncLane<kZ, kU, kB> c;
    c.init(on, ent, on ? nnz : 0u, band_start, out, mem + lane, mem + (kEncRows + 4u) * 32u + lane * kRingPitch);
    while (__any_sync(0xFFFFFFFFu, c.u != 64u)) {
        c.round(band_start);
        c.round(band_start);
        if (c.e.n >= kSumsMax) {
            c.over += c.e.n - (kSumsMax - 512u);
            c.e.n = kSumsMax - 512u;
        }
    }
    if (on) out[c.e.n] = c.e.sum;
    return on ? c.e.n + c.over + 5u : 0u;
}

#ifdef __CUDACC__
// ---------------------------------------------------------------- the bytes
// The whole warp calls this: the n + 5 coder bytes of sums[0..n] to out. Four
// digits at a time: A[w] = sum D[4w + i] 256^(3-i), i = 0..3, has at most 57
// bits; its lower word is added to the upper one of A[w + 1] and stands for bytes
// 4w + 4..4w + 7, the upper word of A[0] for the first four. A sum of two words
// carries at most one, so a step of 32 words takes its carries from two ballots.
__device__ __forceinline__ void enc_resolve(const uint32_t *sums, uint32_t n, uint8_t *out, uint32_t lane) {
    const int32_t words = (int32_t)(n >> 2) + 1;   // A[0..words)
    uint32_t cin = 0, hi0 = 0;   // carry and A's upper word from the step below (less significant)
    // words -1..words-1, from the last; lane l holds word base + l
    for (int32_t base = ((words + 32) & ~31) - 33; base >= -1; base -= 32) {
        const int32_t w = base + (int32_t)lane;
        uint64_t a = 0;
        if (w >= 0 && w < words) {
            const uint32_t k = 4u * (uint32_t)w;
            const uint4 v = *reinterpret_cast<const uint4 *>(sums + k);
            uint32_t prev = k ? sums[k - 1u] : 0u;
            const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                a = (a << 8) + (k + i <= n ? x[i] - prev : 0u);
                prev = x[i];
            }
        }
        uint32_t hi = __shfl_down_sync(0xFFFFFFFFu, (uint32_t)(a >> 32), 1);
        hi = lane == 31u ? hi0 : hi;
        hi0 = __shfl_sync(0xFFFFFFFFu, (uint32_t)(a >> 32), 0);
        const uint64_t t = (uint64_t)(uint32_t)a + hi;
        const uint32_t gen = __brev(__ballot_sync(0xFFFFFFFFu, t >> 32 != 0u));
        const uint32_t pro = __brev(__ballot_sync(0xFFFFFFFFu, (uint32_t)t == 0xFFFFFFFFu)) | gen;
        const uint64_t c = (uint64_t)pro + gen + cin;   // carries: lane 31 is bit 0
        const uint32_t into = (uint32_t)c ^ pro ^ gen;
        cin = (uint32_t)(c >> 32);
        const uint32_t r = (uint32_t)t + ((into >> (31u - lane)) & 1u);
        if (w >= -1 && w < words) {
            const uint32_t b = 4u * (uint32_t)(w + 1);
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i)
                if (b + i < n + 5u) out[b + i] = (uint8_t)(r >> (24u - 8u * i));
        }
    }
}
#endif

// ---------------------------------------------------------------- lengths alone
// A decision multiplies the interval by c / 4096, c the probability of the symbol
// it codes, up to the split's rounding down by less than one: with the interval r
// at 2^24 or more, -log2 of the factor lies within 4096 log2(e) / (2^24 c) of
// 12 - log2 c, above it below the split and below it above. So the bits L by
// which a list's decisions shrink the interval are known, to about a hundredth
// of a bit, from their probabilities alone, without the interval: in any order,
// a lane per context. And the renormalisations leave the interval in
// [2^24, 2^32), so their number is L / 8 rounded down unless L is that close to a
// multiple of 8 (one atom in a thousand), where the coder has to run.
//
// Costs are in 2^-26 bits, rounded to the nearest; a table entry is a cost and
// the most that the true one can differ from it.
constexpr uint32_t kCostOne = 1u << 26;    // one bit
constexpr uint32_t kCostSlack = 1u;        // of the rounding, either way
constexpr uint32_t kCostBypass = 6u;       // a bypass decision: one bit and at most 1.45 2^-24 more
struct EncCosts {
    uint2 one[4096];     // [c]: cost, error
    uint2 eight[4096];   // [q]: eight zeros from q = 4096 - p: cost, error << 16 | q after them
};

// The encoder's tables on the device.
struct EncTables {
    EncCosts costs;
    uint32_t place[32768];   // scan position -> index in the forward transform's tile | quantiser class << 16
};

#ifdef __CUDACC__
struct EncSize {   // least and most bits are cost - lo and cost + hi
    uint64_t cost;
    uint32_t lo, hi;
};

// Significance decisions of band b of the lane's atom: up to eight and four zeros
// and the nonzero a round, as enc_lanes. ROW: lanes 8i..8i+7 hold an atom's bands.
template <bool ROW>
__device__ __forceinline__ EncSize enc_size_bands(const EncCosts &T, const uint32_t *ent, uint32_t nnz, uint32_t b,
                                                  const uint32_t *band_start, uint32_t *ring) {
    EncSize r{0, 0, 0};
    const uint32_t eob = nnz ? (ent[nnz - 1u] & 0xFFFFu) + 1u : 0u;
    const uint32_t beg = band_start[b];
    auto first = [&](uint32_t at) {   // the first entry from scan position at on
        uint32_t lo = 0;
        for (uint32_t hi = nnz; lo < hi;) {
            const uint32_t mid = (lo + hi) >> 1;
            if ((ent[mid] & 0xFFFFu) < at) lo = mid + 1u;
            else hi = mid;
        }
        return lo;
    };
    uint32_t e = first(beg);
    uint32_t e1;
    if (ROW) {
        e1 = __shfl_down_sync(0xFFFFFFFFu, e, 1);
        e1 = b == 7u ? nnz : e1;
    } else {
        e1 = first(band_start[b + 1u]);
    }
    const uint32_t end = band_start[b + 1u] < eob ? band_start[b + 1u] : eob;
    bool live = beg < end;
    const uint32_t j0 = e & ~3u;
#pragma unroll
    for (uint32_t k = 0; k < kRingAhead; ++k)
        if (live && j0 + 4u * k < e1) ring_copy(ring + (j0 + 4u * k) % kRing, ent + j0 + 4u * k);
    ring_commit();
    ring_wait<0>();
    uint32_t p = live && e < e1 ? ring[e % kRing] & 0xFFFFu : end;
    uint32_t rem = live ? p - beg : 0u, q = 2048u;
    if (live) {   // the slack of every zero, or eight of them, and of every nonzero
        r.lo = (end - beg) * kCostSlack;
        r.hi = (e1 - e) * kCostSlack;
    }
    auto round = [&]() {
        const uint32_t nx = ring[(e + 1u) % kRing] & 0xFFFFu;
        uint32_t sum = 0;   // at most 64 bits: eight zeros cost 30 at most, four 20
        {
            const uint2 v = T.eight[q];
            const bool on = rem >= 8u;
            sum += on ? v.x : 0u;
            r.hi += on ? v.y >> 16 : 0u;
            q = on ? v.y & 0xFFFFu : q;
            rem -= on ? 8u : 0u;
        }
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            const uint2 v = T.one[4096u - q];
            const bool on = rem > (uint32_t)y;
            sum += on ? v.x : 0u;
            r.hi += on ? v.y : 0u;
            q = on ? q - (q >> 5) : q;
        }
        rem -= rem < 4u ? rem : 4u;
        const bool ev = live && rem == 0u, hit = ev && e < e1;
        const uint2 v = T.one[q];
        sum += hit ? v.x : 0u;
        r.lo += hit ? v.y : 0u;
        q += hit ? (4096u - q) >> 5 : 0u;
        e += hit ? 1u : 0u;
        const uint32_t np = e < e1 ? nx : end;
        rem = hit ? np - p - 1u : rem;
        p = hit ? np : p;
        live = live && (!ev || hit);
        const uint32_t j = (e & ~3u) + 4u * (kRingAhead - 1u);
        if (hit && (e & 3u) == 0u && j < e1) ring_copy(ring + j % kRing, ent + j);
        r.cost += sum;
    };
    while (__any_sync(0xFFFFFFFFu, live)) {
        round();
        round();
        ring_commit();
        ring_wait<4>();
    }
    ring_wait<0>();   // the ring is the next atom's
    return r;
}

// The other decisions: lane k of each sixteen steps unary context k through its
// atom's list, lane j counts the bypass decisions of every sixteenth entry.
__device__ __forceinline__ EncSize enc_size_rest(const EncCosts &T, const uint32_t *ent, uint32_t nnz,
                                                 uint32_t lane) {
    EncSize r{0, 0, 0};
    const uint32_t l = lane & 15u;
    const uint32_t clane = l < 12u ? l : 0xFFFFu, clane1 = clane + 1u;
    const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, nnz);
    uint32_t ctx = 2048u, nx = l < nnz ? __ldg(ent + l) : 0u;
    for (uint32_t i0 = 0; i0 < most; i0 += 16u) {
        const int32_t lv = (int32_t)nx >> 16;
        const uint32_t m = (uint32_t)(lv < 0 ? -lv : lv);   // 0 past the list's end
        nx = i0 + 16u + l < nnz ? __ldg(ent + i0 + 16u + l) : 0u;
        uint32_t bits;
        const uint32_t tail = m ? enc_tail(m, false, &bits) : 0u;
        r.cost += (uint64_t)tail * kCostOne;
        r.hi += tail * kCostBypass;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t sum = 0;   // eight decisions of at most 7.05 bits
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t mj = __shfl_sync(0xFFFFFFFFu, m, h * 8 + j, 16);
                const bool has = mj > clane, b = mj > clane1;
                const uint2 v = T.one[b ? 4096u - ctx : ctx];
                sum += has ? v.x : 0u;
                r.lo += has ? (b ? v.y : kCostSlack) : 0u;
                r.hi += has ? (b ? kCostSlack : v.y) : 0u;
                const uint32_t nc = ctx + (uint32_t)((int32_t)((b ? 31u : 4096u) - ctx) >> 5);
                ctx = has ? nc : ctx;
            }
            r.cost += sum;
        }
    }
    return r;
}
#endif

}  // namespace vcg
