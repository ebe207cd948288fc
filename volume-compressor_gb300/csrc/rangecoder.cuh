// Adaptive binary range coder and coefficient context coder (device): one
// atom per GPU thread, alone in its warp (few atoms) or a lane of it (many). The
// encoders that a launch runs are in rc_encode.cuh; the lockstep one here writes
// the atoms whose sums outgrow their slot.
//
// Bit-exact with the reference's coder (src/vc/vc.c:344-560): 12-bit P(0),
// shift-5 adaptation, LZMA-style carry-less low with a cached byte, 16-bit EOB
// in bypass bits, 8 significance contexts by frequency band + 12 unary
// magnitude contexts, EG0 escape tail and sign in bypass bits, contexts reset
// per atom. Two facts keep the per-bit work branch-light: a probability never
// leaves [31, 4065], so starting from range >= 2^24 one renormalisation byte
// always suffices (the reference's while-loops run at most once); and the scan
// order is sorted by frequency, so the significance band is non-decreasing
// along the scan and only one band context is live at a time.
#pragma once
#include <stdint.h>

namespace vcg {

constexpr uint32_t kTop = 1u << 24;

// ---------------------------------------------------------------- decoder
// Stream bytes of one lane: up to four unconsumed bytes at the top of `cur`
// (`nb` bits), refilled from the next aligned word `pf`, which is always
// already loaded, so a renormalisation never waits on memory. Words are read
// big-endian-ordered; bytes outside [0, len) read as zero and words wholly
// outside the stream are never loaded. A decision consumes at most one byte,
// so refilling whenever cur runs empty keeps a byte ready for the next one.
struct ByteStream {
    const uint32_t *wp;   // aligned word containing stream byte 0
    int32_t lim0;         // len + misalignment: bytes of the stream + lead-in
    uint32_t wi;          // index of the word in pf
    uint32_t cur, pf;
    uint32_t nb;          // valid bits in cur

    __device__ __forceinline__ uint32_t word(uint32_t i) const {
        const int32_t lim = lim0 - 4 * (int32_t)i;   // stream bytes (from the front) in word i
        const uint32_t raw = lim > 0 ? __ldg(wp + i) : 0u;
        const uint32_t w = __byte_perm(raw, 0, 0x0123);
        return lim >= 4 ? w : (lim <= 0 ? 0u : w & (0xFFFFFFFFu << (8 * (4 - lim))));
    }
    __device__ __forceinline__ void init(const uint8_t *p, uint32_t len) {
        const uintptr_t a = (uintptr_t)p;
        const uint32_t mis = (uint32_t)(a & 3u);
        wp = reinterpret_cast<const uint32_t *>(a - (uintptr_t)mis);
        lim0 = (int32_t)(len + mis);
        cur = word(0) << (8 * mis);
        nb = 32u - 8u * mis;
        wi = 1;
        pf = word(1);
    }
    // code = code << sh | next sh bits of the stream (sh = 0 or 8)
    __device__ __forceinline__ void shift(uint32_t &code, uint32_t sh) {
        code = __funnelshift_l(cur, code, sh);
        cur <<= sh;
        nb -= sh;
    }
    __device__ __forceinline__ void refill() {
        cur = pf;
        nb = 32u;
        pf = word(++wi);
    }
    __device__ __forceinline__ void refill_if(bool need) {
        cur = need ? pf : cur;
        nb = need ? 32u : nb;
        wi = need ? wi + 1u : wi;
        if (need) pf = word(wi);
    }
};

// Adaptive decision with P(0) = prob / 4096 (src/vc/vc.c:414-430): the split
// point (range * prob) >> 12 is the high word of range * (prob << 20), and the
// two adaptation rules are one: prob += ((bit ? 31 : 4096) - prob) >> 5 with an
// arithmetic shift (for bit = 1 it equals -(prob >> 5)). A bypass decision
// (src/vc/vc.c:431-441) is the split range >> 1 without adaptation.
__device__ __forceinline__ uint32_t rc_split(uint32_t range, uint32_t prob) { return __umulhi(range, prob << 20); }
__device__ __forceinline__ uint32_t rc_adapt(uint32_t prob, bool bit) {
    return prob + (uint32_t)((int32_t)((bit ? 31u : 4096u) - prob) >> 5);
}

// One atom per thread, for warps that decode a single atom (latency path):
// plain branches, contexts in registers. Calls sink(scan_position, level) for
// every nonzero level in scan order (src/vc/vc.c:545-560); returns 0, or 1 for
// a malformed stream (escape prefix longer than 32 ones, which no encoder
// output contains).
template <class Sink>
__device__ __forceinline__ int rc_decode_levels_lane(const uint8_t *src, uint32_t len, const uint32_t *band_start,
                                                     Sink &&sink) {
    ByteStream s;
    s.init(src, len);
    uint32_t code = 0, range = 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        s.shift(code, 8);
        if (s.nb == 0) s.refill();
    }
    auto renorm = [&]() {
        if (range < kTop) {
            range <<= 8;
            s.shift(code, 8);
            if (s.nb == 0) s.refill();
        }
    };
    auto bit = [&](uint32_t &prob) -> bool {
        const uint32_t r0 = rc_split(range, prob);
        const bool b = code >= r0;
        code = b ? code - r0 : code;
        range = b ? range - r0 : r0;
        prob = rc_adapt(prob, b);
        renorm();
        return b;
    };
    auto bypass = [&]() -> bool {
        range >>= 1;
        const bool b = code >= range;
        code = b ? code - range : code;
        renorm();
        return b;
    };
    uint32_t eob = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) eob = (eob << 1) | (uint32_t)bypass();
    if (eob > 32768u) eob = 32768u;   // src/vc/vc.c:549
    uint32_t mag[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) mag[k] = 2048u;
    for (int b = 0; b < 8; ++b) {
        const uint32_t beg = band_start[b];
        if (beg >= eob) break;
        const uint32_t end = band_start[b + 1] < eob ? band_start[b + 1] : eob;
        uint32_t sig = 2048u;
        for (uint32_t p = beg; p < end; ++p) {
            if (!bit(sig)) continue;
            uint32_t m = 0;   // unary magnitude, then EG0 escape (src/vc/vc.c:491-506)
#pragma unroll
            for (int k = 0; k < 12; ++k) {
                if (!bit(mag[k])) {
                    m = (uint32_t)k + 1u;
                    break;
                }
            }
            if (m == 0) {
                uint32_t ones = 0;
                while (bypass()) {
                    if (++ones > 32u) return 1;
                }
                uint32_t x = 1;
                for (uint32_t i = 0; i < ones; ++i) x = (x << 1) | (uint32_t)bypass();
                m = 11u + x;
            }
            const bool neg = bypass();
            sink(p, (neg ? 0u - m : m) & 0xFFFFu);
        }
    }
    return 0;
}

// ---------------------------------------------------------------- lockstep decoder
// The lanes of a warp walk the scan positions together, each lane decoding its
// own atom. The significance band and the unary-magnitude index are then
// warp-uniform, so every context is a register with a static index and every
// decision is the same instruction stream for all lanes. The significance step
// runs unpredicated (a lane past its EOB decodes garbage that is never used;
// its reads stay inside its stream); magnitude, escape and sign steps are
// predicated on the lanes that need them, and warp votes end them as soon as no
// lane needs another one.
constexpr uint32_t kFull = 0xFFFFFFFFu;

__device__ __forceinline__ bool ls_ctx(bool on, uint32_t &code, uint32_t &range, uint32_t &prob, ByteStream &s) {
    const uint32_t r0 = rc_split(range, prob);
    const bool b = code >= r0;
    const uint32_t nr = b ? range - r0 : r0;
    const uint32_t nc = b ? code - r0 : code;
    const uint32_t np = rc_adapt(prob, b);
    range = on ? nr : range;
    code = on ? nc : code;
    prob = on ? np : prob;
    const uint32_t sh = (on && nr < kTop) ? 8u : 0u;
    range <<= sh;
    s.shift(code, sh);
    return b;
}

__device__ __forceinline__ bool ls_byp(bool on, uint32_t &code, uint32_t &range, ByteStream &s) {
    const uint32_t r0 = range >> 1;
    const bool b = code >= r0;
    code = (on && b) ? code - r0 : code;
    range = on ? r0 : range;
    const uint32_t sh = (on && r0 < kTop) ? 8u : 0u;
    range <<= sh;
    s.shift(code, sh);
    return b;
}

__device__ __forceinline__ void ls_keep(ByteStream &s) { s.refill_if(s.nb == 0); }

// Every lane of the warp must call this together. `active` lanes decode the
// stream src[0..len); the others take part predicated off. Same results as
// rc_decode_levels_lane for each active lane.
template <class Sink>
__device__ __forceinline__ int rc_decode_levels_warp(const uint8_t *src, uint32_t len, bool active,
                                                     const uint32_t *band_start, Sink &&sink) {
    ByteStream s;
    s.init(active ? src : nullptr, active ? len : 0u);
    uint32_t code = 0, range = 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        s.shift(code, 8);
        s.refill_if(s.nb == 0);
    }
    uint32_t eob = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        eob = (eob << 1) | (uint32_t)ls_byp(true, code, range, s);
        s.refill_if(s.nb == 0);
    }
    if (!active) eob = 0;
    if (eob > 32768u) eob = 32768u;
    const uint32_t eob_max = __reduce_max_sync(kFull, eob);
    uint32_t mag[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) mag[k] = 2048u;
    bool bad = false;
    for (int b = 0; b < 8; ++b) {
        uint32_t sig = 2048u;
        const uint32_t pend = band_start[b + 1] < eob_max ? band_start[b + 1] : eob_max;
        for (uint32_t p = band_start[b]; p < pend; ++p) {
            const uint32_t r0 = rc_split(range, sig);
            const bool one = code >= r0;
            code = one ? code - r0 : code;
            range = one ? range - r0 : r0;
            sig = rc_adapt(sig, one);
            const uint32_t sh = range < kTop ? 8u : 0u;
            range <<= sh;
            s.shift(code, sh);
            const bool nz = one && p < eob && !bad;
            ls_keep(s);
            if (!__any_sync(kFull, nz)) continue;
            // unary magnitude: every lane with a nonzero takes step 0, so it needs
            // no vote; the escape vote is taken with the last step
            uint32_t m = 0;
            bool go = nz, esc = false;
#pragma unroll
            for (int k = 0; k < 12; ++k) {
                if (k > 0 && !__any_sync(kFull, go)) break;
                const bool more = ls_ctx(go, code, range, mag[k], s);
                m = (go && !more) ? (uint32_t)k + 1u : m;
                go = go && more;
                ls_keep(s);
                if (k == 11) esc = __any_sync(kFull, go);
            }
            if (esc) {   // escape: EG0 tail in bypass bits (rare)
                uint32_t ones = 0, x = 1, rem = 0;
                bool pre = go, suf = false;
                while (__any_sync(kFull, pre || suf)) {
                    const bool bit = ls_byp(pre || suf, code, range, s);
                    ls_keep(s);
                    if (pre) {
                        if (bit) {
                            if (++ones > 32u) { bad = true; pre = false; }
                        } else {
                            pre = false;
                            suf = ones != 0;
                            rem = ones;
                        }
                    } else if (suf) {
                        x = (x << 1) | (uint32_t)bit;
                        suf = --rem != 0;
                    }
                }
                m = go ? 11u + x : m;
            }
            const bool emit = nz && !bad;
            const bool neg = ls_byp(emit, code, range, s);
            ls_keep(s);
            if (emit) sink(p, (neg ? 0u - m : m) & 0xFFFFu);
        }
    }
    return bad ? 1 : 0;
}

// ---------------------------------------------------------------- per-lane decoder
// Each lane of a warp decodes its own atom (src/vc/vc.c:491-506, 545-560) in
// rounds that all lanes take together. A round is: up to kZ zeros of the
// significance run at once (optional), four adaptive decisions of whatever
// context the lane is at (the significance of the next position, or the next
// step of the unary magnitude), a few escape bits if a lane of the warp is in an
// escape, and the sign bit with the store of a finished level. A lane whose
// state has no part in a piece of the round sits it out.
//
// What bounds it on GB300 is the integer ALU (16 lanes per SM sub-partition: an
// instruction takes it two cycles) and the chain of one decision, so the round
// is written for few ALU instructions and short dependences (measured there: a
// multiply high 8.8 cycles, a compare and a select on it 8, but a compare and
// an instruction guarded by it 18, a branch 18-23): selects instead of guards
// wherever the next decision waits for the result, no branch inside a round.
// * A zero only shrinks the range, so a run of zeros without renormalisation
//   is a chain of multiplies whose splits all exceed max(code, 2^24 - 1); the
//   first one that does not ends it, and the lane goes on decision by decision.
// * Four decisions take at most four stream bytes: they come from one register
//   (a byte permute with a running selector); the next words of the stream are
//   loaded a round or more before they are needed.
// * The state is the shared-memory address of the context in use, so the step
//   after a one is an addition, and the context after it is always prefetched.
// * What a lane may meet near the end of its stream or of a band (bytes past
//   the end read as zero, a fresh significance context, the EOB) is left to a
//   second form of the round (END), taken when a lane of the warp is near one.
// Measured on the 32,768 atoms of the 1024^3 benchmark volume, with the warps
// placed as in rc_lanes.cuh: 5.57 ms at target 10, 3.55 at 20, 0.65 at 100. Before
// (one decision a step, whatever its kind, 82 instructions) 8.2 ms at target 10;
// at 20 and 100 the two were set side by side only on 1,024 of the atoms,
// replicated: 6.15 -> 2.85 and 1.30 -> 0.56.
constexpr uint32_t kLaneDone = 15u;
constexpr uint32_t kLaneRows = 17u;          // shared-memory rows of a warp: 13 contexts, and rows only prefetched
constexpr uint32_t kLaneRow = 128u;          // bytes of a row: a word per lane
constexpr int kEscBits = 4;                  // escape bits a round takes
// Stream bytes from which on more make no difference, and whose distances fit 31
// bits: an atom takes less than 2 MiB (32,768 positions of 13 decisions of at most
// 8 bits, an escape of 65 and a sign).
constexpr uint32_t kLaneMaxLen = 1u << 30;
constexpr uint32_t kLaneSel = 0x2107u;       // permute selector: code << 8 | first byte of the window

#ifdef __CUDA_ARCH__
// Operands: %0 range %1 code %2 selector %3 probability in use %4 probability
// after a one %5 context address %6 positions left in the band %7 address of a
// finished magnitude (0: none) %8 stream window %9 address of the lane's row 0
#define VC_LANE_Z(T0, T1)                                                                                            \
    "sub.u32 u, 4096, pz;\n\tshl.b32 v, pz, 20;\n\tmul.hi.u32 " T1 ", " T0 ", v;\n\tshr.u32 u, u, 5;\n\t"            \
    "add.u32 pz, pz, u;\n\tsetp.gt.and.u32 z, " T1 ", th, s;\n\tselp.u32 %0, " T1 ", %0, z;\n\t"                     \
    "selp.u32 %3, pz, %3, z;\n\t@z sub.u32 %6, %6, 1;\n\t"
#define VC_LANE_Z6                                                                                                   \
    "setp.eq.u32 s, %5, %9;\n\tsetp.gt.and.u32 s, %6, 6, s;\n\tmax.u32 th, %1, 0xffffff;\n\tmov.u32 t0, %0;\n\t"     \
    "mov.u32 pz, %3;\n\t" VC_LANE_Z("t0", "t1") VC_LANE_Z("t1", "t2") VC_LANE_Z("t2", "t3") VC_LANE_Z("t3", "t4")    \
    VC_LANE_Z("t4", "t5") VC_LANE_Z("t5", "t6")
// one adaptive decision: a = takes part, b / z = a one / a zero, zs / zl = a
// zero of the significance / of the magnitude
#define VC_LANE_U(GO)                                                                                                \
    "shl.b32 v, %3, 20;\n\tmul.hi.u32 t, %0, v;\n\tld.shared.u32 n2, [%5+256];\n\t"                                  \
    "sub.u32 u, 4096, %3;\n\tshr.u32 u, u, 5;\n\tadd.u32 p0, %3, u;\n\tshr.u32 u, %3, 5;\n\tsub.u32 p1, %3, u;\n\t"  \
    "setp.ge.and.u32 b|z, %1, t, a;\n\tselp.u32 tz, t, %0, a;\n\tsub.u32 u, %0, t;\n\tsub.u32 v, %1, t;\n\t"         \
    "selp.u32 %0, u, tz, b;\n\tselp.u32 %1, v, %1, b;\n\t"                                                           \
    "setp.lt.u32 q, %0, 0x1000000;\n\tshl.b32 u, %0, 8;\n\tprmt.b32 v, %1, %8, %2;\n\tselp.u32 %0, u, %0, q;\n\t"    \
    "selp.u32 %1, v, %1, q;\n\t@q sub.u32 %2, %2, 1;\n\t"                                                            \
    "selp.u32 u, p1, p0, b;\n\t@a st.shared.u32 [%5], u;\n\tselp.u32 %3, %4, p0, b;\n\tselp.u32 %4, n2, %4, b;\n\t"  \
    "setp.eq.and.u32 zs|zl, %5, %9, z;\n\t@zl mov.u32 %7, %5;\n\t@zs sub.u32 %6, %6, 1;\n\t"                         \
    "add.u32 u, %5, 128;\n\tselp.u32 %5, u, %5, b;\n\tsetp.ne.and.u32 a, %5, l, b;\n\t" GO
#define VC_LANE_GO "or.pred a, a, zs;\n\t"
#define VC_LANE_GO_END "setp.ne.and.u32 s, %6, 0, zs;\n\tor.pred a, a, s;\n\t"
#define VC_LANE_BLOCK(ZEROS, GO)                                                                                     \
    asm volatile("{\n\t.reg .pred a,b,z,s,q,zs,zl;\n\t.reg .u32 t,u,v,l,th,pz,p0,p1,n2,tz,t0,t1,t2,t3,t4,t5,t6;\n\t" \
                 "add.u32 l, %9, 1664;\n\t" ZEROS                                                                    \
                 "setp.lt.u32 a, %5, l;\n\tsetp.ne.and.u32 a, %6, 0, a;\n\t"                                         \
                 VC_LANE_U(GO) VC_LANE_U(GO) VC_LANE_U(GO) VC_LANE_U(GO) "}"                                         \
                 : "+r"(range), "+r"(code), "+r"(sel), "+r"(pr), "+r"(nx), "+r"(sa), "+r"(left), "+r"(m)             \
                 : "r"(w), "r"(base)                                                                                 \
                 : "memory")
#endif

struct RcLane {
    const uint8_t *wp, *end;      // next stream word to load; end of the stream
    uint32_t a0, a1, a2, pf, o;   // stream words from the one in use, the one loaded last (raw), bits of a0 used
    uint32_t code, range;
    uint32_t pr, nx;              // probability of the context in use, and of the one after a one
    uint32_t base, sa;            // row 0 of the lane (significance), row of the context in use (kEsc, kDone)
    uint32_t left;                // positions from the current one to the end of its band or the EOB
    uint32_t m;                   // row address of a finished magnitude whose sign is due, else 0
    uint32_t x, mag;              // escape: ones of the prefix, then suffix bits due (bit 31 set); value so far
    uint32_t eob, bend, bi;       // EOB, end of the current band (EOB at most), band
    uint32_t *dst;                // coefficient list (scan position | level << 16)
    uint32_t n, cap, bad;         // entries decoded (all, also past cap); list capacity; malformed
    uint32_t c;                   // kLaneDone once the atom is decoded
    static constexpr uint32_t kEsc = 13u * kLaneRow, kDone = 14u * kLaneRow;
#ifndef __CUDA_ARCH__
    uint32_t sig0;                // (host: row 0; rows 1-12 are S[0], S[st], ...)
    uint32_t *hS, hst;
    uint32_t row_ld(uint32_t a) const {
        const uint32_t r = (a - base) / kLaneRow;
        return r == 0 ? sig0 : r <= 12u ? hS[(r - 1u) * hst] : 2048u;
    }
    void row_st(uint32_t a, uint32_t v) {
        const uint32_t r = (a - base) / kLaneRow;
        if (r == 0) sig0 = v;
        else if (r <= 12u) hS[(r - 1u) * hst] = v;
    }
#endif

    __device__ __forceinline__ static uint32_t be(uint32_t v) { return __byte_perm(v, 0, 0x0123); }
    __device__ __forceinline__ static uint32_t stream_mask(int rem) {   // of a word with rem stream bytes from its first on
        return rem >= 4 ? 0xFFFFFFFFu : rem <= 0 ? 0u : 0xFFFFFFFFu << (8 * (4 - rem));
    }
    __device__ __forceinline__ uint32_t load_word() {   // raw word at wp if it holds a stream byte
        const uint32_t v = (int)(end - wp) > 0 ? __ldg(reinterpret_cast<const uint32_t *>(wp)) : 0u;
        wp += 4;
        return v;
    }
    // nothing of the lane is near an end any more; only where no stream word is due (o < 32)
    __device__ __forceinline__ void finish() {
        sa = base + kDone;
        left = 0x40000000u;
        end = wp + 64;
        c = kLaneDone;
    }

    // bstart: the 9-entry band table followed by a copy of its last entry.
    // S: device: the lane's word of the warp's kLaneRows rows, which are st = 32
    // words apart (row 0 the significance context, row c the one of magnitude
    // step c); host: 12 words st apart
    __device__ __forceinline__ void init(const uint8_t *s, uint32_t l, bool active, const uint32_t *bstart,
                                         uint32_t *S, uint32_t st, uint32_t *d, uint32_t cp) {
        const uint32_t len = !active ? 0u : l < kLaneMaxLen ? l : kLaneMaxLen;
        end = s + len;
        uint32_t cd = 0, at = 5;
#pragma unroll
        for (uint32_t i = 0; i < 5; ++i) cd = (cd << 8) | (i < len ? (uint32_t)__ldg(s + i) : 0u);
        uint32_t rg = 0xFFFFFFFFu, e = 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) {   // 16-bit EOB in bypass bits (src/vc/vc.c:520-525)
            rg >>= 1;
            const bool b = cd >= rg;
            cd = b ? cd - rg : cd;
            e = (e << 1) | (b ? 1u : 0u);
            if (rg < kTop) {
                rg <<= 8;
                cd = (cd << 8) | (at < len ? (uint32_t)__ldg(s + at) : 0u);
                ++at;
            }
        }
        if (e > 32768u) e = 32768u;   // src/vc/vc.c:549
        code = cd;
        range = rg;
        eob = e;
        const uint32_t mis = (uint32_t)((uintptr_t)(s + at) & 3u);
        wp = s + at - mis;
        o = 8u * mis;
        const int rem = (int)(end - wp);
        a0 = be(load_word()) & stream_mask(rem);
        a1 = be(load_word()) & stream_mask(rem - 4);
        a2 = be(load_word()) & stream_mask(rem - 8);
        pf = load_word();
        bi = 0;
        bend = bstart[1] < e ? bstart[1] : e;
        left = bend;
#ifdef __CUDA_ARCH__
#pragma unroll
        for (uint32_t k = 0; k < kLaneRows; ++k) S[k * st] = 2048u;
        base = (uint32_t)__cvta_generic_to_shared(S);
#else
        hS = S;
        hst = st;
        sig0 = 2048u;
        for (uint32_t k = 0; k < 12; ++k) S[k * st] = 2048u;
        base = kLaneRow;
#endif
        pr = nx = 2048u;
        m = x = mag = 0;
        dst = d;
        n = 0;
        cap = cp;
        bad = 0;
        c = 0;
        sa = base;
        if (!active || !e) {
            o = 0;
            finish();
        }
    }

    // a lane whose next round may meet the end of its band (a round takes at most
    // kZ + 5 positions), or whose stream word in use is not a0; near_end: or which
    // may meet the end of its stream in one of two rounds (a word each)
    template <int kZ>
    __device__ __forceinline__ bool near_band() const {
        return left < (uint32_t)(kZ + 6) || o >= 32u;
    }
    template <int kZ>
    __device__ __forceinline__ bool near_end() const {
        return (int)(end - wp) < 16 || near_band<kZ>();
    }
    __device__ __forceinline__ void next_word_end() {
        a0 = a1;
        a1 = a2;
        a2 = be(pf) & stream_mask((int)(end - wp) + 4);
        pf = load_word();
        o -= 32u;
    }
    __device__ __forceinline__ void renorm(uint32_t w, uint32_t &sel) {
        const bool q = range < kTop;
        const uint32_t c1 = __byte_perm(code, w, sel);
        range = q ? range << 8 : range;
        code = q ? c1 : code;
        sel -= q ? 1u : 0u;
    }
    __device__ __forceinline__ bool bypass(bool on, uint32_t w, uint32_t &sel) {   // src/vc/vc.c:431-441
        const uint32_t t = range >> 1;
        const bool b = on && code >= t;
        code = b ? code - t : code;
        range = on ? t : range;
        renorm(w, sel);
        return b;
    }

    // One round of every lane of the warp. END: a lane may be near an end
    // (near_end<kZ>). ESC: with escape bits.
    template <int kZ, bool END, bool ESC>
    __device__ __forceinline__ void round(const uint32_t *bstart) {
        static_assert(kZ == 0 || kZ == 6, "zeros taken at once");
        if (END)
            while (o >= 32u) next_word_end();
        uint32_t w = __funnelshift_l(a1, a0, o);
        const uint32_t w1 = __funnelshift_l(a2, a1, o);
        uint32_t sel = kLaneSel;
#ifdef __CUDA_ARCH__
        if (kZ == 0) {
            if (END) VC_LANE_BLOCK("", VC_LANE_GO_END);
            else VC_LANE_BLOCK("", VC_LANE_GO);
        } else {
            if (END) VC_LANE_BLOCK(VC_LANE_Z6, VC_LANE_GO_END);
            else VC_LANE_BLOCK(VC_LANE_Z6, VC_LANE_GO);
        }
#else
        if (sa == base && left > (uint32_t)kZ) {
            const uint32_t th = code > kTop - 1u ? code : kTop - 1u;
            for (int i = 0; i < kZ; ++i) {
                const uint32_t t = __umulhi(range, pr << 20);
                if (t <= th) break;
                range = t;
                pr = rc_adapt(pr, false);
                --left;
            }
        }
        bool go = sa < base + kEsc && left != 0;
        for (int i = 0; i < 4 && go; ++i) {
            const uint32_t t = rc_split(range, pr), n2 = row_ld(sa + 2u * kLaneRow);
            const bool b = code >= t;
            code = b ? code - t : code;
            range = b ? range - t : t;
            row_st(sa, rc_adapt(pr, b));
            renorm(w, sel);
            if (b) {
                pr = nx;
                nx = n2;
                sa += kLaneRow;
                go = sa != base + kEsc;
            } else if (sa == base) {
                pr = sig0;
                --left;
                go = left != 0;
            } else {
                m = sa;
                go = false;
            }
        }
#endif
        // bytes taken by the four decisions; the window moves on by them
        const uint32_t used = 8u * (kLaneSel - sel);
        w = used == 32u ? w1 : __funnelshift_l(w1, w, used);
        sel = kLaneSel;
        if (ESC && __any_sync(0xFFFFFFFFu, sa == base + kEsc)) {   // exponential-Golomb escape: a few bits a round, in selects
#pragma unroll
            for (int i = 0; i < kEscBits; ++i) {
                const bool on = sa == base + kEsc && m == 0 && x != 33u, suffix = (int32_t)x < 0;
                const bool b = bypass(on, w, sel);
                const uint32_t xn = suffix ? x - 1u : (b ? x + 1u : x | 0x80000000u);   // prefix ends: its ones are due
                const uint32_t mn = suffix ? 2u * mag + (b ? 1u : 0u) : 1u;
                const bool fin = on && xn == 0x80000000u;   // no suffix bit due any more
                m = fin ? base + ((11u + mn) & 0xFFFFu) * kLaneRow : m;
                x = on ? (fin ? 0u : xn) : x;
                mag = on ? mn : mag;
            }
            if (x == 33u) {   // a prefix longer than any level needs: malformed, without a part in what
                bad = 1;      // follows and at its end, where END finishes it (the state is left as it
                end = wp;     // is: with x or sa written here 32,768 atoms at target 10 take 6.0 ms, not 5.6)
            }
        }
        // sign bit and store of a finished level, then the significance of the next position
        const uint32_t pos = bend - left;
#ifdef __CUDA_ARCH__
        asm volatile(
            "{\n\t.reg .pred on, b, q, e;\n\t.reg .u32 t, u, v, sg, n1;\n\t.reg .u64 d;\n\t"
            "ld.shared.u32 sg, [%12];\n\tld.shared.u32 n1, [%12+128];\n\t"
            "setp.ne.u32 on, %7, 0;\n\tshr.u32 t, %0, 1;\n\tsetp.ge.and.u32 b, %1, t, on;\n\tsub.u32 u, %1, t;\n\t"
            "selp.u32 %1, u, %1, b;\n\tselp.u32 %0, t, %0, on;\n\tsetp.lt.u32 q, %0, 0x1000000;\n\tshl.b32 u, %0, 8;\n\t"
            "prmt.b32 v, %1, %9, %2;\n\tselp.u32 %0, u, %0, q;\n\tselp.u32 %1, v, %1, q;\n\t@q sub.u32 %2, %2, 1;\n\t"
            "sub.u32 u, %7, %12;\n\tshr.u32 u, u, 7;\n\tneg.s32 v, u;\n\tselp.u32 u, v, u, b;\n\t"
            "prmt.b32 u, %10, u, 0x5410;\n\tsetp.lt.and.u32 e, %8, %11, on;\n\tmad.wide.u32 d, %8, 4, %13;\n\t"
            "@e st.global.u32 [d], u;\n\t@on add.u32 %8, %8, 1;\n\t@on sub.u32 %6, %6, 1;\n\t"
            "selp.u32 %5, %12, %5, on;\n\tselp.u32 %3, sg, %3, on;\n\tselp.u32 %4, n1, %4, on;\n\tmov.u32 %7, 0;\n\t}"
            : "+r"(range), "+r"(code), "+r"(sel), "+r"(pr), "+r"(nx), "+r"(sa), "+r"(left), "+r"(m), "+r"(n)
            : "r"(w), "r"(pos), "r"(cap), "r"(base), "l"(dst)
            : "memory");
#else
        if (m != 0) {
            const uint32_t mg = (m - base) / kLaneRow;
            const bool b = bypass(true, w, sel);
            if (n < cap) dst[n] = ((b ? 0u - mg : mg) << 16) | pos;
            ++n;
            --left;
            sa = base;
            pr = sig0;
            nx = row_ld(base + kLaneRow);
            m = 0;
        }
#endif
        o += used + 8u * (kLaneSel - sel);
        if (!END) {
#ifdef __CUDA_ARCH__
            asm volatile(
                "{\n\t.reg .pred c;\n\t.reg .u32 t;\n\tsetp.ge.u32 c, %0, 32;\n\tselp.u32 %1, %2, %1, c;\n\t"
                "selp.u32 %2, %3, %2, c;\n\tprmt.b32 t, %4, 0, 0x0123;\n\tselp.u32 %3, t, %3, c;\n\t"
                "@c ld.global.nc.u32 %4, [%5];\n\t@c add.u64 %5, %5, 4;\n\t@c sub.u32 %0, %0, 32;\n\t}"
                : "+r"(o), "+r"(a0), "+r"(a1), "+r"(a2), "+r"(pf), "+l"(wp));
#else
            if (o >= 32u) next_word_end();
#endif
        } else {
            while (o >= 32u) next_word_end();
            const bool malformed = x == 33u;
            if (malformed || (left == 0 && sa == base)) {   // or the end of the band: a fresh context, or the EOB
                if (malformed || bend == eob) {   // (past the round's last load: finish() lifts the guard of load_word())
                    x = 0;
                    finish();
                } else {
                    ++bi;
                    const uint32_t e = bstart[bi + 1u] < eob ? bstart[bi + 1u] : eob;
                    left = e - bend;
                    bend = e;
                    pr = 2048u;
#ifndef __CUDA_ARCH__
                    sig0 = 2048u;
#endif
                }
            }
        }
    }

    // rounds of every lane of the warp until some lane has met an end (whole
    // warp; call until all lanes are done): two at a time, with escape bits in
    // the second. A lane is done only through the last round here, so that the
    // loop before it ends when no live lane is left to end it.
    template <int kZ>
    __device__ __forceinline__ void rounds(const uint32_t *bstart) {
        while (!__any_sync(0xFFFFFFFFu, near_end<kZ>())) {
            round<kZ, false, false>(bstart);
            if (__any_sync(0xFFFFFFFFu, near_band<kZ>())) break;
            round<kZ, false, true>(bstart);
        }
        round<kZ, true, true>(bstart);
    }
    // two rounds, or one where a lane may meet an end (whole warp): what
    // tests/host_decoders.cpp steps a lane with; the kernels run rounds()
    __device__ __forceinline__ void step(const uint32_t *bstart, uint32_t *S, uint32_t st) {
        (void)S;
        (void)st;
        if (!__any_sync(0xFFFFFFFFu, near_end<6>())) {
            round<6, false, false>(bstart);
            if (!__any_sync(0xFFFFFFFFu, near_band<6>())) {
                round<6, false, true>(bstart);
                return;
            }
        }
        round<6, true, true>(bstart);
    }
};

// ---------------------------------------------------------------- latency decoder
// One atom on one lane when few atoms share the GPU, so that the dependency
// chain of one decision is all that counts, and whose stream does not fit
// rc_decode_levels_sm's shared memory: both outcomes of a decision (the
// new range renormalised, the adapted probability) are computed before the
// compare, which then only selects; the byte fetch is predicated, not
// branched; and a significance decision takes one branch (a one, or the end of
// the band). Same results as rc_decode_levels_lane; measured on GB300 with one
// atom per SM sub-partition 44 ns per decision against 57 ns. With several
// warps per sub-partition its extra instructions make it slower, so it serves
// only the latency-bound case.
__device__ __forceinline__ uint32_t ld_u8_if(bool on, const uint8_t *ptr, uint32_t old) {
#ifdef __CUDA_ARCH__
    uint32_t v = old;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.global.nc.u8 %0, [%1];\n\t}"
                 : "+r"(v) : "l"(ptr), "r"((uint32_t)on));
    return v;
#else
    return on ? *ptr : old;
#endif
}
struct RcIn {
    const uint8_t *src;
    uint32_t pos, len, nxt;   // next byte to fetch (nxt: its value, 0 past the end)
};

__device__ __forceinline__ uint32_t rc_take_if(bool ren, uint32_t c1, RcIn &in) {
    const uint32_t nx = in.nxt;
    const uint32_t np = in.pos + (ren ? 1u : 0u);
    in.pos = np;
    in.nxt = ld_u8_if(ren && np < in.len, in.src + np, ren ? 0u : nx);
    return ren ? (c1 << 8) | nx : c1;
}

__device__ __forceinline__ bool rc_bit_lat(uint32_t &code, uint32_t &range, uint32_t &p, RcIn &in) {
    const uint32_t r0 = __umulhi(range, p << 20);
    const uint32_t p0 = p + ((4096u - p) >> 5), p1 = p - (p >> 5);
    const uint32_t n1 = range - r0;
    const bool ren0 = r0 < kTop, ren1 = n1 < kTop;
    const uint32_t rr0 = ren0 ? r0 << 8 : r0, rr1 = ren1 ? n1 << 8 : n1;
    const bool b = code >= r0;
    const uint32_t c1 = b ? code - r0 : code;
    range = b ? rr1 : rr0;
    p = b ? p1 : p0;
    code = rc_take_if(b ? ren1 : ren0, c1, in);
    return b;
}

__device__ __forceinline__ bool rc_bypass_lat(uint32_t &code, uint32_t &range, RcIn &in) {
    const uint32_t r0 = range >> 1;
    const bool b = code >= r0;
    const uint32_t c1 = b ? code - r0 : code;
    const bool ren = r0 < kTop;
    range = ren ? r0 << 8 : r0;
    code = rc_take_if(ren, c1, in);
    return b;
}

template <class Sink>
__device__ __forceinline__ int rc_decode_levels_lat(const uint8_t *src, uint32_t len, const uint32_t *band_start,
                                                    Sink &&sink) {
    RcIn in;
    in.src = src;
    in.len = len;
    uint32_t code = 0;
#pragma unroll
    for (uint32_t i = 0; i < 5; ++i) code = (code << 8) | (i < len ? (uint32_t)__ldg(src + i) : 0u);
    in.pos = 5;
    in.nxt = 5 < len ? __ldg(src + 5) : 0u;
    uint32_t range = 0xFFFFFFFFu, eob = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) eob = (eob << 1) | (rc_bypass_lat(code, range, in) ? 1u : 0u);
    if (eob > 32768u) eob = 32768u;   // src/vc/vc.c:549
    uint32_t mag[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) mag[k] = 2048u;
    for (int bnd = 0; bnd < 8; ++bnd) {
        uint32_t p = band_start[bnd];
        if (p >= eob) break;
        const uint32_t lim = band_start[bnd + 1] < eob ? band_start[bnd + 1] : eob;
        uint32_t sig = 2048u;
        for (;;) {
            const bool one = rc_bit_lat(code, range, sig, in);
            if (!(one | (p + 1u == lim))) {
                ++p;
                continue;
            }
            if (one) {
                uint32_t m = 0;   // unary magnitude, then EG0 escape (src/vc/vc.c:491-506)
#pragma unroll
                for (int k = 0; k < 12; ++k) {
                    if (!rc_bit_lat(code, range, mag[k], in)) {
                        m = (uint32_t)k + 1u;
                        break;
                    }
                }
                if (m == 0) {
                    uint32_t ones = 0;
                    while (rc_bypass_lat(code, range, in)) {
                        if (++ones > 32u) return 1;
                    }
                    uint32_t x = 1;
                    for (uint32_t i = 0; i < ones; ++i) x = (x << 1) | (rc_bypass_lat(code, range, in) ? 1u : 0u);
                    m = 11u + x;
                }
                const bool neg = rc_bypass_lat(code, range, in);
                sink(p, (neg ? 0u - m : m) & 0xFFFFu);
            }
            if (++p == lim) break;
        }
    }
    return 0;
}

// ---------------------------------------------------------------- latency decoder, staged stream
// One atom on one thread with its stream in shared memory. A warp that decodes
// one atom issues at most one integer-ALU instruction every two cycles, a
// branch costs it 18-23 cycles, and an instruction guarded by a fresh compare
// 14 before it can start (measured on GB300), so:
// * Zeros of a significance run are taken four at a time while they are likely
//   (probability of a zero above kRunProb): a zero without renormalisation only
//   replaces the range by the split, so four of them are a chain of four
//   multiplies, and the last split above max(code, 2^24 - 1) shows all four.
//   Where it is not, selects take the zeros before the first that is not.
// * A decision is selects only. The renormalisation multiplies the range by 256
//   or 1 (the multiply pipe is otherwise idle) and permutes the next stream byte
//   into the code under a running selector; an eight-byte window of the stream
//   is loaded once per run and per four magnitude steps.
// Measured (512 atoms of the 1024^3 benchmark volume, one per SM sub-partition;
// before: one decision at a time, masks for selects): 2.69 -> 2.25 ms at target
// 10, 1.87 -> 1.26 at 20, 0.43 -> 0.25 at 100, 8.56 -> 7.47 ms for 64 atoms at q
// 0.17. One, two, three, six or eight zeros at a time, or other bounds on their
// probability, were slower at one of these.
constexpr uint32_t kRunZeros = 4;
constexpr uint32_t kRunProb = 2560;     // of 4096
constexpr uint32_t kStagePad = 16;      // zero bytes staged after a stream
// whether a stream and those fit in room bytes (of a length near 2^32 their sum wraps)
__host__ __device__ __forceinline__ bool stage_fits(uint32_t len, uint32_t room) {
    return room >= kStagePad && len <= room - kStagePad;
}

// byte i of a staged stream (words are kept most significant byte first)
__device__ __forceinline__ uint32_t stage_at(uint32_t i) { return i ^ 3u; }

// the whole warp stages a stream and the zero bytes after it
__device__ __forceinline__ void stage_stream(uint8_t *stage, const uint8_t *src, uint32_t len, uint32_t lane) {
    for (uint32_t i0 = 0; i0 < len + kStagePad; i0 += 8u * 32u) {   // 8 independent byte loads per lane in flight
        uint32_t b[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            const uint32_t i = i0 + k * 32u + lane;
            b[k] = i < len ? (uint32_t)__ldg(src + i) : 0u;
        }
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            const uint32_t i = i0 + k * 32u + lane;
            if (i < len + kStagePad) stage[stage_at(i)] = (uint8_t)b[k];
        }
    }
}

struct RcSm {
    const uint8_t *s;        // device: staged words; host: the plain stream
    uint32_t len, pos;       // stream length; stream byte at the start of the window
    uint32_t w0, w1, sel;    // window, selector of its next byte (kLaneSel: the first)
    uint32_t code, range;

    // window at the first byte not taken; bytes past the end read as zero
    __device__ __forceinline__ void load() {
        const uint32_t np = pos + (kLaneSel - sel);
        pos = np < len ? np : len;
#ifdef __CUDA_ARCH__
        const uint32_t *W = reinterpret_cast<const uint32_t *>(s + (pos & ~3u));
        const uint32_t a = W[0], b = W[1], c = W[2], sh = 8u * pos;
        w0 = __funnelshift_l(b, a, sh);
        w1 = __funnelshift_l(c, b, sh);
#else
        for (uint32_t i = 0; i < 4; ++i) {
            w0 = (w0 << 8) | (pos + i < len ? s[pos + i] : 0u);
            w1 = (w1 << 8) | (pos + 4u + i < len ? s[pos + 4u + i] : 0u);
        }
#endif
        sel = kLaneSel;
    }
    // four bytes at hand again after at most four taken since load()
    __device__ __forceinline__ void advance() {
        const uint32_t used = kLaneSel - sel;
        w0 = used == 4u ? w1 : __funnelshift_l(w1, w0, 8u * used);
        pos += used;
        sel = kLaneSel;
    }
    __device__ __forceinline__ void renorm() {
#ifdef __CUDA_ARCH__
        asm("{\n\t.reg .pred n;\n\t.reg .u32 f, c;\n\tsetp.lt.u32 n, %0, 0x1000000;\n\tselp.u32 f, 256, 1, n;\n\t"
            "prmt.b32 c, %1, %3, %2;\n\tmul.lo.u32 %0, %0, f;\n\tselp.u32 %1, c, %1, n;\n\t@n sub.u32 %2, %2, 1;\n\t}"
            : "+r"(range), "+r"(code), "+r"(sel)
            : "r"(w0));
#else
        if (range < kTop) {
            range <<= 8;
            code = __byte_perm(code, w0, sel);
            --sel;
        }
#endif
    }
    __device__ __forceinline__ bool bit(uint32_t &p) {
        const uint32_t t = rc_split(range, p);
        const bool b = code >= t;
        const uint32_t rt = range - t, ct = code - t;
        code = b ? ct : code;
        range = b ? rt : t;
        p = rc_adapt(p, b);
        renorm();
        return b;
    }
    __device__ __forceinline__ bool bypass() {
        const uint32_t t = range >> 1;
        const bool b = code >= t;
        const uint32_t ct = code - t;
        code = b ? ct : code;
        range = t;
        renorm();
        return b;
    }
};

// s: device: the staged stream (byte i at s[stage_at(i)], s word-aligned,
// kStagePad zero bytes after the last); host: the plain stream
template <class Sink>
__device__ __forceinline__ int rc_decode_levels_sm(const uint8_t *s, uint32_t len, const uint32_t *band_start,
                                                   Sink &&sink) {
    RcSm q;
    q.s = s;
    q.len = len;
    q.pos = 0;
    q.sel = kLaneSel;
    q.load();
    q.code = (q.w0 << 8) | (q.w1 >> 24);   // the first five bytes; the very first is shifted out
    q.sel = kLaneSel - 5u;
    q.load();
    q.range = 0xFFFFFFFFu;
    uint32_t eob = 0;
#pragma unroll 1
    for (int i = 0; i < 16; ++i) {
        eob = (eob << 1) | (q.bypass() ? 1u : 0u);
        q.load();
    }
    if (eob > 32768u) eob = 32768u;   // src/vc/vc.c:549
    uint32_t mag[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) mag[k] = 2048u;
    for (int bnd = 0; bnd < 8; ++bnd) {
        if (band_start[bnd] >= eob) break;
        const uint32_t lim = band_start[bnd + 1] < eob ? band_start[bnd + 1] : eob;
        uint32_t left = lim - band_start[bnd];   // positions of the band from the current one on
        uint32_t sig = 2048u;
        while (left) {
            q.load();
            bool one;
            if (sig > kRunProb && left > kRunZeros) {
                const uint32_t th = q.code > kTop - 1u ? q.code : kTop - 1u;
                uint32_t t[kRunZeros + 1], p[kRunZeros + 1];
                for (;;) {
                    t[0] = q.range;
                    p[0] = sig;
#pragma unroll
                    for (uint32_t j = 0; j < kRunZeros; ++j) {
                        t[j + 1] = rc_split(t[j], p[j]);
                        p[j + 1] = p[j] + ((4096u - p[j]) >> 5);
                    }
                    if (!(t[kRunZeros] > th && left > 2u * kRunZeros)) break;
                    q.range = t[kRunZeros];
                    sig = p[kRunZeros];
                    left -= kRunZeros;
                }
#pragma unroll
                for (uint32_t j = 1; j < kRunZeros; ++j) {   // the zeros before the decision that is none
                    const bool ok = t[j] > th;
                    q.range = ok ? t[j] : q.range;
                    sig = ok ? p[j] : sig;
                    left -= ok ? 1u : 0u;
                }
                one = q.bit(sig);
                --left;
            } else {
                do {
                    one = q.bit(sig);
                    --left;
                } while (!one && left && q.sel != kLaneSel - 4u);
            }
            if (!one) continue;
            q.load();
            uint32_t m = 0;   // unary magnitude, then EG0 escape (src/vc/vc.c:491-506)
#pragma unroll
            for (int k = 0; k < 12; ++k) {
                if (k == 4 || k == 8) q.load();
                if (!q.bit(mag[k])) {
                    m = (uint32_t)k + 1u;
                    break;
                }
            }
            if (m == 0) {
                q.load();
                uint32_t ones = 0;
                while (q.bypass()) {
                    if (++ones > 32u) return 1;
                    q.load();
                }
                q.load();
                uint32_t x = 1;
                for (uint32_t i = 0; i < ones; ++i) {
                    x = (x << 1) | (q.bypass() ? 1u : 0u);
                    q.load();
                }
                m = 11u + x;
            }
            q.advance();
            const bool neg = q.bypass();
            sink(lim - left - 1u, (neg ? 0u - m : m) & 0xFFFFu);
        }
    }
    return 0;
}

// ---------------------------------------------------------------- encoder
// WRITE = false only tracks the interval width: the byte count of the
// reference encoder equals its number of shift-low calls (renormalisation
// steps plus the 5 flush steps), which does not depend on `low`.
template <bool WRITE>
struct RcEnc {
    uint64_t low;
    uint32_t range, pending, nbytes;
    uint32_t cache;
    uint8_t *out;
    uint32_t cap;   // bytes stored at most (the count goes on past it)

    __device__ __forceinline__ void init(uint8_t *o, uint32_t c) {
        low = 0; range = 0xFFFFFFFFu; pending = 1; nbytes = 0; cache = 0; out = o; cap = c;
    }
    __device__ __forceinline__ void shift_low() {   // src/vc/vc.c:369-380
        if (!WRITE) { ++nbytes; return; }
        if ((uint32_t)(low >> 32) != 0u || low < 0xFF000000ull) {
            uint32_t carry = (uint32_t)(low >> 32);
            uint32_t c = cache;
            do {
                if (nbytes < cap) out[nbytes] = (uint8_t)(c + carry);
                ++nbytes;
                c = 0xFFu;
            } while (--pending);
            cache = (uint32_t)(low >> 24) & 0xFFu;
        }
        ++pending;
        low = (low << 8) & 0xFFFFFFFFull;
    }
    __device__ __forceinline__ void flush() {
#pragma unroll 1
        for (int i = 0; i < 5; ++i) shift_low();
    }
    // shift_low for the lanes with ren, the others unchanged, without a branch
    // around the common case: a byte leaves (cache + carry) unless the top byte
    // is 0xFF without carry; the 0xFF bytes held back before it (pending - 1 of
    // them, rarely any) follow as 0xFF + carry.
    __device__ __forceinline__ void shift_low_if(bool ren) {
        if (!WRITE) { nbytes += ren ? 1u : 0u; return; }
        const uint32_t hi = (uint32_t)(low >> 32);
        const bool emit = ren && (hi != 0u || low < 0xFF000000ull);
        if (emit && nbytes < cap) out[nbytes] = (uint8_t)(cache + hi);
        if (emit && pending > 1u) {
            const uint8_t fill = (uint8_t)(0xFFu + hi);
            for (uint32_t j = 1; j < pending; ++j)
                if (nbytes + j < cap) out[nbytes + j] = fill;
        }
        nbytes = emit ? nbytes + pending : nbytes;
        cache = emit ? (uint32_t)(low >> 24) & 0xFFu : cache;
        pending = ren ? (emit ? 1u : pending + 1u) : pending;
        low = ren ? (low << 8) & 0xFFFFFFFFull : low;
    }
};

// ---------------------------------------------------------------- lockstep encoder
// Predicated adaptive (src/vc/vc.c:381-393) and bypass (src/vc/vc.c:394-398)
// encoder decisions; lanes with on = false keep their state.
template <bool WRITE>
__device__ __forceinline__ void enc_ctx(bool on, bool bit, RcEnc<WRITE> &e, uint32_t &prob) {
    const uint32_t r0 = rc_split(e.range, prob);
    if (WRITE && on && bit) e.low += r0;
    const uint32_t nrange = bit ? e.range - r0 : r0;
    const uint32_t nprob = rc_adapt(prob, bit);
    const bool ren = on && nrange < kTop;
    e.shift_low_if(ren);
    e.range = on ? (ren ? nrange << 8 : nrange) : e.range;
    prob = on ? nprob : prob;
}

template <bool WRITE>
__device__ __forceinline__ void enc_byp(bool on, bool bit, RcEnc<WRITE> &e) {
    const uint32_t r0 = e.range >> 1;
    if (WRITE && on && bit) e.low += r0;
    const bool ren = on && r0 < kTop;
    e.shift_low_if(ren);
    e.range = on ? (ren ? r0 << 8 : r0) : e.range;
}

// Every lane of the warp must call this together; `active` lanes encode their
// list ent[0..nnz) (scan position | level << 16, 16-byte aligned) and return
// the coder byte count (inactive lanes return 0): the reference encoder's bytes
// (src/vc/vc.c:471-490, 512-544). At most `cap` bytes are stored.
template <bool WRITE>
__device__ __forceinline__ uint32_t rc_encode_levels_warp(const uint32_t *ent, uint32_t nnz, bool active,
                                                          const uint32_t *band_start, uint8_t *out,
                                                          uint32_t cap = 0xFFFFFFFFu) {
    RcEnc<WRITE> e;
    e.init(out, cap);
    if (!active) nnz = 0;
    auto load4 = [&](uint32_t j) -> uint4 {
        return j < nnz ? __ldg(reinterpret_cast<const uint4 *>(ent + j)) : make_uint4(0, 0, 0, 0);
    };
    const uint32_t eob = nnz ? (ent[nnz - 1] & 0xFFFFu) + 1u : 0u;
#pragma unroll
    for (int i = 15; i >= 0; --i) enc_byp(active, (eob >> i) & 1u, e);
    const uint32_t eob_max = __reduce_max_sync(kFull, eob);
    uint4 g = load4(0), gn = load4(4);
    uint32_t gi = 0, i = 0, cur = g.x;
    uint32_t mag[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) mag[k] = 2048u;
    for (int b = 0; b < 8; ++b) {
        uint32_t sig = 2048u;
        const uint32_t pend = band_start[b + 1] < eob_max ? band_start[b + 1] : eob_max;
        for (uint32_t p = band_start[b]; p < pend; ++p) {
            const bool on = p < eob;
            const bool nz = on && p == (cur & 0xFFFFu);
            enc_ctx(on, nz, e, sig);
            if (!__any_sync(kFull, nz)) continue;
            const int32_t lv = (int16_t)(cur >> 16);
            const uint32_t m = (uint32_t)(lv < 0 ? -lv : lv);
            // every lane with a nonzero takes unary step 0, so it needs no vote;
            // the escape vote is taken with the last step
            bool go = nz, esc = false;
#pragma unroll
            for (int k = 0; k < 12; ++k) {
                if (k > 0 && !__any_sync(kFull, go)) break;
                const bool one = m > (uint32_t)k + 1u;   // unary: 1 while more remains
                enc_ctx(go, one, e, mag[k]);
                go = go && one;
                if (k == 11) esc = __any_sync(kFull, go);
            }
            if (esc) {   // escape: EG0 of m - 12 in bypass bits (rare)
                const uint32_t x1 = go ? m - 11u : 2u;
                const uint32_t nb = 31u - __clz(x1);
                uint32_t step = 0;
                const uint32_t total = go ? 2u * nb + 1u : 0u;
                while (__any_sync(kFull, step < total)) {
                    const bool on2 = step < total;
                    const bool one = step < nb ? true : (step == nb ? false : ((x1 >> (2u * nb - step)) & 1u) != 0);
                    enc_byp(on2, one, e);
                    ++step;
                }
            }
            enc_byp(nz, lv < 0, e);
            // the lane's list advances past this entry
            i = nz ? i + 1u : i;
            const uint32_t gi1 = nz ? gi + 1u : gi;
            const bool refill = gi1 == 4u;
            g = refill ? gn : g;
            if (refill) gn = load4(i + 4u);
            gi = refill ? 0u : gi1;
            cur = gi == 0u ? g.x : gi == 1u ? g.y : gi == 2u ? g.z : g.w;
        }
    }
    if (active) e.flush();
    return active ? e.nbytes : 0u;
}

}  // namespace vcg
