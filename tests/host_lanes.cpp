// Host build of the per-lane range decoder (volume-compressor_gb300/csrc/
// rangecoder.cuh, RcLane) in the loop that the kernels run it in, decode_lanes of
// rc_lanes.cuh, with single-lane stand-ins for the CUDA intrinsics (the lanes of
// a warp are alike). Test infrastructure: every stream of the input file must end
// within a bounded number of warp votes, with the oracle's status and levels and
// without a load of a word that holds no stream byte
// (tests/test_host_lanes.py writes the file).
//
// Input (little-endian): u32 n; per stream: u32 len, u32 bad, u32 nent, then
// len stream bytes, then nent entries (scan position | level << 16, scan order).
// With a second argument, that many bytes are claimed past each stream, of which
// the first 2 MiB are there, and zero: more than an atom takes.
// Output: one line per form of the loop, "<name> <streams that differ> <streams
// without an end> <streams with a load outside> <streams>".
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <vector>

#define __device__
#define __host__
#define __forceinline__ inline
#define __global__
#define __constant__

static inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
// A load of a word without a stream byte (or of a byte outside the stream) is
// counted and gives ones instead.
static const uint8_t *g_lo, *g_hi;
static uint64_t g_outside;
static inline bool inside(const void *p, size_t n) {
    const bool in = (const uint8_t *)p < g_hi && (const uint8_t *)p + n > g_lo;
    g_outside += !in;
    return in;
}
static inline uint32_t __ldg(const uint32_t *p) { return inside(p, 4) ? *p : 0xFFFFFFFFu; }
static inline uint8_t __ldg(const uint8_t *p) { return inside(p, 1) ? *p : 0xFFu; }
static inline uint32_t __byte_perm(uint32_t x, uint32_t y, uint32_t s) {
    const uint64_t v = ((uint64_t)y << 32) | x;
    uint32_t r = 0;
    for (int i = 0; i < 4; ++i) r |= (uint32_t)((v >> (8 * ((s >> (4 * i)) & 7u))) & 0xFFu) << (8 * i);
    return r;
}
static inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t sh) {
    return (uint32_t)(((((uint64_t)hi << 32) | lo) << (sh & 31u)) >> 32);
}
static inline int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
// One lane: the warp is this lane. A position costs at most four decisions a round
// and an escape's 65 bits four a round, each round at most four votes: 32,768
// positions of 16 + 4 rounds take 2.6 million.
static uint64_t g_votes;
constexpr uint64_t kVotes = 4000000;
struct Endless {};
static inline bool __any_sync(uint32_t, bool v) {
    if (++g_votes > kVotes) throw Endless();
    return v;
}
static inline uint32_t __reduce_max_sync(uint32_t, uint32_t v) { return v; }
struct uint2 { uint32_t x, y; };
struct uint4 { uint32_t x, y, z, w; };
static inline uint4 make_uint4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) { return uint4{a, b, c, d}; }
static inline uint4 __ldg(const uint4 *p) { return *p; }

#include "rangecoder.cuh"

using namespace vcg;

static void band_table(uint32_t *bs) {   // first scan position of each significance band
    uint32_t cnt[94] = {0};
    for (int a = 0; a < 32; ++a)
        for (int b = 0; b < 32; ++b)
            for (int c = 0; c < 32; ++c) cnt[a + b + c]++;
    uint32_t pos = 0;
    int b = 0;
    bs[0] = 0;
    for (int f = 0; f < 94; ++f) {
        int bb = f * 8 / 96;
        if (bb > 7) bb = 7;
        while (b < bb) bs[++b] = pos;
        pos += cnt[f];
    }
    while (b < 8) bs[++b] = pos;
}

struct Result {
    bool ended;
    uint32_t bad;
    uint64_t outside;
    std::vector<uint32_t> ent;
};

template <int kZ>
static Result decode(const uint8_t *src, uint32_t len, size_t there, const uint32_t *bs) {
    const uint32_t cap = 32768;   // VCD_MAX_ENTRIES
    std::vector<uint32_t> dst(cap);
    uint32_t S[12];
    RcLane L;
    g_votes = g_outside = 0;
    g_lo = src;
    g_hi = src + there;
    bool ended = true;
    try {
        L.init(src, len, true, bs, S, 1, dst.data(), cap);
        while (__any_sync(0xFFFFFFFFu, L.c != kLaneDone)) L.template rounds<kZ>(bs);
    } catch (const Endless &) {
        ended = false;
    }
    Result r{ended, L.bad, g_outside, {}};
    for (uint32_t i = 0; i < L.n && i < cap; ++i)
        if (dst[i] >> 16) r.ent.push_back(dst[i]);   // (a raster has no entry for a crafted level 0)
    return r;
}

int main(int argc, char **argv) {
    if (argc < 2) return 2;
    FILE *f = fopen(argv[1], "rb");
    if (!f) return 2;
    const uint32_t more = argc > 2 ? (uint32_t)strtoul(argv[2], nullptr, 0) : 0u;
    const size_t pad = more ? 2u << 20 : 0u;
    uint32_t n = 0;
    if (fread(&n, 4, 1, f) != 1) return 2;
    uint32_t bs[10];   // the band table and a copy of its end, as the kernels hold it
    band_table(bs);
    bs[9] = bs[8];
    const char *names[2] = {"dense", "zeros"};
    int diff[2] = {0, 0}, endless[2] = {0, 0}, outside[2] = {0, 0};
    for (uint32_t k = 0; k < n; ++k) {
        uint32_t h[3];
        if (fread(h, 4, 3, f) != 3) return 2;
        const uint32_t len = h[0], bad = h[1], nent = h[2], mis = k & 3u;
        std::vector<uint8_t> in(len);
        if (len && fread(in.data(), 1, len, f) != len) return 2;
        std::vector<uint32_t> want(nent);
        if (nent && fread(want.data(), 4, nent, f) != nent) return 2;
        // whole words that hold a stream byte, and nothing after them
        const size_t words = (mis + len + pad + 3u) / 4u;
        uint32_t *buf = new uint32_t[words ? words : 1];
        memset(buf, 0xA5, 4 * (words ? words : 1));
        uint8_t *src = reinterpret_cast<uint8_t *>(buf) + mis;
        if (len) memcpy(src, in.data(), len);
        memset(src + len, 0, pad);
        const Result r[2] = {decode<0>(src, len + more, len + pad, bs), decode<6>(src, len + more, len + pad, bs)};
        for (int d = 0; d < 2; ++d) {
            endless[d] += !r[d].ended;
            outside[d] += r[d].outside != 0;
            const bool same = r[d].ended && (r[d].bad != 0) == (bad != 0) &&
                              (bad || (r[d].ent.size() == nent &&
                                       (!nent || memcmp(r[d].ent.data(), want.data(), 4ull * nent) == 0)));
            diff[d] += !same;
        }
        delete[] buf;
    }
    fclose(f);
    for (int d = 0; d < 2; ++d) printf("%s %d %d %d %u\n", names[d], diff[d], endless[d], outside[d], n);
    return 0;
}
