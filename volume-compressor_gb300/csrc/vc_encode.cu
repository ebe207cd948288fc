// Whole-volume encode on the device: LOD pyramid, rate control, canonical
// placement and archive assembly (the composition vc_encode is defined as in
// include/vc.h). Host work is limited to the bisection decisions, the 128-byte
// header and the L1 hash table (a few entries per LOD).
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "k_ds.cuh"
#include "k_encode.cuh"
#include "kernels.cuh"
#include "rc_encode.cuh"
#include "vc_device.h"

using namespace vcg;

static const uint64_t kChunk = 32768;   // atoms per forward/coder launch (4 GiB of list scratch)

static const EncTables *enc_dev() { return (const EncTables *)g_dev.enc; }

static inline float f_of(uint32_t b) { float f; memcpy(&f, &b, 4); return f; }
static inline uint32_t b_of(float f) { uint32_t b; memcpy(&b, &f, 4); return b; }

#define CK(call, what)                                 \
    do {                                               \
        cudaError_t e_ = (call);                       \
        if (e_ != cudaSuccess) {                       \
            vcd_set_error(what, e_);                   \
            return vcd_status_of(e_);                  \
        }                                              \
    } while (0)

struct EncState {
    vcd_ctx *c;
    Layout lay;
    const uint8_t *lvol[8];
    uint32_t dims[8][3];
    uint32_t *ent, *meta, *len;          // lists and meta: LOD0's, or a chunk's
    uint32_t *ent2, *meta2;              // the coarser LODs', beside them (null: none)
    uint32_t *doubt, *doubt2;            // a size pass's scratch beside meta and meta2
    uint32_t *sums;                      // the coder's sums, kSums words an atom
    bool whole;                          // lists and sums of every atom are kept: one coder pass
    uint64_t *pos;
    uint8_t *dc, *arc;
    unsigned long long *red;             // a size pass's totals: bytes, atoms present, atoms in doubt
    RcJob::Pass size_pass;
    uint32_t sets;                       // quantisers a size pass takes at once, LOD0's lists of each after the other
    vcd_quant *qtab;          // device, per LOD
    vcd_quant qh;             // host staging
    // LOD0 forward transform kept across passes, packed (null when it does not fit)
    uint32_t *coef;
    uint32_t *coef_dc;
    uint64_t coef_n;
    bool coef_valid;
};

// Quantiser constants of `lod` at q, into the device table.
static void set_q(EncState &S, int lod, float q) {
    vch_quant_consts(q, &S.qh);
    cudaMemcpyAsync(S.qtab + lod, &S.qh, sizeof(vcd_quant), cudaMemcpyHostToDevice, S.c->stream);
}

enum EncPass { kSizes, kCode, kWrite };

// Forward + coder passes over canonical atoms [a0, a1) (any mix of LODs, each at
// the q in the device table) on stream st with list and metadata scratch ent,
// meta (kChunk atoms). kSizes: lengths into len and the totals. kCode: lengths,
// and the sums (of canonical atom a at slot a) for a resolve once the payloads'
// places are known. kWrite: sums, a chunk's at a time, and payloads into the
// archive. One launch pair per kChunk atoms: a coder launch costs about one
// atom's serial coding time however many atoms it holds.
static void resolve_range(EncState &S, uint64_t c0, uint64_t n, const uint32_t *ent, const uint32_t *meta,
                          const uint32_t *sums, cudaStream_t st) {
    ResolveJob W;
    memset(&W, 0, sizeof W);
    W.n_atoms = n;
    W.meta = meta;
    W.ent = ent;
    memcpy(W.band_start, g_dev.band_start, sizeof W.band_start);
    W.len = S.len + c0;
    W.sums = sums;
    W.rest = meta == S.meta ? S.doubt : S.doubt2;
    W.arc = S.arc;
    W.pos = S.pos;
    W.canon_first = c0;
    W.lay = S.lay;
    const bool prof = vcd_prof_on();
    if (prof) cudaEventRecord(S.c->ev[5], st);
    launch_resolve(W, g_dev.num_sms, st);
    if (prof) {
        cudaEventRecord(S.c->ev[1], st);
        cudaEventSynchronize(S.c->ev[1]);
        vcd_prof_add("encode_resolve", vcd_elapsed(S.c->ev[5], S.c->ev[1]), 2, 0, 0, n);
    }
}

// forward pass over canonical atoms [c0, c0 + n)
static void fwd_chunk(EncState &S, uint64_t c0, uint64_t n, cudaStream_t st, uint32_t *ent, uint32_t *meta,
                      uint32_t sets = 1) {
    FwdJob F;
    memset(&F, 0, sizeof F);   // fields this pass does not use stay null
    F.lay = S.lay;
    memcpy(F.vol, S.lvol, sizeof F.vol);
    memcpy(F.dims, S.dims, sizeof F.dims);
    F.first = c0;
    F.n_atoms = n;
    F.q = S.qtab;
    F.sets = sets;   // more than one only from kept transforms
    F.place = enc_dev()->place;
    F.ent = ent;
    F.meta = meta;
    F.coef = S.coef;
    F.coef_dc = S.coef_dc;
    F.coef_n = S.coef_n;
    F.coef_store = !S.coef_valid;
    const bool from_cache = S.coef && S.coef_valid && c0 + n <= S.coef_n;
    const bool prof = vcd_prof_on();
    if (prof) cudaEventRecord(S.c->ev[4], st);
    if (from_cache) launch_quant_cached(F, g_dev.num_sms, st);
    else launch_fwd(F, g_dev.num_sms, st);
    if (S.coef && c0 < S.coef_n && c0 + n >= S.coef_n) S.coef_valid = true;   // LOD0 transform kept
    if (prof) {
        cudaEventRecord(S.c->ev[5], st);
        cudaEventSynchronize(S.c->ev[5]);
        // forward: volume bytes in (the lists it writes are scratch, not counted)
        if (from_cache)   // coefficients in, lists out (scratch, not counted)
            vcd_prof_add("quant_cached", vcd_elapsed(S.c->ev[4], S.c->ev[5]), 1, n * sets * 131072ull, 0, n * sets);
        else
            vcd_prof_add("fwd_dct_quant", vcd_elapsed(S.c->ev[4], S.c->ev[5]), 1, n * 32768ull, 0, n);
    }
}

// coder pass over the lists of canonical atoms [c0, c0 + n); of the long ones too, with `longs`
static RcJob code_chunk(EncState &S, uint64_t c0, uint64_t n, EncPass pass, cudaStream_t st, uint32_t *ent,
                        uint32_t *meta, uint32_t *sums, bool longs = true) {
    RcJob R;
    memset(&R, 0, sizeof R);
    R.n_atoms = n;
    R.meta = meta;
    R.ent = ent;
    memcpy(R.band_start, g_dev.band_start, sizeof R.band_start);
    R.len = S.len + c0;
    if (pass == kSizes) {
        R.n_atoms = n * S.sets;
        R.per = n;
        R.costs = &enc_dev()->costs;
        R.doubt = meta == S.meta ? S.doubt : S.doubt2;
        R.pass = S.size_pass;
        R.totals = S.red;
    } else {
        // without room for sums the payloads are coded from the lists (kWrite)
        R.sums = pass == kCode ? sums + c0 * kSums : sums;
        R.longs = meta == S.meta ? S.doubt : S.doubt2;
        launch_gather_dc(meta, n, S.dc + c0, R.longs, st);
    }
    const bool prof = vcd_prof_on();
    if (prof) cudaEventRecord(S.c->ev[5], st);
    if (pass == kSizes || R.sums) launch_rc_encode(R, g_dev.num_sms, st);
    if (longs && R.sums) launch_rc_long(R, g_dev.num_sms, st);
    if (prof) {
        cudaEventRecord(S.c->ev[1], st);
        cudaEventSynchronize(S.c->ev[1]);
        vcd_prof_add(pass == kSizes ? "rc_encode_size" : "rc_encode_write", vcd_elapsed(S.c->ev[5], S.c->ev[1]), 1, 0,
                     0, n);
    }
    if (pass == kWrite) resolve_range(S, c0, n, ent, meta, R.sums, st);
    return R;
}

static void run_range(EncState &S, uint64_t a0, uint64_t a1, EncPass pass, cudaStream_t st, uint32_t *ent,
                      uint32_t *meta, uint32_t *sums = nullptr) {
    for (uint64_t c0 = a0; c0 < a1; c0 += kChunk) {
        const uint64_t n = a1 - c0 < kChunk ? a1 - c0 : kChunk;
        fwd_chunk(S, c0, n, st, ent, meta);
        code_chunk(S, c0, n, pass, st, ent, meta, sums);
    }
}

// The same over all atoms: LOD0 on the context's stream and the coarser LODs
// beside it on the second stream, with their own list scratch. The coarser LODs
// are few atoms but the finest-quantised ones (q down to 0.05): one of them is a
// serial coder chain longer than a whole LOD0 pass, so run after LOD0 it would
// add its length. Where each range is one chunk and LOD0 more than the coder's
// groups hold, both coders fill the GPU and only get in each other's way (one
// after the other 13.9 ms at 1024^3, side by side 12 to 25). Serial under
// per-stage measurement (its events are per stream).
static void run_split(EncState &S, uint64_t na0, uint64_t total, uint64_t chunk, EncPass pass) {
    vcd_ctx *c = S.c;
    // chunks of a kWrite have their own sums on each stream
    uint32_t *sums2 = pass == kWrite && S.sums ? S.sums + chunk * kSums : S.sums;
    if (!S.ent2) {
        run_range(S, 0, total, pass, c->stream, S.ent, S.meta, S.sums);
        return;
    }
    const bool first = total - na0 <= kChunk && na0 <= kChunk;
    const bool alone = first && na0 > enc_group_atoms(g_dev.num_sms);
    cudaStream_t side = vcd_prof_on() ? NULL : vcd_side_stream(c), st1 = side && !alone ? side : c->stream;
    auto fork = [&]() {   // the side stream goes on after the work queued so far
        if (!side) return;
        cudaEventRecord(c->chunk_ev[0], c->stream);
        cudaStreamWaitEvent(side, c->chunk_ev[0], 0);
    };
    // A forward CTA takes nearly all shared memory of an SM, so beside a coder it
    // waits for the coder's CTAs: where one chunk holds each range, both forward
    // passes go first and only the coders run side by side.
    if (first) {
        fwd_chunk(S, na0, total - na0, c->stream, S.ent2, S.meta2);
        fwd_chunk(S, 0, na0, c->stream, S.ent, S.meta);
    }
    if (!alone) fork();
    if (first) {
        const bool late = pass == kCode && alone;   // the long atoms of both then go side by side, after the coders
        const RcJob R1 = code_chunk(S, na0, total - na0, pass, st1, S.ent2, S.meta2, sums2, !late);
        const RcJob R0 = code_chunk(S, 0, na0, pass, c->stream, S.ent, S.meta, S.sums, !late);
        if (late) {
            fork();
            launch_rc_long(R1, g_dev.num_sms, side ? side : c->stream);
            launch_rc_long(R0, g_dev.num_sms, c->stream);
        }
    } else {
        run_range(S, na0, total, pass, st1, S.ent2, S.meta2, sums2);
        run_range(S, 0, na0, pass, c->stream, S.ent, S.meta, S.sums);
    }
    if (side) {
        cudaEventRecord(c->chunk_ev[1], side);
        cudaStreamWaitEvent(c->stream, c->chunk_ev[1], 0);
    }
}

extern "C" int vcd_encode(const uint8_t *vol, int on_dev, vcd_encode_info *info, uint8_t **out, size_t *out_len) {
    vcd_ctx *c = vcd_thread_ctx();
    if (!c) return 4;
    cudaStream_t st = c->stream;
    EncState S;
    memset(&S, 0, sizeof S);
    S.c = c;
    const int nlod = info->nlod;
    S.lay.nlod = nlod;
    uint64_t nvox[8], pyr_bytes = 0, pyr_vox = 0, total_atoms = 0;
    uint32_t d[3] = {info->nx, info->ny, info->nz};
    for (int l = 0; l < nlod; ++l) {
        if (l) for (int k = 0; k < 3; ++k) d[k] = (d[k] + 1) / 2;
        memcpy(S.dims[l], d, sizeof d);
        nvox[l] = (uint64_t)d[0] * d[1] * d[2];
        if (l) pyr_bytes += (nvox[l] + 255) & ~255ull, pyr_vox += nvox[l];
        S.lay.acx[l] = (d[0] + 31) / 32; S.lay.acy[l] = (d[1] + 31) / 32; S.lay.acz[l] = (d[2] + 31) / 32;
        S.lay.base[l] = total_atoms;
        total_atoms += (uint64_t)S.lay.acx[l] * S.lay.acy[l] * S.lay.acz[l];
    }
    S.lay.base[nlod] = total_atoms;
    for (int l = nlod + 1; l <= 8; ++l) S.lay.base[l] = total_atoms;

    // ---- buffers
    void *p;
    if (on_dev) {
        S.lvol[0] = vol;
    } else {
        CK(vcd_scratch(c, VCD_BUF_VOL, nvox[0], &p), "encode volume");
        CK(vcd_copy_from_host(c, p, vol, nvox[0]), "volume upload");
        S.lvol[0] = (const uint8_t *)p;
    }
    CK(vcd_scratch(c, VCD_BUF_PYR, pyr_bytes + 16, &p), "pyramid");
    cudaEventRecord(c->ev[6], st);   // device work starts (input already on the device)
    const bool prof = vcd_prof_on();
    {
        uint8_t *q = (uint8_t *)p;
        for (int l = 1; l < nlod; ++l) {
            launch_ds2x(S.lvol[l - 1], S.dims[l - 1][0], S.dims[l - 1][1], S.dims[l - 1][2], q, info->ds_method,
                        info->ds_alpha, g_dev.num_sms, st);
            S.lvol[l] = q;
            q += (nvox[l] + 255) & ~255ull;   // 256-byte aligned levels (vector loads)
        }
    }
    if (prof && nlod > 1) {   // pyramid: every coarser voxel reads its (up to) 8 children
        cudaEventRecord(c->ev[5], st);
        cudaEventSynchronize(c->ev[5]);
        vcd_prof_add("downsample", vcd_elapsed(c->ev[6], c->ev[5]), (uint64_t)(nlod - 1), nvox[0] + pyr_vox - nvox[nlod - 1],
                     pyr_vox, pyr_vox);
    }
    const uint64_t na0 = S.lay.base[1];
    const uint64_t chunk = total_atoms < kChunk ? total_atoms : kChunk;
    // a rate control of few atoms takes three quantisers at once
    bool three = !info->fixed_q && 3 * na0 <= size_sets_atoms(g_dev.num_sms);
    uint64_t lists = three && 3 * na0 > chunk ? 3 * na0 : chunk;
    S.sets = 1;
    if (lists > chunk && vcd_scratch(c, VCD_BUF_EENT, lists * VCD_MAX_ENTRIES * 4 + 16, &p) != cudaSuccess) {
        three = false;   // no room: one at a time
        lists = chunk;
    }
    CK(vcd_scratch(c, VCD_BUF_EENT, lists * VCD_MAX_ENTRIES * 4 + 16, &p), "coefficient lists");
    S.ent = (uint32_t *)p;
    // quant table (8 LODs) | meta (lists) | doubt (1 + lists) | len (all atoms or lists) | dc (all atoms)
    size_t q_b = 8 * sizeof(vcd_quant), meta_b = lists * 4, doubt_b = (lists + 1) * 4, n_len = total_atoms > lists ? total_atoms : lists,
           len_b = n_len * 4;
    size_t dc_b = total_atoms + 16;
    CK(vcd_scratch(c, VCD_BUF_EMETA, q_b + meta_b + doubt_b + len_b + dc_b + 64, &p), "encode metadata");
    S.qtab = (vcd_quant *)p;
    S.meta = (uint32_t *)((uint8_t *)p + q_b);
    S.doubt = S.meta + lists;
    S.len = S.doubt + lists + 1;
    S.dc = (uint8_t *)(S.len + n_len);
    CK(vcd_scratch(c, VCD_BUF_POS, (total_atoms + 1) * 8, &p), "placement");
    S.pos = (uint64_t *)p;
    CK(vcd_scratch(c, VCD_BUF_RED, 128, &p), "totals");
    S.red = (unsigned long long *)p;
    // keep LOD0's forward transform (128 KiB per atom) for the passes after the first when it takes at most half the
    // free memory
    auto keep_coef = [&]() {
        size_t fr = 0, tot = 0;
        const size_t cb = (size_t)na0 * 131072 + (size_t)na0 * 4 + 64;
        if (cudaMemGetInfo(&fr, &tot) == cudaSuccess && (c->cap[VCD_BUF_COEF] >= cb || cb <= fr / 2) &&
            vcd_scratch(c, VCD_BUF_COEF, cb, &p) == cudaSuccess) {
            S.coef = (uint32_t *)p;
            S.coef_dc = (uint32_t *)((uint8_t *)p + (size_t)na0 * 131072);
            S.coef_n = na0;
        }
        cudaGetLastError();
    };
    if (!info->fixed_q) keep_coef();
    {   // One coder pass for all where the lists and sums of every atom have room (256 KiB an atom, the sums
        // in at most half the free memory): else one for the sizes and one, a chunk at a time, for the bytes.
        size_t fr = 0, tot = 0;
        const uint64_t n1 = total_atoms - na0, n1c = n1 < kChunk ? n1 : kChunk;
        const size_t all_b = (size_t)total_atoms * kSums * 4;
        void *pe = NULL, *pm = NULL;
        if (n1 && vcd_scratch(c, VCD_BUF_EENT2, n1c * VCD_MAX_ENTRIES * 4 + 16, &pe) == cudaSuccess &&
            vcd_scratch(c, VCD_BUF_EMETA2, n1c * 8 + 16, &pm) == cudaSuccess) {
            S.ent2 = (uint32_t *)pe;
            S.meta2 = (uint32_t *)pm;
            S.doubt2 = S.meta2 + n1c;
        }
        if (na0 <= kChunk && n1 <= kChunk && (S.ent2 || !n1) && cudaMemGetInfo(&fr, &tot) == cudaSuccess &&
            (c->cap[VCD_BUF_ESUM] >= all_b || all_b <= fr / 2) &&
            vcd_scratch(c, VCD_BUF_ESUM, all_b, &p) == cudaSuccess) {
            S.whole = true;
            S.sums = (uint32_t *)p;
        } else if (vcd_scratch(c, VCD_BUF_ESUM, (size_t)(chunk + (S.ent2 ? n1c : 0)) * kSums * 4, &p) == cudaSuccess) {
            S.sums = (uint32_t *)p;
        }
        cudaGetLastError();
    }
    if (info->fixed_q && !S.whole) keep_coef();   // one pass keeps nothing

    // ---- rate control on LOD0 (bisection over float bit patterns of [0.05, 4096]):
    // the q visited whose ratio is nearest the target, the larger of two as near.
    // A pass that leaves d atoms in doubt knows its bytes up to d. Those atoms are
    // coded where that decides the next step or is likely to decide the best, or
    // after the last step for a q that may still be the nearest.
    struct Visit { float q; unsigned long long bytes, present, doubt; } v[24];
    const double target = (double)info->target_ratio;
    auto measure = [&](Visit *m, uint32_t sets, RcJob::Pass pass) -> cudaError_t {
        cudaError_t e = cudaSuccess;
        S.size_pass = pass;
        S.sets = sets;
        if (pass != RcJob::kDoubt && (e = cudaMemsetAsync(S.red, 0, 24 * sets, st)) != cudaSuccess) return e;
        if (pass != RcJob::kDoubt)
            for (uint32_t k = 0; k < sets; ++k) set_q(S, (int)k, m[k].q);
        if (pass == RcJob::kDoubt || sets > 1) {
            if (pass != RcJob::kDoubt) fwd_chunk(S, 0, na0, st, S.ent, S.meta, sets);   // else the lists are at hand
            code_chunk(S, 0, na0, kSizes, st, S.ent, S.meta, nullptr);
        } else {
            run_range(S, 0, na0, kSizes, st, S.ent, S.meta);
        }
        S.sets = 1;
        unsigned long long h[9];
        if ((e = cudaMemcpyAsync(h, S.red, 24 * sets, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
        if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
        for (uint32_t k = 0; k < sets; ++k) {
            m[k].bytes = h[3 * k];
            m[k].present = h[3 * k + 1];
            m[k].doubt = pass == RcJob::kNear ? h[3 * k + 2] : 0;
        }
        return cudaSuccess;
    };
    auto ratio = [](const Visit &m, unsigned long long more) {
        return (double)(32768ull * m.present) / (double)(m.bytes + more);
    };
    uint32_t lo = b_of(0.05f), hi = b_of(4096.0f);
    float best_q = 1.0f;
    double best_err = INFINITY;
    uint64_t present = 0, best_bytes = 0;
    int nv = 0;
    const int steps = info->fixed_q ? 0 : 24;
    while (nv < steps) {
        // Once the transform is kept, a step of few atoms takes as long with three
        // quantisers as with one: its own and both that the next step may come to
        // (540 atoms: 0.26 and 0.25 ms). Not in the first steps, where one of those
        // is a much finer one than either step needs.
        const uint32_t mid = lo + (hi - lo) / 2;
        const uint32_t sets = three && S.coef_valid && nv >= 3 && nv + 1 < steps ? 3 : 1;
        Visit m[3];
        m[0].q = f_of(mid);
        m[1].q = f_of(mid + (hi - mid) / 2);   // after lo = mid
        m[2].q = f_of(lo + (mid - lo) / 2);    // after hi = mid
        CK(measure(m, sets, RcJob::kNear), "rate control pass");
        present = m[0].present;
        if (present == 0) break;
        for (uint32_t k = 0, end = 0; !end;) {
            // the doubt of a pass this near is likely to matter, and its lists are at hand
            const double want = (double)(32768ull * m[k].present) / target;
            if (m[k].doubt && ((ratio(m[k], m[k].doubt) < target) != (ratio(m[k], 0) < target) ||
                               fabs((double)m[k].bytes - want) <= 4.0 * (double)m[k].doubt))
                CK(measure(m, sets, na0 <= kChunk ? RcJob::kDoubt : RcJob::kExact), "rate control pass");
            const uint32_t at = b_of(m[k].q);
            const bool below = ratio(m[k], 0) < target;
            if (below) lo = at; else hi = at;
            v[nv++] = m[k];
            end = k || sets == 1;
            k = below ? 1 : 2;
        }
    }
    auto consider = [&](const Visit &m) {
        const double err = fabs(ratio(m, 0) - target);
        if (err < best_err || (err == best_err && m.q > best_q)) {
            best_err = err;
            best_q = m.q;
            best_bytes = m.bytes;
        }
    };
    for (int i = 0; i < nv; ++i)
        if (!v[i].doubt) consider(v[i]);
    for (;;) {   // the nearest that one in doubt can be, until none can be nearer than the best
        int near = -1;
        double near_err = best_err;
        for (int i = 0; i < nv; ++i) {
            const double e = v[i].doubt ? fmin(fabs(ratio(v[i], 0) - target), fabs(ratio(v[i], v[i].doubt) - target))
                                        : INFINITY;
            if (v[i].doubt && e <= near_err) near = i, near_err = e;
        }
        if (near < 0) break;
        CK(measure(&v[near], 1, RcJob::kExact), "rate control pass");
        consider(v[near]);
    }
    S.size_pass = RcJob::kExact;
    info->q0 = best_q;
    info->present0 = present;
    info->bytes0 = best_bytes;
    float qs[8];
    if (info->fixed_q) {
        for (int l = 0; l < nlod; ++l) qs[l] = vch_clamp_q(info->q[l]);
        info->q0 = qs[0];
    } else {
        float q = best_q;
        for (int l = 0; l < nlod; ++l) { qs[l] = vch_clamp_q(q < 0.05f ? 0.05f : q); q = q * 0.6f; }
    }

    // ---- every atom at its LOD's q: coded, or its size (LODs 1.. together in one pass)
    for (int l = 0; l < nlod; ++l) set_q(S, l, qs[l]);
    if (S.whole) {
        run_split(S, na0, total_atoms, chunk, kCode);
    } else {
        CK(cudaMemsetAsync(S.red, 0, 24, st), "totals reset");
        run_split(S, na0, total_atoms, chunk, kSizes);
    }

    // ---- canonical placement: exclusive scan of consumed bytes
    const uint64_t head = 128 + 16 * info->l1_cap;
    PlaceJob P;
    memset(&P, 0, sizeof P);
    P.n_total = total_atoms;
    P.pos = S.pos;
    P.len = S.len;
    P.dc = S.dc;
    P.lay = S.lay;
    if (prof) cudaEventRecord(c->ev[4], st);
    launch_consume(P, st);
    launch_scan_u64(S.pos, total_atoms, head, S.pos + total_atoms, st);
    if (prof) {   // lengths in, consumed bytes out, scanned in place
        cudaEventRecord(c->ev[5], st);
        cudaEventSynchronize(c->ev[5]);
        vcd_prof_add("encode_place", vcd_elapsed(c->ev[4], c->ev[5]), 2, total_atoms * 12, total_atoms * 16, total_atoms);
    }
    uint64_t *pos_h = (uint64_t *)malloc((total_atoms + 1) * 8);
    if (!pos_h) return 3;
    cudaError_t e = cudaMemcpyAsync(pos_h, S.pos, (total_atoms + 1) * 8, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { free(pos_h); vcd_set_error("placement", e); return vcd_status_of(e); }
    const uint64_t total = pos_h[total_atoms];

    // ---- archive: zeroed, payloads + slots on the device, head on the host
    e = vcd_scratch(c, VCD_BUF_ARC, total + 16, &p);
    // no room: what is held for speed alone goes first, the kept transform, then the
    // sums, the coarser LODs' lists and those of more than a chunk (the payloads are
    // then coded from lists made anew, a chunk at a time)
    auto give_back = [&](int slot) {
        cudaStreamSynchronize(st);
        cudaFree(c->buf[slot]);
        c->buf[slot] = NULL;
        c->cap[slot] = 0;
    };
    if (e == cudaErrorMemoryAllocation && S.coef) {
        give_back(VCD_BUF_COEF);
        S.coef = S.coef_dc = NULL;
        S.coef_n = 0;
        S.coef_valid = false;
        e = vcd_scratch(c, VCD_BUF_ARC, total + 16, &p);
    }
    if (e == cudaErrorMemoryAllocation && (S.sums || S.ent2 || lists > chunk)) {
        for (int slot : {(int)VCD_BUF_ESUM, (int)VCD_BUF_EENT2, (int)VCD_BUF_EMETA2}) give_back(slot);
        S.sums = S.ent2 = S.meta2 = S.doubt2 = NULL;
        S.whole = false;
        if (lists > chunk) give_back(VCD_BUF_EENT);
        e = vcd_scratch(c, VCD_BUF_ARC, total + 16, &p);
        void *pe = S.ent;
        if (e == cudaSuccess) e = vcd_scratch(c, VCD_BUF_EENT, chunk * VCD_MAX_ENTRIES * 4 + 16, &pe);
        S.ent = (uint32_t *)pe;
    }
    if (e != cudaSuccess) { free(pos_h); vcd_set_error("archive buffer", e); return vcd_status_of(e); }
    S.arc = (uint8_t *)p;
    P.arc = S.arc;
    cudaMemsetAsync(S.arc, 0, total, st);
    if (S.whole) {
        // (side by side: each may hold atoms past their slots, coded from their lists,
        // whose time is one atom's chain)
        cudaStream_t side = S.ent2 && !prof ? vcd_side_stream(c) : NULL;
        if (side) {
            cudaEventRecord(c->chunk_ev[0], st);
            cudaStreamWaitEvent(side, c->chunk_ev[0], 0);
        }
        if (S.ent2) resolve_range(S, na0, total_atoms - na0, S.ent2, S.meta2, S.sums + na0 * kSums, side ? side : st);
        resolve_range(S, 0, na0, S.ent, S.meta, S.sums, st);
        if (side) {
            cudaEventRecord(c->chunk_ev[1], side);
            cudaStreamWaitEvent(st, c->chunk_ev[1], 0);
        }
    } else {
        run_split(S, na0, total_atoms, chunk, kWrite);
    }
    if (prof) cudaEventRecord(c->ev[4], st);
    launch_slots(P, st);
    if (prof) {   // one 16-byte slot per atom
        cudaEventRecord(c->ev[5], st);
        cudaEventSynchronize(c->ev[5]);
        vcd_prof_add("encode_slots", vcd_elapsed(c->ev[4], c->ev[5]), 1, total_atoms * 21, total_atoms * 16, total_atoms);
    }
    cudaEventRecord(c->ev[7], st);   // device work ends (the archive head and copy-out follow)

    uint8_t *hd = (uint8_t *)calloc(head, 1);
    if (!hd) { free(pos_h); return 3; }
    uint32_t w32[9] = {0x00314356u, 1u, 32u, 1u, 32u, (uint32_t)nlod, info->nx, info->ny, info->nz};
    memcpy(hd, w32, sizeof w32);
    memcpy(hd + 36, &info->target_ratio, 4);
    uint64_t regions = 0;
    const uint64_t mask = info->l1_cap - 1;
    for (int l = 0; l < nlod; ++l) {   // regions in creation order (raster of regions)
        uint32_t nrx = (S.lay.acx[l] + 31) / 32, nry = (S.lay.acy[l] + 31) / 32, nrz = (S.lay.acz[l] + 31) / 32;
        for (uint32_t rz = 0; rz < nrz; ++rz)
            for (uint32_t ry = 0; ry < nry; ++ry)
                for (uint32_t rx = 0; rx < nrx; ++rx) {
                    uint64_t key = vch_region_key(l, rz, ry, rx);
                    uint64_t blk = pos_h[S.lay.region_first(l, rz * 32, ry * 32, rx * 32)];
                    uint64_t i = vch_mix64(key) & mask;
                    while (1) {
                        uint64_t bref;
                        memcpy(&bref, hd + 128 + i * 16 + 8, 8);
                        if (!bref) break;
                        i = (i + 1) & mask;
                    }
                    memcpy(hd + 128 + i * 16, &key, 8);
                    memcpy(hd + 128 + i * 16 + 8, &blk, 8);
                    ++regions;
                }
    }
    uint64_t h64[4] = {info->l1_cap, regions, 128, total};
    memcpy(hd + 40, h64, sizeof h64);
    for (int l = 0; l < nlod; ++l) memcpy(hd + 72 + 4 * l, &qs[l], 4);
    free(pos_h);
    e = cudaMemcpyAsync(S.arc, hd, head, cudaMemcpyHostToDevice, st);
    uint8_t *res = (uint8_t *)malloc(total);
    if (!res) { cudaStreamSynchronize(st); free(hd); return 3; }
    if (e == cudaSuccess) e = vcd_copy_to_host(c, res, S.arc, total);   // after the head on the same stream
    if (e == cudaSuccess) e = cudaGetLastError();
    free(hd);
    if (e != cudaSuccess) { free(res); vcd_set_error("archive assembly", e); return vcd_status_of(e); }
    c->last_ms = vcd_elapsed(c->ev[6], c->ev[7]);
    // a large transform cache or sums are not kept between encodes (more than 1/8 of the device memory)
    for (int b : {(int)VCD_BUF_COEF, (int)VCD_BUF_ESUM}) {
        size_t fr = 0, tot = 0;
        if (c->buf[b] && cudaMemGetInfo(&fr, &tot) == cudaSuccess && c->cap[b] > tot / 8) {
            cudaFree(c->buf[b]);
            c->buf[b] = NULL;
            c->cap[b] = 0;
        }
        cudaGetLastError();
    }
    *out = res;
    *out_len = total;
    return 0;
}

// ---------------------------------------------------------------- writer batches
// Independent atoms (box rasters or stacked single atoms) through the same
// forward and coder kernels as the whole-volume encoder, with one coder pass:
// per chunk of at most kWChunk atoms a forward pass and a coder pass, the lengths
// back to the host for the packing offsets, and a resolve into the packed buffer,
// which is copied into the thread's pinned buffer.
static const uint64_t kWChunk = 8192;

extern "C" int vcd_encode_segments(const vcd_seg *segs, int nseg, const float *qs, int nq, uint8_t **pay,
                                   uint64_t *pay_bytes) {
    vcd_ctx *c = vcd_thread_ctx();
    if (!c) return 4;
    if (nq < 1 || nq > 256) return 2;
    cudaStream_t st = c->stream;
    void *p;
    const size_t q_b = ((size_t)nq * sizeof(vcd_quant) + 255) & ~(size_t)255;
    CK(vcd_scratch(c, VCD_BUF_EMETA, q_b + kWChunk * (4 + 4 + 8 + 1 + 4) + 256, &p), "writer metadata");
    vcd_quant *qtab = (vcd_quant *)p;
    uint32_t *dmeta = (uint32_t *)((uint8_t *)p + q_b);
    uint32_t *dlen = dmeta + kWChunk;
    uint64_t *doff = (uint64_t *)(dlen + kWChunk);
    uint32_t *drest = (uint32_t *)(doff + kWChunk);   // 1 + kWChunk
    uint8_t *dqsel = (uint8_t *)(drest + 1 + kWChunk);
    vcd_quant *qh = (vcd_quant *)malloc((size_t)nq * sizeof(vcd_quant));
    uint64_t *offh = (uint64_t *)malloc(kWChunk * sizeof(uint64_t));
    if (!qh || !offh) { free(qh); free(offh); return 3; }
    for (int i = 0; i < nq; ++i) vch_quant_consts(qs[i], &qh[i]);
    cudaError_t e = cudaEventRecord(c->ev[6], st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(qtab, qh, (size_t)nq * sizeof(vcd_quant), cudaMemcpyHostToDevice, st);
    uint64_t total = 0;
    for (int sg = 0; sg < nseg && e == cudaSuccess; ++sg) {
        const vcd_seg &S = segs[sg];
        const uint64_t acx = S.nx / 32, acy = S.ny / 32, acz = S.nz / 32, na = acx * acy * acz;
        if (!na) continue;
        if ((e = vcd_scratch(c, VCD_BUF_VOL, (size_t)S.nx * S.ny * S.nz + 16, &p)) != cudaSuccess) break;
        const uint8_t *dvol = (const uint8_t *)p;
        if ((e = vcd_copy_from_host(c, p, S.vox, (size_t)S.nx * S.ny * S.nz)) != cudaSuccess) break;
        Layout lay;
        memset(&lay, 0, sizeof lay);
        lay.nlod = 1;
        for (int l = 1; l <= 8; ++l) lay.base[l] = na;
        lay.acx[0] = (uint32_t)acx; lay.acy[0] = (uint32_t)acy; lay.acz[0] = (uint32_t)acz;
        for (uint64_t c0 = 0; c0 < na && e == cudaSuccess; c0 += kWChunk) {
            const uint64_t n = na - c0 < kWChunk ? na - c0 : kWChunk;
            if ((e = vcd_scratch(c, VCD_BUF_EENT, n * VCD_MAX_ENTRIES * 4 + 16, &p)) != cudaSuccess) break;
            uint32_t *ent = (uint32_t *)p;
            if ((e = cudaMemcpyAsync(dqsel, S.qsel + c0, n, cudaMemcpyHostToDevice, st)) != cudaSuccess) break;
            FwdJob F;
            memset(&F, 0, sizeof F);
            F.lay = lay;
            F.vol[0] = dvol;
            F.dims[0][0] = S.nx; F.dims[0][1] = S.ny; F.dims[0][2] = S.nz;
            F.first = c0;
            F.n_atoms = n;
            F.q = qtab;
            F.qsel = dqsel;
            F.place = enc_dev()->place;
            F.ent = ent;
            F.meta = dmeta;
            launch_fwd(F, g_dev.num_sms, st);
            if ((e = vcd_scratch(c, VCD_BUF_ESUM, n * kSums * 4, &p)) != cudaSuccess) break;
            RcJob R;
            memset(&R, 0, sizeof R);
            R.n_atoms = n;
            R.meta = dmeta;
            R.ent = ent;
            memcpy(R.band_start, g_dev.band_start, sizeof R.band_start);
            R.len = dlen;
            R.sums = (uint32_t *)p;
            R.longs = drest;
            if ((e = cudaMemsetAsync(drest, 0, 4, st)) != cudaSuccess) break;
            launch_rc_encode(R, g_dev.num_sms, st);
            launch_rc_long(R, g_dev.num_sms, st);
            if ((e = cudaMemcpyAsync(S.len + c0, dlen, n * 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
                (e = cudaStreamSynchronize(st)) != cudaSuccess)
                break;
            uint64_t bytes = 0;
            for (uint64_t i = 0; i < n; ++i) {
                offh[i] = bytes;
                S.off[c0 + i] = total + bytes;
                bytes += S.len[c0 + i];
            }
            if ((e = vcd_scratch(c, VCD_BUF_WPACK, bytes + 16, &p)) != cudaSuccess) break;
            uint8_t *dpack = (uint8_t *)p;
            if ((e = cudaMemcpyAsync(doff, offh, n * 8, cudaMemcpyHostToDevice, st)) != cudaSuccess) break;
            ResolveJob W;
            memset(&W, 0, sizeof W);
            W.n_atoms = n;
            W.meta = dmeta;
            W.ent = ent;
            memcpy(W.band_start, R.band_start, sizeof W.band_start);
            W.len = dlen;
            W.sums = R.sums;
            W.arc = dpack;
            W.dst_off = doff;
            W.rest = drest;
            launch_resolve(W, g_dev.num_sms, st);
            if (total + bytes > c->wpin_cap) {   // grow the pinned output, keeping what it holds
                if ((e = cudaStreamSynchronize(st)) != cudaSuccess) break;
                size_t want = (total + bytes) + (total + bytes) / 2 + (1 << 20);
                uint8_t *np_ = NULL;
                if ((e = vcd_malloc_host((void **)&np_, want)) != cudaSuccess) break;
                if (c->wpin) {
                    memcpy(np_, c->wpin, total);
                    cudaFreeHost(c->wpin);
                }
                c->wpin = np_;
                c->wpin_cap = want;
            }
            if (bytes && (e = cudaMemcpyAsync(c->wpin + total, dpack, bytes, cudaMemcpyDeviceToHost, st)) != cudaSuccess)
                break;
            // offh and the staging are reused by the next chunk
            if ((e = cudaStreamSynchronize(st)) != cudaSuccess) break;
            total += bytes;
        }
    }
    if (e == cudaSuccess) e = cudaEventRecord(c->ev[7], st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    free(qh);
    free(offh);
    if (e != cudaSuccess) {
        vcd_set_error("writer batch", e);
        return vcd_status_of(e);
    }
    c->last_ms = vcd_elapsed(c->ev[6], c->ev[7]);
    *pay = c->wpin;
    *pay_bytes = total;
    return 0;
}
