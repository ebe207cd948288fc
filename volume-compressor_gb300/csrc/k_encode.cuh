// Encode kernel interfaces (private).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "vc_internal.h"

namespace vcg {

constexpr uint64_t kL2Bytes = 32768ull * 16ull;   // one region's slot block
constexpr uint32_t kMetaZero = 1u << 31;           // meta: all-zero atom
constexpr uint32_t kMetaLong = 1u << 30;           // more coder bytes than a slot of sums holds (launch_rc_encode)
// meta = nnz (bits 0-15, up to 32768) | dc << 16 | kMetaLong | kMetaZero

// Canonical append order: LOD-major, atoms in raster (z, y, x) order.
struct Layout {
    int nlod;
    uint64_t base[9];
    uint32_t acx[8], acy[8], acz[8];

    __host__ __device__ void coords(uint64_t a, int &lod, uint32_t &az, uint32_t &ay, uint32_t &ax) const {
        lod = 0;
        while (lod + 1 < nlod && a >= base[lod + 1]) ++lod;
        uint64_t l = a - base[lod];
        ax = (uint32_t)(l % acx[lod]);
        ay = (uint32_t)((l / acx[lod]) % acy[lod]);
        az = (uint32_t)(l / ((uint64_t)acx[lod] * acy[lod]));
    }
    __host__ __device__ bool first_in_region(uint64_t a) const {
        int lod;
        uint32_t az, ay, ax;
        coords(a, lod, az, ay, ax);
        return ((az | ay | ax) & 31u) == 0;
    }
    __host__ __device__ uint64_t region_first(int lod, uint32_t az, uint32_t ay, uint32_t ax) const {
        return base[lod] + ((uint64_t)(az & ~31u) * acy[lod] + (ay & ~31u)) * acx[lod] + (ax & ~31u);
    }
};

// Forward pass over canonical atoms [first, first + n_atoms) of the pyramid
// (any mix of LODs).
struct FwdJob {
    Layout lay;
    const uint8_t *vol[8];       // LOD volumes (x fastest)
    uint32_t dims[8][3];         // nx, ny, nz per LOD
    uint64_t first;              // canonical index of this launch's first atom
    uint64_t n_atoms;
    const vcd_quant *q;          // per-LOD quantiser constants (device, [lod]); kept transforms: per set
    uint32_t sets;               // kept transforms: all n_atoms with q[0], then all with q[1], ...
    const uint8_t *qsel;         // optional: per atom (this launch) index into q instead of its LOD
    const uint32_t *place;       // scan position -> index in the transform's tile | quantiser class << 16 (EncTables)
    uint32_t *ent;               // per atom VCD_MAX_ENTRIES slots: scan position | level << 16
    uint32_t *meta;              // per atom
    // coefficient cache of canonical atoms [0, coef_n): 32768 packed words per
    // atom in scan order (coef_pack: magnitude, quantiser class, sign), and
    // dc | kMetaZero per atom; coef_store != 0 fills it, else atoms below
    // coef_n are quantised from it
    uint32_t *coef;
    uint32_t *coef_dc;
    uint64_t coef_n;
    int coef_store;
};

struct EncCosts;

// Coder pass over the lists of n_atoms atoms: lengths, and sums or totals.
struct RcJob {
    uint64_t n_atoms;
    uint32_t *meta;
    const uint32_t *ent;
    uint32_t band_start[9];
    uint32_t *len;                       // payload bytes per atom ([dc] + coder bytes; 0 = zero atom)
    uint32_t *sums;                      // kSums words per atom, what k_resolve makes the bytes of; null: lengths alone
    uint32_t *longs;                     // with sums: 1 + n_atoms words: how many atoms are kMetaLong (0 before), which
    // lengths alone
    const EncCosts *costs;
    uint32_t *doubt;                     // scratch, 1 + n_atoms words: how many atoms only the coder can size, which
    // both the lengths and the coder for those in doubt; the lengths alone, where
    // an atom in doubt may be a byte longer than its length says; the coder alone
    enum Pass { kExact, kNear, kDoubt } pass;
    unsigned long long *totals;          // bytes, atoms present and atoms in doubt are added here, for every set
    uint64_t per;                        // of `per` atoms its own three (sets of more than size_sets_atoms: one set)
};

// Payloads from the sums of a coder pass.
struct ResolveJob {
    uint64_t n_atoms;
    const uint32_t *meta;
    const uint32_t *ent;                 // the lists, for atoms coded from them
    uint32_t band_start[9];
    const uint32_t *len;
    const uint32_t *sums;                // null: code every atom from its list
    uint32_t *rest;                      // scratch, 1 + n_atoms words: how many atoms are coded from their lists, which
    uint8_t *arc;
    const uint64_t *dst_off;             // optional: per atom (this launch) payload offset in arc
    const uint64_t *pos;                 // else: canonical exclusive scan of consumed bytes
    uint64_t canon_first;                // canonical index of this chunk's first atom
    Layout lay;
};

struct PlaceJob {
    uint64_t n_total;
    uint64_t *pos;                       // in: consume; out after scan: cursor before each atom
    const uint32_t *len;
    const uint8_t *dc;
    uint8_t *arc;
    Layout lay;
};

void launch_fwd(const FwdJob &J, int num_sms, cudaStream_t s);
// atoms that are all LOD0 with kept coefficients: quantise and compact only
void launch_quant_cached(const FwdJob &J, int num_sms, cudaStream_t s);
void launch_rc_encode(const RcJob &J, int num_sms, cudaStream_t s);
// after launch_rc_encode with sums: the atoms that it has marked kMetaLong, their
// lengths, and their bytes in their slots (before J.longs is used again)
void launch_rc_long(const RcJob &J, int num_sms, cudaStream_t s);
struct EncTables;
void enc_tables(EncTables *t, const vcd_tables *vt);   // on the host
// atoms that a pass for lengths takes as sets, or at once four a CTA, at most
uint64_t size_sets_atoms(int num_sms);
// atoms that a coder pass runs as groups at most
uint64_t enc_group_atoms(int num_sms);
void launch_resolve(const ResolveJob &J, int num_sms, cudaStream_t s);
void launch_consume(const PlaceJob &J, cudaStream_t s);
void launch_slots(const PlaceJob &J, cudaStream_t s);
// *zero: a word set to 0
void launch_gather_dc(const uint32_t *meta, uint64_t n, uint8_t *dc, uint32_t *zero, cudaStream_t s);

}  // namespace vcg
