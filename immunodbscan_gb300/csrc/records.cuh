// records.cuh -- what the bucket and segment-join kernels share: bin numbering, the
// records of the distance kernels, and the size of the join table.
#pragma once
#include "idb_internal.cuh"

namespace idb {

namespace {

struct BinGeom {
    uint32_t Gv, Gj, NL, Lmin, VW, JW, K;
    __device__ __forceinline__ bool in_range(uint32_t L) const { return L >= Lmin && L - Lmin < NL; }
    // sub-bucket index: ((((r*Gv + v)*Gj + j)*NL + L-Lmin)*K + class
    __device__ __forceinline__ uint32_t bin(uint32_t r, uint32_t v, uint32_t j, uint32_t L,
                                            uint32_t c) const {
        return (((r * Gv + v) * Gj + j) * NL + (L - Lmin)) * K + c;
    }
};

// Record of one unique.
//  planes (fast path; Hamming and the diagonal edit-distance test): Bp bit planes x W words; bit i of word
//    p*W + i/32 is bit p of the code of residue i.  Hamming distance of two
//    records = sum over words of popc(OR_p (x_p ^ y_p)).
//  codes (other Levenshtein and the generic path): one code byte per residue.
// Codes are a bijection of the byte values present, so equality of codes is
// equality of bytes.

// Bit planes of one sequence (L <= 128): bit i of wd[p][w] is bit p of the
// code of residue 32w + i; positions past L keep code 0.  Residues are read 4
// at a time.
__device__ __forceinline__ void build_planes(const uint8_t *s, uint32_t L, const uint8_t *cm,
                                             uint32_t (&wd)[5][4]) {
#pragma unroll
    for (int p = 0; p < 5; ++p)
#pragma unroll
        for (int w = 0; w < 4; ++w) wd[p][w] = 0;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        if (32u * w >= L) break;
        uint32_t cw[8];
        load_chunk32(s, L, (uint32_t)w, cw);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t i0 = 32u * w + 4u * k;
            const uint32_t v = cw[k];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const uint32_t c = i0 + b < L ? (uint32_t)cm[(v >> (8 * b)) & 0xFFu] : 0u;
#pragma unroll
                for (int p = 0; p < 5; ++p) wd[p][w] |= ((c >> p) & 1u) << (4 * k + b);
            }
        }
    }
}

// Bit planes as a record of NR 16-byte words: word p*W + w.
template <int NR>
__device__ __forceinline__ void flatten_planes(const uint32_t (&wd)[5][4], int planes, uint32_t W,
                                               uint4 (&rec)[NR]) {
    uint32_t flat[4 * NR];
#pragma unroll
    for (int k = 0; k < 4 * NR; ++k) flat[k] = 0;
#pragma unroll
    for (int p = 0; p < 5; ++p)
#pragma unroll
        for (int w = 0; w < 4; ++w)
            if (p < planes && (uint32_t)w < W) {
                const uint32_t k = (uint32_t)p * W + w;
#pragma unroll
                for (int kk = 0; kk < 4 * NR; ++kk)
                    if ((uint32_t)kk == k) flat[kk] = wd[p][w];
            }
#pragma unroll
    for (int q = 0; q < NR; ++q)
        rec[q] = make_uint4(flat[4 * q], flat[4 * q + 1], flat[4 * q + 2], flat[4 * q + 3]);
}

// The record of one unique (fast paths: at most NR 16-byte words): bit planes, or
// code bytes (planes == 0).
template <int NR>
__device__ __forceinline__ void build_small_record(const uint8_t *s, uint32_t L,
                                                   const uint8_t *cm, int planes, uint32_t W,
                                                   uint4 (&rec)[NR]) {
    if (planes > 0) {
        uint32_t wd[5][4];
        build_planes(s, L, cm, wd);
        flatten_planes<NR>(wd, planes, W, rec);
    } else {
        GlobalReader rd(s, L);
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            uint32_t wv[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const uint32_t i0 = q * 16 + e * 4;
                const uint32_t v = i0 < L ? rd.next() : 0u;
                uint32_t acc = 0;
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const uint32_t c = i0 + t < L ? (uint32_t)cm[(v >> (8 * t)) & 0xFFu] : 0u;
                    acc |= c << (8 * t);
                }
                wv[e] = acc;
            }
            rec[q] = make_uint4(wv[0], wv[1], wv[2], wv[3]);
        }
    }
}

// Gene bitsets as the side records hold them.  Wide lists whose genes in use fit
// (64 V, 30 J): the genes no unique has are left out, order kept.
struct GeneSide {
    const uint64_t *bits;
    const unsigned long long *used;   // null: the first word as it is
    uint32_t W;
    __device__ __forceinline__ uint64_t row(uint32_t r) const {
        const uint64_t *b = bits + (size_t)r * W;
        if (!used) return b[0];
        uint64_t out = 0;
        uint32_t base = 0;
        for (uint32_t w = 0; w < W; ++w) {
            for (uint64_t v = b[w]; v; v &= v - 1) out |= 1ull << (base + rank_in(w, lowest_bit64(v)));
            base += (uint32_t)popc64(used[w]);
        }
        return out;
    }
    __device__ __forceinline__ uint32_t rank_in(uint32_t w, int bit) const {
        return (uint32_t)popc64(used[w] & ((1ull << bit) - 1ull));
    }
    // place of gene g in row()
    __device__ __forceinline__ uint32_t place(uint32_t g) const {
        if (!used) return g;
        uint32_t base = 0;
        for (uint32_t w = 0; w < g / 64; ++w) base += (uint32_t)popc64(used[w]);
        return base + rank_in(g / 64, (int)(g % 64));
    }
};

__device__ __forceinline__ uint32_t seg_count(const int16_t *eps_tab, uint32_t NL, uint32_t li) {
    const int e = eps_tab[(size_t)li * NL + li];
    return e < 0 ? 1u : (uint32_t)e + 1u;
}

// A replayed plan whose data has more entries or bin pairs than it was captured
// for: the fill kernels drop what does not fit, but bin pairs may still name
// entries past the capacity, and the true count runs past the bin pairs.  Called
// by each kernel that fills the bin pairs (none of them reads their count): no
// bin pair is left for the predictor, the schedule and the distance kernels, and
// the host is told.
__device__ __forceinline__ void drop_overgrown(Counters *ctr, uint64_t cap_bp, uint64_t cap_entries) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    const uint32_t over = (ctr->n_binpairs > cap_bp ? kErrBinPairOverflow : 0u) |
                          (ctr->n_entries > cap_entries ? kErrEntryOverflow : 0u);
    if (over) {
        atomicOr(&ctr->error, over);
        ctr->n_binpairs = 0;
    }
}

// Slots of the join table in use: about 1.5 slots per possible key (join_smax
// per unique), a power of two, at most the allocation.  The allocation is sized
// for every row being unique; the uniques are counted on the device, so the
// table a call probes (and clears) is the smaller one they need.
__device__ __forceinline__ uint32_t join_mask(uint32_t nu, uint32_t smax, uint64_t cap_mask) {
    const uint64_t want = max((3ull * smax * nu + 1) / 2, 1024ull);
    uint64_t c = 1024;
    while (c < want) c <<= 1;
    return (uint32_t)min(c - 1, cap_mask);
}

}  // namespace
}  // namespace idb
