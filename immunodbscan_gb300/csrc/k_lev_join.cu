// k_lev_join.cu -- candidate pairs of the edit-distance search by segment join.
//
// The buckets (k_buckets.cu) score every pair of a (repertoire, V, J) whose
// lengths are close: on a deep repertoire only one scored pair in a hundred to a
// thousand is a neighbour.  Here a pair is scored only if it shares a segment.
// Let n be the longer length, S = eps(n) + 1, and y (length n) cut into S
// segments [k n/S, (k+1) n/S).  If x (length m = n - g) is within e = eps(n)
// edits of y, take an alignment and the first segment k such that the segments
// up to and including k hold at most k edits in total: the segments before k
// hold exactly k, so segment k is untouched, x holds it shifted by delta with
// |delta| <= k (the edits to its left) and |delta + g| <= e - k (the edits to
// its right).  (The multi-match-aware substring selection of G. Li, D. Deng,
// J. Wang, J. Feng, "Pass-Join: a partition-based method for similarity
// joins", PVLDB 5(3), 2011, derived here for the longer string cut.)
//
// Every unique is indexed under its S segments (key: repertoire, n, k, a hash of
// the segment's codes) and looks up, for every length n it may pair with, the
// substrings at the shifts above.  A key's group holds the uniques indexed
// under it (class 0) and those that looked it up: class 1 from the same length
// with a shift, class 1 + g from a length g shorter.  The group's bin pairs are
// class 0 against itself and every other class against class 0.  For two
// uniques of one length the one with the larger id counts as the one cut.  A
// pair is emitted from its first (k, delta) only (lev_join_ok, lev_diag.cuh).
//
// Bound by the latency of random look-ups (one 32-byte sector each): the table
// of a million uniques stays in L2.  Whole calls, buckets against join with the
// same pair test: 1M rows with skewed gene usage, eps 2: 38.9e9 pairs 41.2 ms,
// 0.17e9 pairs 3.4 ms; 2M rows, eps min(3, 0.15 L): 10.5e9 pairs 32.4 ms, 1.2e9
// pairs 13.7 ms (0.15e9 of them neighbours).
#include "records.cuh"

namespace idb {

namespace {

constexpr int kThreads = 256;

struct LevJoinGeom {
    uint32_t NL, Lmin, nc, smax;
    int dLmax;
    const int16_t *eps_tab;
    // eps of a length pair, -1 when it has no neighbours
    __device__ __forceinline__ int eps(uint32_t m, int g) const {
        const uint32_t a = m - Lmin, b = a + (uint32_t)g;
        if (a >= NL || b >= NL) return -1;
        const int e = eps_tab[(size_t)a * NL + b];
        return e >= g ? e : -1;
    }
};

// Bits [pos, pos + len) of a plane's words, moved down to bit 0 (word w of them).
template <int W>
__device__ __forceinline__ uint32_t sub_bits(const uint32_t (&pl)[4], uint32_t pos, uint32_t len, int w) {
    const uint32_t q = (pos >> 5) + (uint32_t)w, sh = pos & 31u;
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int k = 0; k < W; ++k) {
        if ((uint32_t)k == q) lo = pl[k];
        if ((uint32_t)k == q + 1) hi = pl[k];
    }
    const uint32_t n = len - 32u * (uint32_t)w;
    return __funnelshift_r(lo, hi, sh) & (n >= 32 ? 0xFFFFFFFFu : (1u << n) - 1u);
}

// Key of the substring [pos, pos + len) as segment k of a length-n sequence.
// Codes are a bijection of the bytes, so equal substrings share a key; two
// different ones that do only make a group larger.
template <int W>
__device__ __forceinline__ unsigned long long sub_key(const uint32_t (&wd)[5][4], uint32_t r, uint32_t n,
                                                      uint32_t k, uint32_t pos, uint32_t len) {
    unsigned long long h = mix64(0x5E6A1F00ull, ((unsigned long long)r << 16) | (n << 2) | k);
#pragma unroll
    for (int w = 0; w < W; ++w) {
        if (32u * (uint32_t)w >= len) break;
        unsigned long long acc = 0;
#pragma unroll
        for (int p = 0; p < 5; ++p)
            acc = acc * 0x9E3779B97F4A7C15ull + sub_bits<W>(wd[p], pos, len, w);
        h = mix64(h, acc);
    }
    return ((unsigned long long)r << 40) | ((unsigned long long)n << 32) |
           ((unsigned long long)k << 30) | (h >> 34);
}

__device__ __forceinline__ uint32_t key_slot(unsigned long long key, uint32_t mask) {
    return (uint32_t)(mix64(key, 0x51ull) & mask);
}

// Slot of a key, kNone if no unique is indexed under it.
__device__ __forceinline__ uint32_t find_key(const unsigned long long *tkey, uint32_t mask,
                                             unsigned long long key) {
    uint32_t sl = key_slot(key, mask);
    for (uint32_t it = 0; it <= mask && it < kSpinCap; ++it) {
        const unsigned long long cur = __ldg(tkey + sl);
        if (cur == key) return sl;
        if (cur == ~0ull) break;
        sl = (sl + 1) & mask;
    }
    return kNone;
}

// The look-ups of a unique of length m: visit(class, key, shift index).
template <int W, typename F>
__device__ __forceinline__ void for_probes(const LevJoinGeom &g, const uint32_t (&wd)[5][4], uint32_t r,
                                           uint32_t m, F visit) {
    for (int gap = 0; gap <= g.dLmax; ++gap) {
        const int e = g.eps(m, gap);
        if (e < 0) continue;
        const uint32_t n = m + (uint32_t)gap, S = (uint32_t)e + 1u;
        for (int k = 0; k <= e; ++k) {
            const uint32_t s = (uint32_t)k * n / S, len = (uint32_t)(k + 1) * n / S - s;
            const int lo = max(-k, -gap - (e - k)), hi = min(k, e - k - gap);
            for (int d = lo; d <= hi; ++d) {
                const int pos = (int)s + d;
                if ((gap == 0 && d == 0) || pos < 0 || (uint32_t)pos + len > m) continue;
                visit(gap == 0 ? 1u : 1u + (uint32_t)gap,
                      sub_key<W>(wd, r, n, (uint32_t)k, (uint32_t)pos, len), (uint32_t)(d - lo));
            }
        }
    }
}

__global__ void __launch_bounds__(kThreads)
k_ljoin_clear(Counters *ctr, uint32_t smax, uint32_t nc, uint64_t cap_mask,
              unsigned long long *__restrict__ key, uint32_t *__restrict__ cnt, unsigned long long *stamp) {
    stamp_begin(stamp);
    const uint32_t n = join_mask(ctr->n_uniques, smax, cap_mask) + 1u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ctr->n_jslots = n;
        ctr->n_binpairs = 0;
        ctr->n_entries = 0;
        ctr->join_pairs = 0;
    }
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint64_t i = t0; i < n; i += stride) key[i] = ~0ull;
    for (uint64_t i = t0; i < (uint64_t)n * nc / 4; i += stride)   // n is a multiple of 1024
        reinterpret_cast<uint4 *>(cnt)[i] = make_uint4(0u, 0u, 0u, 0u);
}

// Uniques indexed under their segments.  The count before an entry's increment
// is its rank in class 0 of the key's group.
template <int W>
__global__ void __launch_bounds__(kThreads)
k_ljoin_insert(LevJoinGeom g, Counters *ctr, const uint32_t *__restrict__ urow,
               const uint32_t *__restrict__ ulen, const uint32_t *__restrict__ urep,
               const uint8_t *__restrict__ seq, const int64_t *__restrict__ seq_off,
               const uint8_t *__restrict__ codemap, unsigned long long *tkey, uint32_t *tcnt,
               uint32_t *__restrict__ islot, uint32_t *__restrict__ irank) {
    __shared__ uint8_t cm[256];
    for (int k = threadIdx.x; k < 256; k += blockDim.x) cm[k] = codemap[k];
    __syncthreads();
    const uint32_t nu = ctr->n_uniques, mask = ctr->n_jslots - 1u;
    const uint32_t stride = gridDim.x * blockDim.x, lane = threadIdx.x & 31;
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < nu; u += stride) {
        const uint32_t row = urow[u], L = ulen[u], r = urep[u];
        const uint32_t S = (uint32_t)(g.eps(L, 0) + 1);
        uint32_t wd[5][4];
        build_planes(seq + seq_off[row], S ? L : 0u, cm, wd);
        for (uint32_t k = 0; k < 4; ++k) {
            uint32_t sl = kNone;
            if (k < S) {
                const uint32_t s = k * L / S;
                const unsigned long long key = sub_key<W>(wd, r, L, k, s, (k + 1) * L / S - s);
                sl = key_slot(key, mask);
                for (uint32_t it = 0;; ++it) {
                    if (it > mask || it >= kSpinCap) {
                        atomicOr(&ctr->error, kErrHashStall);
                        sl = kNone;
                        break;
                    }
                    unsigned long long cur = *((volatile unsigned long long *)&tkey[sl]);
                    if (cur == ~0ull) {
                        cur = atomicCAS(&tkey[sl], ~0ull, key);
                        if (cur == ~0ull) break;   // this entry created the key
                    }
                    if (cur == key) break;
                    sl = (sl + 1) & mask;
                }
            }
            islot[(size_t)u * 4 + k] = sl;
            // one count increment per key among the lanes here together
            const uint32_t am = __activemask();
            const uint32_t grp = __match_any_sync(am, sl);
            const int leader = __ffs(grp) - 1;
            uint32_t base = 0;
            if (lane == (uint32_t)leader && sl != kNone)
                base = atomicAdd(&tcnt[(size_t)sl * g.nc], (uint32_t)__popc(grp));
            base = __shfl_sync(am, base, leader);
            if (k < S) irank[(size_t)u * g.smax + k] = base + (uint32_t)__popc(grp & ((1u << lane) - 1u));
        }
    }
}

// Class sizes of the look-ups that find their key.
template <int W>
__global__ void __launch_bounds__(kThreads)
k_ljoin_probe(LevJoinGeom g, const Counters *__restrict__ ctr, const uint32_t *__restrict__ urow,
              const uint32_t *__restrict__ ulen, const uint32_t *__restrict__ urep,
              const uint8_t *__restrict__ seq, const int64_t *__restrict__ seq_off,
              const uint8_t *__restrict__ codemap, const unsigned long long *__restrict__ tkey,
              uint32_t *tcnt) {
    __shared__ uint8_t cm[256];
    for (int k = threadIdx.x; k < 256; k += blockDim.x) cm[k] = codemap[k];
    __syncthreads();
    const uint32_t nu = ctr->n_uniques, mask = ctr->n_jslots - 1u;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < nu; u += stride) {
        const uint32_t L = ulen[u];
        uint32_t wd[5][4];
        build_planes(seq + seq_off[urow[u]], L, cm, wd);
        for_probes<W>(g, wd, urep[u], L, [&](uint32_t c, unsigned long long key, uint32_t) {
            const uint32_t sl = find_key(tkey, mask, key);
            if (sl != kNone) atomicAdd(&tcnt[(size_t)sl * g.nc + c], 1u);
        });
    }
}

// Places of the groups' entries and bin pairs: a slot is a group when two
// uniques are indexed under its key, or one is and another looked it up.  As
// for the Hamming join, block sums and a counter atomic instead of a scan.
__global__ void __launch_bounds__(kThreads)
k_ljoin_groups(Counters *ctr, uint32_t nc, const uint32_t *__restrict__ tcnt,
               uint32_t *__restrict__ start, uint32_t *__restrict__ bpidx, uint32_t *__restrict__ cur) {
    __shared__ uint2 s_w[8];
    __shared__ uint2 s_base;
    const uint32_t ns = ctr->n_jslots;   // a multiple of the block size
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned long long pairs = 0;
    for (uint32_t h0 = blockIdx.x * blockDim.x; h0 < ns; h0 += gridDim.x * blockDim.x) {
        const uint32_t h = h0 + threadIdx.x;
        const uint32_t *c = tcnt + (size_t)h * nc;
        const uint32_t c0 = c[0];
        uint32_t looked = 0, bps = 0, entries = 0;
        if (c0) {
            for (uint32_t q = 1; q < nc; ++q) { looked += c[q]; bps += c[q] != 0; }
            bps += c0 >= 2;
            if (bps) {
                entries = c0 + looked;
                pairs += (unsigned long long)c0 * (c0 - 1) / 2 + (unsigned long long)c0 * looked;
            }
        }
        uint32_t bi = bps, ei = entries;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t tb = __shfl_up_sync(0xFFFFFFFFu, bi, d);
            const uint32_t te = __shfl_up_sync(0xFFFFFFFFu, ei, d);
            if (lane >= (uint32_t)d) { bi += tb; ei += te; }
        }
        if (lane == 31) s_w[wid] = make_uint2(bi, ei);
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t tb = 0, te = 0;
            for (uint32_t w = 0; w < blockDim.x / 32; ++w) {
                const uint2 x = s_w[w];
                s_w[w] = make_uint2(tb, te);
                tb += x.x;
                te += x.y;
            }
            if (tb) s_base = make_uint2(atomicAdd(&ctr->n_binpairs, tb), atomicAdd(&ctr->n_entries, te));
        }
        __syncthreads();
        if (bps) {
            uint32_t pos = s_base.y + s_w[wid].y + ei - entries;
            start[h] = pos;
            bpidx[h] = s_base.x + s_w[wid].x + bi - bps;
            for (uint32_t q = 0; q < nc; ++q) {
                cur[(size_t)h * nc + q] = pos;
                pos += c[q];
            }
        } else {
            start[h] = kNone;
        }
        __syncthreads();
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) pairs += __shfl_xor_sync(0xFFFFFFFFu, pairs, d);
    if (lane == 0 && pairs) atomicAdd(&ctr->join_pairs, pairs);
}

// Entries: the record and side record {V bits, J bits with the shift index in
// the top two bits, unique id} of every unique in every group it belongs to.
template <int RSC, int W>
__global__ void __launch_bounds__(kThreads)
k_ljoin_fill(LevJoinGeom g, const Counters *__restrict__ ctr, const uint32_t *__restrict__ urow,
             const uint32_t *__restrict__ ulen, const uint32_t *__restrict__ urep,
             const uint8_t *__restrict__ seq, const int64_t *__restrict__ seq_off,
             const uint8_t *__restrict__ codemap, const unsigned long long *__restrict__ tkey,
             const uint32_t *__restrict__ islot, const uint32_t *__restrict__ irank,
             const uint32_t *__restrict__ start, uint32_t *cur, GeneSide gv, GeneSide gj,
             uint4 *__restrict__ ent_rec,
             uint4 *__restrict__ ent_meta, const uint32_t *__restrict__ ucopies,
             uint32_t *__restrict__ ent_copies, int planes, uint64_t cap_entries, uint32_t *err) {
    __shared__ uint8_t cm[256];
    for (int k = threadIdx.x; k < 256; k += blockDim.x) cm[k] = codemap[k];
    __syncthreads();
    const uint32_t nu = ctr->n_uniques, mask = ctr->n_jslots - 1u;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < nu; u += stride) {
        const uint32_t row = urow[u], L = ulen[u];
        uint32_t wd[5][4];
        build_planes(seq + seq_off[row], L, cm, wd);
        uint4 rec[RSC];
        flatten_planes<RSC>(wd, planes, (uint32_t)W, rec);
        const uint64_t vb = gv.row(row);
        const uint32_t copies = ucopies[u];
        const uint32_t jb = (uint32_t)gj.row(row) & 0x3FFFFFFFu;
        auto put = [&](uint64_t pos, uint32_t shift) {
            if (pos >= cap_entries) { atomicOr(err, kErrEntryOverflow); return; }
            ent_meta[pos] = make_uint4((uint32_t)vb, (uint32_t)(vb >> 32), jb | (shift << 30), u);
            ent_copies[pos] = copies;
#pragma unroll
            for (int q = 0; q < RSC; ++q) ent_rec[pos * RSC + q] = rec[q];
        };
        const uint32_t S = (uint32_t)(g.eps(L, 0) + 1);
        for (uint32_t k = 0; k < S; ++k) {
            const uint32_t sl = islot[(size_t)u * 4 + k];
            if (sl == kNone) continue;
            const uint32_t s0 = start[sl];
            if (s0 != kNone) put((uint64_t)s0 + irank[(size_t)u * g.smax + k], 0u);
        }
        for_probes<W>(g, wd, urep[u], L, [&](uint32_t c, unsigned long long key, uint32_t shift) {
            const uint32_t sl = find_key(tkey, mask, key);
            if (sl != kNone) put(atomicAdd(&cur[(size_t)sl * g.nc + c], 1u), shift);
        });
    }
}

// Bin pairs of every group: class 0 with itself, every other class with class 0.
__global__ void __launch_bounds__(kThreads)
k_ljoin_bp_fill(LevJoinGeom g, Counters *ctr, const unsigned long long *__restrict__ tkey,
                const uint32_t *__restrict__ tcnt, const uint32_t *__restrict__ start,
                const uint32_t *__restrict__ bpidx, uint32_t TX, uint64_t cap_bp, uint64_t cap_entries,
                BinPair *__restrict__ out) {
    drop_overgrown(ctr, cap_bp, cap_entries);
    const uint32_t ns = ctr->n_jslots;
    for (uint32_t h = blockIdx.x * blockDim.x + threadIdx.x; h < ns; h += gridDim.x * blockDim.x) {
        uint32_t pos = start[h];
        if (pos == kNone) continue;
        uint32_t at = bpidx[h];
        const unsigned long long key = tkey[h];
        const uint32_t n = (uint32_t)(key >> 32) & 0xFFu, k = (uint32_t)(key >> 30) & 3u;
        const uint32_t s0 = pos, c0 = tcnt[(size_t)h * g.nc];
        const int e = g.eps(n, 0);
        for (uint32_t c = 0; c < g.nc; ++c) {
            const uint32_t m = tcnt[(size_t)h * g.nc + c], first = pos;
            pos += m;
            if (c == 0 ? m < 2 : m == 0) continue;
            if (at >= cap_bp) { ++at; continue; }   // flagged above
            BinPair P;
            P.a_start = first; P.a_n = m; P.b_start = s0; P.b_n = c0;
            P.ncx = (m + TX - 1) / TX;
            P.la = (uint16_t)(c > 1 ? n - (c - 1) : n); P.lb = (uint16_t)n;
            P.v = (uint16_t)k;                      // segment of the group
            P.j = (uint16_t)(e + 1);                // segments of length n
            P.eps = (int16_t)e;
            P.same = c == 0;
            const uint64_t cost = c == 0 ? (uint64_t)m * (m - 1) / 2 : (uint64_t)m * c0;
            P.cls = (uint8_t)(cost ? 63 - __clzll((long long)cost) : 0);
            P.cost_lo = (uint32_t)min(cost, (uint64_t)0xFFFFFFFFu);
            out[at++] = P;
        }
    }
}

LevJoinGeom lev_geom(const Plan &P, const Buffers &B) {
    return LevJoinGeom{P.NL, P.Lmin, P.join_classes, P.join_smax, P.dLmax, B.eps_tab};
}

template <int W>
void ljoin_build(const Plan &P, const Buffers &B, cudaStream_t s) {
    const LevJoinGeom g = lev_geom(P, B);
    k_ljoin_insert<W><<<grid_wave(k_ljoin_insert<W>, P.N, kThreads), kThreads, 0, s>>>(
        g, B.ctr, B.urow, B.ulen, B.urep, B.seq, B.seq_off, B.codemap, B.jn_key, B.jn_cnt, B.jn_islot,
        B.jn_cur);
    k_ljoin_probe<W><<<grid_wave(k_ljoin_probe<W>, P.N, kThreads), kThreads, 0, s>>>(
        g, B.ctr, B.urow, B.ulen, B.urep, B.seq, B.seq_off, B.codemap, B.jn_key, B.jn_cnt);
}

template <int RSC, int W>
void ljoin_fill(const Plan &P, const Buffers &B, cudaStream_t s) {
    auto kern = k_ljoin_fill<RSC, W>;
    kern<<<grid_wave(kern, P.N, kThreads), kThreads, 0, s>>>(
        lev_geom(P, B), B.ctr, B.urow, B.ulen, B.urep, B.seq, B.seq_off, B.codemap, B.jn_key, B.jn_islot,
        B.jn_cur, B.jn_start, B.jn_pos, GeneSide{B.vbits, P.compact ? B.ctr->used_v : nullptr, P.VW},
        GeneSide{B.jbits, P.compact ? B.ctr->used_j : nullptr, P.JW}, B.ent_rec, B.ent_meta, B.ucopies, B.ent_copies, (int)P.B,
        P.cap_entries, &B.ctr->error);
}

}  // namespace

void launch_lev_join(const Plan &P, const Buffers &B, cudaStream_t s) {
    const uint64_t slots = B.jn_mask + 1;
    k_ljoin_clear<<<grid_wave(k_ljoin_clear, slots * P.join_classes / 4, kThreads), kThreads, 0, s>>>(
        B.ctr, P.join_smax, P.join_classes, B.jn_mask, B.jn_key, B.jn_cnt, B.stamp(1));
    switch (P.W) {
        case 1: ljoin_build<1>(P, B, s); break;
        case 2: ljoin_build<2>(P, B, s); break;
        case 3: ljoin_build<3>(P, B, s); break;
        default: ljoin_build<4>(P, B, s); break;
    }
    k_ljoin_groups<<<grid_wave(k_ljoin_groups, slots, kThreads), kThreads, 0, s>>>(
        B.ctr, P.join_classes, B.jn_cnt, B.jn_start, B.jn_bpidx, B.jn_pos);
}

void launch_lev_join_fill(const Plan &P, const Buffers &B, cudaStream_t s) {
    if (P.B <= 2) {
        switch (P.W) {
            case 1: ljoin_fill<1, 1>(P, B, s); break;
            case 2: ljoin_fill<1, 2>(P, B, s); break;
            case 3: ljoin_fill<2, 3>(P, B, s); break;
            default: ljoin_fill<2, 4>(P, B, s); break;
        }
    } else {
        switch (P.W) {
            case 1: ljoin_fill<2, 1>(P, B, s); break;
            case 2: ljoin_fill<3, 2>(P, B, s); break;
            case 3: ljoin_fill<4, 3>(P, B, s); break;
            default: ljoin_fill<5, 4>(P, B, s); break;
        }
    }
}

void launch_lev_join_binpairs(const Plan &P, const Buffers &B, cudaStream_t s) {
    k_ljoin_bp_fill<<<grid_wave(k_ljoin_bp_fill, B.jn_mask + 1, kThreads), kThreads, 0, s>>>(
        lev_geom(P, B), B.ctr, B.jn_key, B.jn_cnt, B.jn_start, B.jn_bpidx, P.TX, P.cap_binpairs,
        P.cap_entries, B.bp);
}

}  // namespace idb
