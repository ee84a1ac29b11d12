// distance_common.cuh -- what the distance kernels share: their arguments, where
// neighbour pairs go (the edge list, or the two sweeps of the streamed mode), the
// work queue of tiled units, batches of hits and the small bin pairs' helpers.
#pragma once
#include "idb_internal.cuh"

namespace idb {

struct DistArgs {
    const BinPair *bp;
    const uint32_t *unit_base;
    const uint4 *rec;
    const uint32_t *ent_uid;
    const uint32_t *urow;
    const uint64_t *vbits, *jbits;
    uint32_t VW, JW;
    uint32_t rs16;                   // record size in 16-byte words
    uint32_t TX, TY, q;
    uint32_t A;                      // number of codes (Levenshtein)
    uint2 *edges;
    uint64_t cap_edges;
    uint32_t chunk_log;              // edge slots a warp reserves at a time: 1 << chunk_log
    Counters *ctr;
    unsigned long long *bp_cycles;   // optional per bin-pair cycle log
    const uint4 *meta;               // per entry {sigV lo, sigV hi, sigJ, uid}
    int sig_exact;                   // signatures decide canonicity exactly
    const uint32_t *small_list;      // schedule positions of the small bin pairs (from the
                                     // front) and of the tiny ones (from small_cap - 1 down)
    uint32_t small_cap;
    // segment join: a hit is a neighbour pair if the V and J sets intersect and no
    // lower segment (edit distance: no earlier look-up) holds, whose group emits it
    int join;
    int vj_meta;                     // the join's side records hold the V and J bits
    // where neighbour pairs go: kSinkEdges = the edge list; kSinkCount /
    // kSinkGrow = the two sweeps of the streamed mode (no edge list kept)
    uint32_t sink;
    uint32_t *cnt;                   // copies-weighted neighbour counts (count sweep)
    const uint32_t *ucopies;
    const uint32_t *ecopies;         // the same per entry
    uint32_t *parent;                // union-find forest (grow sweep)
    uint32_t *bmin;                  // minimum core neighbour of a non-core unique
};

// Hamming on 2- and 5-plane records (hamming.cuh)
void launch_hamming_2(const Plan &P, const DistArgs &a, int grid, cudaStream_t s);
void launch_hamming_5(const Plan &P, const DistArgs &a, int grid, cudaStream_t s);
// Levenshtein with eps <= kLevDiagMaxEps on 2- and 5-plane records (lev_diag.cuh)
void launch_lev_diag_2(const Plan &P, const DistArgs &a, int grid, cudaStream_t s);
void launch_lev_diag_5(const Plan &P, const DistArgs &a, int grid, cudaStream_t s);

namespace {

constexpr int kWarps = 4;            // warps per block
constexpr int kYB = 32;              // y-records staged per batch (a lane's hits: one word)

// Streamed mode, for neighbour graphs larger than the edge memory allowed: the
// distance work runs twice and no pair is stored.  The count sweep adds each
// side's copies to the other's count (rule S5); after the core flags, the grow
// sweep merges core-core pairs into the union-find forest (link to the smaller
// root, as the reference's union_a_and_b does, cuda/PSDBSCAN.hcu:76-107) and
// keeps for every non-core unique its minimum core neighbour (atomicMin: the
// same border rule as the edge-list path).  Both are order-independent.
__device__ __forceinline__ uint32_t sweep_find(uint32_t *p, uint32_t x) {
    volatile uint32_t *vp = p;
    while (true) {   // parent[y] <= y of a core y: x strictly decreases
        const uint32_t px = vp[x];
        if (px >= x) return px == x ? x : kNone;   // kNone: not a core's parent
        const uint32_t ppx = vp[px];
        if (ppx >= px) return ppx == px ? px : kNone;
        vp[x] = ppx;   // path halving
        x = ppx;
    }
}

__device__ __noinline__ void sink_streamed(const DistArgs &a, uint32_t lo, uint32_t hi) {
    // parents carry the core flag; equal ones (stale or not) are one component
    const uint32_t plo = __ldcg(a.parent + lo), phi = __ldcg(a.parent + hi);
    const uint32_t nlo = plo & kNonCore, nhi = phi & kNonCore;
    if (nlo != nhi) {
        atomicMin(&a.bmin[nlo ? lo : hi], nlo ? hi : lo);
        return;
    }
    if (nlo || plo == phi) return;
    uint32_t x = plo, y = phi, it = 0;
    for (; it < kSpinCap; ++it) {
        uint32_t rx = sweep_find(a.parent, x), ry = sweep_find(a.parent, y);
        if (rx == ry) break;
        if (rx < ry) { const uint32_t t = rx; rx = ry; ry = t; }
        if (rx == kNone) { it = kSpinCap; break; }
        if (atomicCAS(&a.parent[rx], rx, ry) == rx) break;   // hook the larger root
        x = rx;
        y = ry;
    }
    if (it == kSpinCap) atomicOr(&a.ctr->error, kErrUnionStall);
}

// One neighbour pair (lo < hi, unique ids) at edge slot `slot`.
__device__ __forceinline__ void put_edge(const DistArgs &a, uint64_t slot, uint32_t lo, uint32_t hi) {
    if (a.sink == kSinkEdges) {
        if (slot < a.cap_edges) a.edges[slot] = make_uint2(lo, hi);
    } else if (a.sink == kSinkGrow) {
        sink_streamed(a, lo, hi);
    }
}

// Copies-weighted counts (rule S5) of one neighbour pair (copies clo, chi), and a
// smaller neighbour for the larger id (any one will do, so a plain store): the
// forest the unions start from (k_core).
__device__ __forceinline__ void count_pair(const DistArgs &a, uint32_t lo, uint32_t hi, uint32_t clo,
                                           uint32_t chi) {
    if (a.sink == kSinkGrow) return;
    atomicAdd(&a.cnt[lo], chi);
    atomicAdd(&a.cnt[hi], clo);
    a.parent[hi] = lo;
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Edge writer: each warp reserves a chunk of 1 << chunk_log slots at a time; slots
// a warp does not fill are set to the sentinel (x = kNone) at the end.
struct EdgeWriter {
    uint64_t base;     // kNoChunk = no chunk held
    uint32_t fill;
    uint32_t written;
    static constexpr uint64_t kNoChunk = ~0ull;

    __device__ void init() { base = kNoChunk; fill = 0; written = 0; }

    __device__ void pad(const DistArgs &a, int lane) {
        if (base == kNoChunk || a.sink != kSinkEdges) return;
        for (uint32_t t = fill + lane; t < 1u << a.chunk_log; t += 32) {
            const uint64_t slot = base + t;
            if (slot < a.cap_edges) a.edges[slot] = make_uint2(kNone, kNone);
        }
    }

    // warp-uniform call; lanes with ok=true append (lo, hi).  The byte and the
    // Myers kernels leave the counts of a stored list to k_count: per pair they
    // cost more here, where a lane waits for both ends' copies.
    template <bool COUNT>
    __device__ void append(const DistArgs &a, int lane, bool ok, uint32_t lo, uint32_t hi) {
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, ok);
        if (!m) return;
        const Bulk bk = reserve(a, lane, (uint32_t)__popc(m));
        if (ok) {
            put_edge(a, slot_of(bk, (uint32_t)__popc(m & lanemask_lt())), lo, hi);
            if (COUNT || a.sink == kSinkCount)
                count_pair(a, lo, hi, __ldg(&a.ucopies[lo]), __ldg(&a.ucopies[hi]));
        }
    }

    // Bulk append, warp-uniform: the warp appends T edges at logical positions
    // 0..T-1 (each lane knows its own); the room left in the held chunk is
    // used first, then as many new chunks as needed, reserved with one atomic.
    struct Bulk { uint64_t b0, nb; uint32_t room; };
    __device__ Bulk reserve(const DistArgs &a, int lane, uint32_t T) {
        const uint32_t chunk = 1u << a.chunk_log;
        Bulk k;
        k.room = base == kNoChunk ? 0u : chunk - fill;
        k.b0 = base + fill;
        k.nb = kNoChunk;
        if (T > k.room) {
            const uint32_t nch = (T - k.room + chunk - 1) >> a.chunk_log;
            uint32_t nb = 0;
            if (lane == 0) nb = atomicAdd(&a.ctr->edge_reserved, nch << a.chunk_log);
            nb = __shfl_sync(0xFFFFFFFFu, nb, 0);
            if ((uint64_t)nb + ((uint64_t)nch << a.chunk_log) > a.cap_edges && lane == 0)
                atomicOr(&a.ctr->error, kErrEdgeOverflow);
            k.nb = nb;
            base = (uint64_t)nb + ((uint64_t)(nch - 1) << a.chunk_log);
            fill = (T - k.room) - ((nch - 1) << a.chunk_log);
        } else {
            fill += T;
        }
        written += T;
        return k;
    }
    __device__ __forceinline__ uint64_t slot_of(const Bulk &k, uint32_t i) const {
        return i < k.room ? k.b0 + i : k.nb + (i - k.room);
    }
};

// lowest common gene of two uniques in one column, -1 if none
__device__ __forceinline__ int lowest_common(const uint64_t *bits, uint32_t W, uint32_t rx,
                                             uint32_t ry) {
    for (uint32_t w = 0; w < W; ++w) {
        const uint64_t c = bits[(size_t)rx * W + w] & bits[(size_t)ry * W + w];
        if (c) return (int)(w * 64) + lowest_bit64(c);
    }
    return -1;
}

__device__ __forceinline__ bool canonical(const DistArgs &a, const BinPair &P, uint32_t ux,
                                          uint32_t uy) {
    const uint32_t rx = a.urow[ux], ry = a.urow[uy];
    return lowest_common(a.vbits, a.VW, rx, ry) == (int)P.v &&
           lowest_common(a.jbits, a.JW, rx, ry) == (int)P.j;
}

// V and J sets of two uniques (by id) intersect.
__device__ __forceinline__ bool vj_intersect(const DistArgs &a, uint32_t ux, uint32_t uy) {
    const uint32_t rx = a.urow[ux], ry = a.urow[uy];
    return lowest_common(a.vbits, a.VW, rx, ry) >= 0 && lowest_common(a.jbits, a.JW, rx, ry) >= 0;
}

// The same from the side records: {V genes below the bin's V gene (64 bits), J
// genes below its J gene, unique id}.  Exact signatures (V genes <= 64, J genes
// <= 32) decide by themselves: no lower gene is shared.
__device__ __forceinline__ bool canonical_meta(const DistArgs &a, const BinPair &P, const uint4 &mx,
                                               const uint4 &my) {
    if (a.sig_exact) return ((mx.x & my.x) | (mx.y & my.y) | (mx.z & my.z)) == 0;
    return canonical(a, P, mx.w, my.w);
}

// Warp-cooperative lookup of the bin pair that owns unit u (largest i with
// unit_base[i] <= u); 32-ary search.
__device__ __forceinline__ uint32_t find_binpair(const uint32_t *base, uint32_t n, uint32_t u,
                                                 int lane) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 32) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t idx = lo + (uint32_t)lane * step;
        const bool ok = idx < hi && __ldg(base + idx) <= u;
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, ok);
        const uint32_t t = 31 - __clz(m);
        lo = lo + t * step;
        hi = min(hi, lo + step);
    }
    const uint32_t idx = lo + lane;
    const bool ok = idx < hi && __ldg(base + idx) <= u;
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, ok);
    return lo + (31 - __clz(m));
}

struct Unit {
    BinPair P;
    uint32_t xbase, nx, ybase, ny;
    uint32_t bpi;             // index of the bin pair in schedule order
    long long t0;             // clock64 at the start (profiling only)
};

__device__ __forceinline__ bool next_unit(const DistArgs &a, uint32_t n_units, uint32_t n_bp,
                                          int lane, Unit &U) {
    uint32_t u = 0;
    if (lane == 0) u = atomicAdd(&a.ctr->unit_cursor, 1u);
    u = __shfl_sync(0xFFFFFFFFu, u, 0);
    if (u >= n_units) return false;
    const uint32_t i = find_binpair(a.unit_base, n_bp, u, lane);
    U.bpi = i;
    if (a.bp_cycles) U.t0 = clock64();
    U.P = a.bp[i];
    const uint64_t k = u - a.unit_base[i];
    uint32_t cx, cy;
    if (U.P.same) {
        tri_decode(k, U.P.ncx, a.q, cx, cy);
    } else {
        cy = (uint32_t)(k / U.P.ncx);
        cx = (uint32_t)(k % U.P.ncx);
    }
    U.xbase = cx * a.TX;
    U.nx = min(a.TX, U.P.a_n - U.xbase);
    U.ybase = cy * a.TY;
    const uint32_t bn = U.P.same ? U.P.a_n : U.P.b_n;
    U.ny = min(a.TY, bn - U.ybase);
    return true;
}

// profiling: device cycles spent on each bin pair (learned-schedule training data)
__device__ __forceinline__ void log_unit(const DistArgs &a, const Unit &U, int lane) {
    if (a.bp_cycles && lane == 0)
        atomicAdd(&a.bp_cycles[U.bpi], (unsigned long long)(clock64() - U.t0));
}

// pairs of the unit that the method evaluates (y after x for a same-bin pair)
__device__ __forceinline__ uint64_t unit_pairs(const Unit &U, uint32_t xpos) {
    if (!U.P.same) return U.ny;
    const uint32_t lo = max(U.ybase, xpos + 1), hi = U.ybase + U.ny;
    return hi > lo ? hi - lo : 0;
}

__device__ __forceinline__ void finish(const DistArgs &a, EdgeWriter &ew, uint64_t pairs,
                                       int lane) {
    ew.pad(a, lane);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) pairs += __shfl_xor_sync(0xFFFFFFFFu, pairs, d);
    if (lane == 0) {
        if (pairs) atomicAdd(&a.ctr->pairs_evaluated, (unsigned long long)pairs);
        if (ew.written) atomicAdd(&a.ctr->n_edges, ew.written);
    }
}

// Pair p of a small bin pair -> (i, j).  One bin: i < j < n, ordered by j
// (pairs of j start at j(j-1)/2).  Two bins: i = p mod n, j = p div n.
__device__ __forceinline__ void small_pair(uint32_t p, bool same, uint32_t n, uint32_t &i,
                                           uint32_t &j) {
    if (same) {
        uint32_t jj = (uint32_t)((1.0f + sqrtf(8.0f * (float)p + 1.0f)) * 0.5f);
        while (jj > 1 && jj * (jj - 1) / 2 > p) --jj;
        while (jj * (jj + 1) / 2 <= p) ++jj;
        j = jj;
        i = p - jj * (jj - 1) / 2;
    } else {
        j = p / n;
        i = p - j * n;
    }
}

// Small bin pairs of a warp: the warp claims up to kSmallBatch schedule positions
// with one atomic, each lane loads one of their bin pairs, and while one bin
// pair is scored the next one's records are prefetched into L1 (a small bin
// pair is otherwise a chain of dependent loads: position, bin pair, records).
// When there are fewer than two claims a warp, the claims get smaller instead,
// so that no warp works through a chain while others have nothing.
constexpr uint32_t kSmallBatch = 16;

__device__ __forceinline__ uint32_t small_batch(uint32_t n_small) {
    return min(kSmallBatch, max(1u, n_small / (2u * gridDim.x * kWarps)));
}

__device__ __forceinline__ BinPair shfl_binpair(const BinPair &p, int src) {
    static_assert(sizeof(BinPair) % 4 == 0, "BinPair words");
    constexpr int NWD = (int)(sizeof(BinPair) / 4);
    uint32_t w[NWD];
    memcpy(w, &p, sizeof(BinPair));
#pragma unroll
    for (int k = 0; k < NWD; ++k) w[k] = __shfl_sync(0xFFFFFFFFu, w[k], src);
    BinPair q;
    memcpy(&q, w, sizeof(BinPair));
    return q;
}

__device__ __forceinline__ void prefetch_l1(const void *p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}
constexpr uint32_t kOff = 0x40000000u;   // score of a masked x-entry (never a hit)

// What a tiled unit keeps of its entries in the warp's shared memory.
struct TileSlice {
    uint4 *xm, *ym;          // side records of the x-entries and of the batch's y-entries
    uint32_t *xcp, *ycp;     // their copies
    uint32_t *xs, *ys;       // sums of the neighbours' copies (ys: small bin pairs only)

    __device__ __forceinline__ void begin_x(const DistArgs &a, uint32_t i, uint32_t entry) const {
        xm[i] = __ldg(a.meta + entry);
        xcp[i] = __ldg(a.ecopies + entry);
        xs[i] = 0u;
    }
    __device__ __forceinline__ void begin_y(const DistArgs &a, uint32_t t, uint32_t entry) const {
        ym[t] = __ldg(a.meta + entry);
        ycp[t] = __ldg(a.ecopies + entry);
    }
    // after the unit's last batch: one count update per x-entry
    __device__ __forceinline__ void end_x(const DistArgs &a, uint32_t n, int lane) const {
        __syncwarp();
        for (uint32_t i = (uint32_t)lane; i < n; i += 32)
            if (xs[i]) atomicAdd(&a.cnt[xm[i].w], xs[i]);
        __syncwarp();
    }
};

// 32 x 32 bit transpose over the warp: bit k of lane i becomes bit i of lane k.
__device__ __forceinline__ uint32_t transpose32(uint32_t m, int lane) {
    uint32_t mask = 0x0000FFFFu;
#pragma unroll
    for (int j = 16; j; j >>= 1, mask ^= mask << j) {
        const uint32_t o = __shfl_xor_sync(0xFFFFFFFFu, m, j);
        m = (lane & j) ? (m & ~mask) | ((o & ~mask) >> j) : (m & mask) | ((o & mask) << j);
    }
    return m;
}

// The neighbour pairs of a batch: bit t of hits[r] = x-entry 32 r + lane with
// y-entry t.  One bulk append for the warp, and the counts of both sides: a
// lane's hits give its x-entries' sums, the transposed bits the y-entries',
// so that an entry costs one count update per unit or batch instead of one per
// pair (a pass over the edge list afterwards took 1.8 ms for 0.15e9 pairs,
// nearly all of it atomics).  Most entries have one copy: a sum is a popcount
// plus what the others add.  Out of line: one copy for every unit loop.
template <int RX>
__device__ __noinline__ void emit_batch(const DistArgs &a, EdgeWriter &ew, const TileSlice &T,
                                        const uint32_t (&hits)[RX], uint32_t nb, int lane) {
    uint32_t c = 0;
#pragma unroll
    for (int r = 0; r < RX; ++r) c += (uint32_t)__popc(hits[r]);
    uint32_t incl = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t n = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += n;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    if (total == 0) return;
    const EdgeWriter::Bulk bk = ew.reserve(a, lane, total);
    const bool count = a.sink != kSinkGrow;
    const uint32_t uy_lane = (uint32_t)lane < nb ? T.ym[lane].w : 0u;
    const uint32_t ymult = __ballot_sync(0xFFFFFFFFu, (uint32_t)lane < nb && T.ycp[lane] > 1);
    uint32_t i = incl - c, ysum = 0, yhint = kNone;
#pragma unroll
    for (int r = 0; r < RX; ++r) {
        const uint32_t h = hits[r], x = 32u * r + (uint32_t)lane;
        if (!__any_sync(0xFFFFFFFFu, h)) continue;
        const uint32_t ux = T.xm[x].w;
        for (uint32_t b = h; b; b &= b - 1) {
            const uint32_t uy = T.ym[__ffs(b) - 1].w;
            put_edge(a, ew.slot_of(bk, i++), min(ux, uy), max(ux, uy));
        }
        if (!count) continue;
        if (h) {
            uint32_t s = (uint32_t)__popc(h);
            for (uint32_t b = h & ymult; b; b &= b - 1) s += T.ycp[__ffs(b) - 1] - 1u;
            T.xs[x] += s;
            const uint32_t uy = T.ym[__ffs(h) - 1].w;
            if (uy < ux) a.parent[ux] = uy;
        }
        const uint32_t m = transpose32(h, lane);
        const uint32_t xmult = __ballot_sync(0xFFFFFFFFu, T.xcp[x] > 1);
        if (m) {
            ysum += (uint32_t)__popc(m);
            for (uint32_t b = m & xmult; b; b &= b - 1) ysum += T.xcp[32 * r + __ffs(b) - 1] - 1u;
            yhint = min(yhint, T.xm[32 * r + __ffs(m) - 1].w);
        }
    }
    if (ysum) {
        atomicAdd(&a.cnt[uy_lane], ysum);
        if (yhint < uy_lane) a.parent[uy_lane] = yhint;
    }
}

// Inclusive sum over the lanes, and the total.
__device__ __forceinline__ uint32_t warp_incl_sum(uint32_t v, int lane, uint32_t *total) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t n = __shfl_up_sync(0xFFFFFFFFu, v, d);
        if (lane >= d) v += n;
    }
    *total = __shfl_sync(0xFFFFFFFFu, v, 31);
    return v;
}

// The neighbour pairs of a small bin pair (n x-entries, m y-entries, at most 32
// each; same: pairs of the n): bit k of a lane's word is pair lane + 32 k.  One
// bulk append; the counts are summed in shared memory, one update per entry.
__device__ __noinline__ void emit_pair_bits(const DistArgs &a, EdgeWriter &ew, const TileSlice &T, int lane,
                                            uint32_t bits, bool same, uint32_t n, uint32_t m,
                                            uint32_t xstart, uint32_t ystart) {
    const uint32_t c = (uint32_t)__popc(bits);
    uint32_t total;
    const uint32_t incl = warp_incl_sum(c, lane, &total);
    if (total == 0) return;
    const EdgeWriter::Bulk bk = ew.reserve(a, lane, total);
    const bool count = a.sink != kSinkGrow;
    __syncwarp();
    if ((uint32_t)lane < n) T.begin_x(a, lane, xstart + lane);
    if (!same && (uint32_t)lane < m) {
        T.begin_y(a, lane, ystart + lane);
        T.ys[lane] = 0u;
    }
    __syncwarp();
    const uint4 *ym = same ? T.xm : T.ym;
    const uint32_t *ycp = same ? T.xcp : T.ycp;
    uint32_t *ys = same ? T.xs : T.ys;
    uint32_t k = incl - c;
    for (uint32_t b = bits; b; b &= b - 1) {
        const uint32_t p = (uint32_t)lane + 32u * ((uint32_t)__ffs(b) - 1u);
        uint32_t i, j;
        small_pair(p, same, n, i, j);
        const uint32_t ux = T.xm[i].w, uy = ym[j].w, lo = min(ux, uy), hi = max(ux, uy);
        put_edge(a, ew.slot_of(bk, k++), lo, hi);
        if (count) {
            atomicAdd(&T.xs[i], ycp[j]);
            atomicAdd(&ys[j], T.xcp[i]);
            a.parent[hi] = lo;     // any smaller neighbour (k_core)
        }
    }
    T.end_x(a, n, lane);
    if (!same && (uint32_t)lane < m && T.ys[lane]) atomicAdd(&a.cnt[T.ym[lane].w], T.ys[lane]);
    __syncwarp();
}

// The neighbour pairs of the lanes' own tiny bin pairs (an entry of the bin with
// another; bit of pair (i, j) as in small_pair): every pair is a constant bit,
// so ids, copies and sums stay in registers and an entry costs one count update.
__device__ __noinline__ void emit_tiny_bits(const DistArgs &a, EdgeWriter &ew, int lane, uint32_t bits,
                                            uint32_t n, uint32_t start) {
    const uint32_t c = (uint32_t)__popc(bits);
    uint32_t total;
    const uint32_t incl = warp_incl_sum(c, lane, &total);
    if (total == 0) return;
    const EdgeWriter::Bulk bk = ew.reserve(a, lane, total);
    if (bits == 0) return;
    const bool count = a.sink != kSinkGrow;
    uint32_t k = incl - c;
    uint32_t uid[kTinySide], cp[kTinySide], sum[kTinySide], hint[kTinySide];
#pragma unroll
    for (uint32_t i = 0; i < kTinySide; ++i) {
        uid[i] = i < n ? __ldg(&a.meta[start + i].w) : 0u;
        cp[i] = i < n ? __ldg(&a.ecopies[start + i]) : 0u;
        sum[i] = 0u;
        hint[i] = kNone;
    }
#pragma unroll
    for (uint32_t j = 1; j < kTinySide; ++j)
#pragma unroll
        for (uint32_t i = 0; i < j; ++i)
            if ((bits >> (j * (j - 1) / 2 + i)) & 1u) {
                put_edge(a, ew.slot_of(bk, k++), min(uid[i], uid[j]), max(uid[i], uid[j]));
                sum[i] += cp[j];
                sum[j] += cp[i];
                hint[i] = min(hint[i], uid[j]);
                hint[j] = min(hint[j], uid[i]);
            }
    if (!count) return;
#pragma unroll
    for (uint32_t i = 0; i < kTinySide; ++i)
        if (sum[i]) {
            atomicAdd(&a.cnt[uid[i]], sum[i]);
            if (hint[i] < uid[i]) a.parent[uid[i]] = hint[i];
        }
}

template <typename K>
int occupancy_grid(K kernel, size_t smem) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kWarps * 32, smem);
    if (per_sm < 1) per_sm = 1;
    return per_sm * sm_count();
}

template <typename K>
void run(K kernel, const DistArgs &a, size_t smem, int grid, cudaStream_t s) {
    if (smem > 48 * 1024) allow_dynamic_smem(reinterpret_cast<const void *>(kernel));
    if (grid <= 0) grid = occupancy_grid(kernel, smem);
    kernel<<<grid, kWarps * 32, smem, s>>>(a);
}

}  // namespace
}  // namespace idb
