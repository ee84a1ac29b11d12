// distance_common.cuh -- what the distance kernels share: their arguments, where
// neighbour pairs go (the edge list, or the two sweeps of the streamed mode), the
// work queue of tiled units, deferred hits and the small bin pairs' helpers.
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
    Counters *ctr;
    unsigned long long *bp_cycles;   // optional per bin-pair cycle log
    uint32_t *bp_hits;
    const uint4 *meta;               // per entry {sigV lo, sigV hi, sigJ, uid}
    int sig_exact;                   // signatures decide canonicity exactly
    const uint32_t *small_list;      // schedule positions of the small bin pairs (from the
                                     // front) and of the tiny ones (from small_cap - 1 down)
    uint32_t small_cap;
    // segment join: a hit is a neighbour pair if the V and J sets intersect and
    // no lower segment is identical (that segment's group emits it)
    int join;
    int vj_meta;                     // the join's side records hold the V and J bits
    // where neighbour pairs go: kSinkEdges = the edge list; kSinkCount /
    // kSinkGrow = the two sweeps of the streamed mode (no edge list kept)
    uint32_t sink;
    uint32_t *cnt;                   // copies-weighted neighbour counts (count sweep)
    const uint32_t *ucopies;
    const uint32_t *ucore;           // core flags (grow sweep)
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
constexpr int kYB = 64;              // y-records staged per batch

// Streamed mode, for neighbour graphs larger than the edge memory allowed: the
// distance work runs twice and no pair is stored.  The count sweep adds each
// side's copies to the other's count (rule S5); after the core flags, the grow
// sweep merges core-core pairs into the union-find forest (link to the smaller
// root, as the reference's union_a_and_b does, cuda/PSDBSCAN.hcu:76-107) and
// keeps for every non-core unique its minimum core neighbour (atomicMin: the
// same border rule as the edge-list path).  Both are order-independent.
__device__ __forceinline__ uint32_t sweep_find(uint32_t *p, uint32_t x) {
    volatile uint32_t *vp = p;
    while (true) {   // parent[y] <= y: x strictly decreases
        const uint32_t px = vp[x];
        if (px == x) return x;
        const uint32_t ppx = vp[px];
        if (ppx == px) return px;
        vp[x] = ppx;   // path halving
        x = ppx;
    }
}

__device__ __noinline__ void sink_streamed(const DistArgs &a, uint32_t lo, uint32_t hi) {
    if (a.sink == kSinkCount) {
        atomicAdd(&a.cnt[lo], __ldg(&a.ucopies[hi]));
        atomicAdd(&a.cnt[hi], __ldg(&a.ucopies[lo]));
        return;
    }
    const uint32_t clo = a.ucore[lo], chi = a.ucore[hi];
    if (clo != chi) {
        atomicMin(&a.bmin[clo ? hi : lo], clo ? lo : hi);
        return;
    }
    if (!clo) return;
    uint32_t x = lo, y = hi, it = 0;
    for (; it < kSpinCap; ++it) {
        uint32_t rx = sweep_find(a.parent, x), ry = sweep_find(a.parent, y);
        if (rx == ry) break;
        if (rx < ry) { const uint32_t t = rx; rx = ry; ry = t; }
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
    } else {
        sink_streamed(a, lo, hi);
    }
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Edge writer: each warp reserves kEdgeChunk slots at a time; slots a warp
// does not fill are set to the sentinel (x = kNone) before it moves on.
struct EdgeWriter {
    uint64_t base;     // kNone64 = no chunk held
    uint32_t fill;
    uint32_t written;
    static constexpr uint64_t kNoChunk = ~0ull;

    __device__ void init() { base = kNoChunk; fill = 0; written = 0; }

    __device__ void pad(const DistArgs &a, int lane) {
        if (base == kNoChunk || a.sink != kSinkEdges) return;
        for (uint32_t t = fill + lane; t < kEdgeChunk; t += 32) {
            const uint64_t slot = base + t;
            if (slot < a.cap_edges) a.edges[slot] = make_uint2(kNone, kNone);
        }
    }

    // warp-uniform call; lanes with ok=true append (lo, hi)
    __device__ void append(const DistArgs &a, int lane, bool ok, uint32_t lo, uint32_t hi) {
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, ok);
        if (!m) return;
        const uint32_t n = __popc(m);
        if (base == kNoChunk || fill + n > kEdgeChunk) {
            pad(a, lane);
            uint32_t b = 0;
            if (lane == 0) b = atomicAdd(&a.ctr->edge_reserved, kEdgeChunk);
            b = __shfl_sync(0xFFFFFFFFu, b, 0);
            base = b;
            fill = 0;
            if ((uint64_t)b + kEdgeChunk > a.cap_edges && lane == 0)
                atomicOr(&a.ctr->error, kErrEdgeOverflow);
        }
        if (ok) put_edge(a, base + fill + __popc(m & lanemask_lt()), lo, hi);
        fill += n;
        written += n;
    }

    // Bulk append, warp-uniform: the warp appends T edges at logical positions
    // 0..T-1 (each lane knows its own); the room left in the held chunk is
    // used first, then as many new chunks as needed, reserved with one atomic.
    struct Bulk { uint64_t b0; uint32_t f0; uint64_t nb; };
    __device__ Bulk reserve(const DistArgs &a, int lane, uint32_t T) {
        Bulk k;
        k.f0 = base == kNoChunk ? kEdgeChunk : fill;
        k.b0 = base;
        k.nb = kNoChunk;
        const uint32_t room = kEdgeChunk - k.f0;
        if (T > room) {
            const uint32_t nch = (T - room + kEdgeChunk - 1) / kEdgeChunk;
            uint32_t nb = 0;
            if (lane == 0) nb = atomicAdd(&a.ctr->edge_reserved, nch * kEdgeChunk);
            nb = __shfl_sync(0xFFFFFFFFu, nb, 0);
            if ((uint64_t)nb + (uint64_t)nch * kEdgeChunk > a.cap_edges && lane == 0)
                atomicOr(&a.ctr->error, kErrEdgeOverflow);
            k.nb = nb;
            base = (uint64_t)nb + (uint64_t)(nch - 1) * kEdgeChunk;
            fill = (T - room) - (nch - 1) * kEdgeChunk;
        } else {
            fill = k.f0 + T;
        }
        written += T;
        return k;
    }
    __device__ __forceinline__ uint64_t slot_of(const Bulk &k, uint32_t i) const {
        const uint32_t room = kEdgeChunk - k.f0;
        return i < room ? k.b0 + k.f0 + i : k.nb + (i - room);
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

// Bulk append of a lane's edges given as bits: bit b stands for pair index
// p0 + stride*b of a small or tiny bin pair (i, j from the pair index; the
// unique ids from the side records).  Warp-uniform.
__device__ __forceinline__ void emit_pair_bits(const DistArgs &a, EdgeWriter &ew, int lane,
                                               uint32_t bits, uint32_t p0, uint32_t stride,
                                               bool same, uint32_t n, uint32_t xstart,
                                               uint32_t ystart) {
    const uint32_t c = (uint32_t)__popc(bits);
    uint32_t incl = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += t;
    }
    const uint32_t T = __shfl_sync(0xFFFFFFFFu, incl, 31);
    if (T == 0) return;
    const EdgeWriter::Bulk bk = ew.reserve(a, lane, T);
    uint32_t k = incl - c;
    for (uint32_t b = bits; b; b &= b - 1) {
        const uint32_t p = p0 + stride * ((uint32_t)__ffs(b) - 1u);
        uint32_t i, j;
        small_pair(p, same, n, i, j);
        const uint32_t ux = __ldg(&a.meta[xstart + i].w), uy = __ldg(&a.meta[ystart + j].w);
        put_edge(a, ew.slot_of(bk, k++), min(ux, uy), max(ux, uy));
    }
}

// Small bin pairs of a warp: the warp claims kSmallBatch schedule positions
// with one atomic, each lane loads one of their bin pairs, and while one bin
// pair is scored the next one's records are prefetched into L1 (a small bin
// pair is otherwise a chain of dependent loads: position, bin pair, records).
constexpr uint32_t kSmallBatch = 16;

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
// Deferred hits: the tiled loops only record, per lane, (y index in the staged
// chunk, hit bits) in a small shared-memory queue; the queue is drained here when
// a lane's queue is full or the chunk ends, with every lane taking part.
constexpr int kHitQ = 8;   // queued (y, hits) records per lane
constexpr uint32_t kOff = 0x40000000u;   // score of a masked x-entry (never a hit)

// The queue holds (y index in the chunk, hit bits) per lane.  Hits are
// compacted over the whole warp before they are written: each lane first keeps
// the bits of its own queue that are edges (check(r, t, my): x-entry 32 r + lane
// against y-entry t of the chunk, whose side record is my; `decided`: the
// hits were checked when they were queued), then one warp scan gives every
// lane its place in one bulk append.
template <typename Check>
__device__ __forceinline__ void drain_hits(const DistArgs &a, EdgeWriter &ew, uint32_t *q,
                                           uint32_t qn, const uint4 *xm, const uint4 *ym, int lane,
                                           bool decided, Check check) {
    uint32_t c = 0;
    for (uint32_t k = 0; k < qn; ++k) {
        const uint32_t e = q[k * 32 + lane];
        uint32_t keep = e & 0xFFu;
        if (!decided) {
            const uint32_t t = e >> 8;
            const uint4 my = ym[t];
            for (uint32_t b = keep; b; b &= b - 1) {
                const uint32_t r = (uint32_t)__ffs(b) - 1u;
                if (!check(r, t, my)) keep &= ~(1u << r);
            }
            q[k * 32 + lane] = (t << 8) | keep;
        }
        c += (uint32_t)__popc(keep);
    }
    uint32_t incl = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t n = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += n;
    }
    const uint32_t T = __shfl_sync(0xFFFFFFFFu, incl, 31);
    if (T == 0) return;
    const EdgeWriter::Bulk bk = ew.reserve(a, lane, T);
    uint32_t i = incl - c;
    for (uint32_t k = 0; k < qn; ++k) {
        const uint32_t e = q[k * 32 + lane];
        const uint32_t uy = ym[e >> 8].w;
        for (uint32_t b = e & 0xFFu; b; b &= b - 1) {
            const uint32_t r = (uint32_t)__ffs(b) - 1u;
            const uint32_t ux = xm[32 * r + lane].w;
            put_edge(a, ew.slot_of(bk, i++), min(ux, uy), max(ux, uy));
        }
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
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (grid <= 0) grid = occupancy_grid(kernel, smem);
    kernel<<<grid, kWarps * 32, smem, s>>>(a);
}

}  // namespace
}  // namespace idb
