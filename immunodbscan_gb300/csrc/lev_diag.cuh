// lev_diag.cuh -- the neighbour search for edit distances up to kLevDiagMaxEps.
//
// Reference: the anti-diagonal DP of levenshtein_distance
// (cuda/PSDBSCAN.hcu:246-290), one block per pair.  Here a pair costs no
// recurrence over columns: both sequences are bit planes (as for Hamming), the
// mismatch masks of the few diagonals an alignment within eps can visit are
// BP logic operations per word each, and the furthest-reaching test on them
// (lev_diag, bitops.cuh) is exact, so it needs no filter in front of it.
//
// Integer-pipe bound (eps 2, equal lengths, one word, 5 planes: 15 LOP3 for three
// masks + 14 for the test).  The y-records are staged with one copy per diagonal,
// already shifted, so the tiled loop reads them as 16-byte broadcasts and does
// no shifts per pair; RX x-entries per lane share every broadcast.  Against the
// filters + Myers kernel it replaces for these eps (whole calls): 200,000
// nucleotide rows, eps 2: 15.2 -> 1.5 ms; 1M rows with skewed gene usage, eps 2
// (38.9e9 pairs): 95.9 -> 41.2 ms; 2M rows, eps min(3, 0.15 L): 72.0 -> 32.4 ms.
#pragma once
#include "distance_common.cuh"

namespace idb {

namespace {

// A unit with at most this many x-entries is scored pair by pair: a pair read from
// L1 costs about twice a tiled one, and a tile would leave 3/4 of the lanes idle.
constexpr uint32_t kThinX = 8;

template <int BP, int W>
struct LevShape {
    static constexpr int NW = BP * W;            // words per record
    static constexpr int R16 = (NW + 3) / 4;     // 16-byte words per record
    static constexpr int YMax = NW;              // 16-byte words of a staged y (4 diagonals)
    // y-records staged per batch, so that a block's static shared memory stays
    // below 48 KB
    static constexpr int YB = NW <= 15 ? kYB : 16;
};

template <int BP, int W>
__device__ __forceinline__ void load_planes(const uint4 *src, uint32_t (&v)[BP * W]) {
#pragma unroll
    for (int q = 0; q < LevShape<BP, W>::R16; ++q) {
        const uint4 u = __ldg(src + q);
        const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (4 * q + e < BP * W) v[4 * q + e] = w4[e];
    }
}

// One pair straight from its records, any admissible (eps, length gap): 0 iff
// within eps.  Out of line: the small bin pairs' lanes may hold different ones.
template <int BP, int W>
__device__ __noinline__ uint32_t lev_pair(const uint4 *xr, const uint4 *yr, uint32_t e, uint32_t g) {
    uint32_t x[BP * W], y[BP * W];
    load_planes<BP, W>(xr, x);
    load_planes<BP, W>(yr, y);
    switch (e * 4 + g) {
        case 0: return lev_planes<BP, W, 0, 0>(x, y);
        case 4: return lev_planes<BP, W, 1, 0>(x, y);
        case 5: return lev_planes<BP, W, 1, 1>(x, y);
        case 8: return lev_planes<BP, W, 2, 0>(x, y);
        case 9: return lev_planes<BP, W, 2, 1>(x, y);
        case 10: return lev_planes<BP, W, 2, 2>(x, y);
        case 12: return lev_planes<BP, W, 3, 0>(x, y);
        case 13: return lev_planes<BP, W, 3, 1>(x, y);
        case 14: return lev_planes<BP, W, 3, 2>(x, y);
        case 15: return lev_planes<BP, W, 3, 3>(x, y);
    }
    return 1u;
}

// Is a pair of a segment-join group that is within eps to be emitted from this
// group?  Its V and J sets must intersect, and the group's (segment k, shift)
// must be the first, in the order of the look-ups (k_lev_join.cu), at which x
// (the shorter; of two equal lengths the smaller unique id) holds a segment of
// y.  P.v is the segment, P.j the segment count.  mx, my: side records.
template <int BP, int W>
__device__ __noinline__ bool lev_join_ok(const DistArgs &a, const BinPair &P, const uint4 *xr,
                                         const uint4 *yr, const uint4 &mx, const uint4 &my) {
    const int m = P.la, n = P.lb, gap = n - m, S = P.j, e = S - 1, kg = P.v;
    int dg = 0;   // the group's shift
    if (P.same) {
        if (mx.w > my.w) { const uint4 *t = xr; xr = yr; yr = t; }
    } else {
        if (gap == 0 && mx.w >= my.w) return false;   // found from the other side (or itself)
        dg = max(-kg, -gap - (e - kg)) + (int)(mx.z >> 30);
    }
    if (a.vj_meta) {
        if (((mx.x & my.x) | (mx.y & my.y)) == 0 || (mx.z & my.z & 0x3FFFFFFFu) == 0) return false;
    } else if (!vj_intersect(a, mx.w, my.w)) {
        return false;
    }
    uint32_t x[BP * W], y[BP * W];
    load_planes<BP, W>(xr, x);
    load_planes<BP, W>(yr, y);
    for (int k = 0; k <= kg; ++k) {
        const int s = k * n / S, len = (k + 1) * n / S - s;
        const int lo = max(-k, -gap - (e - k)), hi = min(k, e - k - gap);
        for (int d = lo; d <= hi; ++d) {
            const int pos = s + d;
            if (pos < 0 || pos + len > m) continue;
            uint32_t diff[W];
#pragma unroll
            for (int w = 0; w < W; ++w) diff[w] = 0;
#pragma unroll
            for (int p = 0; p < BP; ++p) {
                uint32_t in[W], sh[W];
#pragma unroll
                for (int w = 0; w < W; ++w) in[w] = y[p * W + w];
                shift_words<W>(in, -d, sh);            // bit i: y[i - d]
#pragma unroll
                for (int w = 0; w < W; ++w) diff[w] |= x[p * W + w] ^ sh[w];
            }
            uint32_t any = 0;
#pragma unroll
            for (int w = 0; w < W; ++w) {
                const int a0 = max(pos - 32 * w, 0), a1 = min(pos + len - 32 * w, 32);
                if (a0 < a1) any |= diff[w] & (low_mask32(a1) & ~low_mask32(a0));
            }
            const bool here = k == kg && d == dg;
            if (any == 0) return here;
            if (here) return false;   // the key was shared by its hash only
        }
    }
    return false;
}

template <int BP, int W>
__device__ __forceinline__ bool lev_is_edge(const DistArgs &a, const BinPair &P, uint32_t xrow, uint32_t yrow,
                                            const uint4 &mx, const uint4 &my) {
    constexpr int R16 = LevShape<BP, W>::R16;
    if (!a.join) return canonical_meta(a, P, mx, my);
    return lev_join_ok<BP, W>(a, P, a.rec + (size_t)xrow * R16, a.rec + (size_t)yrow * R16, mx, my);
}

// A warp's shared memory.
struct LevSlice {
    uint4 *sy;       // staged y-records, one shifted copy per diagonal
    uint32_t *seg;   // segment join: masks of the look-ups (LevLookups)
    TileSlice T;
};

// The look-ups of a length pair (k_lev_join.cu) are the cells of the diagonal test:
// segment k at shift delta is diagonal d = -delta, and x holds it iff the mask of
// diagonal d has no bit in x's positions of the segment.  A unit keeps, in the
// order of the look-ups, those position masks, then (equal lengths) the masks
// of the unshifted segments for pairs taken the other way round.
template <int E, int G, int W>
struct LevLookups {
    using Dg = LevDiags<E, G>;
    static constexpr int count() {
        int n = 0;
        for (int k = 0; k <= E; ++k)
            for (int d = G + Dg::lo; d >= -Dg::lo; --d) n += Dg::cell(d, k);
        return n;
    }
    static constexpr int n = count();
    static constexpr int words = (n + E + 1) * W;
    // lanes write the masks; returns a bit per look-up that lies inside x
    static __device__ __forceinline__ uint32_t fill(uint32_t *seg, int m, int len_y, int lane) {
        uint32_t valid = 0;
        int idx = 0;
#pragma unroll
        for (int k = 0; k <= E; ++k) {
            const int s = k * len_y / (E + 1), t = (k + 1) * len_y / (E + 1);
#pragma unroll
            for (int d = G + Dg::lo; d >= -Dg::lo; --d) {
                if (!Dg::cell(d, k)) continue;
                const int a = s - d, b = t - d;
                if (a >= 0 && b <= m) valid |= 1u << idx;
#pragma unroll
                for (int w = 0; w < W; ++w)
                    if (lane == w) seg[idx * W + w] = word_mask(a, b, w);
                ++idx;
            }
#pragma unroll
            for (int w = 0; w < W; ++w)
                if (lane == w) seg[(n + k) * W + w] = word_mask(s, t, w);
        }
        return valid;
    }
    // bits of word w at positions [a, b)
    static __device__ __forceinline__ uint32_t word_mask(int a, int b, int w) {
        const int a0 = min(max(a - 32 * w, 0), 32), b0 = min(max(b - 32 * w, 0), 32);
        return low_mask32(b0) & ~low_mask32(a0);
    }
    // number of the first look-up of segment kg
    static __device__ __forceinline__ uint32_t base(int kg) {
        uint32_t n = 0;
#pragma unroll
        for (int k = 0; k < E; ++k)
#pragma unroll
            for (int d = G + Dg::lo; d >= -Dg::lo; --d)
                if (Dg::cell(d, k) && k < kg) ++n;
        return n;
    }
    // Emitted here: of the look-ups that hold (valid: lies inside x), the group's
    // own is the first.  D: the pair's mismatch masks.
    static __device__ __forceinline__ bool first(const uint32_t (&D)[Dg::n][W], const uint32_t *seg,
                                                 uint32_t valid, uint32_t own, bool swapped) {
        uint32_t holds = 0;
        int idx = 0;
#pragma unroll
        for (int k = 0; k <= E; ++k)
#pragma unroll
            for (int d = G + Dg::lo; d >= -Dg::lo; --d) {
                if (!Dg::cell(d, k)) continue;
                uint32_t any = 0;
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    if (G == 0 && d != 0)
                        any |= (swapped ? D[(G == 0 ? -d : d) + Dg::lo][w] : D[d + Dg::lo][w]) &
                               seg[(swapped ? n + k : idx) * W + w];
                    else
                        any |= D[d + Dg::lo][w] & seg[idx * W + w];
                }
                if (any == 0) holds |= 1u << idx;
                ++idx;
            }
        return ((holds & valid) & (0xFFFFFFFFu >> (31 - own))) == 1u << own;
    }
};

// One tiled unit: 32*RX x-entries in registers against the unit's y-entries.
template <int BP, int W, int RX, int E, int G>
__device__ __forceinline__ void lev_unit(const DistArgs &a, EdgeWriter &ew, const Unit &U,
                                         const LevSlice &S, int lane, uint64_t &pairs) {
    using Sh = LevShape<BP, W>;
    using Dg = LevDiags<E, G>;
    constexpr int NW = Sh::NW;
    constexpr int Y16 = (Dg::n * NW + 3) / 4;    // 16-byte words of a staged y
    static_assert(Y16 <= Sh::YMax, "staged y-record size");
    using Lk = LevLookups<E, G, W>;
    const bool same = U.P.same != 0;
    uint32_t x[RX][NW];
    // segment join: the group's look-up, plus a per-entry shift for the classes
    // that looked it up (the group's own uniques: no shift, the middle one)
    const int kg = U.P.v;
    const uint32_t own = Lk::base(kg) + (same ? (uint32_t)min(kg, E - kg) : 0u);
    const uint32_t valid = a.join ? Lk::fill(S.seg, U.P.la, U.P.lb, lane) : 0u;
    // Segment join: may a pair within eps be emitted from this group?  (V and J
    // sets intersect; of equal lengths the smaller id looks the larger one up.)
    auto join_edge = [&](const uint32_t (&D)[Dg::n][W], const uint4 &mx, const uint4 &my) {
        if (a.vj_meta && (((mx.x & my.x) | (mx.y & my.y)) == 0 || (mx.z & my.z & 0x3FFFFFFFu) == 0)) return false;
        if (G == 0 && !same && mx.w >= my.w) return false;
        return Lk::first(D, S.seg, valid, own + (same ? 0u : mx.z >> 30), G == 0 && same && mx.w > my.w);
    };
#pragma unroll
    for (int r = 0; r < RX; ++r) {
        const uint32_t xi = (uint32_t)r * 32 + lane;
        const bool ok = xi < U.nx;
        const uint32_t row = U.P.a_start + U.xbase + (ok ? xi : 0);
        load_planes<BP, W>(a.rec + (size_t)row * Sh::R16, x[r]);
        S.T.begin_x(a, xi, row);
        if (ok) pairs += unit_pairs(U, U.xbase + xi);
    }
    const uint32_t yrow0 = (same ? U.P.a_start : U.P.b_start) + U.ybase;
    // same bin: y-entries at or before the first x-entry pair with nothing
    const uint32_t y0 = (same && U.xbase >= U.ybase) ? min(U.ny, U.xbase - U.ybase + 1) : 0u;
    for (uint32_t yb = y0; yb < U.ny; yb += Sh::YB) {
        const uint32_t nb = min((uint32_t)Sh::YB, U.ny - yb);
        __syncwarp();
        for (uint32_t t = lane; t < nb; t += 32) {
            uint32_t y[NW], o[4 * Y16];
            load_planes<BP, W>(a.rec + (size_t)(yrow0 + yb + t) * Sh::R16, y);
#pragma unroll
            for (int q = 0; q < Dg::n; ++q)
#pragma unroll
                for (int p = 0; p < BP; ++p) {
                    uint32_t in[W], sh[W];
#pragma unroll
                    for (int w = 0; w < W; ++w) in[w] = y[p * W + w];
                    shift_words<W>(in, q - Dg::lo, sh);
#pragma unroll
                    for (int w = 0; w < W; ++w) o[q * NW + p * W + w] = sh[w];
                }
#pragma unroll
            for (int k = Dg::n * NW; k < 4 * Y16; ++k) o[k] = 0u;
#pragma unroll
            for (int k = 0; k < Y16; ++k)
                S.sy[t * Y16 + k] = make_uint4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
            S.T.begin_y(a, t, yrow0 + yb + t);
        }
        __syncwarp();
        // y-entries inside the unit's own x range (same bin) need the mask of the
        // x-entries before them; they come first in the chunk
        uint32_t tdiag = 0;
        if (same && U.ybase + yb < U.xbase + U.nx) tdiag = min(nb, U.xbase + U.nx - (U.ybase + yb));
        uint32_t hits[RX];                // bit t: within eps of y-entry t of the batch
#pragma unroll
        for (int r = 0; r < RX; ++r) hits[r] = 0u;
        for (uint32_t t = 0; t < nb; ++t) {
            uint32_t y[4 * Y16];
#pragma unroll
            for (int k = 0; k < Y16; ++k) {
                const uint4 v = S.sy[t * Y16 + k];
                y[4 * k] = v.x; y[4 * k + 1] = v.y; y[4 * k + 2] = v.z; y[4 * k + 3] = v.w;
            }
            uint32_t sc[RX];
#pragma unroll
            for (int r = 0; r < RX; ++r) {
                uint32_t D[Dg::n][W];
#pragma unroll
                for (int q = 0; q < Dg::n; ++q)
#pragma unroll
                    for (int w = 0; w < W; ++w) {
                        uint32_t d = x[r][w] ^ y[q * NW + w];
#pragma unroll
                        for (int p = 1; p < BP; ++p) d |= x[r][p * W + w] ^ y[q * NW + p * W + w];
                        D[q][w] = d;
                    }
                sc[r] = lev_diag<W, E, G>(D);
            }
            if (t < tdiag) {
                const uint32_t nact = U.ybase + yb + t - U.xbase;   // x-entries before y
#pragma unroll
                for (int r = 0; r < RX; ++r)
                    if ((uint32_t)r * 32 + lane >= nact) sc[r] |= kOff;
            }
#pragma unroll
            for (int r = 0; r < RX; ++r)
                if (sc[r] == 0) hits[r] |= 1u << t;
        }
        uint32_t any = 0;
#pragma unroll
        for (int r = 0; r < RX; ++r) {    // lanes past the unit's end hold a copy of its first entry
            if ((uint32_t)r * 32 + lane >= U.nx) hits[r] = 0u;
            any |= hits[r];
        }
        if (__any_sync(0xFFFFFFFFu, any)) {
            // Which hits are emitted here.  Checked per batch, not in the loop
            // above, where one hit in a warp would make all of it wait for the
            // check (2M rows, 0.15e9 neighbours: 9.2 against 7.4 ms).
#pragma unroll
            for (int r = 0; r < RX; ++r) {
                const uint4 mx = S.T.xm[32 * r + lane];
                for (uint32_t b = hits[r]; b; b &= b - 1) {
                    const uint32_t t = (uint32_t)__ffs(b) - 1u;
                    const uint4 my = S.T.ym[t];
                    bool ok;
                    if (a.join) {
                        const uint32_t *ys = reinterpret_cast<const uint32_t *>(S.sy + t * Y16);
                        uint32_t D[Dg::n][W];
#pragma unroll
                        for (int q = 0; q < Dg::n; ++q)
#pragma unroll
                            for (int w = 0; w < W; ++w) {
                                uint32_t d = x[r][w] ^ ys[q * NW + w];
#pragma unroll
                                for (int p = 1; p < BP; ++p) d |= x[r][p * W + w] ^ ys[q * NW + p * W + w];
                                D[q][w] = d;
                            }
                        ok = join_edge(D, mx, my) && (a.vj_meta || vj_intersect(a, mx.w, my.w));
                    } else {
                        ok = canonical_meta(a, U.P, mx, my);
                    }
                    if (!ok) hits[r] &= ~(1u << t);
                }
            }
            emit_batch<RX>(a, ew, S.T, hits, nb, lane);
        }
    }
    S.T.end_x(a, U.nx, lane);
}

// A unit whose x-chunk fills at most one 32-lane block takes the one-block loop.
template <int BP, int W, int RX, int E, int G>
__device__ __forceinline__ void lev_unit_rx(const DistArgs &a, EdgeWriter &ew, const Unit &U,
                                            const LevSlice &S, int lane, uint64_t &pairs) {
    if (RX > 1 && U.nx <= 32) lev_unit<BP, W, 1, E, G>(a, ew, U, S, lane, pairs);
    else lev_unit<BP, W, RX, E, G>(a, ew, U, S, lane, pairs);
}

// Pairs of n x-entries with m y-entries, at most 32 each (same: pairs of the n),
// lanes taking pairs and reading their records from L1.
template <int BP, int W>
__device__ __forceinline__ void lev_pair_block(const DistArgs &a, EdgeWriter &ew, const TileSlice &T,
                                               const BinPair &P, bool same, uint32_t xstart, uint32_t n,
                                               uint32_t ystart, uint32_t m, int lane) {
    constexpr int R16 = LevShape<BP, W>::R16;
    const uint32_t npairs = same ? n * (n - 1) / 2 : n * m;
    uint32_t rmask = 0;           // bit i: the lane's pair of round i is an edge
    for (uint32_t p0 = 0; p0 < npairs; p0 += 32) {
        const uint32_t p = p0 + lane;
        if (p >= npairs) break;
        uint32_t i, j;
        small_pair(p, same, n, i, j);
        const uint32_t xrow = xstart + i, yrow = ystart + j;
        if (lev_pair<BP, W>(a.rec + (size_t)xrow * R16, a.rec + (size_t)yrow * R16, (uint32_t)P.eps,
                            (uint32_t)(P.lb - P.la)) == 0 &&
            lev_is_edge<BP, W>(a, P, xrow, yrow, __ldg(a.meta + xrow), __ldg(a.meta + yrow)))
            rmask |= 1u << (p0 >> 5);
    }
    __syncwarp();
    emit_pair_bits(a, ew, T, lane, rmask, same, n, m, xstart, ystart);
}

// Small bin pairs (at most kSmallSide entries a side): a warp each, lanes take
// pairs and read their records from L1 (the next bin pair's are prefetched).
template <int BP, int W>
__device__ __forceinline__ void lev_small_all(const DistArgs &a, EdgeWriter &ew, const TileSlice &T, int lane,
                                              uint64_t &pairs) {
    constexpr int R16 = LevShape<BP, W>::R16;
    const uint32_t n_small = a.ctr->n_small, batch = small_batch(n_small);
    for (;;) {
        uint32_t s0 = 0;
        if (lane == 0) s0 = atomicAdd(&a.ctr->small_cursor, batch);
        s0 = __shfl_sync(0xFFFFFFFFu, s0, 0);
        if (s0 >= n_small) break;
        const uint32_t cnt = min(batch, n_small - s0);
        uint32_t myidx = 0;
        BinPair myP;
        memset(&myP, 0, sizeof(BinPair));
        if ((uint32_t)lane < cnt) {
            myidx = a.small_list[s0 + lane];
            myP = a.bp[myidx];
        }
        for (uint32_t k = 0; k < cnt; ++k) {
            if (k + 1 < cnt) {
                const uint32_t na = __shfl_sync(0xFFFFFFFFu, myP.a_start, k + 1);
                const uint32_t nn = __shfl_sync(0xFFFFFFFFu, myP.a_n, k + 1);
                const uint32_t nb = __shfl_sync(0xFFFFFFFFu, myP.b_start, k + 1);
                const uint32_t nm = __shfl_sync(0xFFFFFFFFu, myP.b_n, k + 1);
                if ((uint32_t)lane < nn) prefetch_l1(a.rec + (size_t)(na + lane) * R16);
                if ((uint32_t)lane < nm) prefetch_l1(a.rec + (size_t)(nb + lane) * R16);
            }
            const BinPair P = shfl_binpair(myP, (int)k);
            const uint32_t idx = __shfl_sync(0xFFFFFFFFu, myidx, k);
            const long long t0 = a.bp_cycles ? clock64() : 0;
            const bool same = P.same != 0;
            const uint32_t n = P.a_n, npairs = same ? n * (n - 1) / 2 : n * P.b_n;
            const uint32_t ystart = same ? P.a_start : P.b_start;
            if (lane == 0) pairs += npairs;
            lev_pair_block<BP, W>(a, ew, T, P, same, P.a_start, n, ystart, P.b_n, lane);
            if (a.bp_cycles && lane == 0)
                atomicAdd(&a.bp_cycles[idx], (unsigned long long)(clock64() - t0));
        }
    }
}

// Tiny bin pairs (at most kTinyPairs pairs): one lane takes every pair of one of
// them, 32 at a time.
template <int BP, int W>
__device__ __forceinline__ void lev_tiny_all(const DistArgs &a, EdgeWriter &ew, int lane,
                                             uint64_t &pairs) {
    constexpr int R16 = LevShape<BP, W>::R16;
    const uint32_t n_tiny = a.ctr->n_tiny;
    for (;;) {
        uint32_t s0 = 0;
        if (lane == 0) s0 = atomicAdd(&a.ctr->tiny_cursor, 32u);
        s0 = __shfl_sync(0xFFFFFFFFu, s0, 0);
        if (s0 >= n_tiny) break;
        const long long t0 = a.bp_cycles ? clock64() : 0;
        const bool act = s0 + (uint32_t)lane < n_tiny;
        uint32_t idx = 0;
        BinPair P;
        memset(&P, 0, sizeof(BinPair));
        if (act) {
            idx = a.small_list[a.small_cap - 1u - (s0 + (uint32_t)lane)];
            P = a.bp[idx];
        }
        const bool same = P.same != 0;
        const uint32_t n = P.a_n, np = same ? n * (n - 1) / 2 : n * P.b_n;
        const uint32_t ystart = same ? P.a_start : P.b_start;
        pairs += np;
        static_assert(kTinyPairs <= 32, "tiny pair mask");
        uint32_t emask = 0;
        for (uint32_t p = 0; p < np; ++p) {
            uint32_t i, j;
            small_pair(p, same, n, i, j);
            const uint32_t xrow = P.a_start + i, yrow = ystart + j;
            if (lev_pair<BP, W>(a.rec + (size_t)xrow * R16, a.rec + (size_t)yrow * R16, (uint32_t)P.eps,
                                (uint32_t)(P.lb - P.la)) == 0 &&
                lev_is_edge<BP, W>(a, P, xrow, yrow, __ldg(a.meta + xrow), __ldg(a.meta + yrow)))
                emask |= 1u << p;
        }
        __syncwarp();
        // two bins: their pairs one by one (few: most tiny groups are one bin's)
        emit_tiny_bits(a, ew, lane, same ? emask : 0u, n, P.a_start);
        __syncwarp();
        uint32_t rest = same ? 0u : emask;
        for (uint32_t it = 0; it < kTinyPairs && __any_sync(0xFFFFFFFFu, rest); ++it) {
            uint32_t ux = 0, uy = 0;
            if (rest) {
                const uint32_t p = (uint32_t)__ffs(rest) - 1u;
                ux = __ldg(&a.meta[P.a_start + p % n].w);
                uy = __ldg(&a.meta[ystart + p / n].w);
            }
            ew.append<true>(a, lane, rest != 0, min(ux, uy), max(ux, uy));
            rest &= rest - 1;
        }
        if (a.bp_cycles) {   // the batch's cycles, shared out by pairs
            const uint32_t tot = __reduce_add_sync(0xFFFFFFFFu, np);
            const unsigned long long dt = (unsigned long long)(clock64() - t0);
            if (act) atomicAdd(&a.bp_cycles[idx], dt * np / (tot ? tot : 1u));
        }
    }
}

template <int BP, int W, int RX>
__global__ void __launch_bounds__(kWarps * 32, (W <= 2 ? 4 : 3))
k_lev_diag(const __grid_constant__ DistArgs a) {
    using Sh = LevShape<BP, W>;
    __shared__ uint4 sy[kWarps][Sh::YB * Sh::YMax];
    __shared__ uint4 sym[kWarps][32];
    __shared__ uint4 sxm[kWarps][32 * RX];
    __shared__ uint32_t seg[kWarps][LevLookups<3, 0, W>::words];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t n_units = a.ctr->n_units, n_bp = a.ctr->n_binpairs;
    __shared__ uint32_t scp[kWarps][2 * 32 * RX + 2 * 32];   // copies and sums (TileSlice)
    const LevSlice S{sy[wid], seg[wid],
                     {sxm[wid], sym[wid], scp[wid], scp[wid] + 2 * 32 * RX, scp[wid] + 32 * RX,
                      scp[wid] + 2 * 32 * RX + 32}};
    EdgeWriter ew;
    ew.init();
    uint64_t pairs = 0;
    Unit U;
    while (next_unit(a, n_units, n_bp, lane, U)) {
        if (!U.P.same && U.nx <= kThinX) {   // too few x-entries for the lanes: pair by pair
            if (lane == 0) pairs += (uint64_t)U.nx * U.ny;
            for (uint32_t y = 0; y < U.ny; y += 32)
                lev_pair_block<BP, W>(a, ew, S.T, U.P, false, U.P.a_start + U.xbase, U.nx,
                                      U.P.b_start + U.ybase + y, min(32u, U.ny - y), lane);
            log_unit(a, U, lane);
            continue;
        }
        switch ((uint32_t)U.P.eps * 4 + (uint32_t)(U.P.lb - U.P.la)) {
            case 0: lev_unit_rx<BP, W, RX, 0, 0>(a, ew, U, S, lane, pairs); break;
            case 4: lev_unit_rx<BP, W, RX, 1, 0>(a, ew, U, S, lane, pairs); break;
            case 5: lev_unit_rx<BP, W, RX, 1, 1>(a, ew, U, S, lane, pairs); break;
            case 8: lev_unit_rx<BP, W, RX, 2, 0>(a, ew, U, S, lane, pairs); break;
            case 9: lev_unit_rx<BP, W, RX, 2, 1>(a, ew, U, S, lane, pairs); break;
            case 10: lev_unit_rx<BP, W, RX, 2, 2>(a, ew, U, S, lane, pairs); break;
            case 12: lev_unit_rx<BP, W, RX, 3, 0>(a, ew, U, S, lane, pairs); break;
            case 13: lev_unit_rx<BP, W, RX, 3, 1>(a, ew, U, S, lane, pairs); break;
            case 14: lev_unit_rx<BP, W, RX, 3, 2>(a, ew, U, S, lane, pairs); break;
            case 15: lev_unit_rx<BP, W, RX, 3, 3>(a, ew, U, S, lane, pairs); break;
        }
        log_unit(a, U, lane);
    }
    lev_small_all<BP, W>(a, ew, S.T, lane, pairs);
    lev_tiny_all<BP, W>(a, ew, lane, pairs);
    finish(a, ew, pairs, lane);
}

template <int BP>
void launch_lev_diag(const Plan &P, const DistArgs &a, int grid, cudaStream_t s) {
    switch (P.W) {
        case 1:
            if (P.RX == 2) run(k_lev_diag<BP, 1, 2>, a, 0, grid, s);
            else run(k_lev_diag<BP, 1, 1>, a, 0, grid, s);
            break;
        case 2: run(k_lev_diag<BP, 2, 1>, a, 0, grid, s); break;
        case 3: run(k_lev_diag<BP, 3, 1>, a, 0, grid, s); break;
        default: run(k_lev_diag<BP, 4, 1>, a, 0, grid, s); break;
    }
}

}  // namespace
}  // namespace idb
