// hamming.cuh -- the neighbour search for Hamming distances on bit-plane records:
// tiled units, small bin pairs pair-parallel, tiny ones a lane each; with bucket
// or segment-join candidates.
//
// Reference: half_hamming_core_points / fuse_hamming_clusters
// (cuda/PSDBSCAN.hcu:585-657, 664-742).
#pragma once
#include "distance_common.cuh"

namespace idb {

namespace {

// Segment join with the gene bits in the side records: V and J sets intersect,
// segment k (the group's) is identical and no lower segment is, read from the
// difference words d[w] (bit i of word w: residue 32w+i differs) of the
// length-L pair split into S segments.  Groups are keyed by a hash of the
// segment, so the test on segment k itself keeps a shared key of two different
// segments from emitting a pair twice.
template <int W>
__device__ __forceinline__ bool join_meta_ok(const uint4 &mx, const uint4 &my, const uint32_t (&d)[W],
                                             uint32_t L, uint32_t S, uint32_t k) {
    if (((mx.x & my.x) | (mx.y & my.y)) == 0) return false;
    if ((mx.z & my.z & 0x3FFFFFFFu) == 0) return false;
    for (uint32_t kk = 0; kk <= k; ++kk) {
        const uint32_t lo = kk * L / S, hi = (kk + 1) * L / S;
        uint32_t any = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const uint32_t a0 = max(lo, 32u * w), a1 = min(hi, 32u * w + 32u);
            if (a0 < a1) {
                const uint32_t n = a1 - a0;
                const uint32_t m = (n >= 32 ? 0xFFFFFFFFu : ((1u << n) - 1u)) << (a0 - 32u * w);
                any |= d[w] & m;
            }
        }
        if (kk < k && any == 0) return false;   // identical (or empty) lower segment: emitted there
        if (kk == k && any != 0) return false;  // segment k differs: a shared key only
    }
    return true;
}

// A small bin pair (at most kSmallSide entries a side), pair-parallel: lane l
// holds entry l of each side; each round the lanes take 32 pairs and fetch
// the two records by shuffles.  Canonicity of a hit is decided from the side
// records (global loads: hits are rare).
template <int BP, int W, int EM, bool JN>
__device__ __forceinline__ void hamming_small(const DistArgs &a, EdgeWriter &ew, const TileSlice &T,
                                              const BinPair &P, uint32_t idx, int lane, uint64_t &pairs) {
    constexpr int NW = BP * W;
    constexpr int R16 = (NW + 3) / 4;
    const long long t0 = a.bp_cycles ? clock64() : 0;
    const bool same = P.same != 0;
    const uint32_t n = P.a_n, m = same ? P.a_n : P.b_n;
    const uint32_t ystart = same ? P.a_start : P.b_start;
    uint32_t xr[NW], yr[NW];
    {
        const uint4 *src = a.rec + (size_t)(P.a_start + ((uint32_t)lane < n ? lane : 0)) * R16;
        const uint4 *srcy = a.rec + (size_t)(ystart + ((uint32_t)lane < m ? lane : 0)) * R16;
#pragma unroll
        for (int q = 0; q < R16; ++q) {
            const uint4 v = __ldg(src + q);
            const uint4 u = same ? v : __ldg(srcy + q);
            const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
            const uint32_t u4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (4 * q + e < NW) { xr[4 * q + e] = w4[e]; yr[4 * q + e] = u4[e]; }
        }
    }
    const uint32_t npairs = same ? n * (n - 1) / 2 : n * m;
    if (lane == 0) pairs += npairs;
    const uint32_t thr = EM == 0 ? (uint32_t)max(P.eps, 0) : 0u;
    const bool neg = EM == 0 && P.eps < 0;
    static_assert(kSmallSide * kSmallSide <= 32 * 32, "small round mask");
    uint32_t rmask = 0;           // bit k: the lane's pair of round k is an edge
    for (uint32_t p0 = 0; p0 < npairs && !neg; p0 += 32) {
        const uint32_t p = p0 + lane;
        const bool act = p < npairs;
        uint32_t i = 0, j = 0;
        if (act) small_pair(p, same, n, i, j);
        uint32_t sc;
        uint32_t dw[W];
        if (W == 1) {
            uint32_t d = __shfl_sync(0xFFFFFFFFu, xr[0], i) ^ __shfl_sync(0xFFFFFFFFu, yr[0], j);
#pragma unroll
            for (int q = 1; q < BP; ++q)
                d |= __shfl_sync(0xFFFFFFFFu, xr[q], i) ^ __shfl_sync(0xFFFFFFFFu, yr[q], j);
            dw[0] = d;
            sc = EM == 2 ? d : (EM == 1 ? (d & (d - 1u)) : (uint32_t)__popc(d));
        } else {
            uint32_t dist = 0;
#pragma unroll
            for (int w = 0; w < W; ++w) {
                uint32_t d = __shfl_sync(0xFFFFFFFFu, xr[w], i) ^ __shfl_sync(0xFFFFFFFFu, yr[w], j);
#pragma unroll
                for (int q = 1; q < BP; ++q)
                    d |= __shfl_sync(0xFFFFFFFFu, xr[q * W + w], i) ^
                         __shfl_sync(0xFFFFFFFFu, yr[q * W + w], j);
                dw[w] = d;
                dist += __popc(d);
            }
            sc = dist;
        }
        if (act && sc <= thr) {
            const uint4 mx = __ldg(a.meta + P.a_start + i), my = __ldg(a.meta + ystart + j);
            bool ok;
            if (JN) ok = join_meta_ok<W>(mx, my, dw, P.la, P.j, P.v);
            else ok = canonical_meta(a, P, mx, my);
            rmask |= (uint32_t)ok << (p0 >> 5);
        }
    }
    // every round's edges of the lane, one bulk append for the warp
    emit_pair_bits(a, ew, T, lane, rmask, same, n, m, P.a_start, ystart);
    if (a.bp_cycles && lane == 0)
        atomicAdd(&a.bp_cycles[idx], (unsigned long long)(clock64() - t0));
}

template <int BP, int W, int EM, bool JN>
__device__ __forceinline__ void hamming_small_all(const DistArgs &a, EdgeWriter &ew, const TileSlice &T,
                                                  int lane, uint64_t &pairs) {
    constexpr int R16 = (BP * W + 3) / 4;
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
        for (uint32_t g = 0; g < cnt; ++g) {
            if (g + 1 < cnt) {
                const uint32_t na = __shfl_sync(0xFFFFFFFFu, myP.a_start, g + 1);
                const uint32_t nn = __shfl_sync(0xFFFFFFFFu, myP.a_n, g + 1);
                const uint32_t nb = __shfl_sync(0xFFFFFFFFu, myP.b_start, g + 1);
                const uint32_t nm = __shfl_sync(0xFFFFFFFFu, myP.b_n, g + 1);
                const uint32_t ns = __shfl_sync(0xFFFFFFFFu, (uint32_t)myP.same, g + 1);
                if ((uint32_t)lane < nn) prefetch_l1(a.rec + (size_t)(na + lane) * R16);
                if (!ns && (uint32_t)lane < nm) prefetch_l1(a.rec + (size_t)(nb + lane) * R16);
            }
            const BinPair P = shfl_binpair(myP, (int)g);
            hamming_small<BP, W, EM, JN>(a, ew, T, P, __shfl_sync(0xFFFFFFFFu, myidx, g), lane, pairs);
        }
    }
}

// Tiny bin pairs (a bin with itself, at most kTinySide entries): lane l takes
// every pair of the l-th bin pair of a batch of 32, so the latency of loading
// a bin pair and its records is paid once per 32 bin pairs.  Records are read
// per pair from L1 (a tiny bin's records share one or two cache lines).
template <int BP, int W, int EM, bool JN>
__device__ __forceinline__ void hamming_tiny_all(const DistArgs &a, EdgeWriter &ew, int lane,
                                                 uint64_t &pairs) {
    constexpr int NW = BP * W;
    constexpr int R16 = (NW + 3) / 4;
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
        const uint32_t n = P.a_n;
        const uint32_t np = (EM == 0 && P.eps < 0) ? 0u : n * (n - 1) / 2;
        pairs += n * (n - 1) / 2;
        const uint32_t thr = EM == 0 ? (uint32_t)max((int)P.eps, 0) : 0u;
        const uint4 *rec = a.rec + (size_t)P.a_start * R16;
        // pass 1: each lane scores its bin pair's pairs and keeps the edges
        // as bits of pair indices (at most 28 pairs)
        static_assert(kTinySide * (kTinySide - 1) / 2 <= 32, "tiny pair mask");
        uint32_t emask = 0;
        for (uint32_t p = 0; p < np; ++p) {
            uint32_t i, j;
            small_pair(p, true, n, i, j);
            uint32_t xw[4 * R16], yw[4 * R16];
#pragma unroll
            for (int q = 0; q < R16; ++q) {
                const uint4 u = __ldg(rec + (size_t)i * R16 + q), v = __ldg(rec + (size_t)j * R16 + q);
                xw[4 * q] = u.x; xw[4 * q + 1] = u.y; xw[4 * q + 2] = u.z; xw[4 * q + 3] = u.w;
                yw[4 * q] = v.x; yw[4 * q + 1] = v.y; yw[4 * q + 2] = v.z; yw[4 * q + 3] = v.w;
            }
            uint32_t dw[W], dist = 0;
#pragma unroll
            for (int w = 0; w < W; ++w) {
                uint32_t d = xw[w] ^ yw[w];
#pragma unroll
                for (int q = 1; q < BP; ++q) d |= xw[q * W + w] ^ yw[q * W + w];
                dw[w] = d;
                dist += __popc(d);
            }
            const uint32_t sc = W == 1 && EM == 2 ? dw[0] : (W == 1 && EM == 1 ? (dw[0] & (dw[0] - 1u)) : dist);
            if (sc > thr) continue;
            const uint4 mx = __ldg(a.meta + P.a_start + i), my = __ldg(a.meta + P.a_start + j);
            bool ok;
            if (JN) ok = join_meta_ok<W>(mx, my, dw, P.la, P.j, P.v);
            else ok = canonical_meta(a, P, mx, my);
            emask |= (uint32_t)ok << p;
        }
        // pass 2: one bulk append for the warp
        __syncwarp();
        emit_tiny_bits(a, ew, lane, emask, n, P.a_start);
        __syncwarp();
        if (a.bp_cycles) {
            // the batch's cycles, shared out by pairs (every lane takes part in
            // the reduction; lanes past the list's end hold n = 0)
            const uint32_t mine = n * (n - 1) / 2;
            const uint32_t tot = __reduce_add_sync(0xFFFFFFFFu, mine);
            const unsigned long long dt = (unsigned long long)(clock64() - t0);
            if (act) atomicAdd(&a.bp_cycles[idx], dt * mine / (tot ? tot : 1u));
        }
    }
}

// The y loop of one Hamming unit.  FULL: every r-block of the lane's x-entries
// is inside the unit, so all RX chains run without branches; otherwise the
// chains of r-blocks past the unit's end are skipped.
template <int BP, int W, int RX, int EM, bool FULL, bool JN>
__device__ __forceinline__ void hamming_unit_y(const DistArgs &a, EdgeWriter &ew, const Unit &U,
                                               const uint32_t (&x)[RX][BP * W],
                                               uint32_t valid, uint4 *sy, const TileSlice &T,
                                               const uint32_t *sseg, int lane) {
    constexpr int NW = BP * W;
    constexpr int R16 = (NW + 3) / 4;
    const uint32_t rb = (U.nx + 31) >> 5;   // r-blocks holding entries
    const uint32_t jk = U.P.v;              // segment join: the group's segment
    // a pair is a hit iff its score <= thr (score: d&(d-1) for eps 1, d for
    // eps 0, the popcount otherwise); masked entries score >= kOff.  Lanes past
    // the unit's end hold a copy of its first entry; their hits are dropped.
    const uint32_t thr = EM == 0 ? (uint32_t)max(U.P.eps, 0) : 0u;
    const bool neg = EM == 0 && U.P.eps < 0;       // no pair can be a neighbour
    const uint32_t same = U.P.same;
    const uint32_t yrow0 = (same ? U.P.a_start : U.P.b_start) + U.ybase;
    // same bin: y-entries at or before the first x-entry pair with nothing
    const uint32_t y0 = (same && U.xbase >= U.ybase) ? min(U.ny, U.xbase - U.ybase + 1) : 0u;
    for (uint32_t yb = y0; yb < U.ny && !neg; yb += kYB) {
        const uint32_t nb = min((uint32_t)kYB, U.ny - yb);
        const uint4 *src = a.rec + (size_t)(yrow0 + yb) * R16;
        for (uint32_t t = lane; t < nb * R16; t += 32) sy[t] = __ldg(src + t);
        if ((uint32_t)lane < nb) T.begin_y(a, lane, yrow0 + yb + lane);
        __syncwarp();
        uint32_t hits[RX];                // bit t: a hit with y-entry t of the batch
#pragma unroll
        for (int r = 0; r < RX; ++r) hits[r] = 0u;
        // y-entries inside the unit's own x range (same bin) need the mask of the
        // x-entries before them; they come first in the chunk (y ascending, all
        // after xbase), the rest pair with every x-entry of the unit
        uint32_t tdiag = 0;
        if (same && U.ybase + yb < U.xbase + U.nx)
            tdiag = min(nb, U.xbase + U.nx - (U.ybase + yb));
        auto score = [&](uint32_t t, uint32_t (&sc)[RX]) {
            uint32_t y[NW];
#pragma unroll
            for (int q = 0; q < R16; ++q) {
                const uint4 v = sy[t * R16 + q];
                const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (4 * q + e < NW) y[4 * q + e] = w4[e];
            }
            // FULL: all RX chains without branches (independent, interleaved);
            // otherwise only the r-blocks that hold entries (warp-uniform test)
#pragma unroll
            for (int r = 0; r < RX; ++r) {
                if (!FULL && r >= rb) { sc[r] = kOff; continue; }
                if (W == 1) {
                    uint32_t d = x[r][0] ^ y[0];
#pragma unroll
                    for (int p = 1; p < BP; ++p) d |= x[r][p] ^ y[p];
                    sc[r] = (EM == 2 ? d : (EM == 1 ? (d & (d - 1u)) : (uint32_t)__popc(d)));
                } else {
                    uint32_t dist = 0;
#pragma unroll
                    for (int w = 0; w < W; ++w) {
                        uint32_t d = x[r][w] ^ y[w];
#pragma unroll
                        for (int p = 1; p < BP; ++p) d |= x[r][p * W + w] ^ y[p * W + w];
                        dist += __popc(d);
                    }
                    sc[r] = dist;
                }
            }
        };
        auto record = [&](uint32_t t, const uint32_t (&sc)[RX]) {
            // with exact signatures a hit outside its canonical bin is dropped
            // here: sig_x & sig_y must be empty
            const uint4 ym = T.ym[t];
            const uint32_t bit = 1u << t;
#pragma unroll
            for (int r = 0; r < RX; ++r)
                if (sc[r] <= thr) {
                    bool ok = true;
                    if (JN) {
                        // segment join: V and J sets intersect, the group's
                        // segment is identical and no lower one is (masks of
                        // segment kk, word w at sseg[4 kk + w])
                        const uint4 m = T.xm[32 * r + lane];
                        ok = ((m.x & ym.x) | (m.y & ym.y)) != 0 && (m.z & ym.z & 0x3FFFFFFFu) != 0;
                        if (ok) {
                            const uint32_t *yw = reinterpret_cast<const uint32_t *>(sy + t * R16);
                            uint32_t dk = 0, l0 = 0, l1 = 0, l2 = 0;
#pragma unroll
                            for (int w = 0; w < W; ++w) {
                                uint32_t d = x[r][w] ^ yw[w];
#pragma unroll
                                for (int p = 1; p < BP; ++p) d |= x[r][p * W + w] ^ yw[p * W + w];
                                dk |= d & sseg[4 * jk + w];
                                l0 |= d & sseg[w];
                                l1 |= d & sseg[4 + w];
                                l2 |= d & sseg[8 + w];
                            }
                            ok = dk == 0 && (jk < 1 || l0 != 0) && (jk < 2 || l1 != 0) &&
                                 (jk < 3 || l2 != 0);
                        }
                    } else if (a.sig_exact) {
                        const uint4 m = T.xm[32 * r + lane];
                        ok = ((m.x & ym.x) | (m.y & ym.y) | (m.z & ym.z)) == 0;
                    }
                    if (ok) hits[r] |= bit;
                }
        };
        for (uint32_t t = 0; t < tdiag; ++t) {
            uint32_t sc[RX];
            score(t, sc);
            const uint32_t nact = U.ybase + yb + t - U.xbase;   // x-entries before y
#pragma unroll
            for (int r = 0; r < RX; ++r)
                if ((uint32_t)r * 32 + lane >= nact) sc[r] |= kOff;
            uint32_t z = sc[0];
#pragma unroll
            for (int r = 1; r < RX; ++r) z = min(z, sc[r]);
            if (z <= thr) record(t, sc);
        }
        uint32_t t = tdiag;
        for (; t + 1 < nb; t += 2) {      // two y-entries per step: twice the chains
            uint32_t sa[RX], sb[RX];
            score(t, sa);
            score(t + 1, sb);
            uint32_t za = sa[0], zb = sb[0];
#pragma unroll
            for (int r = 1; r < RX; ++r) { za = min(za, sa[r]); zb = min(zb, sb[r]); }
            if (za <= thr) record(t, sa);
            if (zb <= thr) record(t + 1, sb);
        }
        if (t < nb) {
            uint32_t sc[RX];
            score(t, sc);
            uint32_t z = sc[0];
#pragma unroll
            for (int r = 1; r < RX; ++r) z = min(z, sc[r]);
            if (z <= thr) record(t, sc);
        }
        uint32_t any = 0;
#pragma unroll
        for (int r = 0; r < RX; ++r) {
            if (!((valid >> r) & 1u)) hits[r] = 0u;
            any |= hits[r];
        }
        if (__any_sync(0xFFFFFFFFu, any)) {
            if (!JN && !a.sig_exact) {   // wide gene lists: the bin of the lowest common genes only
#pragma unroll
                for (int r = 0; r < RX; ++r)
                    for (uint32_t b = hits[r]; b; b &= b - 1)
                        if (!canonical(a, U.P, T.xm[32 * r + lane].w, T.ym[__ffs(b) - 1].w)) hits[r] &= ~(b & (0u - b));
            }
            emit_batch<RX>(a, ew, T, hits, nb, lane);
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Hamming, fast path.  BP planes x W words per record; RX x-entries per lane.
// EM: 0 = popcount test, 1 = eps == 1 (d & (d-1)) == 0, 2 = eps == 0.
// ---------------------------------------------------------------------------
template <int BP, int W, int RX, int EM, bool JN>
__global__ void __launch_bounds__(kWarps * 32, (W == 1 && RX <= 2 ? 6 : (W == 1 && RX <= 4 ? 5 : 4)))
k_hamming(const __grid_constant__ DistArgs a) {
    constexpr int NW = BP * W;                 // words per record used
    constexpr int R16 = (NW + 3) / 4;          // 16-byte words per record
    __shared__ uint4 sy[kWarps][kYB * R16];
    __shared__ uint4 sym[kWarps][kYB];            // y side records
    __shared__ uint4 sxm[kWarps][32 * RX];        // x side records
    __shared__ uint32_t sseg[kWarps][16];         // segment join: masks of segment kk, word w
    __shared__ uint32_t scp[kWarps][2 * 32 * RX + 2 * kYB];   // copies and sums (TileSlice)
    static_assert(RX <= 8 && kYB <= 32, "hit words");
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t n_units = a.ctr->n_units, n_bp = a.ctr->n_binpairs;
    const TileSlice T{sxm[wid], sym[wid], scp[wid], scp[wid] + 2 * 32 * RX, scp[wid] + 32 * RX,
                      scp[wid] + 2 * 32 * RX + kYB};
    EdgeWriter ew;
    ew.init();
    uint64_t pairs = 0;
    Unit U;
    while (next_unit(a, n_units, n_bp, lane, U)) {
        uint32_t x[RX][NW];
        uint32_t valid = 0;
#pragma unroll
        for (int r = 0; r < RX; ++r) {
            const uint32_t xi = (uint32_t)r * 32 + lane;
            const bool ok = xi < U.nx;
            valid |= (uint32_t)ok << r;
            const uint4 *src = a.rec + (size_t)(U.P.a_start + U.xbase + (ok ? xi : 0)) * R16;
#pragma unroll
            for (int q = 0; q < R16; ++q) {
                const uint4 v = __ldg(src + q);
                const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (4 * q + e < NW) x[r][4 * q + e] = w4[e];
            }
            if (ok) pairs += unit_pairs(U, U.xbase + xi);
            T.begin_x(a, xi, U.P.a_start + U.xbase + (ok ? xi : 0));
        }
        if (JN && lane < 16) {
            // segment kk = lane / 4 of length la split into j segments, word w = lane % 4
            const uint32_t kk = (uint32_t)lane >> 2, w = (uint32_t)lane & 3u;
            const uint32_t L = U.P.la, S = U.P.j;
            const uint32_t lo = kk < S ? kk * L / S : 0u, hi = kk < S ? (kk + 1) * L / S : 0u;
            const uint32_t a0 = max(lo, 32u * w), a1 = min(hi, 32u * w + 32u);
            uint32_t m = 0;
            if (a0 < a1) {
                const uint32_t n = a1 - a0;
                m = (n >= 32 ? 0xFFFFFFFFu : ((1u << n) - 1u)) << (a0 - 32u * w);
            }
            sseg[wid][lane] = m;
        }
        __syncwarp();
        if (U.nx == (uint32_t)(32 * RX))
            hamming_unit_y<BP, W, RX, EM, true, JN>(a, ew, U, x, valid, sy[wid], T, sseg[wid], lane);
        else
            hamming_unit_y<BP, W, RX, EM, false, JN>(a, ew, U, x, valid, sy[wid], T, sseg[wid], lane);
        T.end_x(a, U.nx, lane);
        log_unit(a, U, lane);
    }
    // then the small bin pairs (they also fill the tail of the tiled work)
    hamming_small_all<BP, W, EM, JN>(a, ew, T, lane, pairs);
    hamming_tiny_all<BP, W, EM, JN>(a, ew, lane, pairs);
    finish(a, ew, pairs, lane);
}

// The segment join and the buckets are separate instantiations, so the
// bucket path's hot loop carries none of the join's per-hit tests (and the
// instruction cache holds one of them, not both).
template <int BP, int W, int RX, bool JN>
void run_hamming_jn(const Plan &P, const DistArgs &a, int grid, cudaStream_t s) {
    if (P.hamming_eps_mode == 2) run(k_hamming<BP, W, RX, 2, JN>, a, 0, grid, s);
    else if (P.hamming_eps_mode == 1 && W == 1) run(k_hamming<BP, W, RX, 1, JN>, a, 0, grid, s);
    else run(k_hamming<BP, W, RX, 0, JN>, a, 0, grid, s);
}

template <int BP, int W, int RX>
void run_hamming(const Plan &P, const DistArgs &a, int grid, cudaStream_t s) {
    if (P.join) run_hamming_jn<BP, W, RX, true>(P, a, grid, s);
    else run_hamming_jn<BP, W, RX, false>(P, a, grid, s);
}

template <int BP>
void launch_hamming(const Plan &P, const DistArgs &a, int grid, cudaStream_t s) {
    const int RX = (int)P.RX;
    switch (P.W) {
        case 1:
            if (RX == 2 && P.join) run_hamming_jn<BP, 1, 2, true>(P, a, grid, s);
            else if (RX == 8) run_hamming<BP, 1, 8>(P, a, grid, s);
            else run_hamming<BP, 1, 4>(P, a, grid, s);
            break;
        case 2: run_hamming<BP, 2, 4>(P, a, grid, s); break;
        case 3: run_hamming<BP, 3, 4>(P, a, grid, s); break;
        default: run_hamming<BP, 4, 4>(P, a, grid, s); break;
    }
}

}  // namespace
}  // namespace idb
