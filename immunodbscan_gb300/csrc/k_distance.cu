// k_distance.cu -- the neighbour search (rule S4), one persistent launch.
//
// Reference: half_core_points / half_hamming_core_points
// (cuda/PSDBSCAN.hcu:585-657, 751-833) and their second sweep fuse_clusters /
// fuse_hamming_clusters (:664-742, 840-931).  The reference runs one block per
// pair with an anti-diagonal DP and a __syncthreads per diagonal, twice.  Here
// the distance work is done once: every neighbour pair becomes an edge of the
// neighbour graph, and core marking and cluster growth run on that graph.
//
// Work decomposition
//  * A work unit is an x-chunk of TX = 32*RX entries of bin A against a y-chunk
//    of TY entries of bin B (B = A for a same-bin pair; then only pairs with
//    y after x in the bin are kept).  Units are numbered in schedule order (heavy
//    bin pairs first) and handed out by an atomic queue; each warp owns a unit.
//  * Lane l holds x-entries l, l+32, ... of the chunk in registers.  The
//    y-records are staged into the warp's shared memory with coalesced 128-bit
//    loads and read back as broadcasts, so a y-record costs two shared loads
//    per RX pairs.
//  * Hamming (fast path): residues are bit-sliced (Bp planes of W 32-bit
//    words); a pair costs Bp*W XOR/OR plus a population test.
//  * Levenshtein, eps <= 3 at every admissible length pair (fast path): the
//    diagonal test of lev_diag.cuh.
//  * Levenshtein, larger eps (fast path): Myers/Hyyro bit-parallel recurrence
//    with the x-pattern's match masks (Peq) in shared memory and the y-text
//    broadcast; the value on the diagonal through (m, n) is checked every 4
//    columns and a warp leaves a y early once all its pairs exceed eps (the
//    diagonal value never decreases, so the early exit is exact).
//  * A neighbour pair is kept only in the bin of its lowest common V gene and
//    lowest common J gene, so a pair that shares several bins counts once.
//  * Segment joins: the "bins" are groups of uniques that share a whole segment
//    (Hamming, eps <= 2) or in which one holds a segment of the other at a small
//    shift (edit distance, eps <= 3); a pair is kept only in the group of its
//    lowest identical segment, or of its first look-up that holds, and only if
//    its V and J sets intersect.
//  * Bin pairs of at most 32 entries a side are scored pair-parallel (Hamming:
//    records by shuffles; edit distance: from L1), and those of at most 28 pairs
//    by one lane (Hamming: a bin with itself).
//  * With bit planes a lane's hits are bits of a batch of 32 y-entries, written as
//    one bulk append with both sides' counts; the byte and the Myers kernels
//    append each round's hits, and k_count sums their counts from the list.
#include "distance_common.cuh"

namespace idb {

namespace {

constexpr uint32_t kLevQ = 256;          // queued candidate pairs per warp (Levenshtein)

// ---------------------------------------------------------------------------
// Levenshtein, fast path.  Codes records (one byte per residue, RS bytes);
// pattern <= 32*W residues; RX patterns per lane.
// ---------------------------------------------------------------------------
template <int W, int RX>
__global__ void __launch_bounds__(kWarps * 32, 4)
k_levenshtein(DistArgs a) {
    extern __shared__ uint32_t smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t A = a.A;
    const uint32_t peq_words = RX * A * W * 32;          // per warp
    const uint32_t ybuf_words = kYB * a.rs16 * 4;        // per warp
    const uint32_t meta_words = (kYB + 32 * RX) * 4;     // per warp
    constexpr uint32_t kCW = 8;                          // count words: 4 codes each, A <= 32
    uint32_t *peq = smem + wid * (peq_words + ybuf_words + meta_words + kYB +
                                  kCW * (kYB + 32 * RX) + kLevQ);
    uint4 *sy = reinterpret_cast<uint4 *>(peq + peq_words);
    uint4 *sym = sy + kYB * a.rs16;                      // y side records
    uint4 *sxm = sym + kYB;                              // x side records
    uint32_t *spres = reinterpret_cast<uint32_t *>(sxm + 32 * RX);   // y residue sets
    uint32_t *sycnt = spres + kYB;                       // y residue counts [kYB][kCW]
    uint32_t *sxcnt = sycnt + kCW * kYB;                 // x residue counts [RX][kCW][32]
    uint32_t *lq = sxcnt + kCW * 32 * RX;                // queued candidate pairs [kLevQ]
    const uint32_t cw = (A + 3) / 4;                     // count words in use
    const uint32_t n_units = a.ctr->n_units, n_bp = a.ctr->n_binpairs;
    EdgeWriter ew;
    ew.init();
    uint64_t pairs = 0, cols = 0;
    Unit U;
    while (next_unit(a, n_units, n_bp, lane, U)) {
        const int m = U.P.la, n = U.P.lb, eps = U.P.eps;
        const int dg = n - m;
        uint32_t xpos[RX];
        bool xval[RX];
        uint32_t xpres[RX];        // set of residue codes of each x-entry (A <= 32)
        // Peq[r][c][w][lane]
        for (uint32_t k = 0; k < (uint32_t)RX * A * W; ++k) peq[k * 32 + lane] = 0u;
        for (uint32_t k = 0; k < (uint32_t)RX * kCW; ++k) sxcnt[k * 32 + lane] = 0u;
        __syncwarp();
#pragma unroll
        for (int r = 0; r < RX; ++r) {
            xpos[r] = U.xbase + r * 32 + lane;
            xval[r] = xpos[r] < U.xbase + U.nx;
            xpres[r] = 0;
            sxm[r * 32 + lane] = __ldg(a.meta + U.P.a_start + (xval[r] ? xpos[r] : U.xbase));
            if (xval[r]) {
                pairs += unit_pairs(U, xpos[r]);
                const uint8_t *codes =
                    reinterpret_cast<const uint8_t *>(a.rec + (size_t)(U.P.a_start + xpos[r]) * a.rs16);
                for (int i = 0; i < m; ++i) {
                    const uint32_t c = __ldg(codes + i);
                    peq[((r * A + c) * W + (i >> 5)) * 32 + lane] |= 1u << (i & 31);
                    xpres[r] |= 1u << c;
                    sxcnt[(r * kCW + (c >> 2)) * 32 + lane] += 1u << (8 * (c & 3));
                }
            }
        }
        uint32_t xcnt[RX][kCW];    // residue counts, one byte per code (lengths < 256)
#pragma unroll
        for (int r = 0; r < RX; ++r)
#pragma unroll
            for (uint32_t k = 0; k < kCW; ++k) xcnt[r][k] = sxcnt[(r * kCW + k) * 32 + lane];
        // An edit changes the set of residues present by at most two (a
        // substitution drops one and adds one, an indel one), so a pair whose
        // sets differ in more than 2*eps residues is not within eps.  Likewise
        // an edit changes the residue counts by at most 2 in total (sum of
        // absolute differences), so a pair with that sum above 2*eps is not.
        const int pres_max = 2 * eps;
        __syncwarp();
        const uint32_t yrow0 = (U.P.same ? U.P.a_start : U.P.b_start) + U.ybase;
        for (uint32_t yb = 0; yb < U.ny; yb += kYB) {
            const uint32_t nb = min((uint32_t)kYB, U.ny - yb);
            const uint4 *src = a.rec + (size_t)(yrow0 + yb) * a.rs16;
            for (uint32_t t = lane; t < nb * a.rs16; t += 32) sy[t] = __ldg(src + t);
            for (uint32_t t = lane; t < nb; t += 32) sym[t] = __ldg(a.meta + yrow0 + yb + t);
            __syncwarp();
            for (uint32_t t = lane; t < nb; t += 32) {
                const uint8_t *yc = reinterpret_cast<const uint8_t *>(sy + t * a.rs16);
                uint32_t *yk = sycnt + t * kCW;
#pragma unroll
                for (uint32_t k = 0; k < kCW; ++k) yk[k] = 0u;
                uint32_t pr = 0;
                for (int j = 0; j < n; ++j) {
                    const uint32_t c = yc[j];
                    pr |= 1u << c;
                    yk[c >> 2] += 1u << (8 * (c & 3));
                }
                spres[t] = pr;
            }
            __syncwarp();
            // 1. filters: the pairs that survive go to a warp queue as
            //    (owner lane, r, t), so the DP below runs with every lane busy
            uint32_t qn = 0;
            for (uint32_t t = 0; t < nb; ++t) {
                const uint32_t ypos = U.ybase + yb + t;
                const uint32_t ypres = spres[t];
                uint32_t ycnt[kCW];
#pragma unroll
                for (uint32_t k = 0; k < kCW; ++k) ycnt[k] = k < cw ? sycnt[t * kCW + k] : 0u;
#pragma unroll
                for (int r = 0; r < RX; ++r) {
                    bool alive = xval[r] && !(U.P.same && ypos <= xpos[r]) &&
                                 __popc(xpres[r] ^ ypres) <= pres_max;
                    if (alive) {
                        uint32_t sad = 0;
#pragma unroll
                        for (uint32_t k = 0; k < kCW; ++k) sad = __vsadu4(xcnt[r][k], ycnt[k]) + sad;
                        alive = (int)sad <= pres_max;
                    }
                    const uint32_t mk = __ballot_sync(0xFFFFFFFFu, alive);
                    if (alive) lq[qn + __popc(mk & lanemask_lt())] = (uint32_t)lane | ((uint32_t)r << 5) | (t << 8);
                    qn += __popc(mk);
                }
                if (qn > kLevQ - 32 * RX || t + 1 == nb) {
                    __syncwarp();
                    // 2. bit-parallel DP of the queued pairs, 32 at a time
                    for (uint32_t k0 = 0; k0 < qn; k0 += 32) {
                        const bool has = k0 + lane < qn;
                        const uint32_t it = has ? lq[k0 + lane] : 0u;
                        const uint32_t owner = it & 31u, r = (it >> 5) & 7u, tt = it >> 8;
                        const uint8_t *yc = reinterpret_cast<const uint8_t *>(sy + tt * a.rs16);
                        uint32_t Pv[W], Mv[W];
#pragma unroll
                        for (int w = 0; w < W; ++w) { Pv[w] = 0xFFFFFFFFu; Mv[w] = 0u; }
                        bool live = has;
                        for (int j = 0; j < n; ++j) {
                            const uint32_t c = yc[j];
                            const uint32_t *pe = peq + ((r * A + c) * W) * 32 + owner;
                            if (W == 1) {
                                myers_step1(Pv[0], Mv[0], pe[0]);
                            } else {
                                int h = 1;
#pragma unroll
                                for (int w = 0; w < W; ++w) h = myers_block(Pv[w], Mv[w], pe[w * 32], h);
                            }
                            if ((j & 3) == 3) {
                                const int col = j + 1;
                                const int i = col - dg;
                                if (i >= 0 && i <= m) {
                                    if (live && myers_value<W>(Pv, Mv, i, col) > eps) {
                                        live = false;
                                        cols += (uint32_t)col;
                                    }
                                    if (!__any_sync(0xFFFFFFFFu, live)) break;
                                }
                            }
                        }
                        bool hit = false;
                        if (live) {
                            cols += (uint32_t)n;
                            hit = myers_value<W>(Pv, Mv, m, n) <= eps;
                        }
                        if (__any_sync(0xFFFFFFFFu, hit)) {
                            bool ok = hit;
                            const uint4 mx = sxm[r * 32 + owner], my = sym[tt];
                            if (ok) ok = canonical_meta(a, U.P, mx, my);
                            ew.append<false>(a, lane, ok, min(mx.w, my.w), max(mx.w, my.w));
                        }
                    }
                    qn = 0;
                    __syncwarp();
                }
            }
            __syncwarp();
        }
        log_unit(a, U, lane);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) cols += __shfl_xor_sync(0xFFFFFFFFu, cols, d);
    if (lane == 0 && cols) atomicAdd(&a.ctr->lev_columns, (unsigned long long)cols);
    finish(a, ew, pairs, lane);
}

// ---------------------------------------------------------------------------
// Generic path (more than 32 distinct residues, or longer than 128): one pair
// per lane, code bytes read from global memory.  Hamming stops once the count
// exceeds eps (cuda/PSDBSCAN.hcu:628-636); Levenshtein is a DP restricted to
// the diagonals |j - i| <= eps with a cut-off once a row exceeds eps.
// ---------------------------------------------------------------------------
__device__ bool generic_lev_leq(const uint8_t *x, int m, const uint8_t *y, int n, int eps) {
    if (eps < 0) return false;
    if (m - n > eps || n - m > eps) return false;
    // D restricted to the band; values above eps are clamped to eps+1
    short row[2][kGenericMaxLen + 1];
    const int big = eps + 1;
    for (int j = 0; j <= n; ++j) row[0][j] = (short)min(j, big);
    int cur = 0;
    for (int i = 1; i <= m; ++i) {
        const int nx = cur ^ 1;
        const int jlo = max(1, i - eps), jhi = min(n, i + eps);
        row[nx][0] = (short)min(i, big);
        if (jlo > 1) row[nx][jlo - 1] = (short)big;
        int rmin = row[nx][0];
        for (int j = jlo; j <= jhi; ++j) {
            int v = row[cur][j - 1] + (x[i - 1] != y[j - 1]);
            const int up = (j <= i - 1 + eps) ? row[cur][j] + 1 : big;
            const int left = row[nx][j - 1] + 1;
            v = min(v, min(up, left));
            v = min(v, big);
            row[nx][j] = (short)v;
            rmin = min(rmin, v);
        }
        if (jhi < n) row[nx][jhi + 1] = (short)big;
        cur = nx;
        if (rmin > eps) return false;
    }
    return row[cur][n] <= eps;
}

template <bool HAM>
__global__ void __launch_bounds__(kWarps * 32)
k_generic(DistArgs a) {
    const int lane = threadIdx.x & 31;
    const uint32_t n_units = a.ctr->n_units, n_bp = a.ctr->n_binpairs;
    EdgeWriter ew;
    ew.init();
    uint64_t pairs = 0;
    Unit U;
    while (next_unit(a, n_units, n_bp, lane, U)) {
        const int m = U.P.la, n = U.P.lb, eps = U.P.eps;
        const uint32_t yrow0 = (U.P.same ? U.P.a_start : U.P.b_start) + U.ybase;
        const uint32_t total = U.nx * U.ny;
        for (uint32_t p0 = 0; p0 < total; p0 += 32) {
            const uint32_t p = p0 + lane;
            bool ok = false;
            uint32_t ux = 0, uy = 0;
            if (p < total) {
                const uint32_t xi = p / U.ny, yi = p % U.ny;
                const uint32_t xpos = U.xbase + xi, ypos = U.ybase + yi;
                if (!(U.P.same && ypos <= xpos)) {
                    ++pairs;
                    const uint8_t *xc =
                        reinterpret_cast<const uint8_t *>(a.rec + (size_t)(U.P.a_start + xpos) * a.rs16);
                    const uint8_t *yc =
                        reinterpret_cast<const uint8_t *>(a.rec + (size_t)(yrow0 + yi) * a.rs16);
                    if (HAM) {
                        int d = 0;
                        ok = eps >= 0;
                        for (int k = 0; k < m && ok; ++k)
                            if (xc[k] != yc[k] && ++d > eps) ok = false;
                    } else {
                        ok = generic_lev_leq(xc, m, yc, n, eps);
                    }
                    if (ok) {
                        ux = a.ent_uid[U.P.a_start + xpos];
                        uy = a.ent_uid[yrow0 + yi];
                        ok = canonical(a, U.P, ux, uy);
                    }
                }
            }
            ew.append<false>(a, lane, ok, min(ux, uy), max(ux, uy));
        }
        log_unit(a, U, lane);
    }
    finish(a, ew, pairs, lane);
}

// ---------------------------------------------------------------------------
// Admissible-pair count (the throughput metric's numerator): unique pairs that
// share a bin (V and J overlap) with an admissible length gap, each counted in
// its canonical bin only.  One pair per lane; run once per workload.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kWarps * 32)
k_count_admissible(DistArgs a) {
    const int lane = threadIdx.x & 31;
    const uint32_t n_units = a.ctr->n_units, n_bp = a.ctr->n_binpairs;
    unsigned long long cnt = 0;
    Unit U;
    while (next_unit(a, n_units, n_bp, lane, U)) {
        const uint32_t yrow0 = (U.P.same ? U.P.a_start : U.P.b_start) + U.ybase;
        const uint32_t total = U.nx * U.ny;
        for (uint32_t p = lane; p < total; p += 32) {
            const uint32_t xi = p / U.ny, yi = p % U.ny;
            const uint32_t xpos = U.xbase + xi, ypos = U.ybase + yi;
            if (U.P.same && ypos <= xpos) continue;
            if (U.P.eps < 0) continue;
            const uint32_t ux = a.ent_uid[U.P.a_start + xpos], uy = a.ent_uid[yrow0 + yi];
            cnt += canonical(a, U.P, ux, uy);
        }
    }
    const uint32_t n_small = a.ctr->n_small, n_tiny = a.ctr->n_tiny;
    for (;;) {
        uint32_t s = 0;
        if (lane == 0) s = atomicAdd(&a.ctr->small_cursor, 1u);
        s = __shfl_sync(0xFFFFFFFFu, s, 0);
        if (s >= n_small + n_tiny) break;
        const uint32_t sidx = s < n_small ? a.small_list[s] : a.small_list[a.small_cap - 1u - (s - n_small)];
        const BinPair P = a.bp[sidx];
        if (P.eps < 0) continue;
        const bool same = P.same != 0;
        const uint32_t ystart = same ? P.a_start : P.b_start;
        const uint32_t npairs = same ? P.a_n * (P.a_n - 1) / 2 : P.a_n * P.b_n;
        for (uint32_t p = lane; p < npairs; p += 32) {
            uint32_t i, j;
            small_pair(p, same, P.a_n, i, j);
            cnt += canonical(a, P, a.ent_uid[P.a_start + i], a.ent_uid[ystart + j]);
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) cnt += __shfl_xor_sync(0xFFFFFFFFu, cnt, d);
    if (lane == 0 && cnt) atomicAdd(&a.ctr->admissible_pairs, cnt);
}

}  // namespace

static DistArgs make_args(const Plan &P, const Buffers &B) {
    DistArgs a;
    a.bp = B.bp_sorted;
    a.unit_base = B.bp_units;
    a.rec = B.ent_rec;
    a.ent_uid = B.ent_uid;
    a.urow = B.urow;
    a.vbits = B.vbits; a.jbits = B.jbits;
    a.VW = P.VW; a.JW = P.JW;
    a.rs16 = P.RS / 16;
    a.TX = P.TX; a.TY = P.TY; a.q = P.TY / P.TX;
    a.A = P.A;
    a.edges = B.edges;
    a.cap_edges = P.cap_edges;
    a.ctr = B.ctr;
    a.bp_cycles = B.bp_cycles;   // set only while profiling
    a.meta = B.ent_meta;
    a.sig_exact = (P.side_exact() && !P.join) ? 1 : 0;
    a.small_list = B.bp_small;
    a.small_cap = (uint32_t)P.cap_binpairs + 1u;
    a.join = P.join ? 1 : 0;
    a.vj_meta = P.side_exact() ? 1 : 0;
    a.sink = kSinkEdges;
    a.cnt = B.cnt;
    a.ucopies = B.ucopies;
    a.ecopies = B.ent_copies;
    a.parent = B.parent;
    a.bmin = B.bmin;
    return a;
}

void launch_count_admissible(const Plan &P, const Buffers &B, cudaStream_t s) {
    DistArgs a = make_args(P, B);
    cudaMemsetAsync(&B.ctr->unit_cursor, 0, sizeof(uint32_t), s);
    cudaMemsetAsync(&B.ctr->small_cursor, 0, sizeof(uint32_t), s);
    cudaMemsetAsync(&B.ctr->tiny_cursor, 0, sizeof(uint32_t), s);
    run(k_count_admissible, a, 0, 0, s);
}

const char *distance_variant_name(const Plan &P) {
    if (!P.fast) return P.hamming ? "k_generic<hamming>" : "k_generic<levenshtein>";
    return P.hamming ? "k_hamming" : (P.lev_diag ? "k_lev_diag" : "k_levenshtein");
}

// Slots a warp reserves at a time.  Every warp may leave most of a chunk unused, and
// when there are few bin pairs nearly every resident warp finds an edge: with 256
// slots each, 20k rows with 15k neighbour pairs reserved 0.6M slots, ran over
// their first list (so the sweep ran twice and the list grew by 134 MB) and were
// streamed under any edge-memory limit below that.  So at most a 64th of an SM's
// share of the list; 256 from 2.5M slots on, where the counter's atomics count.
static uint32_t edge_chunk_log(uint64_t cap_edges) {
    const uint64_t share = cap_edges / (64ull * (uint64_t)sm_count());
    uint32_t lg = 0;
    while ((2u << lg) <= kEdgeChunk && ((2u << lg) <= share || (2u << lg) <= kEdgeChunkMin)) ++lg;
    return lg;
}

void launch_distance(const Plan &P, const Buffers &B, int grid, cudaStream_t s, uint32_t sink) {
    DistArgs a = make_args(P, B);
    a.sink = sink;
    if (sink != kSinkEdges) {   // no list: nothing to overflow
        a.edges = nullptr;
        a.cap_edges = ~0ull;
    }
    a.chunk_log = edge_chunk_log(a.cap_edges);
    if (sink != kSinkGrow) {   // the work queues too; a repeated sweep counts anew
        launch_graph_init(P, B, s);
    } else {
        cudaMemsetAsync(&B.ctr->unit_cursor, 0, sizeof(uint32_t), s);
        cudaMemsetAsync(&B.ctr->small_cursor, 0, sizeof(uint32_t), s);
        cudaMemsetAsync(&B.ctr->tiny_cursor, 0, sizeof(uint32_t), s);
    }
    if (!P.fast) {
        if (P.hamming) run(k_generic<true>, a, 0, grid, s);
        else run(k_generic<false>, a, 0, grid, s);
        return;
    }
    if (P.hamming) {
        if (P.B <= 2) launch_hamming_2(P, a, grid, s);
        else launch_hamming_5(P, a, grid, s);
        return;
    }
    if (P.lev_diag) {
        if (P.B <= 2) launch_lev_diag_2(P, a, grid, s);
        else launch_lev_diag_5(P, a, grid, s);
        return;
    }
    const size_t smem = (size_t)kWarps * ((size_t)P.RX * P.A * P.W * 32 * 4 + (size_t)kYB * P.RS +
                                          16 * ((size_t)kYB + 32 * P.RX) + 4 * (size_t)kYB +
                                          4 * 8 * ((size_t)kYB + 32 * P.RX) + 4 * (size_t)kLevQ);
    switch (P.W) {
        case 1: if (P.RX == 2) run(k_levenshtein<1, 2>, a, smem, grid, s); else run(k_levenshtein<1, 1>, a, smem, grid, s); break;
        case 2: run(k_levenshtein<2, 1>, a, smem, grid, s); break;
        case 3: run(k_levenshtein<3, 1>, a, smem, grid, s); break;
        default: run(k_levenshtein<4, 1>, a, smem, grid, s); break;
    }
}

}  // namespace idb
