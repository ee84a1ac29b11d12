// bitops.cuh -- integer helpers shared by the device kernels and the host-side
// unit tests (compiled by nvcc for sm_103a and by g++ for the CPU tests).
//
// Contents
//  * popcount / find-first-set wrappers
//  * Myers/Hyyro bit-parallel global edit distance on 32-bit blocks
//    (G. Myers, "A fast bit-vector algorithm for approximate string matching
//    based on dynamic programming", J. ACM 46(3), 1999; H. Hyyro, "A bit-vector
//    algorithm for computing Levenshtein and Damerau edit distances", Nordic J.
//    Computing 10, 2003 -- block-based form with a horizontal delta carried
//    between 32-row blocks).  The reference computes the same quantity with a
//    full anti-diagonal DP (cuda/PSDBSCAN.hcu:246-290).
//  * edit distance <= E by furthest-reaching points on mismatch bit masks
//    (E. Ukkonen, "Algorithms for approximate string matching", Information and
//    Control 64, 1985; G. Landau and U. Vishkin, J. Algorithms 10(2), 1989)
//  * closed-form decode of triangular work-unit grids
//  * a step of a walk to the root of a tree that many threads flatten at once
//  * a 64-bit mixing hash for the duplicate table
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define IDB_HD __host__ __device__ __forceinline__
#else
#define IDB_HD inline
#endif

namespace idb {

IDB_HD int popc32(uint32_t x) {
#if defined(__CUDA_ARCH__)
    return __popc(x);
#else
    return __builtin_popcount(x);
#endif
}

IDB_HD int popc64(uint64_t x) {
#if defined(__CUDA_ARCH__)
    return __popcll(x);
#else
    return __builtin_popcountll(x);
#endif
}

// index of the lowest set bit, -1 if none
IDB_HD int lowest_bit64(uint64_t x) {
#if defined(__CUDA_ARCH__)
    return __ffsll((long long)x) - 1;
#else
    return x ? __builtin_ctzll(x) : -1;
#endif
}

IDB_HD uint32_t low_mask32(int i) {   // bits [0, i) set, 0 <= i <= 32
    return i >= 32 ? 0xFFFFFFFFu : ((1u << i) - 1u);
}

// ---------------------------------------------------------------------------
// One column of the bit-parallel edit-distance recurrence for one 32-row block.
// Pv/Mv hold the vertical deltas D[i][j-1]-D[i-1][j-1] = +1 / -1 of the block's
// rows; eq has bit i set iff pattern row i matches the text character.
// h_in is the horizontal delta D[r0][j]-D[r0][j-1] entering from the row above
// the block (+1 for the first block: D[0][j] = j).  Returns the delta leaving
// the block's top bit (row r0+32).
// ---------------------------------------------------------------------------
IDB_HD int myers_block(uint32_t &Pv, uint32_t &Mv, uint32_t eq, int h_in) {
    const uint32_t in_neg = (uint32_t)(h_in < 0);
    const uint32_t in_pos = (uint32_t)(h_in > 0);
    const uint32_t Xv = eq | Mv;
    eq |= in_neg;                            // a -1 entering from above acts like a match
    const uint32_t Xh = (((eq & Pv) + Pv) ^ Pv) | eq;
    uint32_t Ph = Mv | ~(Xh | Pv);
    uint32_t Mh = Pv & Xh;
    const int h_out = (int)(Ph >> 31) - (int)(Mh >> 31);
    Ph = (Ph << 1) | in_pos;
    Mh = (Mh << 1) | in_neg;
    Pv = Mh | ~(Xv | Ph);
    Mv = Ph & Xv;
    return h_out;
}

// Single-block specialisation (pattern <= 32, h_in = +1 always).
IDB_HD void myers_step1(uint32_t &Pv, uint32_t &Mv, uint32_t eq) {
    const uint32_t Xv = eq | Mv;
    const uint32_t Xh = (((eq & Pv) + Pv) ^ Pv) | eq;
    uint32_t Ph = Mv | ~(Xh | Pv);
    uint32_t Mh = Pv & Xh;
    Ph = (Ph << 1) | 1u;
    Mh = Mh << 1;
    Pv = Mh | ~(Xv | Ph);
    Mv = Ph & Xv;
}

// D[i][j] recovered from the vertical deltas of column j (D[0][j] = j).
template <int W>
IDB_HD int myers_value(const uint32_t (&Pv)[W], const uint32_t (&Mv)[W], int i, int j) {
    int d = j;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        int lo = w * 32;
        int take = i - lo;
        if (take <= 0) break;
        uint32_t m = low_mask32(take);
        d += popc32(Pv[w] & m) - popc32(Mv[w] & m);
    }
    return d;
}

// Reference edit distance of two code strings via the block recurrence
// (used by the host unit tests; the kernels inline the same steps).
template <int W>
IDB_HD int myers_distance(const uint8_t *p, int m, const uint8_t *t, int n) {
    uint32_t Pv[W], Mv[W];
#pragma unroll
    for (int w = 0; w < W; ++w) { Pv[w] = 0xFFFFFFFFu; Mv[w] = 0u; }
    for (int j = 0; j < n; ++j) {
        int h = 1;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            uint32_t eq = 0;
            for (int b = 0; b < 32; ++b) {
                int i = w * 32 + b;
                if (i < m && p[i] == t[j]) eq |= 1u << b;
            }
            h = myers_block(Pv[w], Mv[w], eq, h);
        }
    }
    return myers_value<W>(Pv, Mv, m, n);
}

// ---------------------------------------------------------------------------
// Is the edit distance of x (length m) and y (length n = m + G) at most E?
// Decided on the mismatch masks of a few diagonals instead of a column-by-column
// recurrence: bit i of the mask of diagonal d says that x[i] != y[i + d].  An
// alignment with at most E edits from (0,0) to (m,n) only visits the diagonals
// -LO .. G + LO, LO = (E - G) / 2 (leaving further costs more than E to come
// back), and on a diagonal it is always best to have consumed as much of x as
// possible.  "Consumed" is a prefix mask F of x positions:
//   t = D_d & ~F              mismatches not yet passed
//   E = (t - 1) & ~t          prefix up to the first one (all ones if none)
//   G = t ^ (t - 1)           the same with the mismatch itself
// and with one more edit diagonal d starts from G_d (substitution),
// E_{d-1} (a character of y skipped) and G_{d+1} (a character of x skipped);
// the union of prefix masks is the longest, so merging is an OR.  Returns 0 iff
// diagonal G is passed to its end after E edits.
// Positions past an end need no masking.  Both strings are padded with the same
// code, so diagonal G matches there; on a diagonal d < G x is exhausted and more
// prefix gains nothing; on a diagonal d > G the last d - G positions of x lie
// past y's end, and passing them for free saves nothing: the d - G edits (each
// skipping a character of x) back to diagonal G are due either way.
// ---------------------------------------------------------------------------
template <int E, int G>
struct LevDiags {
    static constexpr int lo = (E - G) / 2;       // lowest diagonal is -lo
    static constexpr int n = G + 2 * lo + 1;
    // cells (diagonal d, k edits) on some path within the budget
    static constexpr bool cell(int d, int k) {
        return k >= 0 && (d < 0 ? -d : d) <= k && (d < G ? G - d : d - G) <= E - k;
    }
};

// r = t - 1 over W words, least significant first
template <int W>
IDB_HD void dec_words(const uint32_t (&t)[W], uint32_t (&r)[W]) {
#if defined(__CUDA_ARCH__)
    if (W == 1) {
        r[0] = t[0] - 1u;
    } else if (W == 2) {
        asm("sub.cc.u32 %0, %2, 1; subc.u32 %1, %3, 0;"
            : "=&r"(r[0]), "=r"(r[1 % W]) : "r"(t[0]), "r"(t[1 % W]));
    } else if (W == 3) {
        asm("sub.cc.u32 %0, %3, 1; subc.cc.u32 %1, %4, 0; subc.u32 %2, %5, 0;"
            : "=&r"(r[0]), "=&r"(r[1 % W]), "=r"(r[2 % W])
            : "r"(t[0]), "r"(t[1 % W]), "r"(t[2 % W]));
    } else {
        static_assert(W <= 4, "at most four words");
        asm("sub.cc.u32 %0, %4, 1; subc.cc.u32 %1, %5, 0; subc.cc.u32 %2, %6, 0; subc.u32 %3, %7, 0;"
            : "=&r"(r[0]), "=&r"(r[1 % W]), "=&r"(r[2 % W]), "=r"(r[3 % W])
            : "r"(t[0]), "r"(t[1 % W]), "r"(t[2 % W]), "r"(t[3 % W]));
    }
#else
    uint32_t b = 1;
    for (int w = 0; w < W; ++w) {
        const uint32_t v = t[w];
        r[w] = v - b;
        b = (uint32_t)(v < b);
    }
#endif
}

template <int W, int E, int G>
IDB_HD uint32_t lev_diag(const uint32_t (&D)[LevDiags<E, G>::n][W]) {
    using S = LevDiags<E, G>;
    static_assert(E >= G && G >= 0 && S::lo <= 1, "diagonal test: G <= E <= 3");
    uint32_t pe[S::n][W], pg[S::n][W];       // E and G masks of the previous edit count
    uint32_t last = 0;
#pragma unroll
    for (int k = 0; k <= E; ++k) {
        uint32_t ce[S::n][W], cg[S::n][W];
#pragma unroll
        for (int q = 0; q < S::n; ++q) {
            const int d = q - S::lo;
            if (!S::cell(d, k)) continue;
            uint32_t t[W];
#pragma unroll
            for (int w = 0; w < W; ++w) {
                uint32_t f = 0;
                if (S::cell(d, k - 1)) f |= pg[q][w];
                if (q > 0 && S::cell(d - 1, k - 1)) f |= pe[q > 0 ? q - 1 : 0][w];
                if (q + 1 < S::n && S::cell(d + 1, k - 1)) f |= pg[q + 1 < S::n ? q + 1 : q][w];
                t[w] = D[q][w] & ~f;
            }
            if (k == E) {                    // the one cell left: diagonal G
#pragma unroll
                for (int w = 0; w < W; ++w) last |= t[w];
                continue;
            }
            uint32_t m[W];
            dec_words<W>(t, m);
#pragma unroll
            for (int w = 0; w < W; ++w) {
                ce[q][w] = m[w] & ~t[w];
                cg[q][w] = m[w] ^ t[w];
            }
        }
#pragma unroll
        for (int q = 0; q < S::n; ++q)
            if (k < E && S::cell(q - S::lo, k)) {
#pragma unroll
                for (int w = 0; w < W; ++w) { pe[q][w] = ce[q][w]; pg[q][w] = cg[q][w]; }
            }
    }
    return last;
}

// y's bit plane (W words) moved so that bit i holds position i + d, -3 <= d <= 3
template <int W>
IDB_HD void shift_words(const uint32_t (&y)[W], int d, uint32_t (&r)[W]) {
#pragma unroll
    for (int w = 0; w < W; ++w) {
        if (d == 0) {
            r[w] = y[w];
        } else if (d > 0) {
            const uint32_t up = w + 1 < W ? y[w + 1 < W ? w + 1 : w] : 0u;
            r[w] = (y[w] >> d) | (up << (32 - d));
        } else {
            const uint32_t dn = w > 0 ? y[w > 0 ? w - 1 : 0] : 0u;
            r[w] = (y[w] << -d) | (dn >> (32 + d));
        }
    }
}

// Mismatch masks of two bit-plane records (word p*W + w, BP planes) and the
// test above: 0 iff the edit distance is at most E.
template <int BP, int W, int E, int G>
IDB_HD uint32_t lev_planes(const uint32_t *x, const uint32_t *y) {
    using S = LevDiags<E, G>;
    uint32_t D[S::n][W];
#pragma unroll
    for (int q = 0; q < S::n; ++q)
#pragma unroll
        for (int w = 0; w < W; ++w) D[q][w] = 0;
#pragma unroll
    for (int p = 0; p < BP; ++p) {
        uint32_t yw[W];
#pragma unroll
        for (int w = 0; w < W; ++w) yw[w] = y[p * W + w];
#pragma unroll
        for (int q = 0; q < S::n; ++q) {
            uint32_t r[W];
            shift_words<W>(yw, q - S::lo, r);
#pragma unroll
            for (int w = 0; w < W; ++w) D[q][w] |= x[p * W + w] ^ r[w];
        }
    }
    return lev_diag<W, E, G>(D);
}

// ---------------------------------------------------------------------------
// Work units of a same-bucket (triangular) bucket pair.  The bucket holds n
// entries; x-chunks have TX entries, y-chunks TY = q*TX.  Unit (cx, cy) exists
// iff some y of chunk cy lies above some x of chunk cx, i.e. cx < (cy+1)*q.
// Units are numbered row by row (cy major).
// ---------------------------------------------------------------------------
IDB_HD uint64_t tri_units(uint32_t ncx, uint32_t ncy, uint32_t q) {
    uint64_t s = ncx / q;                  // rows cy < s are unsaturated
    if (s > ncy) s = ncy;
    return (uint64_t)q * s * (s + 1) / 2 + (uint64_t)(ncy - s) * ncx;
}

IDB_HD void tri_decode(uint64_t k, uint32_t ncx, uint32_t q, uint32_t &cx, uint32_t &cy) {
    uint64_t s = ncx / q;
    uint64_t head = (uint64_t)q * s * (s + 1) / 2;
    if (k < head) {
        // largest c with q*c*(c+1)/2 <= k
        double kk = (double)k / (double)q;
#if defined(__CUDA_ARCH__)
        uint64_t c = (uint64_t)((sqrt(8.0 * kk + 1.0) - 1.0) * 0.5);
#else
        uint64_t c = (uint64_t)((__builtin_sqrt(8.0 * kk + 1.0) - 1.0) * 0.5);
#endif
        while (c > 0 && (uint64_t)q * c * (c + 1) / 2 > k) --c;
        while ((uint64_t)q * (c + 1) * (c + 2) / 2 <= k) ++c;
        cy = (uint32_t)c;
        cx = (uint32_t)(k - (uint64_t)q * c * (c + 1) / 2);
    } else {
        uint64_t r = k - head;
        cy = (uint32_t)(s + r / ncx);
        cx = (uint32_t)(r % ncx);
    }
}

// ---------------------------------------------------------------------------
// One step of node u's walk to the root of its tree (parents are smaller than their
// children, a root is its own parent, no root is hooked meanwhile); r is the
// ancestor reached, first u's parent.  False at the root.  A node writes its own
// parent only, at every step: the nodes that walk through u then skip what u has
// walked already, so that a chain of n nodes walked together is flat after about
// log2(n) steps.  Written at the root only, it took sqrt(4 n) (1M rows, each next
// to the one before it: 1.44 against 0.90 ms a call).
// ---------------------------------------------------------------------------
template <typename V>
IDB_HD bool climb(V *parent, uint32_t u, uint32_t &r) {
    const uint32_t pr = parent[r];
    if (pr >= r) return false;
    parent[u] = r = pr;
    return true;
}

// ---------------------------------------------------------------------------
// 64-bit mixing hash (splitmix64 finaliser applied per absorbed word).
// ---------------------------------------------------------------------------
IDB_HD uint64_t mix64(uint64_t h, uint64_t v) {
    h ^= v + 0x9E3779B97F4A7C15ull + (h << 6) + (h >> 2);
    h ^= h >> 30;
    h *= 0xBF58476D1CE4E5B9ull;
    h ^= h >> 27;
    h *= 0x94D049BB133111EBull;
    h ^= h >> 31;
    return h;
}

}  // namespace idb
