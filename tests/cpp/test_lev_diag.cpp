// The diagonal edit-distance test of bitops.cuh against a full dynamic program,
// for every admissible (eps, length gap) and 1 to 4 words, with code 0 (the pad
// code) among the residues and lengths on both sides of a word boundary.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "../../immunodbscan_gb300/csrc/bitops.cuh"

using namespace idb;

static int dp(const std::vector<uint8_t> &x, const std::vector<uint8_t> &y) {
    std::vector<int> row(y.size() + 1);
    for (size_t j = 0; j <= y.size(); ++j) row[j] = (int)j;
    for (size_t i = 1; i <= x.size(); ++i) {
        int diag = row[0];
        row[0] = (int)i;
        for (size_t j = 1; j <= y.size(); ++j) {
            const int up = row[j];
            row[j] = std::min({diag + (x[i - 1] != y[j - 1]), up + 1, row[j - 1] + 1});
            diag = up;
        }
    }
    return row[y.size()];
}

template <int BP, int W>
static void planes(const std::vector<uint8_t> &s, uint32_t *rec) {
    std::memset(rec, 0, 4 * BP * W);
    for (size_t i = 0; i < s.size(); ++i)
        for (int p = 0; p < BP; ++p)
            rec[p * W + i / 32] |= (uint32_t)((s[i] >> p) & 1u) << (i % 32);
}

static long checked = 0;

template <int BP, int W, int E, int G>
static void one(const std::vector<uint8_t> &x, const std::vector<uint8_t> &y) {
    uint32_t rx[BP * W], ry[BP * W];
    planes<BP, W>(x, rx);
    planes<BP, W>(y, ry);
    const bool got = lev_planes<BP, W, E, G>(rx, ry) == 0;
    const bool want = dp(x, y) <= E;
    ++checked;
    if (got != want) {
        std::printf("E=%d G=%d W=%d: got %d want %d\n x:", E, G, W, got, want);
        for (auto c : x) std::printf(" %d", c);
        std::printf("\n y:");
        for (auto c : y) std::printf(" %d", c);
        std::printf("\n");
        std::exit(1);
    }
}

// every pair of strings over `A` letters with lengths m and m + G
template <int E, int G>
static void exhaustive(int A, int m) {
    const int n = m + G;
    long nx = 1, ny = 1;
    for (int i = 0; i < m; ++i) nx *= A;
    for (int i = 0; i < n; ++i) ny *= A;
    std::vector<uint8_t> x(m), y(n);
    for (long a = 0; a < nx; ++a) {
        long v = a;
        for (int i = 0; i < m; ++i) { x[i] = (uint8_t)(v % A); v /= A; }
        for (long b = 0; b < ny; ++b) {
            long u = b;
            for (int i = 0; i < n; ++i) { y[i] = (uint8_t)(u % A); u /= A; }
            one<2, 1, E, G>(x, y);
        }
    }
}

// y from x by E-ish random edits that leave it G longer, and unrelated pairs
template <int BP, int W, int E, int G>
static void random_pairs(std::mt19937 &rng, int A, int trials) {
    const int lens[] = {32 * W - 3, 32 * W - 2, 32 * W - 1, 32 * W, 32 * (W - 1) + 1, 32 * (W - 1) + 2,
                        32 * W - 15, 32 * (W - 1) + 7};
    for (int n : lens) {
        if (n < G) continue;
        for (int k = 0; k < trials; ++k) {
            const int m = n - G;
            std::vector<uint8_t> x(m);
            for (auto &c : x) c = (uint8_t)(rng() % A);
            std::vector<uint8_t> y = x;
            int ins = G, del = 0, sub = 0;
            for (int e = G + (int)(rng() % 3); e + 1 < E + 2 && rng() % 2; ++e) ++sub;
            if (rng() % 2) { ++ins; ++del; }
            for (int i = 0; i < del && !y.empty(); ++i) y.erase(y.begin() + rng() % y.size());
            while ((int)y.size() < n) {
                const size_t at = rng() % 4 == 0 ? (rng() % 2 ? 0 : y.size()) : rng() % (y.size() + 1);
                y.insert(y.begin() + at, (uint8_t)(rng() % A));
            }
            (void)ins;
            for (int i = 0; i < sub && !y.empty(); ++i) y[rng() % y.size()] = (uint8_t)(rng() % A);
            y.resize(n);
            one<BP, W, E, G>(x, y);
        }
    }
}

template <int E, int G>
static void all(std::mt19937 &rng) {
    for (int m = 0; m + G <= 7; ++m)
        if (m + G <= 6 || E <= 2) exhaustive<E, G>(2, m);
    for (int m = 0; m + G <= 5; ++m) exhaustive<E, G>(3, m);
    random_pairs<2, 1, E, G>(rng, 2, 3000);
    random_pairs<2, 1, E, G>(rng, 4, 3000);
    random_pairs<5, 1, E, G>(rng, 20, 2000);
    random_pairs<2, 2, E, G>(rng, 3, 1500);
    random_pairs<5, 2, E, G>(rng, 20, 800);
    random_pairs<2, 3, E, G>(rng, 4, 800);
    random_pairs<5, 3, E, G>(rng, 32, 400);
    random_pairs<2, 4, E, G>(rng, 2, 400);
    random_pairs<5, 4, E, G>(rng, 20, 400);
}

int main() {
    std::mt19937 rng(7);
    all<0, 0>(rng);
    all<1, 0>(rng);
    all<1, 1>(rng);
    all<2, 0>(rng);
    all<2, 1>(rng);
    all<2, 2>(rng);
    all<3, 0>(rng);
    all<3, 1>(rng);
    all<3, 2>(rng);
    all<3, 3>(rng);
    std::printf("ok %ld\n", checked);
    return 0;
}
