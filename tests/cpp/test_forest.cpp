// CPU test of climb (bitops.cuh): a forest flattened by one walk per node, all walks
// one step a round.  Nodes of a round are taken from the largest down, so that
// every step reads what the round before left (a step writes its own node, a
// larger one).  Exit status 0 = every node at its root within the bound.
#include "bitops.cuh"

#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

using namespace idb;

static int flatten(std::vector<uint32_t> parent, const char *what) {
    const uint32_t n = (uint32_t)parent.size();
    std::vector<uint32_t> root(n), at(n);
    for (uint32_t u = 0; u < n; ++u) root[u] = parent[u] == u ? u : root[parent[u]];
    for (uint32_t u = 0; u < n; ++u) at[u] = parent[u];
    std::vector<char> live(n, 1);
    uint32_t left = n, rounds = 0, bound = 4;
    while ((1u << (bound - 3)) < n) ++bound;   // log2(n) rounded up, and a few
    while (left && rounds < 4 * bound) {
        ++rounds;
        for (uint32_t u = n; u-- > 0;)
            if (live[u] && !climb(parent.data(), u, at[u])) { live[u] = 0; --left; }
    }
    int bad = left != 0 || rounds > bound;
    for (uint32_t u = 0; u < n; ++u) bad += parent[u] != root[u];
    if (bad) std::printf("%s n=%u: %u rounds (bound %u), %u left, %d bad\n", what, n, rounds, bound, left, bad);
    return bad;
}

int main() {
    int bad = 0;
    std::mt19937 rng(5);
    for (uint32_t n : {1u, 2u, 3u, 33u, 1000u, 200000u}) {
        std::vector<uint32_t> p(n);
        for (uint32_t u = 0; u < n; ++u) p[u] = u ? u - 1 : 0;
        bad += flatten(p, "chain");
        for (uint32_t u = 0; u < n; ++u) p[u] = u < 7 ? u : u - 7;
        bad += flatten(p, "seven chains");
        for (uint32_t u = 0; u < n; ++u) p[u] = rng() % (u + 1);
        bad += flatten(p, "random forest");
        for (uint32_t u = 0; u < n; ++u) p[u] = u - std::min<uint32_t>(u, rng() % 4);
        bad += flatten(p, "deep forest");
    }
    return bad != 0;
}
