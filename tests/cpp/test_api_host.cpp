// test_api_host.cpp -- idb_api.cu on the CPU, with a stand-in for the CUDA runtime and
// the launchers (fake_cuda.hpp): lifetimes of host tables and what the host does
// on failed allocations and on the sizes the device reports.
// usage: test_api_host <test name>
#include "fake_cuda.hpp"

#include "../../immunodbscan_gb300/csrc/idb_api.cu"

#include <cstdio>

#define CHECK(c)                                                                       \
    do {                                                                               \
        if (!(c)) { std::printf("%s:%d: %s (%s)\n", __FILE__, __LINE__, #c, g_err.c_str()); std::exit(1); } \
    } while (0)

// What the scripted device reports.
struct Script {
    uint32_t lmin = 10, lmax = 12;
    uint32_t join_entries = 100, join_binpairs = 20, bucket_entries = 50, bucket_binpairs = 10;
    unsigned long long join_pairs = 1000, bucket_pairs = 2000;
    bool genes_fit = true;
    uint32_t edge_overflows = 0;     // sweeps that run over their list
    std::vector<int16_t> eps_seen;   // the eps table as the device holds it
} script;

static void note(const char *what, const Plan &P, const Buffers &B) {
    char b[128];
    std::snprintf(b, sizeof b, "%s join=%d compact=%d timing=%d", what, (int)P.join, (int)P.compact, (int)B.timing);
    fake::st().log.push_back(b);
}
static int logged(const std::string &s) {
    int n = 0;
    for (auto &x : fake::st().log) n += x.find(s) != std::string::npos;
    return n;
}

namespace idb {
void launch_survey(const Plan &P, const Buffers &B, cudaStream_t) {
    Counters *c = B.ctr;
    const uint32_t lo = script.lmin, hi = script.lmax;
    fake::push([=] { c->lmax = hi; c->lmin_inv = ~lo; c->used['A' >> 5] |= 0x1Fu << ('A' & 31); });
    (void)P;
}
void launch_check_plan(const Plan &, const Buffers &, cudaStream_t) {}
void launch_const_strings(uint8_t *, int64_t *, uint32_t, cudaStream_t) {}
void launch_call_init(const Plan &, const Buffers &, bool, cudaStream_t) {}
void launch_gene_bits(const Plan &, const Buffers &, bool, uint32_t, cudaStream_t) {}
void launch_dedupe_init(const Plan &P, const Buffers &B, cudaStream_t) {
    const int16_t *e = B.eps_tab;
    const size_t n = (size_t)P.NL * P.NL;
    fake::push([=] { script.eps_seen.assign(e, e + n); });
}
void launch_dedupe_rows(const Plan &, const Buffers &, uint32_t, cudaStream_t) {}
void launch_dedupe_final(const Plan &, const Buffers &, cudaStream_t) {}
void launch_uniques_rows(const Plan &, const Buffers &, uint32_t, cudaStream_t) {}
void launch_uniques_finish(const Plan &, const Buffers &, cudaStream_t) {}
void launch_uniques(const Plan &P, const Buffers &B, cudaStream_t) {
    Counters *c = B.ctr;
    const uint32_t n = P.N;
    fake::push([=] { c->n_uniques = n; });
}
void launch_join_init(const Plan &, const Buffers &, cudaStream_t) {}
void launch_join_insert(const Plan &, const Buffers &, int, cudaStream_t) {}
void launch_buckets(const Plan &P, const Buffers &B, cudaStream_t) {
    note("buckets", P, B);
    Counters *c = B.ctr;
    const bool join = P.join, wide = P.wide, expect = P.compact;
    fake::push([=] {
        c->n_entries = join ? script.join_entries : script.bucket_entries;
        if (join) { c->n_binpairs = script.join_binpairs; c->join_pairs = script.join_pairs; }
        if (wide) c->vj_compact = script.genes_fit;
        if (wide && expect && !script.genes_fit) c->error |= kErrGenesInUse;
    });
}
void launch_bucket_pairs(const Plan &, const Buffers &B, cudaStream_t) {
    Counters *c = B.ctr;
    fake::push([=] { c->bucket_pairs = script.bucket_pairs; });
}
void launch_fill(const Plan &P, const Buffers &B, cudaStream_t) { note("fill", P, B); }
void launch_binpairs(const Plan &P, const Buffers &B, cudaStream_t) {
    Counters *c = B.ctr;
    if (!P.join) fake::push([=] { c->n_binpairs = script.bucket_binpairs; });
}
void launch_binpairs_fill(const Plan &P, const Buffers &B, cudaStream_t) { note("binpairs", P, B); }
void launch_schedule(const Plan &, const Buffers &, cudaStream_t) {}
void launch_distance(const Plan &P, const Buffers &B, int, cudaStream_t, uint32_t) {
    note("distance", P, B);
    Counters *c = B.ctr;
    fake::push([=] {
        c->edge_reserved = 100000;
        if (script.edge_overflows) { --script.edge_overflows; c->error |= kErrEdgeOverflow; }
    });
}
void launch_count_admissible(const Plan &, const Buffers &, cudaStream_t) {}
void launch_graph(const Plan &, const Buffers &, bool, cudaStream_t, cudaEvent_t) {}
void launch_streamed_sweeps(const Plan &P, const Buffers &B, cudaStream_t) { note("streamed", P, B); }
void launch_streamed_labels(const Plan &, const Buffers &, bool, cudaStream_t) {}
void launch_outputs(const Plan &, const Buffers &, cudaStream_t, uint32_t) {}
uint32_t scan_part_needed(uint64_t n) { return (uint32_t)(n / 4096 + 2); }
void launch_features(const Buffers &, uint32_t, float *, cudaStream_t) {}
void launch_mlp_predict(const Buffers &, uint32_t, const void *, cudaStream_t) {}
void launch_mlp_grad(const float *, const float *, uint32_t, const float *, float, float *, float *, cudaStream_t) {}
void launch_adam(float *, const float *, float *, float *, float, int, cudaStream_t) {}
void launch_to_bf16(const float *, void *, cudaStream_t) {}
void launch_mlp_forward_rows(const float *, uint32_t, const void *, float *, cudaStream_t) {}
}  // namespace idb

// A call of `n` rows; the scripted device reads none of the columns.
struct Call {
    std::string seqs, v, j, vg, jg;
    std::vector<int64_t> so, vo, jo, vgo, jgo;
    std::vector<uint32_t> clone, copies;
    std::vector<int32_t> core;
    idb_input in{};
    idb_params prm{};
    idb_output out{};
    idb_stats stats{};
    Call(uint32_t n, uint32_t n_vg, uint32_t n_jg, bool hamming, int eps) {
        so = {0}; vo = {0}; jo = {0}; vgo = {0}; jgo = {0};
        for (uint32_t i = 0; i < n; ++i) {
            seqs += "ABCDEABCDE"; so.push_back((int64_t)seqs.size());
            v += "V1*01"; vo.push_back((int64_t)v.size());
            j += "J1*01"; jo.push_back((int64_t)j.size());
        }
        for (uint32_t g = 0; g < n_vg; ++g) { vg += "V" + std::to_string(g) + "*"; vgo.push_back((int64_t)vg.size()); }
        for (uint32_t g = 0; g < n_jg; ++g) { jg += "J" + std::to_string(g) + "*"; jgo.push_back((int64_t)jg.size()); }
        clone.resize(n); copies.resize(n); core.resize(n);
        in.n_rows = n;
        in.seqs = seqs.data(); in.seq_offsets = so.data();
        in.v_calls = v.data(); in.v_offsets = vo.data();
        in.j_calls = j.data(); in.j_offsets = jo.data();
        in.v_genes = vg.data(); in.v_gene_offsets = vgo.data(); in.n_v_genes = n_vg;
        in.j_genes = jg.data(); in.j_gene_offsets = jgo.data(); in.n_j_genes = n_jg;
        prm.threshold = NAN;
        prm.abs_eps = eps;
        prm.min_pts = 2;
        prm.use_hamming = hamming;
        out.clone_id = clone.data(); out.core = core.data(); out.copies = copies.data();
        out.stats = &stats;
    }
};

static idb_context *context() {
    idb_context *c = nullptr;
    CHECK(idb_context_create(0, &c) == IDB_OK);
    return c;
}

// The tables a call uploads are read by copies that may run as late as the next
// synchronisation: they have to live until then, on error returns too.
static void test_tables_outlive_their_copies() {
    idb_context *c = context();
    Call a(40, 8, 3, false, 2);
    CHECK(idb_cluster(c, &a.in, &a.prm, &a.out) == IDB_OK);
    CHECK(script.eps_seen == std::vector<int16_t>(9, 2));
    // a launch that fails right after the upload of each table
    fake::st().fail_alloc = [](size_t) { fake::st().last = cudaErrorUnknown; return false; };
    Call b(5000, 60, 20, false, 3);
    CHECK(idb_cluster(c, &b.in, &b.prm, &b.out) == IDB_ERR_CUDA);
    fake::st().fail_alloc = nullptr;
    fake::st().last = cudaSuccess;
    CHECK(idb_cluster(c, &b.in, &b.prm, &b.out) == IDB_OK);
    CHECK(script.eps_seen == std::vector<int16_t>(9, 3));
    std::vector<uint64_t> words(5000);
    CHECK(idb_diag_gene_bits(c, b.v.data(), b.vo.data(), 5000, b.vg.data(), b.vgo.data(), 60, words.data()) == IDB_OK);
    CHECK(idb_context_destroy(c) == IDB_OK);
    fake::drain();
}

// A batch plan over a wide gene list, made while the genes in use fitted the side
// records: a run on data that uses more of them plans anew by itself (the
// join for Hamming needs them to fit) and a later run replays that plan.
static void test_batch_run_with_more_genes_in_use() {
    for (const bool hamming : {true, false}) {
        idb_context *c = context();
        Call a(200, 100, 3, hamming, 1);
        a.out.stats = nullptr;
        script = Script();
        CHECK(idb_batch_plan(c, &a.in, &a.prm, &a.out) == IDB_OK);
        fake::st().log.clear();
        CHECK(idb_batch_run(c, &a.stats) == IDB_OK);
        CHECK(a.stats.candidates == 1 && c->plan.compact && fake::st().log.empty());
        script.genes_fit = false;
        CHECK(idb_batch_run(c, &a.stats) == IDB_OK);
        CHECK(!c->plan.compact && a.stats.candidates == (hamming ? 0u : 1u));
        CHECK(a.stats.n_entries == (hamming ? script.bucket_entries : script.join_entries));
        CHECK(logged(std::string("distance join=") + (hamming ? "0" : "1") + " compact=0") == 2);   // and captured
        fake::st().log.clear();
        CHECK(idb_batch_run(c, &a.stats) == IDB_OK);
        script.genes_fit = true;
        CHECK(idb_batch_run(c, &a.stats) == IDB_OK);
        CHECK(fake::st().log.empty());
        CHECK(idb_context_destroy(c) == IDB_OK);
    }
}

// A join whose table, entries or bin pairs the device has no room for: every entry
// point takes the buckets instead, as it would without a join, and gives the join's
// memory back first; without room for the buckets either, out of memory.
static void test_buckets_when_the_join_does_not_fit() {
    struct Short { const char *what; uint32_t entries, binpairs; size_t lo, hi; };
    const Short shorts[] = {{"table", 100, 20, 1000000, 100000000},
                            {"entries", 1000000, 20, 15000000, 100000000},
                            {"bin pairs", 100, 1000000, 15000000, 100000000}};
    for (const bool hamming : {false, true})
        for (const Short &sh : shorts) {
            if (hamming && sh.hi == 100000000 && sh.lo == 1000000) continue;   // its table is smaller
            idb_context *c = context();
            Call a(5000, 60, 20, hamming, hamming ? 2 : 3);
            script = Script();
            CHECK(idb_cluster(c, &a.in, &a.prm, &a.out) == IDB_OK && a.stats.candidates == 1);
            CHECK(idb_context_destroy(c) == IDB_OK);
            c = context();
            script.join_entries = sh.entries;
            script.join_binpairs = sh.binpairs;
            fake::st().fail_alloc = [&](size_t n) { return n >= sh.lo && n < sh.hi; };
            for (int k = 0; k < 3; ++k) {   // eager, eager and captured, replayed
                CHECK(idb_cluster(c, &a.in, &a.prm, &a.out) == IDB_OK);
                CHECK(a.stats.candidates == 0 && a.stats.n_entries == script.bucket_entries);
            }
            CHECK(!c->buf[bJnTab].p && !c->buf[bJnPos].p);
            CHECK(idb_cluster_device(c, &a.in, &a.prm, &a.out) == IDB_OK && a.stats.candidates == 0);
            idb_stats st{};
            idb_output o = a.out;
            o.stats = nullptr;
            CHECK(idb_batch_plan(c, &a.in, &a.prm, &o) == IDB_OK && idb_batch_run(c, &st) == IDB_OK);
            CHECK(st.candidates == 0);
            idb_tuning t{};
            CHECK(idb_autotune(c, &a.in, &a.prm, &t) == IDB_OK && t.n_tried > 0);
            std::vector<float> f(16 * script.bucket_binpairs), y(script.bucket_binpairs);
            uint64_t n = 0;
            CHECK(idb_profile_binpairs(c, &a.in, &a.prm, f.data(), y.data(), y.size(), &n) == IDB_OK);
            CHECK(n == script.bucket_binpairs);
            fake::st().fail_alloc = [](size_t b) { return b >= 20000; };
            CHECK(idb_context_destroy(c) == IDB_OK);
            c = context();
            CHECK(idb_cluster(c, &a.in, &a.prm, &a.out) == IDB_ERR_OUT_OF_MEMORY);
            fake::st().fail_alloc = nullptr;
            CHECK(idb_cluster(c, &a.in, &a.prm, &a.out) == IDB_OK && a.stats.candidates == 1);
            CHECK(idb_context_destroy(c) == IDB_OK);
        }
}

// Which side records hold every gene in use and so decide a hit by themselves.
static void test_side_records_decide() {
    struct { uint32_t gv, gj; bool join, fits, exact; } cases[] = {
        {64, 30, true, true, true},  {64, 30, false, true, true},  {64, 31, true, true, true},
        {64, 31, true, false, false}, {64, 31, false, false, true}, {64, 32, false, false, true},
        {64, 33, false, false, false}, {65, 32, false, false, false}, {65, 32, false, true, true},
        {300, 200, true, true, true}};
    for (const auto &t : cases) {
        Plan P;
        P.Gv = t.gv;
        P.Gj = t.gj;
        P.join = t.join;
        P.wide = t.gv > 64 || t.gj > 30;
        P.compact = P.wide && t.fits;
        CHECK(P.side_exact() == t.exact);
    }
}

// Candidates of a call whose join has many pairs: the buckets are counted and the
// smaller side taken, eagerly and in the plan captured after; the join's time
// stays in the bucket phase (one kernel writes its time stamp).
static void test_candidates_by_pairs() {
    for (const bool buckets_win : {false, true}) {
        idb_context *c = context();
        Call a(500, 8, 3, false, 2);
        script = Script();
        script.join_pairs = kJoinSurePairs + 1;
        script.bucket_pairs = buckets_win ? kJoinSurePairs : kJoinSurePairs + 1;
        fake::st().log.clear();
        CHECK(idb_cluster_device(c, &a.in, &a.prm, &a.out) == IDB_OK);
        CHECK(a.stats.candidates == (buckets_win ? 0u : 1u));
        CHECK(a.stats.n_entries == (buckets_win ? script.bucket_entries : script.join_entries));
        CHECK(c->h_ctr->n_binpairs == (buckets_win ? script.bucket_binpairs : script.join_binpairs));
        CHECK(logged("buckets join=1") == 1 && logged("buckets join=0") == 1);
        CHECK(logged("buckets join=1 compact=0 timing=1") == 1 && logged("buckets join=0 compact=0 timing=0") == 1);
        CHECK(logged(std::string("distance join=") + (buckets_win ? "0" : "1") + " compact=0 timing=1") == 1);
        idb_output o = a.out;
        o.stats = nullptr;
        CHECK(idb_batch_plan(c, &a.in, &a.prm, &o) == IDB_OK);
        CHECK(idb_batch_run(c, &a.stats) == IDB_OK && a.stats.candidates == (buckets_win ? 0u : 1u));
        CHECK(a.stats.n_entries == (buckets_win ? script.bucket_entries : script.join_entries));
        CHECK(idb_context_destroy(c) == IDB_OK);
    }
}

// A sweep that runs over its list is repeated with a longer one, or streamed under
// an edge-memory limit: the distance phase begins with the first sweep.
static void test_repeated_sweeps_keep_the_stamp() {
    for (const int mb : {0, 1, -1}) {
        idb_context *c = context();
        Call a(500, 8, 3, false, 2);
        script = Script();
        script.edge_overflows = mb < 0 ? 0 : 1;
        a.prm.edge_memory_mb = mb;
        fake::st().log.clear();
        CHECK(idb_cluster_device(c, &a.in, &a.prm, &a.out) == IDB_OK);
        CHECK(a.stats.streamed == (mb != 0));
        const std::string at = " join=1 compact=0 timing=";
        CHECK(logged("distance" + at + "1") == (mb >= 0) && logged("distance" + at + "0") == (mb == 0));
        CHECK(logged("streamed" + at + "0") == (mb > 0) && logged("streamed" + at + "1") == (mb < 0));
        CHECK(idb_context_destroy(c) == IDB_OK);
    }
}

// The eps table of a wide length range (2 bytes a pair of lengths) goes to the device
// from where it was made, without a second copy of it on the host.
static void test_long_eps_table() {
    for (const uint32_t lmax : {40u, 3000u}) {
        idb_context *c = context();
        Call a(100, 8, 3, true, 2);
        script = Script();
        script.lmin = 1;
        script.lmax = lmax;
        CHECK(idb_cluster(c, &a.in, &a.prm, &a.out) == IDB_OK);
        CHECK(script.eps_seen == std::vector<int16_t>((size_t)lmax * lmax, 2));
        {
            Pipeline pl;
            pl.c = c;
            CHECK(stage_inputs_and_survey(pl, &a.in, true) == IDB_OK);
            CHECK(derive_plan(pl, &a.prm) == IDB_OK && alloc_fixed(pl) == IDB_OK);
            CHECK(pl.plan_tables.bytes.size() <= 70000);
            CHECK(read_counters(pl) == IDB_OK);
            CHECK(std::memcmp(pl.B.codemap, pl.P.codemap, 256) == 0);
        }
        CHECK(idb_context_destroy(c) == IDB_OK);
    }
}

int main(int argc, char **argv) {
    const std::map<std::string, void (*)()> tests = {
        {"tables_outlive_their_copies", test_tables_outlive_their_copies},
        {"batch_run_with_more_genes_in_use", test_batch_run_with_more_genes_in_use},
        {"buckets_when_the_join_does_not_fit", test_buckets_when_the_join_does_not_fit},
        {"side_records_decide", test_side_records_decide},
        {"candidates_by_pairs", test_candidates_by_pairs},
        {"repeated_sweeps_keep_the_stamp", test_repeated_sweeps_keep_the_stamp},
        {"long_eps_table", test_long_eps_table},
    };
    const auto it = tests.find(argc > 1 ? argv[1] : "");
    if (it == tests.end()) { std::printf("unknown test\n"); return 2; }
    it->second();
    std::printf("ok\n");
    return 0;
}
