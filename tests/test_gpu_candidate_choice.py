"""Paths that only larger calls take: the comparison of the join's pairs with the
buckets' above 2^27 join pairs (both outcomes, eager and replayed), scans of more
than 2,048 tiles, and replays whose unions start from a sample of the edges.
Against the oracle."""
import numpy as np
import pytest

import oracle
from immunodbscan_gb300 import Context, DeviceBatch, cluster_workload, synth
from test_gpu_counts import _dense
from test_gpu_parity import _random_workload, assert_same

pytestmark = pytest.mark.gpu


def _half_shared(n, n_shared, n_v):
    """n rows of 14 residues; the first n_shared have the same first half, one group of
    the join's first segment."""
    rng = np.random.default_rng(n + n_v)
    aa = np.frombuffer(synth.AA, np.uint8)
    s = rng.choice(aa, size=(n, 14))
    s[:n_shared, :7] = s[0, :7]
    near = rng.permutation(n)[: n // 4]          # a quarter one edit from another row
    s[near] = s[rng.integers(0, n, len(near))]
    s[near, rng.integers(0, 14, len(near))] = rng.choice(aa, size=len(near))
    vg = [b"IGHV%d*" % g for g in range(1, n_v + 1)]
    vc = [vg[int(g)] + b"01" for g in rng.integers(0, n_v, n)]
    return synth.from_strings([r.tobytes() for r in s], vc, [b"IGHJ1*01"] * n, vg, [b"IGHJ1*"], abs_eps=1,
                              min_pts=2, use_hamming=False)


@pytest.mark.parametrize("n,n_v,candidates", [(24000, 8, 0), (28000, 1, 1)])
def test_candidates_by_pairs(n, n_v, candidates):
    w = _half_shared(n, 23500, n_v)
    o = oracle.cluster(w, indexed=True)
    with Context(0) as ctx:
        for k in range(3):     # eager, eager and captured, replayed
            g = cluster_workload(w, ctx)
            assert (g.stats.kernel_launches > 0) == (k == 2)
            assert g.stats.candidates == candidates
            assert (g.stats.pairs_evaluated > 1 << 27) == bool(candidates)
            assert_same(g, o, w, f"host call {k}")
            assert g.stats.neighbour_pairs == o.neighbour_pairs
        b = DeviceBatch(w, ctx)
        assert b.cluster_once().candidates == candidates
        b.plan()
        assert b.run().candidates == candidates
        clone, core, copies = b.results()
        assert np.array_equal(clone, o.clone_id) and np.array_equal(core, o.core)
        assert np.array_equal(copies, o.copies)


@pytest.mark.parametrize("hamming", [True, False])
def test_scan_of_more_than_2048_tiles(gpu_ctx, hamming):
    """10 repertoires x 130 V x 60 J genes x 30 lengths x 4 classes: 9.4M buckets."""
    rng = np.random.default_rng(8 + hamming)
    n, n_rep = 6000, 10
    w0 = _random_workload(rng, n, 8, 37, list(b"ACDEFGHIKLMNPQRSTVWY"), hamming, 1, 2, n_fam=400)
    seqs = [w0.seq(i) for i in range(n)]
    vg = [b"TRAV%03d*" % g for g in range(130)]
    jg = [b"TRAJ%02d*" % g for g in range(60)]
    vc = [vg[len(s) * 4 % 130] + b"01, or " + vg[i % 130] + b"01" for i, s in enumerate(seqs)]
    jc = [jg[len(s) * 2 % 60] + b"01, or " + jg[i % 60] + b"01" for i, s in enumerate(seqs)]
    w = synth.from_strings(seqs, vc, jc, vg, jg, abs_eps=1, min_pts=2, use_hamming=hamming,
                           rep_sizes=[n // n_rep] * n_rep)
    lengths = w.lengths()
    assert n_rep * 130 * 60 * (int(lengths.max()) - int(lengths.min()) + 1) * 4 > 2048 * 4096
    w.candidates = 1
    o = oracle.cluster(w, indexed=True)
    g = cluster_workload(w, gpu_ctx)
    assert g.stats.candidates == 0
    assert_same(g, o, w, "buckets")
    assert g.stats.neighbour_pairs == o.neighbour_pairs > 0


def test_replays_with_sampled_unions():
    w = _dense(np.random.default_rng(1), 14000, 6, np.frombuffer(synth.AA, np.uint8), False, 3, 3000)
    o = oracle.cluster(w, indexed=True)
    assert o.neighbour_pairs > 1 << 20
    with Context(0) as ctx:
        for k in range(4):
            g = cluster_workload(w, ctx)
            assert (g.stats.kernel_launches > 0) == (k >= 2)
            assert_same(g, o, w, f"host call {k}")
        b = DeviceBatch(w, ctx)
        b.plan()
        for _ in range(2):
            b.run()
            clone, core, copies = b.results()
            assert np.array_equal(clone, o.clone_id) and np.array_equal(core, o.core)
