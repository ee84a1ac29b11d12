"""Gene lists at the width of the buckets' side records (64 V and 32 J genes, all in
use; a join's hold 30 J genes): hits decided from the first words of the bitsets,
one more gene and from the full ones.  Against the oracle."""
import numpy as np
import pytest

import oracle
from immunodbscan_gb300 import cluster_workload, synth
from test_gpu_parity import _random_workload, assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hamming,eps", [(True, 1), (True, 4), (False, 1), (False, 5)])
@pytest.mark.parametrize("n_v,n_j", [(64, 30), (64, 31), (64, 32), (64, 33), (65, 32)])
def test_lists_at_the_side_records_width(gpu_ctx, hamming, eps, n_v, n_j):
    rng = np.random.default_rng(n_v * n_j + eps)
    n = 4000
    w0 = _random_workload(rng, n, 9, 14, list(b"ACDEFGHIKL"), hamming, eps, 2, n_fam=150)
    seqs = [w0.seq(i) for i in range(n)]
    vg = [b"TRAV%02d*" % g for g in range(n_v)]
    jg = [b"TRAJ%02d*" % g for g in range(n_j)]
    # neighbours mostly share the last genes of the lists or lower ones as well
    vc = [vg[-1 - len(s) % 3] + b"01, or " + vg[i % n_v] + b"01" for i, s in enumerate(seqs)]
    jc = [jg[-1 - len(s) % 2] + b"01, or " + jg[(i // 3) % n_j] + b"01" for i, s in enumerate(seqs)]
    w = synth.from_strings(seqs, vc, jc, vg, jg, abs_eps=eps, min_pts=2, use_hamming=hamming)
    o = oracle.cluster(w, indexed=True)
    for candidates in (0, 1):
        w.candidates = candidates
        g = cluster_workload(w, gpu_ctx)
        assert_same(g, o, w, f"{n_v} V, {n_j} J, candidates={candidates}")
        assert g.stats.neighbour_pairs == o.neighbour_pairs
