"""Reference lists of more than 64 V or 30 J genes: the side records hold the
genes in use, renumbered, when at most 64 V and 30 J genes are; otherwise the
full bitsets decide.  Join and buckets, both distances, against the oracle."""
import numpy as np
import pytest

import oracle
from immunodbscan_gb300 import cluster_workload, synth
from test_gpu_parity import _random_workload, assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hamming", [True, False])
@pytest.mark.parametrize("used_v,used_j", [(5, 3), (64, 30), (65, 30), (64, 31), (140, 44)])
def test_wide_lists(gpu_ctx, hamming, used_v, used_j):
    rng = np.random.default_rng(used_v + used_j)
    n = 4000
    w0 = _random_workload(rng, n, 9, 14, list(b"ACDEFGHIKL"), hamming, 1, 2, n_fam=120)
    seqs = [w0.seq(i) for i in range(n)]
    vg = [b"TRBV%03d*" % g for g in range(150)]
    jg = [b"TRBJ%03d*" % g for g in range(45)]
    v_in = np.sort(rng.choice(150, used_v, replace=False))     # the genes calls name
    j_in = np.sort(rng.choice(45, used_j, replace=False))
    vc, jc = [], []
    for i, s in enumerate(seqs):
        # every gene in use appears; neighbours mostly share a length-dependent gene
        gv = {int(v_in[len(s) % min(4, used_v)])} | set(v_in[rng.choice(used_v, int(rng.integers(0, 3)))].tolist())
        gj = {int(j_in[len(s) % min(2, used_j)])} | set(j_in[rng.choice(used_j, int(rng.integers(0, 2)))].tolist())
        if i < used_v:
            gv.add(int(v_in[i]))
        if i < used_j:
            gj.add(int(j_in[i]))
        vc.append(b", or ".join(vg[g] + b"01" for g in sorted(gv)))
        jc.append(b", or ".join(jg[g] + b"01" for g in sorted(gj)))
    w = synth.from_strings(seqs, vc, jc, vg, jg, abs_eps=1, min_pts=2, use_hamming=hamming)
    o = oracle.cluster(w)
    for candidates in (0, 1):
        w.candidates = candidates
        g = cluster_workload(w, gpu_ctx)
        assert_same(g, o, w, f"wide {used_v}/{used_j} candidates={candidates}")
        assert g.stats.neighbour_pairs == o.neighbour_pairs
        fits = used_v <= 64 and used_j <= 30
        assert g.stats.candidates == (0 if candidates or (hamming and not fits) else 1)
