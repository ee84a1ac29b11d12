"""Hamming eps 0 on sequences of more than one word: rows that agree in their first 32
residues and differ later are no neighbours, in tiny, small and tiled bins, by
the buckets and by the join.  Against the oracle."""
import numpy as np
import pytest

import oracle
from immunodbscan_gb300 import cluster_workload, synth
from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [32, 33, 64, 70, 97, 128])
@pytest.mark.parametrize("alphabet", [b"ACGT", b"ACDEFGHIKLMNPQRSTVWY"])
@pytest.mark.parametrize("n,n_genes", [(900, 60), (900, 6), (900, 1)])
def test_differences_past_the_first_word(gpu_ctx, length, alphabet, n, n_genes):
    rng = np.random.default_rng(length + n_genes)
    alpha = np.frombuffer(alphabet, np.uint8)
    root = rng.choice(alpha, size=length)
    seqs = []
    for i in range(n):
        s = root.copy()
        if i % 3:       # one residue, mostly past the first word
            s[int(rng.integers(min(32, length - 1), length))] = rng.choice(alpha)
        seqs.append(s.tobytes())
    vg = [b"IGHV%02d*" % g for g in range(n_genes + 1)]
    vc = [vg[i % n_genes] + b"01, or " + vg[int(g)] + b"01" for i, g in enumerate(rng.integers(0, n_genes + 1, n))]
    w = synth.from_strings(seqs, vc, [b"IGHJ1*01"] * n, vg, [b"IGHJ1*"], abs_eps=0, min_pts=2, use_hamming=True)
    o = oracle.cluster(w)
    for candidates in (0, 1):
        w.candidates = candidates
        g = cluster_workload(w, gpu_ctx)
        assert_same(g, o, w, f"candidates={candidates}")
        assert g.stats.neighbour_pairs == o.neighbour_pairs
