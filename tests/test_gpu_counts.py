"""Neighbour counts and unions of dense graphs: the distance kernels add each
entry's neighbours' copies per tile, per small and per tiny bin pair, and long
edge lists are merged through a sampled forest.  Families with repeated rows
(copies of 1 to 40), minPts on both sides of the counts that occur, edge lists
below and above the sampled length, eagerly and in streamed mode."""
import numpy as np
import pytest

import oracle
from immunodbscan_gb300 import cluster_workload, synth
from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


def _dense(rng, n_uniques, n_roots, alphabet, hamming, eps, min_pts):
    roots = [rng.choice(alphabet, size=int(rng.integers(13, 16))) for _ in range(n_roots)]
    seqs = []
    for k in range(n_uniques):
        s = roots[int(rng.integers(0, n_roots)) if k % 3 else 0].copy()
        for _ in range(int(rng.integers(0, 3))):
            s[int(rng.integers(0, len(s)))] = rng.choice(alphabet)
        if not hamming and rng.random() < 0.1:
            s = np.delete(s, int(rng.integers(0, len(s))))
        copies = 1 if rng.random() < 0.7 else int(rng.integers(2, 41))
        seqs += [s.astype(np.uint8).tobytes()] * copies
    order = rng.permutation(len(seqs))
    seqs = [seqs[int(i)] for i in order]
    return synth.from_strings(seqs, [b"IGHV1*01"] * len(seqs), [b"IGHJ1*01"] * len(seqs), [b"IGHV1*"],
                              [b"IGHJ1*"], abs_eps=eps, min_pts=min_pts, use_hamming=hamming)


@pytest.mark.parametrize("hamming,eps", [(True, 1), (True, 2), (True, 4), (False, 1), (False, 3)])
@pytest.mark.parametrize("min_pts", [3, 60, 2500])
@pytest.mark.parametrize("n_uniques", [300, 4500])
def test_dense_counts(gpu_ctx, hamming, eps, min_pts, n_uniques):
    rng = np.random.default_rng(n_uniques + 10 * eps + hamming)
    w = _dense(rng, n_uniques, 6, np.frombuffer(b"ACDEFG", np.uint8), hamming, eps, min_pts)
    o = oracle.cluster(w, indexed=True)
    for budget in (0, -1):
        w.edge_memory_mb = budget
        g = cluster_workload(w, gpu_ctx)
        assert_same(g, o, w, f"hamming={hamming} eps={eps} minPts={min_pts} budget={budget}")
        assert g.stats.neighbour_pairs == o.neighbour_pairs


def test_sampled_unions(gpu_ctx):
    """More than 2^20 neighbour pairs, many components and borders."""
    rng = np.random.default_rng(1)
    w = _dense(rng, 14000, 6, np.frombuffer(b"ACDEFGHIKLMNPQRSTVWY", np.uint8), False, 3, 3000)
    o = oracle.cluster(w, indexed=True)
    assert o.neighbour_pairs > (1 << 20)
    g = cluster_workload(w, gpu_ctx)
    assert_same(g, o, w, "sampled unions")
    assert g.stats.neighbour_pairs == o.neighbour_pairs
