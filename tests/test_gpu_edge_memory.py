"""Short neighbour lists: a warp reserves few slots at a time in a short list, so that
pairs which fit an edge-memory limit are kept (one sweep) although nearly every
resident warp finds some, and lists that do run over are grown or streamed.  All
distance kernels, against the oracle."""
import numpy as np
import pytest

import oracle
from immunodbscan_gb300 import Context, cluster_workload, synth
from test_gpu_parity import _random_workload, assert_same


def _check(w, streamed, label):
    o = oracle.cluster(w, indexed=True)
    with Context(0) as ctx:     # no list from an earlier call
        g = cluster_workload(w, ctx)
    assert_same(g, o, w, label)
    assert g.stats.neighbour_pairs == o.neighbour_pairs, label
    assert g.stats.streamed == streamed, label


pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("workload,scale,mb,streamed", [(0, 1.0, 1, 0), (0, 2.0, 1, 0), (0, 4.0, 1, 0), (0, 4.0, 0, 0),
                                                        (2, 0.01, 2, 0), (2, 0.04, 8, 0), (3, 0.01, 1, 1),
                                                        (3, 0.01, 0, 0), (1, 0.05, 0, 0)])
def test_limits(workload, scale, mb, streamed):
    w = synth.workload(workload, scale=scale, seed=5)
    w.edge_memory_mb = mb
    _check(w, streamed, f"workload {workload} x {scale}, {mb} MB")


@pytest.mark.parametrize("hamming,eps,alphabet", [(True, 1, 20), (False, 1, 20), (False, 5, 20), (True, 3, 90),
                                                  (False, 2, 90)])
@pytest.mark.parametrize("mb", [0, 1])
def test_every_kernel(hamming, eps, alphabet, mb):
    """Few rows and many pairs (lists that run over 65,536 slots) or few of them, with
    bit planes, code bytes (eps 5) and more than 32 residue values."""
    rng = np.random.default_rng(eps + alphabet)
    for n_fam in (12, 900):
        w = _random_workload(rng, 8000, 12, 20, list(range(33, 33 + alphabet)), hamming, eps, 2, n_fam=n_fam)
        w.edge_memory_mb = mb
        o = oracle.cluster(w, indexed=True)
        # (8000 rows: a first list of 65,536 slots under either limit)
        _check(w, int(mb > 0 and o.neighbour_pairs > 65536), f"{n_fam} families, {o.neighbour_pairs} pairs")
