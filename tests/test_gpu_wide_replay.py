"""Plans over reference lists of more than 64 V genes, replayed on data that uses
more of them than when the plan was made: with at most 64 genes in use the side
records hold them renumbered (and Hamming joins), with more the full bitsets
decide.  Batch plans plan anew inside the run; host calls run eagerly, also from
row chunks whose join inserts were made before the genes were counted."""
import numpy as np
import pytest

import oracle
from immunodbscan_gb300 import Context, DeviceBatch, cluster_workload, synth
from test_gpu_parity import _random_workload

pytestmark = pytest.mark.gpu

N = 3000


def _pair(hamming):
    rng = np.random.default_rng(3 + hamming)
    w0 = _random_workload(rng, N, 9, 14, list(b"ACDEFGHIKL"), hamming, 1, 2, n_fam=120)
    seqs = [w0.seq(i) for i in range(N)]
    vg = [b"TRBV%03d*" % g for g in range(130)]
    jg = [b"TRBJ%02d*" % g for g in range(20)]
    jc = [jg[len(s) % 2] + b"01" for s in seqs]
    out = []
    for used in (40, 130):   # calls of two names: every column as long
        vc = [vg[len(s) % 4] + b"01, or " + vg[i % used] + b"01" for i, s in enumerate(seqs)]
        out.append(synth.from_strings(seqs, vc, jc, vg, jg, abs_eps=1, min_pts=2, use_hamming=hamming))
    return out


def _same(clone, core, copies, w, label):
    o = oracle.cluster(w)
    assert np.array_equal(copies, o.copies), label
    assert np.array_equal(core, o.core), label
    assert np.array_equal(clone, o.clone_id), label


@pytest.mark.parametrize("hamming", [True, False])
def test_batch_replay_with_more_genes_in_use(hamming):
    few, many = _pair(hamming)
    with Context(0) as ctx:
        b = DeviceBatch(few, ctx)
        b.plan()
        assert b.run().candidates == 1
        _same(*b.results(), few, "planned")
        for k, w in enumerate([many, many, few]):
            b.v.copy_(b.torch.from_numpy(w.v_blob))
            b.torch.cuda.synchronize()
            st = b.run()
            assert st.candidates == (0 if hamming else 1) and st.kernel_launches > 0
            _same(*b.results(), w, f"run {k} after the plan")


@pytest.mark.parametrize("hamming", [True, False])
@pytest.mark.parametrize("row_chunks", [0, 4])
def test_host_replay_with_more_genes_in_use(hamming, row_chunks):
    few, many = _pair(hamming)
    few.row_chunks = many.row_chunks = row_chunks
    with Context(0) as ctx:
        for k, (w, replayed) in enumerate([(few, False), (few, False), (few, True), (many, False), (many, True),
                                           (few, True)]):
            g = cluster_workload(w, ctx)
            assert (g.stats.kernel_launches > 0) == replayed, k
            assert g.stats.candidates == (1 if k < 3 or not hamming else 0), k
            _same(g.clone_id, g.core, g.copies, w, k)
