"""Replays whose data needs more entries or more bin pairs than the plan was
captured for: unrelated rows with one call each are planned, then rows of the same
lengths that form many small families, with ambiguous calls over many genes.
Nothing of such a replay may touch memory past the capacities; a batch replay
reports IDB_ERR_CAPACITY and the context stays usable, a host call runs eagerly
instead and gives the oracle's answer."""
import numpy as np
import pytest

import oracle
from immunodbscan_gb300 import Context, DeviceBatch, IdbError, cluster_workload, learned, synth

pytestmark = pytest.mark.gpu

N = 6000
CAPACITY = 6


def _pair(hamming, eps, candidates):
    """Planned and replayed workload: equal lengths, so every column is as long."""
    rng = np.random.default_rng(100 * eps + 10 * hamming + candidates)
    aa = np.frombuffer(synth.AA, np.uint8)
    length = [18 + (i // 4) % 23 for i in range(N)]
    vg = [b"IGHV%d*" % g for g in range(1, 10)]
    jg = [b"IGHJ%d*" % g for g in range(1, 10)]
    out = []
    for families in (False, True):
        seqs, vc, jc = [], [], []
        for i in range(N):
            if i % 4 == 0 or not families:
                s = rng.choice(aa, size=length[i])
                v, j = rng.integers(1, 10, 2), int(rng.integers(1, 10))
            m = s.copy()
            if families and i % 4:
                m[int(rng.integers(0, len(m)))] = rng.choice(aa)
            seqs.append(m.tobytes())
            if not families:
                v, j = (1, 1), 1
            vc.append(b"IGHV%d*01, or IGHV%d*02" % (v[0], v[1]))
            jc.append(b"IGHJ%d*01" % j)
        w = synth.from_strings(seqs, vc, jc, vg, jg, abs_eps=eps, min_pts=2, use_hamming=hamming)
        w.candidates = candidates
        out.append(w)
    return out


def _assert_oracle(clone, core, copies, w, label):
    o = oracle.cluster(w, indexed=True)
    assert np.array_equal(copies, o.copies), label
    assert np.array_equal(core, o.core), label
    assert np.array_equal(clone, o.clone_id), label


CASES = [(True, 1, 0, 0), (True, 2, 0, 1), (True, 1, 1, 0), (False, 2, 0, 0), (False, 3, 0, 1), (False, 1, 1, 0)]


@pytest.mark.parametrize("hamming,eps,candidates,schedule", CASES)
def test_replay_past_the_capacities(hamming, eps, candidates, schedule):
    wa, wb = _pair(hamming, eps, candidates)
    with Context(0) as ctx:
        if schedule:
            X, T = learned.profile(wb, ctx)
            p, _ = learned.train(X, T, ctx, epochs=3)
            learned.install(ctx, p)
        b = DeviceBatch(wa, ctx, schedule=schedule)
        b.plan()
        b.run()
        _assert_oracle(*b.results(), wa, "planned rows")
        for dst, src in ((b.seq, wb.seq_blob), (b.v, wb.v_blob), (b.j, wb.j_blob)):
            assert dst.numel() == src.size
            dst.copy_(b.torch.from_numpy(src))
        b.torch.cuda.synchronize()
        with pytest.raises(IdbError) as e:
            b.run()
        assert e.value.status == CAPACITY
        b.plan()
        b.run()
        _assert_oracle(*b.results(), wb, "planned again")
    with Context(0) as ctx:
        if schedule:
            learned.install(ctx, p)
        for k in range(3):
            g = cluster_workload(wa, ctx, schedule=schedule)
        assert g.stats.kernel_launches > 0
        g = cluster_workload(wb, ctx, schedule=schedule)
        assert g.stats.kernel_launches == 0
        _assert_oracle(g.clone_id, g.core, g.copies, wb, "eager instead of the replay")
        g = cluster_workload(wb, ctx, schedule=schedule)
        assert g.stats.kernel_launches > 0   # captured by the call before
        _assert_oracle(g.clone_id, g.core, g.copies, wb, "replay of the larger plan")
