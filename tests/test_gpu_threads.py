"""Threads with a context each: calls whose kernels need different amounts of dynamic
shared memory (long and short gene lists; edit distances above 3 on long and short
sequences), in turn and at the same time, against the oracle."""
import threading

import numpy as np
import pytest

import oracle
from immunodbscan_gb300 import Context, cluster_workload, synth
from test_gpu_parity import _random_workload

pytestmark = pytest.mark.gpu


def _workloads():
    out = []
    for k, (n_v, hi, hamming, eps) in enumerate([(400, 16, True, 1), (3, 14, True, 1), (60, 60, False, 5),
                                                 (5, 20, False, 5), (90, 120, False, 6), (40, 30, False, 2)]):
        rng = np.random.default_rng(k)
        w = _random_workload(rng, 1500, hi - 6, hi, list(b"ACDEFGHIKLMNPQRSTVWY"), hamming, eps, 2, n_fam=150)
        seqs = [w.seq(i) for i in range(w.n)]
        vg = [b"IGHV%03d*" % g for g in range(n_v)]
        vc = [vg[len(s) % n_v] + b"01, or " + vg[(7 * i) % n_v] + b"01" for i, s in enumerate(seqs)]
        out.append(synth.from_strings(seqs, vc, [b"IGHJ1*01"] * w.n, vg, [b"IGHJ1*", b"IGHJ2*"], abs_eps=eps,
                                      min_pts=2, use_hamming=hamming))
    return [(w, oracle.cluster(w)) for w in out]


def _call(w, o, ctx):
    g = cluster_workload(w, ctx)
    assert np.array_equal(g.copies, o.copies) and np.array_equal(g.core, o.core)
    assert np.array_equal(g.clone_id, o.clone_id)


def _in_threads(jobs):
    failed = []

    def run(job):
        try:
            job()
        except Exception as e:  # noqa: BLE001  (reported by the main thread)
            failed.append(repr(e))
    threads = [threading.Thread(target=run, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


@pytest.mark.parametrize("big,small", [(0, 1), (4, 3), (2, 3)])
def test_in_turn(big, small):
    """A thread's larger kernels still launch after another thread used smaller ones."""
    ws = _workloads()
    turn = [threading.Semaphore(1), threading.Semaphore(0)]

    def job(me, which):
        def run():
            with Context(0) as ctx:
                for _ in range(2):
                    turn[me].acquire(timeout=60)
                    try:
                        _call(*ws[which], ctx)
                    finally:
                        turn[1 - me].release()
        return run
    _in_threads([job(0, big), job(1, small)])


def test_at_the_same_time():
    ws = _workloads()

    def job(t):
        def run():
            rng = np.random.default_rng(t)
            with Context(0) as ctx:
                for _ in range(25):     # repeats replay the shape's captured sequence
                    w, o = ws[int(rng.integers(0, len(ws)))]
                    for _ in range(int(rng.integers(1, 4))):
                        _call(w, o, ctx)
        return run
    _in_threads([job(t) for t in range(6)])
