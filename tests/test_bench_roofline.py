"""bench.py's integer-operation count of the distance kernel: per pair (Hamming), per
text column (the recurrence), and none where pairs of several eps and length gaps
cost different numbers of operations (the diagonal test)."""
import types

import bench
from immunodbscan_gb300 import synth


def _last(pairs, columns):
    return types.SimpleNamespace(pairs_evaluated=pairs, lev_columns=columns)


def test_distance_work():
    w = synth.workload(2, scale=0.002)
    assert bench.distance_work(w, _last(1000, 0)) == ("k_hamming", "pair", 1000, 8)
    w = synth.workload(3, scale=0.002)
    assert bench.distance_work(w, _last(1000, 70)) == ("k_levenshtein", "pair-column (text residue)", 70, 16)
    for k in (1, 3, 4):     # two words of two planes; one word, eps 2; eps 0 to 3 by length
        w = synth.workload(k, scale=0.002)
        assert bench.distance_work(w, _last(1000, 0)) == ("k_lev_diag", "pair", 1000, None)
