"""Edit distances up to 3 by the diagonal test (furthest-reaching points on
mismatch masks): the routine on the CPU against a full DP, and the kernels
against the oracle at word boundaries, every eps, both plane counts, and bins
from one entry to several tiles."""
import os
import subprocess

import numpy as np
import pytest

import oracle
from immunodbscan_gb300 import synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_diagonal_test_on_cpu(tmp_path):
    exe = tmp_path / "test_lev_diag"
    subprocess.run(["g++", "-O2", "-std=c++17", os.path.join(ROOT, "tests", "cpp", "test_lev_diag.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def _families(rng, n, lo, hi, alphabet, n_fam, edits):
    """Members of n_fam families, each 0..edits random substitutions, insertions
    and deletions (ends included) away from its root, lengths kept in [lo, hi]."""
    roots = [rng.choice(alphabet, size=int(rng.integers(lo, hi + 1))).astype(np.uint8).tolist()
             for _ in range(n_fam)]
    out = []
    for _ in range(n):
        s = list(roots[int(rng.integers(0, n_fam))])
        for _ in range(int(rng.integers(0, edits + 1))):
            kind, p = int(rng.integers(0, 3)), int(rng.integers(0, len(s) + 1))
            p = 0 if rng.random() < 0.15 else (len(s) if rng.random() < 0.15 else p)
            c = int(rng.choice(alphabet))
            if kind == 0 and len(s) < hi:
                s.insert(p, c)
            elif kind == 1 and len(s) > lo:
                del s[min(p, len(s) - 1)]
            elif s:
                s[min(p, len(s) - 1)] = c
        out.append(bytes(s))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("eps", [0, 1, 2, 3])
@pytest.mark.parametrize("lo,hi,alphabet", [(1, 6, b"AC"), (8, 25, b"ACDEFGHIKLMNPQRSTVWY"), (28, 34, b"ACGT"),
                                            (30, 33, b"ACDEFGHIKLMNPQRSTVWY"), (62, 66, b"ACGT"),
                                            (61, 65, b"ACDEFGHIKLMNPQRSTVWY"), (93, 98, b"ACGT"),
                                            (124, 128, b"ACDEFGHIKLMNPQRSTVWY")])
def test_levenshtein_vs_oracle(gpu_ctx, eps, lo, hi, alphabet):
    from immunodbscan_gb300 import cluster_workload
    from test_gpu_parity import assert_same
    rng = np.random.default_rng(1000 * eps + hi)
    seqs = _families(rng, 2600, lo, hi, np.frombuffer(alphabet, np.uint8), 40, 4)
    vg = [b"IGHV%d*" % g for g in range(1, 7)]
    jg = [b"IGHJ%d*" % g for g in range(1, 4)]
    # one crowded V gene (several tiles), some ambiguous calls, some rare genes
    vc = [b"IGHV1*01" if rng.random() < 0.7 else b"IGHV%d*01, or IGHV%d*02" % tuple(rng.integers(1, 7, 2))
          for _ in seqs]
    jc = [b"IGHJ%d*02" % (1 + int(rng.random() < 0.1)) for _ in seqs]
    w = synth.from_strings(seqs, vc, jc, vg, jg, abs_eps=eps, min_pts=3)
    g, o = cluster_workload(w, gpu_ctx), oracle.cluster(w)
    assert_same(g, o, w, f"eps={eps} L={lo}-{hi}")
    assert g.stats.neighbour_pairs == o.neighbour_pairs


@pytest.mark.gpu
def test_eps_varies_with_length(gpu_ctx):
    """min(3, trunc(0.15 L)): bins of eps 0 to 3 in one launch."""
    from immunodbscan_gb300 import cluster_workload
    from test_gpu_parity import assert_same
    rng = np.random.default_rng(5)
    seqs = _families(rng, 6000, 4, 32, np.frombuffer(b"ACDEFGHIKLMNPQRSTVWY", np.uint8), 150, 4)
    w = synth.from_strings(seqs, [b"IGHV1*01"] * 6000, [b"IGHJ1*01"] * 6000, [b"IGHV1*"], [b"IGHJ1*"],
                           threshold=0.15, abs_eps=3, min_pts=4)
    g, o = cluster_workload(w, gpu_ctx), oracle.cluster(w)
    assert_same(g, o, w, "eps by length")
    assert g.stats.neighbour_pairs == o.neighbour_pairs


def _look_ups(m, n, e):
    """(segment start, length, shift) in the order the segment join looks them up
    for a pair of lengths m <= n within e edits (k_lev_join.cu)."""
    g, S, out = n - m, e + 1, []
    for k in range(S):
        s, t = k * n // S, (k + 1) * n // S
        for d in range(max(-k, -g - (e - k)), min(k, e - k - g) + 1):
            if s + d >= 0 and t + d <= m:
                out.append((s, t - s, d))
    return out


@pytest.mark.parametrize("eps", [0, 1, 2, 3])
def test_join_finds_every_pair(eps):
    """Every pair within eps shares a segment of the longer string with the
    shorter one at one of the shifts the join looks up (random families over
    two and four letters, lengths from 0)."""
    rng = np.random.default_rng(eps)
    checked = 0
    for lo, hi, alphabet in [(0, 7, b"AC"), (1, 12, b"ACGT"), (20, 26, b"ACGT")]:
        seqs = [b""] if lo == 0 else []
        seqs += _families(rng, 160, max(lo, 1), hi, np.frombuffer(alphabet, np.uint8), 6, 4)
        for i, a in enumerate(seqs):
            for b in seqs[i:]:
                x, y = (a, b) if len(a) <= len(b) else (b, a)
                if len(y) - len(x) > eps or not oracle.levenshtein_within(x, y, eps):
                    continue
                checked += 1
                for p, q in ((x, y), (y, x)) if len(x) == len(y) else ((x, y),):
                    assert any(p[s + d:s + d + l] == q[s:s + l] for s, l, d in _look_ups(len(p), len(q), eps)), (p, q)
    assert checked > 500


@pytest.mark.gpu
@pytest.mark.parametrize("eps", [1, 2, 3])
@pytest.mark.parametrize("genes", ["narrow", "wide"])
def test_join_and_buckets_agree(gpu_ctx, eps, genes):
    """Groups of every shape: repeats (a unique that looks up its own segment),
    one-letter runs, several repertoires, thin classes against long ones; the
    join and the buckets give the oracle's answer."""
    from immunodbscan_gb300 import cluster_workload
    from test_gpu_parity import assert_same
    rng = np.random.default_rng(70 + eps)
    seqs = _families(rng, 3000, 6, 20, np.frombuffer(b"ACDE", np.uint8), 25, 3)
    seqs += _families(rng, 800, 10, 14, np.frombuffer(b"A", np.uint8), 4, 2)
    seqs += [b"A" * int(k) for k in rng.integers(0, 12, size=200)]
    n_v = 8 if genes == "narrow" else 90
    vg = [b"IGHV%d*" % g for g in range(1, n_v + 1)]
    jg = [b"IGHJ%d*" % g for g in range(1, 4)]
    vc = [b"IGHV%d*01, or IGHV%d*02" % (1 + int(rng.integers(0, 2)), 1 + int(rng.integers(0, n_v)))
          for _ in seqs]
    jc = [b"IGHJ%d*02" % (1 + int(rng.integers(0, 2))) for _ in seqs]
    w = synth.from_strings(seqs, vc, jc, vg, jg, abs_eps=eps, min_pts=3, rep_sizes=[1500, 1500, 1000])
    o = oracle.cluster(w)
    g = cluster_workload(w, gpu_ctx)
    assert_same(g, o, w, f"join eps={eps} {genes}")
    assert g.stats.neighbour_pairs == o.neighbour_pairs and g.stats.candidates == 1
    w.candidates = 1
    b = cluster_workload(w, gpu_ctx)
    assert_same(b, o, w, f"buckets eps={eps} {genes}")
    assert b.stats.neighbour_pairs == o.neighbour_pairs and b.stats.candidates == 0
