"""The forest that unions start from hangs a unique under any smaller neighbour, so a
lineage whose members each neighbour the one before gives a chain as deep as it
is long.  The walk that flattens it on the CPU, step by step, and whole calls on
such lineages."""
import os
import subprocess

import numpy as np
import pytest

from immunodbscan_gb300 import cluster_workload, synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_flattening_walk_on_cpu(tmp_path):
    exe = tmp_path / "test_forest"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "immunodbscan_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "test_forest.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("hamming", [True, False])
@pytest.mark.parametrize("n,n_chains", [(5_000, 1), (1_300_000, 3)])
def test_lineages(gpu_ctx, hamming, n, n_chains):
    """Row i differs from row i + 1 of its lineage in one residue and from every other
    row in more (31 residues change in turn, each by a step of 1 to 19 of 20);
    1.3M rows take the long lists' unions."""
    rng = np.random.default_rng(n + hamming)
    L, aa = 31, np.frombuffer(synth.AA, np.uint8)
    pos, step = np.arange(n) % L, rng.integers(1, 20, n)
    seq = np.empty((n, L), np.uint8)
    for p in range(L):
        seq[:, p] = (int(rng.integers(0, 20)) + np.cumsum(np.where(pos == p, step, 0))) % 20
    w = synth.from_strings([b"A"], [b"IGHV1*01"], [b"IGHJ1*01"], [b"IGHV1*"], [b"IGHJ1*"], abs_eps=1,
                           min_pts=2, use_hamming=hamming)
    w.seq_blob, w.seq_off = aa[seq].reshape(-1), np.arange(n + 1, dtype=np.int64) * L
    for name, call in (("v", w.v_blob), ("j", w.j_blob)):
        setattr(w, name + "_blob", np.tile(call, n))
        setattr(w, name + "_off", np.arange(n + 1, dtype=np.int64) * len(call))
    cut = n // n_chains     # a repertoire each
    w.rep_off = np.array([k * cut for k in range(n_chains)] + [n], np.uint32)
    g = cluster_workload(w, gpu_ctx)
    assert g.n_uniques == n and np.all(g.core == 1) and np.all(g.copies == 1)
    assert g.stats.neighbour_pairs == n - n_chains
    assert np.all(g.clone_id == 1)
