"""The work this framework is measured on: whole clustering calls over seeded synthetic repertoires.

A case names one of the generators of ``immunodbscan_gb300.synth`` (``workload`` 0..4) and a
``scale`` of its full row count, the clustering parameters (``eps`` = absolute edit distance or -1,
``threshold`` = relative edit distance or -1, ``hamming``, ``min_pts``), how many V genes the
reference list holds, and the entry point a program calls:

  host     Interlink(...)               host columns in, host results out (page-locked columns)
  device   DeviceBatch.cluster_once()   columns resident on the device, one eager call
  batch    DeviceBatch.run()            the same columns, planned once and replayed

Every pass returns the three result columns (clone ids, core flags, copies).  They are whole
numbers, so there is nothing for a 64-bit computation to say beyond equality: ``exact`` has none.
"""
import math

import numpy as np
import torch

from immunodbscan_gb300 import Context, DeviceBatch, Interlink, synth

#: full-size rows, mean bytes of a sequence and of a V and a J call, for each generator
SHAPE = {0: (10_000, 15, 48, 40), 1: (200_000, 50, 52, 39), 2: (5_000_000, 15, 48, 39),
         3: (2_000_000, 15, 50, 39), 4: (10_000_000, 15, 48, 43)}


def case(name, workload, scale, api, *, eps=-1, threshold=-1.0, hamming=False, min_pts=2,
         v_genes=50, genes=True, edge_memory_mb=0):
    c = dict(workload=workload, scale=scale, api=api, eps=eps, threshold=threshold,
             hamming=hamming, min_pts=min_pts, v_genes=v_genes, genes=genes,
             edge_memory_mb=edge_memory_mb)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one small sample per call, as an interactive program or a test does: latency
        case("sample-500-host", 0, 0.05, "host", eps=1, hamming=True),
        # one ordinary sample already on the device, a new call each time
        case("sample-10k-device", 0, 1.0, "device", eps=1, hamming=True),
        # the reference's own settings (relative threshold 0.15, edit distance) with a
        # reference gene list of more than one bitset word
        case("relative-20k-host", 3, 0.01, "host", threshold=0.15, v_genes=120),
        # no gene columns configured: every row is compatible with every other
        case("no-genes-20k-host", 0, 2.0, "host", eps=1, genes=False),
        # nucleotide junctions, edit distance 2, replayed
        case("nt-200k-batch", 1, 1.0, "batch", eps=2, min_pts=3, v_genes=60),
        # nucleotide junctions, substitutions only, relative threshold (eps 2 to 7)
        case("nt-100k-hamming-device", 1, 0.5, "device", threshold=0.1, hamming=True, v_genes=60),
        # a cohort of 64 repertoires in one replayed plan: the headline workload
        case("cohort-2.5M-batch", 2, 0.5, "batch", eps=1, hamming=True),
        # a cohort from host memory, copies overlapped with the first phases
        case("cohort-1.3M-host", 2, 0.25, "host", eps=1, hamming=True),
        # a cohort at a relative Hamming threshold (eps 1 to 5)
        case("cohort-500k-relative", 2, 0.1, "device", threshold=0.2, hamming=True),
        # one deep repertoire with skewed gene usage, edit distance 2, replayed: the heaviest
        case("skewed-1M-batch", 3, 0.5, "batch", eps=2),
        # one deep repertoire of many clones, min(3, 0.15 L) edits, one eager call
        case("deep-2M-device", 4, 0.2, "device", eps=3, threshold=0.15, min_pts=4),
        # a dense neighbour graph with no memory for its pairs: two sweeps
        case("skewed-400k-streamed", 3, 0.2, "device", eps=2, edge_memory_mb=-1),
    ]


def _between(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["sample", "sample", "nt", "cohort", "skewed", "deep"])
    api = rng.choice(["host", "device", "batch"])
    v = rng.choice([50, 50, 120])
    if kind == "sample":        # 300 to 40,000 rows, every small eps
        return case(None, 0, _between(rng, 0.03, 4.0), api, eps=rng.randint(0, 3),
                    hamming=rng.random() < 0.5, min_pts=rng.randint(1, 4), v_genes=v,
                    genes=rng.random() < 0.7)
    if kind == "nt":
        if rng.random() < 0.5:
            return case(None, 1, _between(rng, 0.02, 1.0), api, eps=rng.randint(1, 3),
                        hamming=rng.random() < 0.4, min_pts=3, v_genes=v)
        return case(None, 1, _between(rng, 0.02, 0.5), api, threshold=rng.uniform(0.03, 0.12),
                    hamming=rng.random() < 0.5, min_pts=rng.randint(2, 4), v_genes=v)
    if kind == "cohort":        # 64 repertoires, up to the largest listed
        return case(None, 2, _between(rng, 0.005, 0.4), api, eps=rng.randint(0, 2), hamming=True,
                    min_pts=rng.randint(2, 3), v_genes=v)
    if kind == "skewed":
        return case(None, 3, _between(rng, 0.005, 0.35), api, eps=rng.randint(1, 2), v_genes=v,
                    edge_memory_mb=rng.choice([0, 0, -1]))
    return case(None, 4, _between(rng, 0.002, 0.15), api, eps=3,
                threshold=rng.uniform(0.08, 0.2), min_pts=rng.randint(2, 5), v_genes=v)


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _rows(case):
    return max(int(SHAPE[case["workload"]][0] * case["scale"]), 2)


def _cohort(case, seed):
    """Workload 2 cut to the case's row count: its 64 log-uniform sizes come first from the
    seed's generator, and their sum differs from seed to seed."""
    n = _rows(case)
    raw = np.exp(np.random.default_rng(seed).uniform(math.log(5_000), math.log(500_000), size=64))
    w = synth.workload(2, scale=(n + 64) / raw.sum(), seed=seed)
    for name in ("seq", "v", "j"):
        off = getattr(w, name + "_off")[:n + 1]
        setattr(w, name + "_off", off)
        setattr(w, name + "_blob", getattr(w, name + "_blob")[:off[-1]])
    w.rep_off = np.minimum(w.rep_off, n).astype(np.uint32)
    return w


def prepare(case, seed):
    if case["workload"] == 2:
        w = _cohort(case, seed)
    else:
        w = synth.workload(case["workload"], scale=case["scale"], seed=seed)
    w.abs_eps = case["eps"]
    w.threshold = case["threshold"] if case["threshold"] >= 0 else math.nan
    w.use_hamming = case["hamming"]
    w.min_pts = case["min_pts"]
    w.edge_memory_mb = case["edge_memory_mb"]
    if case["v_genes"] > len(w.v_genes):     # names that no call holds
        w.v_genes = w.v_genes + synth.gene_names("IGHV", case["v_genes"])[len(w.v_genes):]
    ctx = Context(0)
    if case["api"] == "host" or not case["genes"]:
        cols = [(_pinned(b), _pinned(o)) for b, o in
                ((w.v_blob, w.v_off), (w.j_blob, w.j_off), (w.seq_blob, w.seq_off))]
        if not case["genes"]:
            cols[0] = cols[1] = None
        sizes = np.diff(w.rep_off).tolist() if w.n_rep > 1 else None
        return {"api": "host", "w": w, "cols": cols, "rep_sizes": sizes, "ctx": ctx}
    batch = DeviceBatch(w, ctx)
    if case["api"] == "batch":
        batch.plan()
    return {"api": case["api"], "batch": batch, "ctx": ctx}


def run(state):
    if state["api"] == "host":
        w, (v, j, seq) = state["w"], state["cols"]
        r = Interlink(v, j, seq, w.n, w.v_genes, w.j_genes, w.threshold, w.min_pts, w.use_hamming,
                      abs_eps=w.abs_eps, rep_sizes=state["rep_sizes"], context=state["ctx"],
                      edge_memory_mb=w.edge_memory_mb)
        return [r.get_clusters(), r.get_cores(), r.get_copies()]
    batch = state["batch"]
    if state["api"] == "batch":
        batch.run()
    else:
        batch.cluster_once()
    return [batch.clone, batch.core, batch.copies]


def work(case):
    """Columns and offsets read once, results written once; the operations are those of hashing
    and joining each row once per segment of its sequence (the pairs depend on the data)."""
    n = _rows(case)
    _, seq, v, j = SHAPE[case["workload"]]
    read = seq + 8 + ((v + j + 16) if case["genes"] else 0)
    return {"bytes": n * (read + 12), "flops": n * read}


def exact(case, seed):
    return None
