"""The work that users of this framework have it do, as cases to time.

A case is one clustering (or one burst of served clusterings) through the
public Python view of the C ABI: FASTA bytes in host memory to the
representatives' FASTA bytes, the cluster array and the sort permutation
(`gsdr.cluster_fasta`, the path of the `cluster` executable), a job whose
reads stay on the device (`gsdr.Job`), or jobs of mixed sizes and thresholds
given to the server (`gsdr.Server`).  Inputs are the seeded synthetic
workloads of the repository's benchmark and tests.  All outputs are bytes and
whole numbers, so there is no 64-bit reference to compare them with.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "gene-sequences-de-redundancy_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import gsdr  # noqa: E402

# recipe: (generator preset, reads and seeds of the named workload, mean read length)
RECIPES = {
    "uniform": (0, 10_000, 2_000, 600),         # 200-1,000 bp
    "lognormal": (1, 200_000, 40_000, 1_700),   # median 1,500 bp, 300-10,000 bp
    "short": (2, 2_000_000, 300_000, 150),      # 150 bp reads
    "long": (3, 300_000, 60_000, 10_340),       # 2-30 kbp, log-uniform
    "serving": (4, 1_000, 200, 2_575),          # 150-5,000 bp
    "serving_drop": (4, 1_000, 200, 1_075),     # 150-2,000 bp, the serving jobs without filters
}
# thresholds of a burst's jobs in turn; below 0.88 the word filter is off
# (drop mode, quadratic), and such jobs are small
BURST_T = (0.95, 0.90, 0.80, 0.95, 0.90, 0.85)
BURST_DROP_READS = 1_500


def _case(name, entry, recipe, reads, t, **kw):
    c = {"entry": entry, "recipe": recipe, "reads": reads, "threshold": t, "batch": 0,
         "pigeon": 0, "variant": 0, "jobs": 1}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest job of the serving recipe: launches and host calls count
        _case("serve_1k_t95", "fasta", "serving", 1_000, 0.95),
        # the 10k-read workload, default threshold
        _case("uniform_10k_t95", "fasta", "uniform", 10_000, 0.95),
        # the same reads through the reference's own form: device-resident
        # reads, one representative per round
        _case("uniform_10k_plain", "job", "uniform", 10_000, 0.95, batch=1),
        # the optional 4-mer position filter in front of the alignment
        _case("uniform_9973_pigeon", "fasta", "uniform", 9_973, 0.95, pigeon=1),
        # the headline workload: 200k reads of 300-10,000 bp
        _case("lognormal_200k_t95", "fasta", "lognormal", 200_000, 0.95),
        # the other parity mode (the SYCL program's rules), shorter words
        _case("lognormal_20011_sycl", "fasta", "lognormal", 20_011, 0.95, variant=1),
        # short reads in a sparse k-mer space (k = 7), half the named workload
        _case("short_1m_t90", "fasta", "short", 1_000_000, 0.90),
        # a large serving job at the default threshold (k = 6)
        _case("serve_100k_t95", "fasta", "serving", 100_000, 0.95),
        # a middle-sized serving job at t = 0.90 (k = 7)
        _case("serve_30k_t90", "fasta", "serving", 30_000, 0.90),
        # long reads at the widest band, filters off (drop mode)
        _case("long_3k_t80", "fasta", "long", 3_000, 0.80),
        # a serving job with the filters off
        _case("serve_drop_1499_t85", "fasta", "serving_drop", 1_499, 0.85),
        # a burst of served jobs, 1k-12k reads, mixed thresholds, four slots
        _case("serve_burst_12", "server", "serving", 12_000, 0.95, jobs=12),
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["uniform", "lognormal", "short", "serving", "serving", "long",
                       "serving_drop", "plain", "options", "burst"])
    if kind == "uniform":
        return _case(None, "fasta", "uniform", _log_size(rng, 1_000, 50_000),
                     rng.choice([0.90, 0.95, 0.97]))
    if kind == "lognormal":
        return _case(None, "fasta", "lognormal", _log_size(rng, 2_000, 200_000),
                     rng.choice([0.95, 0.97]))
    if kind == "short":
        return _case(None, "fasta", "short", _log_size(rng, 10_000, 1_000_000), 0.90)
    if kind == "serving":
        t = rng.choice([0.90, 0.95])
        return _case(None, "fasta", "serving",
                     _log_size(rng, 1_000, 30_000 if t < 0.95 else 100_000), t)
    if kind == "long":
        return _case(None, "fasta", "long", _log_size(rng, 300, 2_500),
                     rng.choice([0.80, 0.85]))
    if kind == "serving_drop":
        return _case(None, "fasta", "serving_drop", _log_size(rng, 300, 1_500),
                     rng.choice([0.80, 0.85]))
    if kind == "plain":
        return _case(None, "job", "uniform", _log_size(rng, 1_000, 10_000),
                     rng.choice([0.90, 0.95]), batch=1)
    if kind == "options":
        if rng.random() < 0.5:
            return _case(None, "fasta", "uniform", _log_size(rng, 1_000, 10_000),
                         rng.choice([0.90, 0.95]), pigeon=1)
        return _case(None, "fasta", "lognormal", _log_size(rng, 2_000, 30_000), 0.95, variant=1)
    return _case(None, "server", "serving", _log_size(rng, 2_000, 12_000), 0.95,
                 jobs=rng.randint(4, 12))


def _fasta(recipe, reads, seed):
    """The recipe's file of `reads` records, seeds in the named workload's
    proportion, in page-locked host memory as a uint8 array."""
    preset, n0, s0, _ = RECIPES[recipe]
    kw = {"n_seeds": max(1, round(s0 * reads / n0))}
    if recipe.startswith("serving"):
        kw.update(len_lo=150, len_hi=2000 if recipe == "serving_drop" else 5000)
    data = gsdr.synth_fasta(preset, n_reads=reads, seed=100_003 * preset + seed, **kw)
    a = torch.empty(len(data), dtype=torch.uint8, pin_memory=True).numpy()
    a[:] = np.frombuffer(data, dtype=np.uint8)
    return a


def _burst_sizes(case):
    """(recipe, reads, threshold) of a burst's jobs, sizes from 1,000 reads
    up to the case's in equal ratios."""
    k, top = case["jobs"], case["reads"]
    out = []
    for i in range(k):
        t = BURST_T[i % len(BURST_T)]
        n = int(round(1_000 * (top / 1_000) ** (i / max(1, k - 1))))
        out.append(("serving_drop", min(n, BURST_DROP_READS), t) if t < 0.88
                   else ("serving", n, t))
    return out


def _out_buffer(recipe, reads):
    """The program's own buffer for the output file: the representatives are
    well under these shares of the input file, whatever the seed."""
    share = 0.5 if recipe in ("lognormal", "short") else 0.9
    return np.zeros(int(share * reads * (RECIPES[recipe][3] + 8)) + (1 << 16), dtype=np.uint8)


def prepare(case, seed):
    opts = {"threshold": case["threshold"], "batch": case["batch"], "pigeon": case["pigeon"],
            "variant": case["variant"]}
    if case["entry"] == "fasta":
        return {"entry": "fasta", "data": _fasta(case["recipe"], case["reads"], seed),
                "opts": gsdr.default_opts(**opts),
                "out": _out_buffer(case["recipe"], case["reads"])}
    if case["entry"] == "job":
        # the reads parsed on the host and uploaded once; the job is run again
        f = gsdr.Fasta.parse(_fasta(case["recipe"], case["reads"], seed).tobytes())
        return {"entry": "job", "job": gsdr.Job(f, gsdr.default_opts(**opts))}
    jobs = [(_fasta(r, n, seed + 7919 * i), t, _out_buffer(r, n))
            for i, (r, n, t) in enumerate(_burst_sizes(case))]
    return {"entry": "server", "server": gsdr.Server(max_inflight=4), "jobs": jobs}


def run(state):
    if state["entry"] == "fasta":
        fa, cluster, order = gsdr.cluster_fasta(state["data"], state["opts"], copy=False)
        state["out"][:fa.size] = fa
        return state["out"], fa.size, cluster, order
    if state["entry"] == "job":
        state["job"].run()
        return state["job"].cluster()
    srv = state["server"]
    ids = {srv.submit(data, t): i for i, (data, t, _) in enumerate(state["jobs"])}
    got = [None] * len(ids)
    while any(g is None for g in got):
        j, status, _ = srv.wait()
        if status != gsdr.OK:
            raise gsdr.GsdrError(status, "served job failed")
        fa, cluster = srv.result(j)
        srv.release(j)
        out = state["jobs"][ids[j]][2]
        out[:len(fa)] = np.frombuffer(fa, dtype=np.uint8)
        got[ids[j]] = (out, len(fa), cluster)
    return got


def work(case):
    """Bytes: the file read once, the cluster array and the permutation
    written once.  What the clustering itself costs (integer work: filter
    words and DP cells) depends on the reads, so no operations are claimed."""
    def one(recipe, reads):
        return reads * (RECIPES[recipe][3] + 8 + 8)

    if case["entry"] == "server":
        return {"bytes": sum(one(r, n) for r, n, _ in _burst_sizes(case)), "flops": 0}
    return {"bytes": one(case["recipe"], case["reads"]), "flops": 0}
