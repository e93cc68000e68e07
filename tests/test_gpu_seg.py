"""The segment alignment kernel (csrc/lcs_seg.cuh) against the oracle's LCS at
the sizes where it can go wrong: pattern lengths around a segment's steps,
text lengths around a word, a lane's words and the group's window, both lane
groupings (few pairs: a whole warp each; many: 8, 16 or 32 lanes), patterns
longer than their text, and pairs decided without any step."""
import numpy as np
import pytest

import gsdr
import oracle_binding as orc

pytestmark = pytest.mark.gpu

CODES = np.frombuffer(b"ACGT", dtype=np.uint8)


def _seq(rng, n):
    return CODES[rng.integers(0, 4, n)].tobytes()


def _copy(rng, s, rate):
    a = np.frombuffer(s, dtype=np.uint8).copy()
    hit = rng.random(len(a)) < rate
    a[hit] = CODES[rng.integers(0, 4, int(hit.sum()))]
    keep = rng.random(len(a)) >= rate / 4
    return a[keep].tobytes() or s[:1]


def _pair(rng, q, T, t):
    """A pattern of about q bases and a text of T: a mutated part of the text
    whose identity straddles t, or unrelated bases."""
    b = _seq(rng, T)
    if rng.random() < 0.7:
        a = _copy(rng, (b + _seq(rng, max(0, q - T)))[:q], float(rng.uniform(0, 2.5 * (1 - t))))
    else:
        a = _seq(rng, q)
    return b, a


def _check(cases, t, rng):
    seqs, pairs = [], []
    for q, T in cases:
        b, a = _pair(rng, q, T, t)
        seqs += [b, a]
        pairs.append((len(seqs) - 1, len(seqs) - 2))
    want = orc.lcs_decisions(seqs, pairs, t)
    got, _ = gsdr.lcs_decide(seqs, pairs, t, mapping=3, greedy=0)
    bad = np.nonzero(got != want)[0]
    assert len(bad) == 0, f"{len(bad)} of {len(pairs)} differ: {[cases[i] for i in bad[:5]]}"
    assert 0 < want.sum() < len(pairs)


EDGES = [1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 383, 384, 385, 511, 512, 513]


@pytest.mark.parametrize("t", [0.80, 0.88, 0.95])
def test_segment_and_word_edges_few_pairs(t):
    rng = np.random.default_rng(int(1000 * t))
    cases = [(q, T) for q in EDGES for T in (q, q + 1, q + 31, q + 32, 2 * q + 5, max(1, q - 1))]
    _check(cases, t, rng)


@pytest.mark.parametrize("t", [0.80, 0.95])
def test_segment_and_word_edges_many_pairs(t):
    # more pairs than half the grid's warps: 8 lanes per pair
    rng = np.random.default_rng(int(1000 * t) + 1)
    cases = [(q + d, T) for q in EDGES[2:] for d in (0, 1, 2, 3)
             for T in (q, q + 1, q + 31, 2 * q + 5, 3 * q + 1, max(1, q - 1))] * 4
    _check(cases, t, rng)


@pytest.mark.parametrize("many", [False, True])
def test_every_window_class(many):
    """Windows from a few words to the kernel's widest (512 words) and past it
    (those pairs run on the systolic kernels)."""
    rng = np.random.default_rng(5 + many)
    cases = []
    for T in (900, 1100, 2000, 2300, 4000, 4200, 8000, 8300, 15800, 16400, 17500):
        for f in (0.35, 0.6, 0.97):
            cases.append((int(T * f), T))
    if many:
        cases += [(int(rng.integers(60, 200)), int(rng.integers(180, 700))) for _ in range(1400)]
    _check(cases, 0.90, rng)
