"""The segment alignment kernel at the edges of its window classes and in the
lane grouping of its narrow runs, against the oracle's LCS.  The windows are
those of seg_words (csrc/lcs_seg.cuh): up to 512 words on the kernel itself, up
to 768 on its wide form (20 words a lane up to 640, 24 above), wider ones on
the systolic kernels."""
import numpy as np
import pytest

import gsdr
import oracle_binding as orc

pytestmark = pytest.mark.gpu

CODES = np.frombuffer(b"ACGT", dtype=np.uint8)
F = np.float32
SEG_STEPS8, SEG_STEPS32, SEG_STRIP, SLOPE_MORE = 128, 256, 96, F(0.6)


def _cut(q, t):
    return int(np.ceil(F(q) * F(t)))


def _seg_words(T, q, c):
    return min((T - c + q - c + 1 + SEG_STEPS32) // 32 + 3, (T + 31) // 32)


def _seg_narrow(T, q, c):
    if c >= q or T <= q:
        return False
    ratio = F(0.23) + F(0.57) * np.log2(F(q) / F(q - c))
    if F(T) < ratio * F(q):
        return False
    strip = int(SEG_STEPS8 * min(F(T) / F(q), ratio + SLOPE_MORE) + 2 * SEG_STRIP) // 32 + 2
    return _seg_words(T, q, c) >= 2 * strip


def _substituted(rng, s, rate):
    a = s.copy()
    hit = rng.random(a.size) < rate
    a[hit] = CODES[rng.integers(0, 4, int(hit.sum()))]
    return a


def _decide(seqs, pairs, t, greedy):
    want = orc.lcs_decisions(seqs, pairs, t)
    got, _ = gsdr.lcs_decide(seqs, pairs, t, mapping=3, greedy=greedy)
    bad = np.nonzero(got != want)[0]
    assert len(bad) == 0, f"{len(bad)} of {len(pairs)} differ, first {bad[:8]}"
    return want


@pytest.mark.parametrize("words", [256, 257, 511, 512, 513, 640, 641, 767, 768, 769])
def test_window_edges(words):
    """Texts 1.2 times their pattern at t = 0.80, both ends of the lengths that
    need `words` words: exact copies (their window grows to its full width),
    copies around the threshold and unrelated bases (rejected)."""
    t = 0.80
    rng = np.random.default_rng(words)
    seqs, pairs = [], []
    for rows in (32 * (words - 3) - 257, 32 * (words - 3) - 226):  # T - c + q - c
        q = int(rows / 0.6)
        T = rows + 2 * _cut(q, t) - q
        assert _seg_words(T, q, _cut(q, t)) == words
        for rate in (0.0, 0.18, 0.27, 0.33, 1.0):
            text = CODES[rng.integers(0, 4, T)]
            at = int(rng.integers(0, T - q + 1))
            seqs += [text.tobytes(), _substituted(rng, text[at:at + q], rate).tobytes()]
            pairs.append((len(seqs) - 1, len(seqs) - 2))
    want = _decide(seqs, pairs, t, greedy=0)
    assert 0 < want.sum() < len(pairs)


@pytest.mark.parametrize("t,ratio,n", [(0.80, 1.55, 2600), (0.90, 2.2, 2600), (0.95, 2.7, 2600)])
def test_narrow_runs_of_eight_lanes(t, ratio, n):
    """More narrow pairs than half the grid's warps, so that eight lanes take a
    pair: unrelated bases around the ratio from which they are accepted, copies,
    and pairs too similar in length for a narrow run beside them."""
    rng = np.random.default_rng(int(1000 * t))
    seqs, pairs, narrow = [], [], 0
    for i in range(n):
        T = int(rng.integers(1700, 2600))
        q = int(T / rng.uniform(0.95 * ratio, 1.5 * ratio)) if i % 9 else int(T * 0.97)
        narrow += _seg_narrow(T, q, _cut(q, t))
        text = CODES[rng.integers(0, 4, T)]
        a = CODES[rng.integers(0, 4, q)]
        if i % 3 == 0:
            a = _substituted(rng, text[T - q:], float(rng.uniform(0, 2 * (1 - t))))
        seqs += [text.tobytes(), a.tobytes()]
        pairs.append((len(seqs) - 1, len(seqs) - 2))
    assert narrow > 1500
    want = _decide(seqs, pairs, t, greedy=1)
    assert 0 < want.sum() < len(pairs)
