"""The word filter by hashed k-mer counts (k_bfilter_hash): short reads in a
sparse k-mer space, at the edges of its tiles (candidates around a multiple of
128, tentatives around a group), with low-complexity reads whose bucket counts
round up and saturate, and on both sides of the rule that chooses it, against
the oracle's clustering."""
import numpy as np
import pytest

import gsdr
import oracle_binding as orc

pytestmark = pytest.mark.gpu


def _check(tmp_path, data, t, word_index=3, **kw):
    _, ocl, _, _ = orc.run_bytes(data, tmp_path, t=t, **({"w": kw["word_length"]}
                                                         if "word_length" in kw else {}))
    f = gsdr.Fasta.parse(data)
    try:
        cl, st = gsdr.clustering(f, gsdr.default_opts(threshold=t, **kw), stats=True)
    finally:
        f.close()
    assert st.word_index == word_index
    np.testing.assert_array_equal(cl, ocl)


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 300, 1000])
def test_candidates_around_a_tile(tmp_path, n):
    _check(tmp_path, gsdr.synth_fasta(2, n_reads=n, seed=70 + n), 0.90)


@pytest.mark.parametrize("batch", [1, 2, 16, 17, 159, 160, 161, 321, 1024])
def test_tentatives_per_pass(tmp_path, batch):
    data = gsdr.synth_fasta(2, n_reads=3000, seed=71, n_seeds=2500)
    _check(tmp_path, data, 0.90, word_index=3 if batch > 1 else 0, batch=batch)


@pytest.mark.parametrize("t,w", [(0.90, 7), (0.92, 7), (0.95, 6), (0.97, 6), (0.97, 5)])
def test_thresholds_and_ragged_lengths(tmp_path, t, w):
    data = gsdr.synth_fasta(0, n_reads=1500, seed=72, n_seeds=900, len_lo=20, len_hi=160)
    _check(tmp_path, data, t, word_length=w)


def test_low_complexity_reads(tmp_path):
    # tandem repeats: a few k-mers with counts of up to 144, next to random reads
    rng = np.random.default_rng(73)
    recs = []
    for i in range(900):
        unit = "".join("ACGT"[x] for x in rng.integers(0, 4, int(rng.integers(1, 6))))
        s = (unit * 150)[:150] if i % 3 else "".join("ACGT"[x] for x in rng.integers(0, 4, 150))
        s = list(s)
        for x in rng.integers(0, 150, int(rng.integers(0, 12))):
            s[x] = "ACGT"[rng.integers(0, 4)]
        recs.append(f">r{i}\n{''.join(s)}\n")
    _check(tmp_path, "".join(recs).encode(), 0.90)


@pytest.mark.parametrize("length", [140, 150, 180, 200, 260])
def test_both_sides_of_the_rule(tmp_path, length):
    # from some length on the job takes the tentative masks instead (the same form)
    data = gsdr.synth_fasta(2, n_reads=1200, seed=74, len_lo=length, len_hi=length)
    _check(tmp_path, data, 0.90, word_filter=4)


@pytest.mark.parametrize("unit", [0, 3, 40, 400])
def test_open_pairs_of_long_lists(tmp_path, unit):
    # lists of up to ~900 k-mers: several loads of a lane's five entries, the
    # largest tables; repeats of `unit` bases raise the counts, so that the
    # presence bits leave pairs open and the tables form their sums
    rng = np.random.default_rng(75)
    recs = []
    for i in range(400):
        base = rng.integers(0, 4, 900) if not unit else np.tile(rng.integers(0, 4, unit), 900)[:900]
        for v in range(3):
            s = base.copy()
            at = rng.integers(0, 900, (8, 20, 30)[v])
            s[at] = rng.integers(0, 4, at.size)
            recs.append(f">r{i}_{v}\n{''.join('ACGT'[x] for x in s[:900 - 7 * v])}\n")
    _check(tmp_path, "".join(recs).encode(), 0.97, word_length=7, word_filter=4)


def test_full_groups_of_tentatives(tmp_path):
    # enough remaining reads for passes that take only full groups of tentatives,
    # and later ones that take R_max; a caller's R is taken as it is
    data = gsdr.synth_fasta(2, n_reads=230_000, seed=76, n_seeds=40_000)
    f = gsdr.Fasta.parse(data)
    try:
        a, sa = gsdr.clustering(f, gsdr.default_opts(threshold=0.90), stats=True)
        b, sb = gsdr.clustering(f, gsdr.default_opts(threshold=0.90, batch=512), stats=True)
    finally:
        f.close()
    assert sa.word_index == sb.word_index == 3
    assert sa.batch == 1024
    np.testing.assert_array_equal(a, b)
