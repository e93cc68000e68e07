"""The bitmap word filter on the tensor cores (k_bfilter_bits) at the edges of
its tiles: passes of 2 to 1,024 tentatives (one to five column tiles, with and
without padding columns) and remain lists around a multiple of 128 rows, every
word length, against the oracle's clustering."""
import numpy as np
import pytest

import gsdr
import oracle_binding as orc

pytestmark = pytest.mark.gpu


def _run(tmp_path, n, t, w, batch, recipe=0, **kw):
    data = gsdr.synth_fasta(recipe, n_reads=n, seed=900 + n, **kw)
    _, ocl, _, _ = orc.run_bytes(data, tmp_path, t=t, w=w)
    f = gsdr.Fasta.parse(data)
    try:
        cl, st = gsdr.clustering(f, gsdr.default_opts(threshold=t, word_length=w, batch=batch,
                                                      word_filter=3), stats=True)
    finally:
        f.close()
    assert st.word_index == 2
    np.testing.assert_array_equal(cl, ocl)


@pytest.mark.parametrize("batch", [2, 15, 16, 17, 239, 240, 241, 480, 481, 1024])
def test_tentatives_per_pass(tmp_path, batch):
    _run(tmp_path, 1600, 0.95, 6, batch, n_seeds=1300, len_lo=150, len_hi=600)


@pytest.mark.parametrize("n", [2, 3, 127, 128, 129, 255, 257, 640])
def test_candidates_around_a_tile(tmp_path, n):
    _run(tmp_path, n, 0.95, 6, 64, n_seeds=max(1, n - 20), len_lo=150, len_hi=600)


@pytest.mark.parametrize("w", [4, 5, 6, 7])
@pytest.mark.parametrize("t", [0.88, 0.97])
def test_word_lengths(tmp_path, w, t):
    _run(tmp_path, 700, t, w, 300, n_seeds=400, len_lo=200, len_hi=2500)


@pytest.mark.parametrize("w,lo,hi", [(5, 150, 300), (5, 700, 900), (6, 150, 700), (6, 1200, 1500),
                                     (6, 2600, 3000), (6, 4600, 5000), (7, 300, 700),
                                     (7, 1500, 2000), (7, 3000, 3500)])
def test_bitmap_depths(tmp_path, w, lo, hi):
    # reads for which a quarter, half or all of the first level, or both levels
    # decide nearly every pair
    _run(tmp_path, 400, 0.95, w, 128, n_seeds=300, len_lo=lo, len_hi=hi)


def _check_reads(tmp_path, reads, t, w):
    data = "".join(f">r{i}\n{s}\n" for i, s in enumerate(reads)).encode()
    _, ocl, _, _ = orc.run_bytes(data, tmp_path, t=t, w=w)
    f = gsdr.Fasta.parse(data)
    try:
        cl, st = gsdr.clustering(f, gsdr.default_opts(threshold=t, word_length=w, word_filter=3,
                                                      batch=0), stats=True)
    finally:
        f.close()
    assert st.word_index == 2
    np.testing.assert_array_equal(cl, ocl)


@pytest.mark.parametrize("w", [6, 7])
def test_reads_that_share_their_kmers(tmp_path, w):
    # two bases only: far more shared k-mers than random reads, so that passes
    # with shortened bitmaps leave most pairs open and later ones lengthen them
    rng = np.random.default_rng(77)
    reads = ["".join("AC"[x] for x in rng.integers(0, 2, int(n)))
             for n in np.sort(rng.integers(300, 420, 1500))[::-1]]
    reads += ["".join("ACGT"[x] for x in rng.integers(0, 4, 290)) for _ in range(300)]
    _check_reads(tmp_path, reads, 0.92, w)


def test_composition_counts_above_16_bits(tmp_path):
    # single-base counts that 16-bit halves do not hold
    a = "A" * 65_537
    _check_reads(tmp_path, [a + "C", a + "G", a, a[:-2] + "CG"] + ["A" * 900] * 3, 0.99999, 6)
