"""gsdr_opts.group_words, the widest window the segment kernel takes, holds for
its narrow runs, for the full window behind one and for the lane-banded pairs
of a small pass too: with a limit of one word every pair of these jobs runs on
the kernels that take it with the segment kernel off, so both step the same
cells.  (Patterns of up to 2,048 bases: one warp per pair, whose early exit
does not depend on timing.)  The clusters are the same at every limit."""
import numpy as np
import pytest

import gsdr

pytestmark = pytest.mark.gpu


def _reads(rng, n):
    """Long and short unrelated reads: a text several times its pattern holds
    enough of it at t = 0.80 for a narrow run."""
    seqs = [rng.integers(0, 4, int(x)) for x in rng.integers(1500, 2000, n // 2)]
    seqs += [rng.integers(0, 4, int(x)) for x in rng.integers(150, 900, n - n // 2)]
    seqs.sort(key=len, reverse=True)
    return ["".join("ACGT"[x] for x in s).encode() for s in seqs]


def _run(seqs, **kw):
    return gsdr.cluster_reads(seqs, gsdr.default_opts(threshold=0.80, **kw), stats=True)


@pytest.mark.parametrize("batch", [1, 64])
def test_one_word_limit_steps_the_cells_of_no_segment_kernel(batch):
    # band_serial: batched passes take no pair to the lane-banded kernel, whose
    # pairs go to the segment kernel where they are few
    seqs = _reads(np.random.default_rng(94), 240)
    off, st_off = _run(seqs, batch=batch, group_words=-1, band_serial=-1)
    one, st_one = _run(seqs, batch=batch, group_words=1, band_serial=-1)
    free, st_free = _run(seqs, batch=batch, band_serial=-1)
    np.testing.assert_array_equal(one, off)
    np.testing.assert_array_equal(free, off)
    assert st_one.pairs_aligned == st_off.pairs_aligned > 0
    assert st_one.cells_computed == st_off.cells_computed
    assert st_free.cells_computed < st_off.cells_computed


def test_few_lane_banded_pairs_stay_within_the_limit():
    # reads of 100-300 bases that differ little: lane-banded pairs only, few in
    # each pass; they stay on the lane-banded kernel where their window in the
    # segment kernel would be above the limit
    data = gsdr.synth_fasta(0, n_reads=600, seed=95, n_seeds=200, len_lo=100, len_hi=300)
    f = gsdr.Fasta.parse(data)
    try:
        got = {w: gsdr.clustering(f, gsdr.default_opts(threshold=0.95, batch=64, group_words=w),
                                  stats=True) for w in (-1, 1, 16, 17, 0)}
    finally:
        f.close()
    for cl, _ in got.values():
        np.testing.assert_array_equal(cl, got[-1][0])
    cells = {w: st.cells_computed for w, (_, st) in got.items()}
    assert cells[1] == cells[-1]
    assert cells[17] == cells[0] != cells[-1]


@pytest.mark.parametrize("batch", [1, 64])
@pytest.mark.parametrize("group_words", [8, 16, 24, 32, 64, 128])
def test_same_clusters_at_every_limit(batch, group_words):
    seqs = _reads(np.random.default_rng(96), 300)
    want, _ = _run(seqs, batch=1, group_words=-1)
    got, _ = _run(seqs, batch=batch, group_words=group_words)
    np.testing.assert_array_equal(got, want)
