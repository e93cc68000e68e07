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
