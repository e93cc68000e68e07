"""Which of the short reads' two word filters a job runs, and the tentative
masks (k_bfilter_mask) forced where the job would take the hashed counts: every
row width, both plane counts, ragged and low-complexity reads, against the
oracle's clustering.  Both forms report word_index 3; the job's buckets
(gsdr_job_filter_form) tell them apart."""
import math

import numpy as np
import pytest

import gsdr
import oracle_binding as orc
from test_gpu_index_filter import repeat_reads

pytestmark = pytest.mark.gpu


def _run(data, t, form, monkeypatch, **kw):
    """(clusters, hash buckets) of a job with GSDR_BFILTER=form."""
    if form is None:
        monkeypatch.delenv("GSDR_BFILTER", raising=False)
    else:
        monkeypatch.setenv("GSDR_BFILTER", form)
    f = gsdr.Fasta.parse(data)
    job = gsdr.Job(f, gsdr.default_opts(threshold=t, **kw))
    try:
        st = job.run()
        assert st.word_index == 3
        return job.cluster(), job.filter_form()[0]
    finally:
        job.close()
        f.close()


def _check_masks(tmp_path, monkeypatch, data, t, w=0, **kw):
    _, ocl, _, _ = orc.run_bytes(data, tmp_path, t=t, w=w)
    masks, none = _run(data, t, "tmasks", monkeypatch, word_length=w, **kw)
    hashed, buckets = _run(data, t, "masks", monkeypatch, word_length=w, **kw)
    assert none == 0 and buckets > 0
    np.testing.assert_array_equal(masks, ocl)
    np.testing.assert_array_equal(hashed, ocl)


# 1, 2, 4 and 8 lanes per row of 16-byte words, with partly used words
@pytest.mark.parametrize("batch", [2, 100, 129, 300, 513, 1024])
def test_row_widths(tmp_path, monkeypatch, batch):
    data = gsdr.synth_fasta(2, n_reads=12000, seed=46)
    _check_masks(tmp_path, monkeypatch, data, 0.90, batch=batch)


@pytest.mark.parametrize("w,batch", [(6, 64), (6, 1024), (7, 300), (5, 0)])
def test_ten_planes(tmp_path, monkeypatch, w, batch):
    data = gsdr.synth_fasta(0, n_reads=2500, seed=51)
    _check_masks(tmp_path, monkeypatch, data, 0.95, w=w, batch=batch)


@pytest.mark.parametrize("w", [4, 5, 6, 7])
def test_word_lengths_ragged_reads(tmp_path, monkeypatch, w):
    data = gsdr.synth_fasta(0, n_reads=2500, seed=47, len_lo=20, len_hi=240, n_seeds=500)
    _check_masks(tmp_path, monkeypatch, data, 0.95, w=w, batch=256)


@pytest.mark.parametrize("t", [0.90, 0.93, 0.97])
def test_thresholds(tmp_path, monkeypatch, t):
    data = gsdr.synth_fasta(0, n_reads=2500, seed=48, len_lo=60, len_hi=240, n_seeds=400)
    _check_masks(tmp_path, monkeypatch, data, t)


@pytest.mark.parametrize("t,batch", [(0.90, 64), (0.90, 0), (0.95, 512)])
def test_low_complexity_open_pairs(tmp_path, monkeypatch, t, batch):
    _check_masks(tmp_path, monkeypatch, repeat_reads(np.random.default_rng(49)), t, batch=batch)


def _buckets(max_len, k, t):
    """hash_buckets (csrc/api.cu): the fewest buckets, in steps of 512, that
    leave the word cutoff of the longest read five deviations above L^2 / H."""
    n = max_len - k + 1
    cut = n - math.ceil(max_len * (1.0 - float(np.float32(t)))) * k
    for h in (1024, 1536, 2048):
        if cut >= 1 and n * n / h + 5.0 * math.sqrt(n * n / h) <= cut:
            return h
    return 0


# at k = 7 and t = 0.90 the masks take the shortest reads (no cutoff to stay
# below) and those of about 330 bases and more
@pytest.mark.parametrize("length", [60, 100, 101, 150, 200, 320, 330, 331, 345, 400])
def test_both_sides_of_the_rule(tmp_path, monkeypatch, length):
    rng = np.random.default_rng(74)
    recs = []
    for i in range(300):
        seed = rng.integers(0, 4, length)
        for v in range(3):
            s = seed.copy()
            at = rng.integers(0, length, v * length // 30)
            s[at] = rng.integers(0, 4, at.size)
            recs.append(f">r{i}_{v}\n{''.join('ACGT'[x] for x in s)}\n")
    data = "".join(recs).encode()
    _, ocl, _, _ = orc.run_bytes(data, tmp_path, t=0.90)
    cl, buckets = _run(data, 0.90, None, monkeypatch, word_filter=4)
    assert buckets == _buckets(length, 7, 0.90)
    assert (buckets == 0) == (length in (60, 330, 331, 400))
    np.testing.assert_array_equal(cl, ocl)


def test_automatic_forms(monkeypatch):
    # 150 bp reads take the hashed counts, 200-1,000 bp reads at t = 0.90 the masks
    short = gsdr.synth_fasta(2, n_reads=2000, seed=98)
    assert _run(short, 0.90, None, monkeypatch)[1] == 1536
    longer = gsdr.synth_fasta(0, n_reads=1500, seed=98)
    assert _run(longer, 0.90, None, monkeypatch)[1] == 0
