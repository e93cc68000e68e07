"""The tuning cache's lines belong to the kernels they were measured on: an
automatic job takes a line of its own kernel generation, and neither a line
without the mark, as older builds wrote them, nor one with another mark.  The
autotuner leaves such lines in the file."""
import numpy as np
import pytest

import gsdr
from gsdr.autotune import autotune

pytestmark = pytest.mark.gpu


def test_lines_of_other_kernels_are_not_applied(tmp_path, monkeypatch):
    data = gsdr.synth_fasta(0, n_reads=1500, seed=97)
    cache = tmp_path / "tune.tsv"
    monkeypatch.setenv("GSDR_TUNE_CACHE", str(cache))
    f = gsdr.Fasta.parse(data)
    try:
        def job():
            return gsdr.clustering(f, gsdr.default_opts(threshold=0.95), stats=True)

        want, st = job()
        assert st.tuned == 0
        res = autotune(data, 0.95, reps=200, runs=1)
        own = cache.read_text().splitlines()[-1]
        assert job()[1].tuned == 1
        knobs = ["64", "3", "32", "0", "0", "0", "0", "9.999"]
        old = "\t".join([res["gpu"], res["bucket"]] + knobs)
        other = "\t".join([own.split("\t")[0] + "x", res["bucket"]] + knobs)
        assert own.split("\t")[0] not in (res["gpu"], other.split("\t")[0])
        cache.write_text(old + "\n" + other + "\n")
        cl, st = job()
        assert st.tuned == 0 and st.batch != 64
        np.testing.assert_array_equal(cl, want)
        autotune(data, 0.95, reps=200, runs=1)
        lines = cache.read_text().splitlines()
        assert old in lines and other in lines and len(lines) == 3
        assert job()[1].tuned == 1
    finally:
        f.close()
