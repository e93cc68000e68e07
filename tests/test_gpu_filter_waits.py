"""The tensor-core word filters' waits end in a status, not a hang: with the
limit at 0 polls (gsdr_set_spin_limit) every hand-over between their warps
gives up at once, the kernels free their tensor memory, set the error flag and
return, the job reports GSDR_ETIMEOUT, and the same job with the default limit
gives the oracle's clusters.  With a few polls a run either ends that way,
with products in flight, or finishes exactly.  Lowering the limit only
shortens waits that are bounded already."""
import numpy as np
import pytest

import gsdr
import oracle_binding as orc

pytestmark = pytest.mark.gpu


def _case(form):
    if form == "hash":  # 150 bp reads, k = 7
        return gsdr.synth_fasta(2, n_reads=6000, seed=99), 0.90
    return gsdr.synth_fasta(0, n_reads=2500, seed=99), 0.95  # bitmaps, k = 6


@pytest.mark.parametrize("form", ["bits", "hash"])
def test_wait_that_runs_out_reports_timeout(tmp_path, form):
    data, t = _case(form)
    _, ocl, _, _ = orc.run_bytes(data, tmp_path, t=t)
    f = gsdr.Fasta.parse(data)
    job = gsdr.Job(f, gsdr.default_opts(threshold=t, batch=64))
    try:
        assert (job.filter_form()[0] > 0) == (form == "hash")
        gsdr.set_spin_limit(0)
        for _ in range(2):
            with pytest.raises(gsdr.GsdrError) as e:
                job.run()
            assert e.value.status == gsdr.ETIMEOUT
        gsdr.set_spin_limit(None)
        assert job.run().word_index == (3 if form == "hash" else 2)
        np.testing.assert_array_equal(job.cluster(), ocl)
    finally:
        gsdr.set_spin_limit(None)
        job.close()
        f.close()


@pytest.mark.parametrize("form", ["bits", "hash"])
@pytest.mark.parametrize("polls", [1, 3])
def test_few_polls_end_in_a_status_or_exactly(form, polls):
    data, t = _case(form)
    f = gsdr.Fasta.parse(data)
    job = gsdr.Job(f, gsdr.default_opts(threshold=t, batch=256))
    try:
        job.run()
        want = job.cluster()
        gsdr.set_spin_limit(polls)
        for _ in range(3):
            try:
                job.run()
            except gsdr.GsdrError as e:
                assert e.status == gsdr.ETIMEOUT
            else:
                np.testing.assert_array_equal(job.cluster(), want)
        gsdr.set_spin_limit(None)
        job.run()
        np.testing.assert_array_equal(job.cluster(), want)
    finally:
        gsdr.set_spin_limit(None)
        job.close()
        f.close()
