"""A job for whose word filter the device has no room: the rows of hashed
k-mer counts give way to the tentative masks, the folded bitmaps to the full
ones, and only a job that does not fit in its smaller form either is refused
(GSDR_ENOMEM).  The clusters are the same.  The full device is a limit on the
size of a device allocation (gsdr_set_alloc_limit), lowered step by step."""
import numpy as np
import pytest

import gsdr

pytestmark = pytest.mark.gpu

MB = 1 << 20


# (recipe, reads, threshold, form of the job with room, its smaller form)
@pytest.mark.parametrize("recipe,n,t,full,small", [
    (2, 30_000, 0.90, (1536, False), (0, False)),   # 150 bp reads, k = 7
    (4, 6_000, 0.95, (0, True), (0, False)),        # 150-5,000 bp, k = 6
    (4, 6_000, 0.90, (0, True), (0, False)),        # k = 7
])
def test_smaller_form_when_the_device_is_full(recipe, n, t, full, small):
    data = gsdr.synth_fasta(recipe, n_reads=n, seed=92, **(
        {"n_seeds": n // 5, "len_lo": 150, "len_hi": 5000} if recipe == 4 else {}))
    f = gsdr.Fasta.parse(data)
    opts = gsdr.default_opts(threshold=t)
    got = {}
    limit = 256 * MB
    try:
        want = gsdr.clustering(f, opts)
        while limit > 0:
            gsdr.set_alloc_limit(limit)
            try:
                job = gsdr.Job(f, opts)
            except gsdr.GsdrError as e:
                assert e.status == gsdr.ENOMEM
                break
            try:
                form = job.filter_form()
                if form not in got:
                    job.run()
                    got[form] = job.cluster()
            finally:
                job.close()
            limit -= MB
    finally:
        gsdr.set_alloc_limit(None)
        f.close()
    assert list(got) == [full, small]
    for cl in got.values():
        np.testing.assert_array_equal(cl, want)


def test_no_limit_again():
    data = gsdr.synth_fasta(2, n_reads=3000, seed=93)
    f = gsdr.Fasta.parse(data)
    try:
        gsdr.set_alloc_limit(1 * MB)
        with pytest.raises(gsdr.GsdrError) as e:
            gsdr.clustering(f, gsdr.default_opts(threshold=0.90))
        assert e.value.status == gsdr.ENOMEM
        gsdr.set_alloc_limit(None)
        assert gsdr.clustering(f, gsdr.default_opts(threshold=0.90)).size == f.n
    finally:
        gsdr.set_alloc_limit(None)
        f.close()
