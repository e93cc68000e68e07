"""gsdr_server_times: a job's run starts once it has room on the device; the
wait for that room is queueing.  With a budget of one byte the jobs that hold
the slots run one after another, so the runs do not overlap: together they take
no longer than the time from the first submission to the last result, and the
waits show in the queued times."""
import time

import numpy as np
import pytest

import gsdr

pytestmark = pytest.mark.gpu


def test_waiting_for_memory_is_not_run_time():
    n_jobs = 4
    data = gsdr.synth_fasta(4, n_reads=8000, seed=91, n_seeds=1600, len_lo=150, len_hi=5000)
    warm = gsdr.Server(max_inflight=1)
    try:
        warm.submit(data, 0.95)
        assert warm.wait(120000)[1] == gsdr.OK
    finally:
        warm.close()
    srv = gsdr.Server(max_inflight=n_jobs, mem_budget=1, express_bytes=-1)
    try:
        t0 = time.perf_counter()
        ids = [srv.submit(data, 0.95) for _ in range(n_jobs)]
        for _ in ids:
            r = srv.wait(120000)
            assert r is not None and r[1] == gsdr.OK
        wall = 1e3 * (time.perf_counter() - t0)
        times = [srv.times(j) for j in ids]
        results = [srv.result(j) for j in ids]
    finally:
        srv.close()
    # (2 ms of slack per job between a release and the recorded end of its run)
    assert sum(run for _, run in times) <= wall + 2.0 * n_jobs, (times, wall)
    assert max(queued for queued, _ in times) >= min(run for _, run in times), times
    for out, cl in results[1:]:
        np.testing.assert_array_equal(cl, results[0][1])
        assert out == results[0][0]
