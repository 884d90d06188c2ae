"""pfc_job_run, the C call that runs a whole search (the Python Job.run walks the same segments itself): the same
hits and totals as Job.run, and what it reports where the caller's buffer is too small."""
import ctypes

import numpy as np
import pytest

pfc = pytest.importorskip("pfcsieve_gb300")

from oracle import oracle as o  # noqa: E402

pytestmark = pytest.mark.gpu
OVERFLOW = -4


def run(job, cap):
    buf = np.zeros(max(cap, 1), dtype=pfc.FACTOR_DTYPE)
    n = ctypes.c_size_t(0)
    rc = pfc.lib().pfc_job_run(job.h, buf.ctypes.data, cap, ctypes.byref(n))
    return rc, n.value, buf


@pytest.mark.parametrize("case,budget", [((1, 101, 9000, 3, 20000), 0), ((5, 101, 3000, 10**6, 10**6 + 50000), 0),
                                         ((2, 101, 20000, 2**40, 2**40 + 20000), 0),
                                         ((1, 101, 9000, 10**6, 10**6 + 8 * 10**6), 24 << 20)])   # several segments
def test_whole_search_and_small_buffers(case, budget):
    with pfc.Context(0, budget=budget) as c:
        with pfc.Job(c, *case) as job:
            want, totals = o.sort_factors(job.run()), job.totals()
        if budget:
            with pfc.Job(c, *case) as job:
                assert job.segment_end(case[3]) < case[4]
        with pfc.Job(c, *case) as job:
            rc, n, buf = run(job, len(want) + 5)
            assert rc == 0 and n == len(want) and job.totals() == totals
            assert np.array_equal(o.sort_factors(buf[:n]), want) and not buf[n:].view(np.uint8).any()
        for cap in {0, len(want) // 2, max(len(want) - 1, 0)}:
            if cap >= len(want):
                continue
            with pfc.Job(c, *case) as job:   # the search goes on to its end and reports its count
                rc, n, buf = run(job, cap)
                assert (rc, n) == (OVERFLOW, len(want)) and job.totals() == totals
            with pfc.Job(c, *case) as job:
                with pytest.raises(pfc.PFCError) as e:
                    job.run(cap=cap)
                assert e.value.code == OVERFLOW and "cap=%d" % len(want) in str(e.value) and "Job.run" in str(e.value)
