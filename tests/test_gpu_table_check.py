"""pfc_job_verify_tables runs the setup that the segments will use: the tensor cores' tiles (merged and paired
words) of each class that takes them, beside the integer pipe's words; and the job works as before after it."""
import numpy as np
import pytest

pfc = pytest.importorskip("pfcsieve_gb300")

from oracle import oracle as o  # noqa: E402

pytestmark = pytest.mark.gpu


# the classes of the p range that set up on the tensor cores
@pytest.mark.parametrize("mode,nmin,lo,hi,classes", [
    (1, 400000, 10**9, 10**9 + 20000, 1), (5, 300000, 2**40, 2**40 + 20000, 1),
    (4, 150000, 2**63, 2**63 + 20000, 1), (2, 600000, 2**64 - 30000, 2**64 - 1, 1),
    (5, 300000, 2**31 - 20000, 2**31 + 20000, 2), (1, 400000, 2**31 - 20000, 2**64 // 3 + 20000, 3),
    (1, 20000, 2**31 - 20000, 2**64 // 3 + 20000, 0)])
def test_the_check_runs_the_tiles(mode, nmin, lo, hi, classes):
    launches, nbytes, totals = [], [], []
    for tc in (False, True):
        with pfc.Context(0) as c:
            c.set_setup_tc(tc)
            with pfc.Job(c, mode, nmin, nmin + 50, lo, hi) as job:
                l0 = c.launches
                nbytes.append(job.verify_tables())
                launches.append(c.launches - l0)
                if hi - lo < 10**6:
                    job.segment(lo, hi)
                    _, s0, _ = job.segment_state()
                    job.segment(lo, hi)   # captured
                    nbytes.append(job.verify_tables())
                    job.segment(lo, hi)   # replayed
                    p, r0, s1 = job.segment_state()
                    assert np.array_equal(np.sort(s0), np.sort(r0))
                    totals.append(job.totals())
                    k = np.argsort(p)
                    hits, _, terms = o.sieve(mode, nmin, nmin + 50, p[k], want_terms=True)
                    assert np.array_equal(r0[k], terms[:, 0])
                    assert len(job.drain_hits()) == 3 * len(hits)
    packs = 0 if not classes else 2 if mode == 5 else 1
    assert launches[1] - launches[0] == packs + classes
    assert len(set(nbytes)) == 1 and len(set(totals)) <= 1


def test_setup_mulmods_is_a_read():
    """The count of the 64-bit words that a search from 2^64/3 on leaves out: the same as with them, without work on
    the device."""
    case = (1, 400000, 400050, 2**63, 2**63 + 20000)
    with pfc.Context(0) as c:
        c.set_setup_tc(False)
        with pfc.Job(c, *case) as job:
            want = job.setup_mulmods(True)
    words, squarings = pfc.setup_program_size(1, 400000, False)
    assert want == words + squarings
    with pfc.Context(0) as c, pfc.Job(c, *case) as job:
        before = c.transfer_bytes(), c.launches
        assert job.setup_mulmods(True) == want and (c.transfer_bytes(), c.launches) == before
