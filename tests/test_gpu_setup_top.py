"""The tensor-core setup of candidates from 2^64/3 on (csrc/setup_tc.cu) against the 64-bit words of the integer
pipe, at both ends of its range of p, one tile and several, every mode, across the class boundary, alone and
in a batch.  Integers: equal, no tolerance."""
import numpy as np
import pytest

pfc = pytest.importorskip("pfcsieve_gb300")

from oracle import oracle as o  # noqa: E402

pytestmark = pytest.mark.gpu
CASES = [(1, 60000, 60100, 2**64 // 3 + 1, 2**64 // 3 + 40000), (1, 400001, 400050, 2**64 - 90000, 2**64 - 1),
         (2, 600000, 600050, 3 * 2**62, 3 * 2**62 + 3000), (4, 150000, 150100, 2**63 - 20000, 2**63 + 20000),
         (5, 300000, 300050, 2**64 - 30000, 2**64 - 1), (5, 90000, 90100, 2**64 // 3 - 20000, 2**64 // 3 + 20000),
         (1, 30000, 30100, 2**63, 2**63 + 20000)]


@pytest.mark.parametrize("case", CASES)
def test_equals_the_integer_setup(case):
    mode, nmin, nmax, lo, hi = case
    out = []
    for tc in (True, False):
        with pfc.Context(0) as c:
            c.set_setup_tc(tc)
            with pfc.Job(c, mode, nmin, nmax, lo, hi) as job:
                job.segment(lo, hi)
                p, s0, s1 = job.segment_state()
                k = np.argsort(p)
                out.append((job.totals(), p[k].tobytes(), s0[k].tobytes(), s1[k].tobytes(), job.setup_mulmods(True),
                            job.verify_tables(), o.sort_factors(job.drain_hits()).tobytes()))
                if tc:   # switched off in the middle of a job: the same segment again
                    c.set_setup_tc(False)
                    job.gen(lo, hi)
                    job.setup()
                    q, r0, _ = job.segment_state()
                    c.set_setup_tc(True)
                    job.gen(lo, hi)
                    job.setup()
                    q2, r2, _ = job.segment_state()
                    assert np.array_equal(r0[np.argsort(q)], r2[np.argsort(q2)])
    assert out[0] == out[1]


def test_batch():
    out = []
    for tc in (True, False):
        with pfc.Context(0) as c:
            c.set_setup_tc(tc)
            with pfc.Batch(c) as b:
                ids = [b.submit(*s) for s in CASES]
                b.run()
                out.append([(b.status(i).status, b.status(i).term_checksum, b.status(i).primecount) for i in ids])
    assert out[0] == out[1] and all(s[0] == 0 for s in out[0])
