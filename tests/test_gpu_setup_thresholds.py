"""The tensor-core setup on both sides of its thresholds (kernels.cuh kTcMinWords32, kTcMinWords64, kTcMinWordsTop):
the smallest programs that take it and the largest that do not, by their packing launches, with the oracle's
residues.  Integers: equal, no tolerance."""
import numpy as np
import pytest

pfc = pytest.importorskip("pfcsieve_gb300")

from oracle import oracle as o  # noqa: E402

pytestmark = pytest.mark.gpu


def words(mode, nmin):
    return pfc.setup_program_size(mode, nmin, True)[0]


def first_at(mode, least):
    """The smallest nmin near which programs reach `least` words (sizes grow by steps with nmin)."""
    lo, hi = 1000, 2000000
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if words(mode, mid) < least else (lo, mid)
    return hi


@pytest.mark.parametrize("mode", [1, 2, 4, 5])
@pytest.mark.parametrize("least,lo,hi", [(240, 10**9, 10**9 + 30000), (240, 3, 9000), (216, 2**31 + 1, 2**31 + 30000),
                                         (216, 2**64 // 3 - 60000, 2**64 // 3), (112, 2**64 // 3 + 1, 2**64 // 3 + 60000),
                                         (112, 2**64 - 60000, 2**64 - 1)])
def test_both_sides(mode, least, lo, hi):
    at = first_at(mode, least)
    for nmin in (at, at - 1):
        takes = words(mode, nmin) >= least
        assert takes == (nmin == at)
        launches = []
        for tc in (True, False):
            with pfc.Context(0) as c:
                c.set_setup_tc(tc)
                with pfc.Job(c, mode, nmin, nmin + 40, lo, hi) as job:
                    l0 = c.launches
                    job.segment(lo, hi)
                    launches.append(c.launches - l0)
                    p, s0, s1 = job.segment_state()
                    k = np.argsort(p)
                    cands = o.candidates(lo, hi)
                    assert np.array_equal(p[k], cands)
                    hits, _, terms = o.sieve(mode, nmin, nmin + 40, cands, want_terms=True)
                    assert np.array_equal(s0[k], terms[:, 0])
                    assert mode != 5 or np.array_equal(s1[k], terms[:, 2])
                    assert np.array_equal(o.sort_factors(job.drain_hits()), hits)
        assert launches[0] - launches[1] == ((2 if mode == 5 else 1) if takes else 0)
