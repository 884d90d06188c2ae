"""Split walks whose last sub-range is far shorter than the others (n lengths just past a multiple of the
sub-ranges' alignment), so that its candidates end while the first sub-range still walks its first residue:
every size class, both kinds of walk, one and two residues, against the oracle.  Integers: equal, no tolerance."""
import numpy as np
import pytest

pfc = pytest.importorskip("pfcsieve_gb300")

from oracle import oracle as o  # noqa: E402

pytestmark = pytest.mark.gpu


def run(case, split, tc):
    mode, nmin, nmax, lo, hi = case
    with pfc.Context(0) as c:
        c.set_split(split)
        c.set_walk_tc(tc)
        with pfc.Job(c, mode, nmin, nmax, lo, hi) as job:
            out = []
            for _ in range(3):   # on the stream, captured, replayed
                l0 = c.launches
                job.segment(lo, hi)
                launches = c.launches - l0
                p, s0, s1 = job.segment_state()
                k = np.argsort(p)
                out.append((p[k], s0[k], s1[k], o.sort_factors(job.drain_hits())))
            return out, launches


# seven sub-ranges of 1,280 steps and one of 40, seven of 2,304 and one of 272 (fewer where their programs cost
# more); the per-step kernels' are of one length
@pytest.mark.parametrize("mode,nmax,tc", [(5, 9101, 1), (1, 9101, 1), (4, 16501, 1), (5, 16501, 0), (1, 16501, 0)])
@pytest.mark.parametrize("lo,hi", [(10**9, 10**9 + 41000), (2**31 - 20000, 2**31 + 21000), (2**40, 2**40 + 55000),
                                   (2**62, 2**62 + 85000), (2**64 - 90000, 2**64 - 1)])
def test_short_last_sub_range(mode, nmax, tc, lo, hi):
    case = (mode, 101, nmax, lo, hi)
    got, launches = run(case, True, tc)
    assert launches > run(case, False, tc)[1], "the walk did not run split"
    cands = o.candidates(lo, hi)
    hits, _, terms = o.sieve(mode, 101, nmax, cands, want_terms=True)
    for p, s0, s1, found in got:
        assert np.array_equal(p, cands) and np.array_equal(s0, terms[:, 0])
        if mode == 5:
            assert np.array_equal(s1, terms[:, 2])
        assert np.array_equal(found, hits)
