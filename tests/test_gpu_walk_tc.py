"""The tensor-core walk (csrc/walk_tc.cu) against the oracle and the per-step kernels, at the edges of its
tiles: candidate counts around a CTA's 128, n lengths around a block, a tile and a supertile, the word
shapes, both size classes, every mode, several launches of one walk, split walks.  Integers: equal, no
tolerance."""
import numpy as np
import pytest

pfc = pytest.importorskip("pfcsieve_gb300")

from oracle import oracle as o  # noqa: E402

pytestmark = pytest.mark.gpu


def segment(mode, nmin, nmax, lo, hi, on, cuts=(), split=False):
    with pfc.Context(0) as ctx:
        ctx.set_walk_tc(2 * on)   # (2: whatever the size)
        ctx.set_split(split)
        with pfc.Job(ctx, mode, nmin, nmax, lo, hi) as job:
            job.gen(lo, hi)
            job.setup()
            at = [nmin, *cuts, nmax]
            for a, b in zip(at, at[1:]):
                job.iterate(a, b)
            job.check()
            p, s0, s1 = job.segment_state()
            order = np.argsort(p)
            return p[order], s0[order], s1[order], job.totals(), o.sort_factors(job.drain_hits())


def same(a, b):
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("mode", [1, 2, 4, 5])
@pytest.mark.parametrize("p", [2**16, 2**31 - 20000, 2**62, 2**64 // 3 - 100000, 2**64 // 3, 2**64 - 60000])
def test_walk_matches_the_oracle(mode, p):
    nmin, nmax = 101, 9000 + p % 7
    hi = p + 50003
    got = segment(mode, nmin, nmax, p, hi, True)
    cands = o.candidates(p, hi)
    assert np.array_equal(got[0], cands)
    hits, _, terms = o.sieve(mode, nmin, nmax, cands, want_terms=True)
    assert np.array_equal(got[1], terms[:, 0])
    if mode == 5:
        assert np.array_equal(got[2], terms[:, 2])
    assert np.array_equal(got[4], hits)


@pytest.mark.parametrize("nmin,length", [(n, k) for n in (201000, 202001, 12899000)
                                         for k in (1, 15, 17, 64, 255, 257, 1025, 4097)] + [(2**31 - 6000, 2049)])
def test_lengths_and_word_shapes(nmin, length):
    for p in (1500000000, 2**45, 2**63 + 2**61):
        args = (1, nmin, nmin + length, p, p + 200000)
        same(segment(*args, True), segment(*args, False))


@pytest.mark.parametrize("mode,p,span,cuts,split", [
    (5, 10**9, 40, (), False), (2, 2**40, 2700, (), False), (5, 10**9, 2800, (), True), (1, 2**40, 60000, (), True),
    (5, 10**8, 150000, (517, 1541, 9000, 20001), False), (2, 2**50, 150000, (517, 1541, 9000, 20001), False),
    (5, 2**64 - 60000, 59999, (517, 1541, 9000, 20001), False), (2, 2**64 // 3 - 30000, 60000, (), True),
    (4, 2**50, 20000, (503, 504, 1009, 1010, 1041), False), (5, 10**9, 20000, (503, 504, 1009, 1010, 1041), False),
    (4, 2**31 - 70000, 150000, (), True), (5, 2**31 - 70000, 150000, (), True),
])
def test_candidate_counts_and_ranges(mode, p, span, cuts, split):
    args = (mode, 500, 30000, p, p + span)
    same(segment(*args, True, cuts=cuts, split=split), segment(*args, False))


@pytest.mark.parametrize("mode", [1, 2, 4, 5])
def test_many_hits(mode):
    """p not far above n: hits in every block, and candidates that n passes (their residue is 0 from there)."""
    args = (mode, 101, 90000, 2**16, 160000)
    same(segment(*args, True), segment(*args, False))


@pytest.mark.parametrize("budget,work", [(0, None), (96 << 20, None), (0, 2e8)])
def test_batches(budget, work):
    """Windows of many searches in one launch: every mode and class, both word shapes, timelines that end in a
    window and that go on, and (small budget) tables that take several passes."""
    searches = [(m, n0, n0 + ln, p, p + span) for m, n0, ln, p, span in (
        (1, 101, 30000, 10**9, 60000), (5, 500, 20000, 2**31 - 40000, 90000), (2, 300000, 90000, 2**50, 30000),
        (4, 200000, 9000, 2**62, 130000), (5, 1000, 12000, 3 * 2**62, 50000), (1, 20000, 70000, 2**40, 9000),
        (4, 101, 300, 10**9, 100000), (2, 101, 200000, 2**64 // 3 + 10**6, 40000))]

    def run(on):
        with pfc.Context(0, budget=budget) as ctx:
            ctx.set_walk_tc(2 * on)
            with pfc.Batch(ctx, work) as batch:
                ids = [batch.submit(*s) for s in searches]
                batch.run()
                out = []
                for i in ids:
                    st = batch.status(i)
                    out.append((st.status, st.term_checksum, st.primecount, st.pairs,
                                o.sort_factors(batch.hits(i)).tobytes()))
                return out

    got = run(True)
    assert got == run(False)
    assert all(r[0] == 0 for r in got) and any(r[4] for r in got)
