"""Small memory budgets: what a search can do without (the tensor cores' setup tiles, the walk's word tables, a
split) makes room for what it needs, so every budget from the least accepted one on is accepted, with the same
result.  Integers: equal, no tolerance."""
import numpy as np
import pytest

pfc = pytest.importorskip("pfcsieve_gb300")

from oracle import oracle as o  # noqa: E402

pytestmark = pytest.mark.gpu

SEARCHES = [(1, 1000001, 1000500, 2**40, 2**40 + 10**6), (1, 1000001, 1000500, 3 * 2**62, 3 * 2**62 + 10**6),
            (5, 400001, 400500, 10**9, 10**9 + 10**6), (5, 101, 60000, 10**9, 10**9 + 2 * 10**5),
            (4, 101, 9000, 2**40, 2**40 + 55000)]
STEPS = [4096 * k for k in range(64)] + [1 << k for k in range(18, 25)]


def job(search, budget):
    """Three segments (on the stream, captured, replayed)."""
    with pfc.Context(0, budget=budget) as c:
        c.set_walk_tc(2)
        with pfc.Job(c, *search) as j:
            hits = []
            for _ in range(3):
                j.segment(*search[3:])
                hits.append(j.drain_hits())
            return (j.totals(), o.sort_factors(np.concatenate(hits)).tobytes()), (c.walk_counts(), c.launches)


def least(run):
    lo, hi = 16 << 20, 256 << 20
    while hi - lo > 1024:
        mid = (lo + hi) // 2
        try:
            run(mid)
            hi = mid
        except pfc.PFCError as e:
            assert e.code == -3   # out of memory
            lo = mid
    return hi


@pytest.mark.parametrize("search", SEARCHES)
def test_every_budget_from_the_least_on(search):
    want, route = job(search, 0)
    at = least(lambda b: job(search, b))
    routes = set()
    for k in STEPS:
        got, r = job(search, at + k)
        assert got == want, k
        routes.add(r)
    assert route in routes or len(routes) > 1
    assert any(r[0][0] == 0 for r in routes), "no budget left the word tables out"
    assert any(r[0][0] >= 3 for r in routes), "no budget took them"
    if search[1] > 10**5:   # tiles, or none: packing launches
        assert len({r[1] for r in routes if r[0][0]}) > 1, "no budget left the tiles out"


def test_words_and_tiles_make_room():
    """Another job and a larger segment on a context that a job's tables have filled."""
    a, b = SEARCHES[2], (1, 101, 9000, 10**9, 10**9 + 20000)

    def both(budget):
        with pfc.Context(0, budget=budget) as c:
            c.set_walk_tc(2)
            out = []
            with pfc.Job(c, *a) as j:
                for hi in (a[3] + 10**5, a[3] + 10**6, a[3] + 10**6):
                    j.segment(a[3], hi)
                    out.append(j.totals())
                with pfc.Job(c, *b) as k:
                    k.segment(*b[3:])
                    out.append(k.totals())
                j.segment(*a[3:])
                out += [j.totals(), o.sort_factors(j.drain_hits()).tobytes()]
            return out

    want = both(0)
    at = least(both)
    for k in STEPS:
        assert both(at + k) == want, k


def batch(searches, budget):
    """One search after another through one batch: each is alone in it."""
    with pfc.Context(0, budget=budget) as c:
        c.set_walk_tc(2)
        with pfc.Batch(c) as b:
            out = []
            for s in searches:
                i = b.submit(*s)
                b.run()
                st = b.status(i)
                if st.status:
                    raise pfc.PFCError(st.status, "batch")
                out.append((st.term_checksum, st.primecount, o.sort_factors(b.hits(i)).tobytes()))
            return out, c.walk_counts()[0], c.launches


@pytest.mark.parametrize("search", SEARCHES[:3])
def test_every_budget_of_a_batch(search):
    want, most, _ = batch([search], 0)
    at = least(lambda b: batch([search], b))
    routes = set()
    for k in [256 * i for i in range(600)] + STEPS:
        got, tc, launches = batch([search], at + k)
        assert got == want, k
        routes.add((tc, launches))
    tcs = {tc for tc, _ in routes}
    assert {0, most} <= tcs, "both walks"
    assert len({n for tc, n in routes if tc == most}) > 1, "no budget left the tiles out"


@pytest.mark.parametrize("search", SEARCHES[:3])
def test_a_batch_gives_its_window_records_back(search):
    """The least budget of a search alone is enough for it after another one as well."""
    small = (1, 101, 9000, 10**9, 10**9 + 20000)
    want = batch([small, search], 0)[0]
    assert batch([small, search], least(lambda b: batch([search], b)))[0] == want


def test_a_job_that_outlives_its_context():
    """Closing the context gives its jobs' buffers back; the job is closed (or collected) after it."""
    for _ in range(3):
        c = pfc.Context(0)
        jobs = [pfc.Job(c, *s) for s in (SEARCHES[4], SEARCHES[3])]
        jobs[0].segment(*SEARCHES[4][3:])
        c.close()
        jobs[0].close()
        del jobs
    assert job(SEARCHES[4], 0)[0][0][1]
