"""Which walk runs (pfc_ctx_walk_counts), in the cases whose tests compare two walks: the tensor-core walk and the
split where they are meant, none where they are switched off, on the stream, captured and replayed, and in
batches with small memory budgets.  Integers: equal, no tolerance."""
import numpy as np
import pytest

pfc = pytest.importorskip("pfcsieve_gb300")

from oracle import oracle as o  # noqa: E402
from tests import test_gpu_split_last as last  # noqa: E402
from tests import test_gpu_walk_tc as tc  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture
def contexts(monkeypatch):
    """The counts of every context that a test opens, as they are when it closes."""
    seen = []

    class Counted(pfc.Context):
        def close(self):
            if self.h:
                seen.append(self.walk_counts())
            super().close()

    monkeypatch.setattr(pfc, "Context", Counted)
    return seen


@pytest.mark.parametrize("on", [0, 1])
@pytest.mark.parametrize("mode", [1, 2, 4, 5])
@pytest.mark.parametrize("p", [2**16, 2**31 - 20000, 2**62, 2**64 // 3 - 100000, 2**64 - 60000])
def test_plain(contexts, mode, p, on):
    tc.segment(mode, 101, 9000 + p % 7, p, p + 50003, on)
    (ntc, nsplit), = contexts
    both = p == 2**31 - 20000   # a launch per size class
    assert (ntc, nsplit) == ((2 if both else 1) if on else 0, 0)


@pytest.mark.parametrize("mode,nmax,p,span", [
    (5, 30000, 10**9, 2800), (1, 30000, 2**40, 60000), (4, 30000, 2**31 - 70000, 150000),
    (5, 30000, 2**31 - 70000, 150000), (2, 200000, 2**62, 60000), (5, 30000, 2**64 // 3 - 30000, 60000)])
def test_split(contexts, mode, nmax, p, span):
    args = (mode, 500, nmax, p, p + span)
    tc.same(tc.segment(*args, True, split=True), tc.segment(*args, False))
    n = 2 if p < 2**31 < p + span else 1
    assert contexts == [(n, n), (0, 0)]


@pytest.mark.parametrize("lo,hi", [(10**9, 10**9 + 41000), (2**40, 2**40 + 55000), (2**62, 2**62 + 85000),
                                   (2**64 - 90000, 2**64 - 1)])
def test_split_on_the_stream_captured_and_replayed(contexts, lo, hi):
    last.run((5, 101, 9101, lo, hi), True, 1)
    assert contexts == [(3, 3)]


@pytest.mark.parametrize("budget", [0, 96 << 20])
def test_batches(contexts, budget):
    tc.test_batches(budget, None)
    on, off = contexts
    # its searches are of class 32, class 64 in both word shapes, and from 2^64/3; small tables take several passes
    assert on[0] >= (8 if budget else 4) and off[0] == 0


@pytest.mark.parametrize("cls,lo", [(0, 10**9), (1, 2**40)])
def test_every_per_step_variant_vs_oracle(contexts, cls, lo):
    """Each compiled variant of the per-step walk, which the tensor-core walk stands in for at these sizes, gives
    the oracle's residues, hits and checksum."""
    hi = lo + 300000
    cands = o.candidates(lo, hi)
    for fused, modes in ((0, (1, 2, 4)), (1, (5,))):
        for mode in modes:
            ohits, osum, terms = o.sieve(mode, 3000, 7001, cands, want_terms=True)
            for v in range({(0, 0): 3, (0, 1): 2, (1, 0): 4, (1, 1): 2}[cls, fused]):
                with pfc.Context(0) as c:
                    c.set_walk_tc(0)
                    c.set_split(False)
                    c.set_walk_variant(cls, fused, v)
                    with pfc.Job(c, mode, 3000, 7001, lo, hi) as job:
                        job.segment(lo, hi)
                        p, s0, s1 = job.segment_state()
                        k = np.argsort(p)
                        assert np.array_equal(p[k], cands) and np.array_equal(s0[k], terms[:, 0]), (mode, v)
                        assert mode != 5 or np.array_equal(s1[k], terms[:, 2]), v
                        assert np.array_equal(o.sort_factors(job.drain_hits()), ohits), (mode, v)
                        assert job.totals()[0] == osum, (mode, v)
    assert all(n == (0, 0) for n in contexts)
