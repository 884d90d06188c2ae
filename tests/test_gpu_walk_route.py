"""Which walk runs (pfc_ctx_walk_counts), in the cases whose tests compare two walks: the tensor-core walk and the
split where they are meant, none where they are switched off, on the stream, captured and replayed, and in
batches with small memory budgets.  Integers: equal, no tolerance."""
import pytest

pfc = pytest.importorskip("pfcsieve_gb300")

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
