"""The device re-verification (csrc/verify.cu) where its two arithmetics and its share lengths change: p on both
sides of 2^31, ranges of a few k, of about the 8 D k per thread from which finite differences run, and of many.
Every hit of the GPU sieve passes, each with a flipped sign or n off by one fails as on the CPU."""
import numpy as np
import pytest

pfc = pytest.importorskip("pfcsieve_gb300")

pytestmark = pytest.mark.gpu


def cpu_fails(mode, nmax, rec):
    try:
        pfc.finalize(mode, nmax, np.array([rec], dtype=pfc.FACTOR_DTYPE), threads=1, verify=True)
        return False
    except pfc.PFCError as e:
        assert e.code == -6
        return True


@pytest.mark.parametrize("mode,nmin,nmax,pmin,pmax", [
    (1, 101, 300, 101, 2 * 10**5), (5, 7900, 8600, 10**6, 2 * 10**6), (1, 16200, 17000, 2**31, 2**31 + 3 * 10**8),
    (5, 15000, 40000, 2**31 - 10**7, 2**31 + 10**8), (2, 101, 2 * 10**6, 2**31, 2**31 + 5 * 10**7),
    (4, 101, 40000, 2**32, 2**32 + 3 * 10**8),
])
def test_verdicts(mode, nmin, nmax, pmin, pmax):
    with pfc.Context(0) as ctx, pfc.Job(ctx, mode, nmin, nmax, pmin, pmax) as job:
        hits = job.run()
        assert len(hits) > 3
        assert not pfc.verify_factors(ctx, mode, nmax, hits).any()
        bad = hits.copy()
        bad["nc"] = -bad["nc"]
        assert pfc.verify_factors(ctx, mode, nmax, bad).all()
        bad = hits[:6].copy()
        bad["nc"] += np.where(bad["nc"] > 0, -1, 1).astype(np.int32)
        assert pfc.verify_factors(ctx, mode, nmax, bad).tolist() == [cpu_fails(mode, nmax, r) for r in bad]
