"""bench.py's figures follow what the library says ran: walks on the tensor cores are priced as their tests, the
others as multiplies, and setups from 2^64/3 on as the tensor cores' from kTcMinWordsTop words on."""
import os
import re
import types

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PEAKS = {"imad": 20e12, "mul_hi": 8e12, "imad_wide": 10e12, "iadd_xor": 40e12}


def test_mixed_roofline_prices_what_ran():
    pytest.importorskip("pfcsieve_gb300")
    import bench
    from pfcsieve_gb300 import serving
    S = serving.Search
    jobs = [S(1, 5000, 6000, 10**9, 10**9 + 10**6), S(1, 5000, 7000, 2**40, 2**40 + 10**6),
            S(1, 5000, 8000, 3 * 2**62, 3 * 2**62 + 10**6)]
    out = {i: types.SimpleNamespace(primecount=1000) for i in range(3)}
    plain = bench.mixed_roofline(jobs, out, 2.0, PEAKS)
    assert bench.mixed_roofline(jobs, out, 2.0, PEAKS, tc_steps=[0, 0, 0]) == plain
    steps, cost = [1e6, 2e6, 3e6], [5.0, 9.0, 16.0]   # multiplies of a step: 2 w + 1, 4 w + 1, 7 w + 2
    for tc in ([1e6, 0, 0], [5e5, 2e6, 0], steps, [9e9] * 3):
        ran = [min(t, s) for t, s in zip(tc, steps)]
        want = (plain["alg_ops"] - sum(t * c for t, c in zip(ran, cost))) / 20e12 + 2.5 * sum(ran) / 40e12
        r = bench.mixed_roofline(jobs, out, 2.0, PEAKS, tc_steps=tc)
        assert abs(r["frac"] - want / 2.0) < 1e-12 and r["achieved"] / r["peak"] == r["frac"]
        assert r["per_step_algorithm"]["frac"] == plain["frac"] and r["alg_ops"] == plain["alg_ops"]
        assert abs(r["walk_steps_on_tensor_cores"] - sum(ran) / 6e6) < 1e-12


def test_setups_from_the_third_class_on():
    pfc = pytest.importorskip("pfcsieve_gb300")
    import bench
    from pfcsieve_gb300 import serving
    src = open(os.path.join(ROOT, "pfcsieve_gb300", "csrc", "kernels.cuh")).read()
    assert bench.TC_MIN_WORDS_TOP == int(re.search(r"kTcMinWordsTop = (\d+);", src).group(1))
    jobs = [serving.Search(1, 60000, 61000, 3 * 2**62, 3 * 2**62 + 10**6)]
    out = {0: types.SimpleNamespace(primecount=10)}
    words, sq = pfc.setup_program_size(1, 60000)
    narrow, nsq = pfc.setup_program_size(1, 60000, wide=False)
    assert words >= bench.TC_MIN_WORDS_TOP
    on, off = (bench.mixed_roofline(jobs, out, 1.0, PEAKS, setup_tc=tc) for tc in (True, False))
    assert on["alg_ops"] == 10 * (words * 11.5 + sq * 18.0 + 1000 * 16.0)
    assert off["alg_ops"] == 10 * (narrow * 18.0 + nsq * 18.0 + 1000 * 16.0)
    assert on["tensor_setup"]["flops"] == 2 * 10 * words * 112 * 8 and off["tensor_setup"] is None
