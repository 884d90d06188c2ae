"""Host threads, each with a context of its own, whose first launches of every kernel fall together."""
import os
import subprocess
import sys

import pytest

pytest.importorskip("pfcsieve_gb300")

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import sys, threading
sys.path.insert(0, ".")
import pfcsieve_gb300 as pfc
searches = [(1, 101, 20000, 10**9, 10**9 + 10**6), (5, 300000, 303000, 2**50, 2**50 + 50000),
            (4, 150000, 153000, 2**63, 2**63 + 50000), (2, 400000, 430000, 10**9, 10**9 + 50000)]
start, out = threading.Barrier(4), [None] * 4

def run(i):
    with pfc.Context(0) as c:
        c.set_walk_tc(2)
        start.wait()
        out[i] = [(r.checksum, r.primecount) for r in (pfc.sieve(*s, threads=2, ctx=c) for s in searches)]

threads = [threading.Thread(target=run, args=(i,)) for i in range(4)]
[t.start() for t in threads]
[t.join() for t in threads]
assert out[0] and all(o == out[0] for o in out), out
print("same")
"""


@pytest.mark.gpu
def test_first_launches_from_several_threads():
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stdout + r.stderr
