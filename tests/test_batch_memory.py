"""Device memory of mixed batches of small lattices, whose loop stage takes optional
scratch: counted in the estimate, and kept within a server's budget.  Each case in
a process of its own, whose memory pool starts empty."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEAD = """
import json
from wloop_b200 import APE, WloopParms
from wloop_b200._native import lib
from wloop_b200.api import Batch, Server, estimate_bytes
n = (32, 16, 16, 16)
p = WloopParms(msl=4, nss=[0, 1, 1, 1], mwlt=8, mwlr=8, op_smear=APE, alpha_ape=0.5, proj_iter=4)
estimate = estimate_bytes(n, 3, p, "mixed")
"""
# what the pool gives out in whole pieces
SLACK = 64 << 20


def run(script):
    r = subprocess.run([sys.executable, "-c", HEAD + script], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return json.loads(r.stdout.splitlines()[-1])


@pytest.mark.gpu
def test_estimate_counts_the_scratch():
    v = run("""
with Batch([(n, 3, p)], "mixed") as b:
    b.generate([1], [0.2])
    b.run()
    held = b.device_bytes
print(json.dumps([estimate, held, lib.wlg_batch_pool_idle_bytes(0)]))
""")
    estimate, held, pool = v
    assert pool <= estimate + SLACK and held <= estimate


@pytest.mark.gpu
def test_server_keeps_the_scratch_within_its_budget():
    """A budget one byte short of the scratch: the request runs without it."""
    v = run("""
with Server(max_inflight=1, max_batch=1) as s:
    s.set_limits(budget_bytes=estimate - 1)
    s.wait(s.submit(n, 3, p, "mixed", seed=1, eps=0.2))
    failed = s.stats()["failed"]
    small = lib.wlg_batch_pool_idle_bytes(0)
    s.set_limits(budget_bytes=estimate)
    s.wait(s.submit(n, 3, p, "mixed", seed=1, eps=0.2))
print(json.dumps([estimate, failed, small, lib.wlg_batch_pool_idle_bytes(0)]))
""")
    estimate, failed, small, full = v
    assert failed == 0
    assert small <= estimate - (256 << 20)  # the scratch of one such lattice: 0.4 GB
    assert small < full <= estimate + SLACK
