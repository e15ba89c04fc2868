"""The mixed temporal-gauge form's packed-FMA Gram product (wloop_b200/csrc/
gpair.cu): its plan on the CPU, and on the GPU the same bits as the kernel that
runs one launch per spatial extent."""
import ctypes as C
import itertools

import numpy as np
import pytest

from tests.test_gram_plan import LATTICES
from tests.test_gram_plan import plan as gram_plan
from wloop_b200 import APE, Context, WloopParms
from wloop_b200._native import WLG_MIXED, lib

KEYS = ("lp", "tq", "ng", "bx", "bxp", "nybp", "nblk", "stages", "block", "ctas", "smem", "cpc",
        "nsplit", "nchunks", "runs", "npass", "nuc", "bytes_a", "bytes_b", "bytes_p")
THREADS = {(2, 12): 256, (2, 8): 384, (3, 8): 256, (3, 6): 384, (4, 6): 256, (4, 4): 384,
           (5, 4): 256, (5, 3): 384, (6, 3): 256, (6, 2): 384, (7, 2): 256, (8, 2): 256}


def plan(n, bc, msl, mwlt, mwlr, budget=0):
    out = (C.c_longlong * 20)()
    rc = lib.wlg_pair_plan_shape((C.c_int * 4)(*n), bc, msl, mwlt, mwlr, budget, out)
    return dict(zip(KEYS, list(out))) if rc == 0 else None


@pytest.mark.parametrize("budget", [0, 1 << 27])
@pytest.mark.parametrize("n", LATTICES)
def test_plans(n, budget):
    for bc, msl, r in itertools.product((0, 3), range(2, 9), (1, min(n[1:]) // 2 + 1)):
        for t in sorted({1, 2, n[0] // 4 + 1, n[0] // 2 + 1}):
            p = plan(n, bc, msl, t, r, budget)
            if p is None:
                assert budget  # one run may not fit a small budget
                continue
            most = THREADS[msl, p["tq"]]
            assert p["block"] % 32 == 0 and p["bx"] * p["ng"] <= p["block"]
            # registers: `most` threads of the kernel fill an SM
            assert p["block"] * p["ctas"] <= most and p["ctas"] >= 1
            assert p["ng"] * p["tq"] >= t > (p["ng"] - 1) * p["tq"]
            assert p["nblk"] * p["bx"] >= n[0] > (p["nblk"] - 1) * p["bx"]
            assert p["bxp"] % 8 == 0 and p["bx"] <= p["bxp"] <= 256
            assert p["nybp"] % 8 == 0 and p["bx"] + t - 1 <= p["nybp"] <= 256
            stage = p["lp"] * (p["bxp"] + p["nybp"]) * 128
            assert stage % 1024 == 0 and 3 <= p["stages"] <= 8
            assert p["smem"] == p["stages"] * stage + 1024
            assert p["ctas"] * (p["smem"] + 1024) <= 228 * 1024
            # the runs of the kernel with one launch per extent
            g = gram_plan(n, bc, msl, t, WLG_MIXED)
            assert (p["cpc"], p["nsplit"], p["nchunks"]) == (g["cpc"], g["nsplit"], g["nchunks"])
            assert p["runs"] * p["npass"] >= p["nsplit"] > p["runs"] * (p["npass"] - 1)
            for k in {0, p["npass"] // 2, p["npass"] - 1}:
                c0 = k * p["runs"] * p["cpc"]
                c1 = min(p["nchunks"], (k + 1) * p["runs"] * p["cpc"])
                assert -(-c1 // 18) - c0 // 18 <= p["nuc"]
            ntile = -(-n[1] * n[2] * n[3] // 32)
            assert p["nuc"] <= 3 * ntile
            nu = n[0] + (0 if bc == 0 else t)
            unit = r * p["lp"] * p["nuc"] * 576 * 8
            assert p["bytes_a"] == unit * n[0] and p["bytes_b"] == unit * nu
            assert p["bytes_p"] == 4 * r * p["runs"] * n[0] * t * msl * msl
            assert p["bytes_a"] + p["bytes_b"] + p["bytes_p"] <= (budget or 4 << 30)


def test_plans_refused():
    n = (64, 32, 32, 32)
    assert plan(n, 3, 6, 24, 16) is not None
    assert plan(n, 3, 1, 24, 16) is None  # one level: the other kernel
    assert plan(n, 3, 6, 24, 16, budget=1 << 20) is None
    assert plan(n, 3, 9, 24, 16) is None and plan(n, 3, 6, 24, 0) is None
    assert plan(n, 1, 6, 24, 16) is None and plan((8, 1, 4, 4), 3, 2, 2, 2) is None


# even and odd level counts, a time slice of 15 and 60 sites, start slices over
# several blocks, extents that leave threads idle, the longest extent
CASES = [((4, 4, 4, 4), 3, 2, 1, 1), ((6, 3, 5, 4), 0, 3, 4, 2), ((33, 4, 4, 4), 0, 4, 16, 3),
         ((40, 4, 6, 4), 3, 7, 21, 3), ((50, 3, 5, 4), 3, 5, 13, 2), ((26, 2, 2, 2), 3, 8, 14, 2),
         ((64, 4, 4, 4), 3, 6, 24, 2), ((20, 8, 8, 8), 0, 2, 11, 4)]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])) + f"_{c[2]}")
def test_same_bits(case):
    n, bc, msl, t, r = case
    p = WloopParms(msl=msl, nss=[0] + [1] * (msl - 1), mwlt=t, mwlr=r, op_smear=APE, alpha_ape=0.5,
                   proj_iter=4)
    with Context(n, bc, "mixed") as c:
        c.set_contract_tuning(variant=11)
        c.generate(2300 + msl, 0.25)
        c.snapshot()
        c.set_profiling(True)
        got = c.measure(p)
        assert c.contract_form == 11
        assert c.kernel_time("contract")[1] == plan(n, bc, msl, t, r)["npass"]
        c.reset_kernel_times()
        c.set_gram_tuning(stages=2)  # asks for one launch per extent
        c.restore()
        ref = c.measure(p)
        assert c.contract_form == 11 and c.kernel_time("contract")[1] == r
    assert np.isfinite(ref).all() and np.array_equal(got, ref)


@pytest.mark.gpu
def test_same_bits_every_time():
    """Blocks of three warps, two per SM, three stages, several passes: the case
    in which a warp once freed a stage before its last read of it."""
    n, p = (48, 24, 24, 24), WloopParms(msl=4, nss=[0, 1, 1, 1], mwlt=12, mwlr=12, op_smear=APE,
                                        alpha_ape=0.5, proj_iter=4)
    shape = plan(n, 3, 4, 12, 12)
    assert shape["block"] == 96 and shape["ctas"] == 2 and shape["npass"] > 1
    with Context(n, 3, "mixed") as c:
        c.generate(5, 0.2)
        c.snapshot()
        c.set_gram_tuning(stages=2)
        ref = c.measure(p)
        c.set_gram_tuning()
        for _ in range(12):
            c.restore()
            assert np.array_equal(c.measure(p), ref)
