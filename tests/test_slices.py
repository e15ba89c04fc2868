"""The FP64 temporal-gauge form's Gram product as exact 8-bit digit products
(wloop_b200/csrc/gslice.cu): its plan on the CPU, and on the GPU the loops
against the oracle and against the FMA kernel, at the edges of its tiles."""
import ctypes as C
import itertools

import numpy as np
import pytest

from tests import oracle as O
from tests.test_gpu_parity import assert_wl_close
from tests.test_gram_plan import LATTICES
from wloop_b200 import APE, Context, WloopParms, generate_links
from wloop_b200._native import lib

KEYS = ("rows_a", "rows_b", "tn", "nmt", "ntiles", "stages", "tmem", "smem", "nuc", "nchunk",
        "kps", "nsplit", "bytes_a", "bytes_b", "acc", "ntile")
P = 7  # digit planes


def plan(n, bc, msl, mwlt, mwlr, budget=0):
    out = (C.c_longlong * 16)()
    rc = lib.wlg_slice_plan_shape((C.c_int * 4)(*n), bc, msl, mwlt, mwlr, budget, out)
    return dict(zip(KEYS, list(out))) if rc == 0 else None


@pytest.mark.parametrize("n", LATTICES)
def test_plans(n):
    for bc, msl, r in itertools.product((0, 3), (1, 2, 3, 5, 6, 8), (1, min(n[1:]) // 2 + 1)):
        for t in sorted({1, 2, n[0] // 2 + 1}):
            p = plan(n, bc, msl, t, r)
            assert p is not None, (n, bc, msl, t, r)
            units = 3 * p["ntile"]
            assert p["rows_a"] == n[0] * msl
            assert p["rows_b"] == (n[0] + (0 if bc == 0 else t)) * msl
            # one MMA operand: N a multiple of 16 up to 256, all classes in TMEM
            assert p["tn"] % 16 == 0 and P * p["tn"] <= p["tmem"] <= 512
            stage = P * 64 * (128 + p["tn"])
            assert 2 <= p["stages"] <= 8
            assert p["stages"] * stage + 1024 <= p["smem"] <= 226 * 1024
            # two CTAs (two TMEM owners) never share an SM
            assert 2 * p["smem"] > 228 * 1024
            # every entry of the band lies in a tile
            tiles = 0
            for m in range(0, p["rows_a"], 128):
                first = (m // msl + 1) * msl
                last = min((min(m + 127, p["rows_a"] - 1) // msl + t + 1) * msl, p["rows_b"])
                tiles += max(0, -(-(last - first) // p["tn"]))
            assert tiles == p["ntiles"] >= 1
            # chunks cover the units, splits the K blocks; 32-bit sums
            assert p["nuc"] * p["nchunk"] >= units > p["nuc"] * (p["nchunk"] - 1)
            assert p["kps"] * p["nsplit"] >= 9 * p["nuc"] > p["kps"] * (p["nsplit"] - 1)
            assert p["kps"] * 64 * P * 128 * 128 < 2 ** 31
            row = 4096  # 9 x 7 x 64 digits, padded
            assert p["bytes_a"] == r * p["nuc"] * p["rows_a"] * row
            assert p["bytes_b"] == r * p["nuc"] * p["rows_b"] * row
            assert p["bytes_a"] + p["bytes_b"] <= 2 << 30


def test_plans_refused():
    n = (64, 32, 32, 32)
    assert plan(n, 3, 6, 24, 16) is not None
    assert plan(n, 3, 6, 24, 16, budget=1 << 20) is None  # one unit does not fit
    assert plan(n, 3, 9, 24, 16) is None and plan(n, 3, 6, 0, 16) is None
    assert plan(n, 3, 6, 24, 0) is None and plan(n, 1, 6, 24, 16) is None
    assert plan((8, 1, 4, 4), 3, 2, 2, 2) is None


# (lattice, bc, levels, t, r): one A tile with few rows; a row count just past
# a tile (132 = 128 + 4); levels that do not divide a tile, several B tiles;
# ragged time slices of 15 and 60 sites; 8 levels and the longest extent
CASES = [((4, 4, 4, 4), 3, 1, 1, 1), ((6, 3, 5, 4), 0, 2, 4, 2), ((22, 4, 4, 4), 3, 6, 5, 3),
         ((33, 4, 4, 4), 0, 4, 16, 2), ((40, 4, 6, 4), 3, 7, 21, 3), ((50, 3, 5, 4), 3, 3, 26, 2),
         ((26, 2, 2, 2), 3, 8, 14, 2)]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])) + f"_{c[2]}")
def test_loops(case):
    n, bc, msl, t, r = case
    p = WloopParms(msl=msl, nss=[0] + [1] * (msl - 1), mwlt=t, mwlr=r, op_smear=APE, alpha_ape=0.5,
                   proj_iter=4)
    u = generate_links(n, bc, 2200 + msl, 0.2)
    uh = O.hyp_links(n, bc, u, *p.alpha_action, p.proj, p.proj_iter)
    ref, ref_abs = O.wloop_sum(n, bc, uh, p, want_abs=True)
    with Context(n, bc, "fp64") as c:
        c.set_contract_tuning(variant=11)
        c.upload(u)
        c.snapshot()
        c.set_profiling(True)
        got = c.measure(p)
        assert c.contract_form == 11
        # one contraction launch per chunk, not per extent
        assert c.kernel_time("contract")[1] == plan(n, bc, msl, t, r)["nchunk"]
        c.set_profiling(False)
        c.restore()
        assert np.array_equal(c.measure(p), got)  # exact sums: no order dependence
        c.set_gram_tuning(stages=2)
        c.restore()
        fma = c.measure(p)
    assert_wl_close(got, ref, ref_abs)
    # the FMA sums: at most 54 N1 N2 N3 roundings each, random in sign; the
    # digits' 2^-54 per column and the lines' common rounding are far smaller
    columns = 54 * n[1] * n[2] * n[3]
    assert np.abs(got - fma).max() <= 4.0 * np.sqrt(columns) * 2.0 ** -53
    assert np.array_equal(got == 0.0, ref == 0.0)


@pytest.mark.gpu
def test_rough_links_leave_the_digits():
    """Spatial links far from unitary (one projection step short of
    convergence on a rough field) could leave the digits' range: the FMA
    kernel measures them."""
    n, bc = (8, 4, 4, 4), 3
    p = WloopParms(msl=2, nss=[0, 2], mwlt=3, mwlr=2, op_smear=1, alpha_hyp=(0.75, 0.6),
                   proj_iter=3)
    u = generate_links(n, bc, 77, 0.1)
    u[:, 1:] *= 1.2  # spatial links of norm 1.2, smeared into level 0 unprojected
    with Context(n, bc, "fp64") as c:
        c.set_contract_tuning(variant=11)
        c.upload(u)
        c.set_profiling(True)
        got = c.wloop_sum(p)
        assert c.contract_form == 11
        assert c.kernel_time("contract")[1] == p.mwlr  # one launch per extent
    ref, ref_abs = O.wloop_sum(n, bc, u, p, want_abs=True)
    assert_wl_close(got, ref, ref_abs)
