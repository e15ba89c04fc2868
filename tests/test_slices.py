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
from wloop_b200.api import Batch

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
            assert p["bytes_a"] + p["bytes_b"] <= 4 << 30


def test_plans_refused():
    n = (64, 32, 32, 32)
    assert plan(n, 3, 6, 24, 16) is not None
    assert plan(n, 3, 6, 24, 16, budget=1 << 20) is None  # one unit does not fit
    assert plan(n, 3, 9, 24, 16) is None and plan(n, 3, 6, 0, 16) is None
    assert plan(n, 3, 6, 24, 0) is None and plan(n, 1, 6, 24, 16) is None
    assert plan((8, 1, 4, 4), 3, 2, 2, 2) is None
    # the 64-bit sums' range
    assert plan((4, 85, 84, 84), 3, 1, 1, 1) is not None
    assert plan((4, 86, 84, 84), 3, 1, 1, 1) is None


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


# the spatial links' norm and whether the digits, scaled, hold lines of two links
@pytest.mark.gpu
@pytest.mark.parametrize("norm,fits", [(1.2, True), (1.7, True), (3.5, True), (4.3, False)])
def test_links_far_from_unitary(norm, fits):
    """Spatial links of norm 1.2 to 4.3 (level 0 is not projected): lines of two of
    them reach up to norm^2, which the digits hold up to 1.98 x 8 when scaled
    (exponents 0 to 3); beyond, the FMA kernel measures."""
    n, bc = (8, 4, 4, 4), 3
    p = WloopParms(msl=2, nss=[0, 2], mwlt=3, mwlr=2, op_smear=APE, alpha_ape=0.5, proj_iter=3)
    u = generate_links(n, bc, 77, 0.01)
    u[:, 1:] *= norm
    with Context(n, bc, "fp64") as c:
        c.set_contract_tuning(variant=11)
        c.upload(u)
        c.set_profiling(True)
        got = c.wloop_sum(p)
        assert c.contract_form == 11
        launches = c.kernel_time("contract")[1]
        c.set_profiling(False)
        c.upload(u)
        c.set_gram_tuning(stages=2)
        fma = c.wloop_sum(p)
    # one launch per chunk, or one per extent
    assert launches == (plan(n, bc, 2, 3, 2)["nchunk"] if fits else p.mwlr)
    ref, ref_abs = O.wloop_sum(n, bc, u, p, want_abs=True)
    assert_wl_close(got, ref, ref_abs)
    columns = 54 * n[1] * n[2] * n[3]
    assert np.abs(got - fma).max() <= 4.0 * np.sqrt(columns) * 2.0 ** -53 * norm ** 4


@pytest.mark.gpu
def test_spatial_hyp_in_a_batch():
    """Spatial HYP leaves links far from unitary: a batch scales such a lattice's
    digits as a context does, with the same bits, also when the next field needs
    another exponent."""
    n, bc = (32, 16, 16, 16), 3
    p = WloopParms(msl=3, nss=[0, 2, 2], mwlt=6, mwlr=5, op_smear=1, alpha_hyp=(0.75, 0.6),
                   proj_iter=4)
    fields = [generate_links(n, bc, 91 + k, eps) for k, eps in enumerate((0.2, 0.05, 0.3))]
    with Context(n, bc, "fp64") as c, Batch([(n, bc, p)], "fp64") as b:
        for u in fields:
            c.upload(u)
            c.set_profiling(True)
            c.reset_kernel_times()
            ref = c.measure(p)
            assert c.contract_form == 11
            c.set_profiling(False)
            for _ in range(2):  # direct, then as a graph
                b.upload(0, u)
                b.run()
                assert np.array_equal(b.result(0), ref)
