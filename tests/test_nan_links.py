"""Fields with a NaN or an infinity in one link: the temporal-gauge form's range
tests see it, so that W is NaN where the loops through that link are."""
import numpy as np
import pytest

from wloop_b200 import APE, Context, WloopParms, generate_links
from wloop_b200.api import Batch

pytestmark = pytest.mark.gpu


# one entry in each column, an infinity, and a link that is NaN throughout
SPOTS = [((0, 0), np.nan), ((2, 1), np.nan), ((1, 2), np.nan), ((1, 0), np.inf),
         ((slice(None), slice(None)), np.nan)]


@pytest.mark.parametrize("spot,value", SPOTS, ids=["col0", "col1", "col2", "inf", "link"])
def test_spatial_link(spot, value):
    """The deviation kernel's threads take several links each here (at most 606208
    threads, 1.5 million links): a NaN among a thread's first links has to outlast
    the finite ones after it."""
    n, bc = (32, 20, 20, 20), 3
    p = WloopParms(msl=2, nss=[0, 0], mwlt=2, mwlr=2, op_smear=APE, alpha_ape=0.5, proj_iter=4,
                   alpha_action=(0.0, 1.0, 0.5))
    u = generate_links(n, bc, 11, 0.2)
    u[5 * 8000 + 1234, 1][spot] = value
    with Context(n, bc, "fp64") as c:
        c.upload(u)
        got = c.wloop_sum(p)
        c.set_gram_tuning(stages=2)  # one launch of FP64 FMAs per extent
        c.upload(u)
        ref = c.wloop_sum(p)
        assert c.contract_form == 11
    assert np.isnan(ref).any() and not np.isnan(ref).all()
    assert np.array_equal(got, ref, equal_nan=True)
    with Batch([(n, bc, p)], "fp64") as b:
        for _ in range(2):  # direct, then as a graph
            b.upload(0, u)
            b.run()
            assert np.array_equal(b.result(0), ref, equal_nan=True)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_temporal_link(precision):
    """Slices of more than 303104 sites, where also the last slice is shared out in
    several sites a thread: the gauge field is refused, and the carried lines
    give NaN from the one start slice whose loops use the link."""
    n, bc = (2, 68, 68, 68), 3
    p = WloopParms(msl=2, nss=[0, 0], mwlt=1, mwlr=1, op_smear=APE, alpha_ape=0.5, proj_iter=4)
    u = generate_links(n, bc, 12, 0.2)
    u[0, 0] = np.nan
    with Context(n, bc, precision) as c:
        c.upload(u)
        got = c.wloop_sum(p).reshape(n[0], -1)
        assert c.contract_form != 11
    assert np.isnan(got[0]).all() and np.isfinite(got[1]).all()
