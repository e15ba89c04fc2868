"""The plaquette sum on both sides of the size where a thread takes all planes
of a site instead of one (75,776 sites on 148 SMs), against the oracle: FP64 to
the rounding of the sum, mixed to the FP32 products' (6 products of unit
matrices per plaquette, 2^-24 each, random over the sites)."""
import pytest

from tests import oracle as O
from wloop_b200 import Context, generate_links

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(3, 2, 5, 2), (18, 16, 16, 16), (19, 16, 16, 16), (21, 16, 17, 15)])
@pytest.mark.parametrize("bc", [0, 3])
def test_plaq(n, bc):
    u = generate_links(n, bc, 77, 0.3)
    ref = O.plaq_sum(n, bc, u)
    for prec, tol in (("fp64", 1e-13), ("mixed", 1e-6)):
        with Context(n, bc, prec) as c:
            c.upload(u)
            got = [c.lnk_plaq_sum() for _ in range(3)]
            assert got[0] == got[1] == got[2]
            assert abs(got[0] - ref) <= tol * abs(ref)
