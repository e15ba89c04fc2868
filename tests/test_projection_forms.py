"""FP64 smearing with every number of projection steps (from 3 on all but the last
run on polynomials of U^dag U) against the oracle, on smooth and rough fields,
with open time (zero links) and without. Bound: an element's error is that of
about 40 rounded products of entries up to 1.8, amplified by at most 1.5 a
step."""
import numpy as np
import pytest

from tests import oracle as O
from wloop_b200 import Context, generate_links

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [0, 1, 2, 3, 4, 7])
@pytest.mark.parametrize("eps,bc", [(0.15, 0), (0.6, 3), (2.5, 3)])
def test_steps(steps, eps, bc):
    n = (6, 3, 5, 4)
    u = generate_links(n, bc, 31, eps)
    tol = 40 * 1.8 * 2.0 ** -53 * 1.5 ** steps
    with Context(n, bc, "fp64") as c:
        for got, ref in (
                (lambda: c.ape_links(0.3, proj=1, piter=steps), O.ape_links(n, u, 0.3, 1, steps)),
                (lambda: c.hyp_spatial_links(0.75, 0.6, proj=1, piter=steps),
                 O.hyp_spatial_links(n, u, 0.75, 0.6, 1, steps))):
            c.upload(u)
            got()
            assert np.abs(c.download() - ref).max() <= tol
