"""Which lattices the FP64 digit product takes unscaled, and how it scales the
others."""
import numpy as np
import pytest

from wloop_b200 import APE, Context, WloopParms, generate_links
from wloop_b200.api import Batch, launch_count

DELTA = 0.0297  # largest |Re| and |Im| of U^dag U - 1


def turn(a, b):
    """A unitary matrix that takes the unit vector a to the unit vector b."""
    frames = []
    for x in (a, b):
        q = np.linalg.qr(np.column_stack([x, np.eye(3)[:, 1:]]))[0].astype(complex)
        q[:, 0] *= q[:, 0].conj() @ x
        frames.append(q)
    return frames[1] @ frames[0].conj().T


def longest_line():
    """Sixteen links, each with U^dag U - 1 at most DELTA in every real and imaginary
    part, and a product as large as such links allow in its first entry."""
    m = DELTA * np.array([[1, 1 + 1j, 1 + 1j], [1 - 1j, 1, 1 + 1j], [1 - 1j, 1 - 1j, 1]])
    lam, vec = np.linalg.eigh(m)
    root = (vec * np.sqrt(1 + lam)) @ vec.conj().T  # stretches vec[:, 2] most
    axis = np.array([1, 0, 0], dtype=complex)
    links = [turn(vec[:, 2], axis) @ root] + [root] * 14
    return links + [np.sqrt(1 + DELTA) * turn(axis, vec[:, 2])]


def test_longest_line():
    links = longest_line()
    for u in links:
        d = u.conj().T @ u - np.eye(3)
        assert max(np.abs(d.real).max(), np.abs(d.imag).max()) < DELTA * (1 + 1e-12)
    # above what the digits hold; the norm of U^dag U - 1 is not 3 DELTA
    assert np.linalg.multi_dot(links)[0, 0].real > 2.2 > 1.98 > (1 + 3 * DELTA) ** 8


@pytest.mark.gpu
def test_bound_holds_every_line():
    n, bc = (2, 30, 30, 30), 3
    p = WloopParms(msl=1, nss=[0], mwlt=1, mwlr=16, op_smear=APE, alpha_ape=0.5, proj_iter=4)
    u = np.zeros((n[0], 30, 30, 30, 4, 3, 3), dtype=np.complex128)
    u[..., :, :] = np.eye(3)
    for x3, link in enumerate(longest_line()):
        u[:, :, :, x3, 3] = link
    u = u.reshape(-1, 4, 3, 3)
    with Context(n, bc, "fp64") as c:
        c.upload(u)
        got = c.wloop_sum(p)
        assert c.contract_form == 11
        c.set_gram_tuning(stages=2)
        c.upload(u)
        fma = c.wloop_sum(p)
    # lines of R links are at most 1.111^R in norm: sums of 54 x 30^3 products
    columns = 54 * 30 ** 3
    assert np.abs(got - fma).max() <= 4.0 * np.sqrt(columns) * 2.0 ** -53 * 2.25 ** 2


@pytest.mark.gpu
def test_another_scale_replays_the_graph():
    """A batch's captured graph serves fields whose lines need another scale, and
    fields that need none: replaying it issues no launches but those that find the
    scale."""
    n, bc = (32, 8, 8, 16), 3
    p = WloopParms(msl=2, nss=[0, 0], mwlt=4, mwlr=2, op_smear=APE, alpha_ape=0.5, proj_iter=4,
                   alpha_action=(0.0, 1.0, 0.5))
    base = generate_links(n, bc, 21, 0.05)
    with Context(n, bc, "fp64") as c, Batch([(n, bc, p)], "fp64") as b:
        for k, norm in enumerate((1.7, 3.5, 1.2, 1.0, 1.7, 1.0)):
            u = base.copy()
            u[:, 1:] *= norm
            c.upload(u)
            ref = c.wloop_sum(p)
            b.upload(0, u)
            before = launch_count()
            b.run()
            if k:
                assert launch_count() - before <= 2
            assert np.array_equal(b.result(0), ref)
