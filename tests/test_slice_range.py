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


def digit_sum(a, b):
    """sum a b from the 7 digits of each, the classes i + j < 7 (gslice.cu)."""
    planes = []
    for x in (a, b):
        v = np.rint(x * 2.0 ** 54).astype(np.int64)  # exact: |x| < 2, 54 bits
        q = []
        for _ in range(6):
            d = ((v + 128) & 255) - 128
            q.append(d)
            v = (v - d) >> 8
        planes.append([v] + q[::-1])
    total = sum(int(planes[0][i] @ planes[1][m - i]) << (8 * (6 - m))
                for m in range(7) for i in range(m + 1))
    return np.longdouble(total) * np.longdouble(2) ** -60


@pytest.mark.parametrize("run,runs", [(96, 72), (576, 48), (2304, 2)])
def test_digits_are_no_further_off_than_fmas(run, runs):
    """Lines as small against the digits' range as the rule of slice_scales admits
    (norm^2 = 1 / (0.08 sqrt(run + runs)), or 1 / 1.1), against sums of the same
    products in FP64 FMAs, in runs as the FMA kernel adds them."""
    rng = np.random.default_rng(run)
    rms = np.sqrt(1.0 / max(1.1, 0.08 * np.sqrt(run + runs)) / 6.0)
    digits, fmas = [], []
    for _ in range(100):
        a, b = np.clip(rng.standard_normal((2, run * runs)) * rms, -1.98, 1.98)
        exact = a.astype(np.longdouble) * b
        digits.append(digit_sum(a, b) - exact.sum())
        acc = np.zeros(runs)
        for col in exact.reshape(runs, run).T:
            acc = (acc + col).astype(np.float64)
        total = 0.0
        for x in acc:
            total += x
        fmas.append(total - exact.sum())
    assert np.linalg.norm(digits) <= np.linalg.norm(fmas)


def loops(u, n, bc, p, **tuning):
    """wloop_sum in FP64 and its contraction launches."""
    with Context(n, bc, "fp64") as c:
        if tuning:
            c.set_gram_tuning(**tuning)
        c.upload(u)
        c.set_profiling(True)
        got = c.wloop_sum(p)
        assert c.contract_form == 11
        return got, c.kernel_time("contract")[1]


@pytest.mark.gpu
@pytest.mark.parametrize("bc", [0, 3])
@pytest.mark.parametrize("norm", [0.25, 1.4])
def test_scales_follow_level_and_extent(norm, bc):
    """Lines of links of one norm have its R-th power: every extent and level keeps
    the bits its own size needs."""
    n, R = (32, 8, 8, 16), 4
    p = WloopParms(msl=2, nss=[0, 1], mwlt=4, mwlr=R, op_smear=APE, alpha_ape=0.0, proj_iter=4)
    u = generate_links(n, bc, 23, 0.2)
    u[:, 1:] *= norm  # level 0; level 1 is the field projected, in SU(3)
    got, launches = loops(u, n, bc, p)
    fma, _ = loops(u, n, bc, p, stages=2)
    assert launches == 1
    # the FMA kernel's plan adds 288 runs of 384 columns: against W of the largest size
    # its rounding is about (sqrt(288 / 3) + sqrt(384 / 288 / 3)) 2^-54; 4 times that
    got, fma = (w.reshape(n[0], R, 4, 2, 2) for w in (got, fma))
    for r in range(R):  # [level 2][level 1], lines of r + 1 links
        size = np.array([[norm ** 2, norm], [norm, 1.0]]) ** (r + 1)
        assert (np.abs(got[:, r] - fma[:, r]) <= 21.0 * 2.0 ** -53 * size).all(), r


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["link", "slice"])
def test_lines_far_apart(where):
    """One link far larger than the rest, or one slice of far smaller links: the
    digits' unit would be too coarse for the others, and the FMA kernel measures."""
    n, bc = (32, 8, 8, 16), 3
    p = WloopParms(msl=1, nss=[0], mwlt=4, mwlr=2, op_smear=APE, alpha_ape=0.5, proj_iter=4)
    u = generate_links(n, bc, 22, 0.2)
    sites = u.reshape(n[0], -1, 4, 3, 3)
    if where == "link":
        sites[5, 77, 2] *= 7.0
    else:
        sites[5, :, 1:] *= 0.1
    got, launches = loops(u, n, bc, p)
    fma, _ = loops(u, n, bc, p, stages=2)
    assert launches == p.mwlr and np.array_equal(got, fma)
