"""The FP64 projection's rounding, against extended precision: no more than that of
the iteration on matrices in FP64, also where a link is far from SU(3)."""
import numpy as np
import pytest

from wloop_b200 import Context


def project(u, steps, real):
    """The iteration of projection.c:120-154 in the arithmetic of `real`."""
    u = u.astype(np.result_type(real, np.complex64))
    one = np.eye(3, dtype=real)
    third = real(1) / real(3)
    u = u / np.sqrt((np.abs(u) ** 2).sum((-1, -2), keepdims=True) * third)
    for _ in range(steps):
        k = np.einsum("...ki,...kj->...ij", u.conj(), u)
        y = np.einsum("...ik,...kj->...ij", u, real(1.5) * one - real(0.5) * k)
        det = (y[..., 0, :] * np.cross(y[..., 1, :], y[..., 2, :])).sum(-1)
        u = y * (1 - 1j * det.imag * third)[..., None, None]
    return u


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [3, 4, 5, 7])
@pytest.mark.parametrize("noise", [0.2, 0.4, 1.5])
def test_error(steps, noise):
    """Spatial links are unit matrices with Gaussian noise; a sweep with alpha = 0
    projects them as they are."""
    n = (8, 8, 8, 8)
    rng = np.random.default_rng(int(10 * noise) + 100 * steps)
    u = np.broadcast_to(np.eye(3), (4096, 4, 3, 3)).astype(np.complex128)
    u[:, 1:] += noise * (rng.standard_normal((4096, 3, 3, 3)) +
                         1j * rng.standard_normal((4096, 3, 3, 3)))
    with Context(n, 3, "fp64") as c:
        c.upload(u)
        c.ape_spatial_links(0.0, proj=1, piter=steps)
        got = c.download()[:, 1:]
    exact = project(u[:, 1:], steps, np.longdouble)
    plain = project(u[:, 1:], steps, np.float64)
    error, bound = (np.linalg.norm((x - exact).astype(np.complex128)) for x in (got, plain))
    # two FP64 evaluations of one formula: their errors differ by their rounding's
    # luck in the few worst links, which carry most of the norm
    assert error <= 1.5 * bound, error / bound
