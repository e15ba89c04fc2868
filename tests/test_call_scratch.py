"""Smearing calls that give their scratch back (keep = 0): small ones take it
from a bounded pool of the device, larger ones from cudaMalloc."""
import threading

import numpy as np
import pytest

from wloop_b200 import Context, generate_links
from wloop_b200._native import lib

LIMIT = 1 << 30


def smear(c, u, keep):
    c.upload(u)
    c.hyp_links(0.75, 0.6, 0.3, keep=keep)
    c.ape_links(0.1, nsweeps=3, keep=keep)
    c.hyp_spatial_links(0.75, 0.6, nsweeps=2, keep=keep)
    return c.download()


@pytest.mark.gpu
@pytest.mark.parametrize("n,precision", [((4, 4, 4, 4), "mixed"), ((8, 5, 6, 7), "fp64"),
                                         ((40, 20, 20, 24), "fp64")])
def test_same_bits_with_and_without_keep(n, precision):
    """The last lattice's HYP scratch (3456 bytes a site) is above the pool's limit,
    its APE and spatial-HYP scratch below."""
    u = generate_links(n, 3, 5, 0.3)
    with Context(n, 3, precision) as c:
        first = smear(c, u, 0)
        assert np.array_equal(smear(c, u, 0), first)
        assert 0 < lib.wlg_batch_pool_idle_bytes(0)
        assert np.array_equal(smear(c, u, 1), first)
        assert np.array_equal(smear(c, u, 0), first)  # takes and gives back what was kept


@pytest.mark.gpu
def test_pool_is_bounded_and_given_back():
    import torch
    n = (32, 16, 16, 20)  # 566 MB of HYP scratch
    u = generate_links(n, 3, 5, 0.3)
    with Context(n, 3, "fp64") as a, Context(n, 3, "fp64") as b, Context((4, 4, 4, 4), 3) as c:
        c.free_scratch()
        before = lib.wlg_batch_pool_idle_bytes(0)
        ref = smear(a, u, 1)
        a.free_scratch()
        out = {}

        def work(k, ctx):
            out[k] = [smear(ctx, u, 0) for _ in range(3)]

        threads = [threading.Thread(target=work, args=(k, x)) for k, x in enumerate((a, b))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert all(np.array_equal(x, ref) for k in out for x in out[k])
        a.sync()
        idle = lib.wlg_batch_pool_idle_bytes(0) - before
        assert 0 < idle <= LIMIT + (64 << 20)
        free = torch.cuda.mem_get_info(0)[0]
        a.free_scratch()
        b.free_scratch()
        assert lib.wlg_batch_pool_idle_bytes(0) <= before
        assert torch.cuda.mem_get_info(0)[0] >= free + idle


@pytest.mark.gpu
@pytest.mark.parametrize("call", [lambda c: c.hyp_links(0.75, 0.6, 0.3),
                                  lambda c: c.ape_links(0.1, nsweeps=3),
                                  lambda c: c.hyp_spatial_links(0.75, 0.6)],
                         ids=["hyp", "ape", "hyp_spatial"])
def test_scratch_comes_from_the_pool_and_returns_at_once(call):
    """The pool of the calls alone (other pools' idle memory stays what it was), and
    another context gives its memory back right after the call."""
    import torch
    n = (32, 16, 16, 20)
    with Context(n, 3, "fp64") as c, Context((4, 4, 4, 4), 3) as other:
        c.generate(3, 0.3)
        c.sync()
        other.free_scratch()
        before = lib.wlg_batch_pool_idle_bytes(0)
        free = torch.cuda.mem_get_info(0)[0]
        call(c)
        idle = lib.wlg_batch_pool_idle_bytes(0) - before
        assert 4 * 163840 * 144 <= idle <= LIMIT  # at least four directions
        other.free_scratch()
        assert lib.wlg_batch_pool_idle_bytes(0) <= before
        assert torch.cuda.mem_get_info(0)[0] >= free - (2 << 20)
