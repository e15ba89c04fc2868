"""The lines of a chunk (up to 4 GiB) belong to a measurement, not to a context: many
contexts share them, and they are given back."""
import threading

import numpy as np
import pytest

from wloop_b200 import APE, Context, WloopParms
from wloop_b200._native import lib

N = (32, 16, 16, 16)
P = WloopParms(msl=4, nss=[0, 1, 1, 1], mwlt=8, mwlr=8, op_smear=APE, alpha_ape=0.5, proj_iter=4)
LINES = {"mixed": 2038431744, "fp64": 3623878656}  # of one measurement (the plans' bytes)


def held(fields):
    """What a context keeps beside the lines: U, the smearing scratch (HYP's 24
    directions, APE's 6), the levels (3 each), first lines and recursion links (3
    each, 40 slices for 32), g and H^-1, the upload's staging; in directions."""
    return (4 + 24 + 6 + 3 * P.msl + 2 * 3 * P.msl * 40 / 32 + 4 * 2 * 40 / 32 + 8) * fields


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_contexts_share_the_lines(precision):
    import torch
    with Context((4, 4, 4, 4), 3) as small:
        small.free_scratch()
        free = torch.cuda.mem_get_info(0)[0]
        contexts = [Context(N, 3, precision) for _ in range(6)]
        try:
            out = []
            for c in contexts:
                c.generate(3, 0.2)
                out.append(c.measure(P))
                assert c.contract_form == 11
            used = free - torch.cuda.mem_get_info(0)[0]
            direction = 131072 * 18 * (4 if precision == "mixed" else 8)
            assert used <= 6 * held(direction) + LINES[precision] + (512 << 20)
            assert all(np.array_equal(x, out[0]) for x in out)
            # two at a time
            again = {}

            def work(k):
                for _ in range(3):
                    contexts[k].generate(3, 0.2)
                    again[k] = contexts[k].measure(P)

            threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
            assert all(np.array_equal(again[k], out[0]) for k in range(2))
            # given back through any context, without a word from the ones that used them
            idle = lib.wlg_batch_pool_idle_bytes(0)
            assert idle >= LINES[precision]
            free = torch.cuda.mem_get_info(0)[0]
            small.free_scratch()
            assert lib.wlg_batch_pool_idle_bytes(0) <= idle - LINES[precision]
            assert torch.cuda.mem_get_info(0)[0] >= free + LINES[precision]
            contexts[0].generate(3, 0.2)
            assert np.array_equal(contexts[0].measure(P), out[0])
        finally:
            for c in contexts:
                c.close()
    # and with the last context
    assert lib.wlg_batch_pool_idle_bytes(0) <= idle - LINES[precision]


@pytest.mark.gpu
def test_idle_lines_are_bounded():
    """Three contexts that measure at once with 3.6 GB each leave at most 9 GiB."""
    with Context((4, 4, 4, 4), 3) as small:
        small.free_scratch()
        before = lib.wlg_batch_pool_idle_bytes(0)
        contexts = [Context(N, 3, "fp64") for _ in range(3)]
        try:
            barrier = threading.Barrier(3)

            def work(c):
                c.generate(3, 0.2)
                barrier.wait()
                for _ in range(4):
                    c.measure(P)

            threads = [threading.Thread(target=work, args=(c,)) for c in contexts]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
            assert 0 < lib.wlg_batch_pool_idle_bytes(0) - before <= 9 << 30
        finally:
            for c in contexts:
                c.close()
