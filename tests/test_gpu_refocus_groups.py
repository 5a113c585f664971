"""A focal stack for the host is rendered and copied in groups of slices
(pfd_refocus): the whole stack equals its slices rendered one at a time, bit for
bit, at one group, two, an uneven last one and the most, into pageable and pinned
memory, and again when a second call follows at once."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,side", [(1, 1024), (3, 1024), (5, 1024), (16, 1025), (7, 2048), (16, 64)])
@pytest.mark.parametrize("pinned", [False, True])
def test_grouped_stack_equals_its_slices(pfd, n, side, pinned):
    w = pfd.make_workload(420, 320, 23.0, 5, seed=3, max_nb=6)
    vds = np.linspace(2.5, 9.0, n).astype(np.float32)
    with pfd.Context(0) as ctx:
        fid = ctx.frame_upload(w.frame.raw, w.centers, w.tilekeys, w.mi, w.mi, w.nb_ids, w.nb_counts)
        want = np.concatenate([ctx.refocus(fid, vds[i:i + 1], side, side) for i in range(n)])
        outs = [torch.full((n, side, side), -7.0, pin_memory=pinned) for _ in range(2)]
        for o, order in zip(outs, (vds, vds[::-1].copy())):
            rc = ctx._L.pfd_refocus(ctx._h, fid, order.ctypes.data_as(ctypes.c_void_p), n, side, side,
                                    ctypes.c_void_p(o.data_ptr()))
            assert rc == 0
        ctx.frame_free(fid)
    assert np.array_equal(outs[0].numpy(), want)
    assert np.array_equal(outs[1].numpy(), want[::-1])
