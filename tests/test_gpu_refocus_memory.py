"""The focal stack's packed micro-images take no device memory of their own: they lie
in the frame's idle state buffer.  A call of a size that the frame has rendered
before allocates nothing, and half-sweeps go on after it as if it had not been."""
import numpy as np
import pytest

from test_gpu_fuse_bands import _Pool
from test_gpu_slots import _grid, _same

pytestmark = pytest.mark.gpu


def test_a_stack_needs_no_memory_beside_the_frame(pfd, oracle):
    rs = np.random.RandomState(2)
    side, base = 16, 24.0
    cen, keys, _, ids, cnt = _grid(rs, 12, 9, side, side, 6, base)
    W, H = int(cen[:, 0].max() + side + 40), int(cen[:, 1].max() + side + 40)
    raw = rs.randint(0, 256, (H, W)).astype(np.uint8)
    P = pfd.PmParams(base=base, patch_size=7, max_iterations=1, top_k=3)
    vd = np.array([3.0, 7.5], np.float32)
    pool = _Pool()
    with pfd.Context(0) as ctx:
        fid = ctx.frame_upload(raw, cen, keys, side, side, ids, cnt)
        first = ctx.refocus(fid, vd, 150, 110)               # before any state
        gray = np.stack([raw[y:y + side, x:x + side] for x, y in oracle.window_origins(cen, side, side)])
        orc = oracle.Oracle(gray, cen, ids, cnt)
        ctx.pm_init(fid, P, 5)
        st = orc.init(P, 5)
        for ph in (0, 1):
            ctx.sync()
            pool.start()
            assert np.array_equal(ctx.refocus(fid, vd, 150, 110), first)
            ctx.sync()
            assert pool.peak() == 0
            ctx.pm_sweep(fid, P, 5, 0, ph)
            st = orc.sweep(P, 5, 0, ph, st)
            for name, g in zip(("plane", "cost", "disp", "sel"), ctx.download(fid)):
                assert _same(g, st[name]), f"phase {ph}: {name}"
        ctx.frame_free(fid)
