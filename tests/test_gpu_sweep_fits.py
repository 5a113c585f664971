"""Half-sweeps of an uploaded state at windows with a blur channel whose quads
nearly fill the shared memory: on one side of the line the slot kernel runs, on
the other, where not even one slot fits, the warp-per-pixel kernel, with and
without allocation.  Every state field equals the CPU oracle's bit for bit."""
import numpy as np
import pytest

from test_gpu_slots import _grid, _same, _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,K,patch,mode", [
    (25, 25, 32, 9, ""), (28, 28, 26, 9, "shifted"), (30, 30, 22, 9, "acmm"), (32, 32, 19, 9, ""),
    (32, 32, 19, 3, "acmm shifted"), (32, 32, 18, 9, ""), (24, 25, 32, 15, "shifted")])
def test_sweep_of_a_window_near_the_limit(pfd, oracle, W, H, K, patch, mode):
    rs = np.random.RandomState(W * 100 + K)
    base = W * 1.45
    cen, keys, gray, ids, cnt = _grid(rs, 7, 5, W, H, K, base)
    V = len(cen)
    blur = rs.randint(0, 256, gray.shape).astype(np.uint8)
    P = pfd.PmParams(base=base, patch_size=patch, max_iterations=1, top_k=5)
    orc = oracle.Oracle(gray, cen, ids, cnt, blur=blur, shifted="shifted" in mode, acmm="acmm" in mode)
    with pfd.Context(0) as ctx:
        ctx.set_ncc_moments("shifted" in mode)
        ctx.set_matcher("acmm" in mode)
        ctx.set_sweep_shape(pfd.SHAPE_AUTOTUNE if patch == 3 else 0)
        fid = ctx.frame_create(int(cen[:, 0].max() + W + 40), int(cen[:, 1].max() + H + 40), cen, keys, W, H, ids, cnt, blur)
        ctx.frame_set_micro_images(fid, gray)
        st = _state(rs, V, W, H, K, base)
        ctx.state_upload(fid, st["plane"], st["cost"], st["disp"], st["sel"])
        # the second half-sweep of each phase uses the vectors that the first one stored
        for sweep, it, ph in ((ctx.pm_sweep, 0, 0), (ctx.pm_sweep_noalloc, 0, 1), (ctx.pm_sweep_noalloc, 1, 0), (ctx.pm_sweep, 1, 1)):
            sweep(fid, P, 18, it, ph)
            st = orc.sweep(P, 18, it, ph, st)
            for name, g in zip(("plane", "cost", "disp", "sel"), ctx.download(fid)):
                assert _same(g, st[name]), f"{it}.{ph}: {name} differs at {np.count_nonzero(np.asarray(g) != st[name])}"
        if patch == 3:
            assert ctx.tuned_sweep_shape(fid, P) == 0
        ctx.frame_free(fid)
