"""Half-sweeps whose micro-images are split between CTAs (pm_slots.cu): view
counts around one and two items per CTA, the smallest frame, an odd number of
pixels, parts near the number of slots, and frames that share a launch.  Every
state field equals the CPU oracle's bit for bit."""
import numpy as np
import pytest

from test_gpu_slots import _grid, _same

pytestmark = pytest.mark.gpu

CTAS = 2 * 148                                           # of the default launch shape


def _check(got, st, what):
    for name, g in zip(("plane", "cost", "disp", "sel"), got):
        assert _same(g, st[name]), f"{what}: {name} differs at {np.count_nonzero(np.asarray(g) != st[name])}"


def _frame(ctx, rs, cols, rows, side, K):
    base = side * 1.45
    cen, keys, gray, ids, cnt = _grid(rs, cols, rows, side, side, K, base)
    fid = ctx.frame_create(int(cen[:, 0].max() + side + 40), int(cen[:, 1].max() + side + 40), cen, keys, side, side, ids, cnt)
    ctx.frame_set_micro_images(fid, gray)
    return fid, (gray, cen, ids, cnt), base


@pytest.mark.parametrize("cols,rows,side", [(2, 1, 19), (2, 2, 11), (2 * CTAS - 1, 1, 12), (2 * CTAS, 1, 12),
                                            (CTAS - 1, 1, 12), (37, 8, 13)])
def test_split_views_match_the_oracle(pfd, oracle, cols, rows, side):
    rs = np.random.RandomState(cols)
    with pfd.Context(0) as ctx:
        fid, args, base = _frame(ctx, rs, cols, rows, side, 3 if cols * rows > 3 else 1)
        P = pfd.PmParams(base=base, patch_size=7, max_iterations=1, top_k=1)
        orc = oracle.Oracle(*args)
        ctx.pm_init(fid, P, 3)
        st = orc.init(P, 3)
        for ph in (0, 1):
            ctx.pm_sweep(fid, P, 3, 0, ph)
            st = orc.sweep(P, 3, 0, ph, st)
            _check(ctx.download(fid), st, f"phase {ph}")
        ctx.frame_free(fid)


def test_frames_of_one_launch_match_the_oracle(pfd, oracle):
    rs = np.random.RandomState(5)
    with pfd.Context(0) as ctx:
        made = [_frame(ctx, rs, c, r, side, 3) for c, r, side in ((2, 2, 19), (20, 6, 12), (5, 4, 15))]
        Ps = [pfd.PmParams(base=m[2], patch_size=7, max_iterations=1, top_k=1) for m in made]
        ctx.patchmatch_batch([m[0] for m in made], Ps, [7, 8, 9])
        for (fid, args, _), P, seed in zip(made, Ps, (7, 8, 9)):
            orc = oracle.Oracle(*args)
            st = orc.init(P, seed)
            for ph in (0, 1):
                st = orc.sweep(P, seed, 0, ph, st)
            _check(ctx.download(fid), st, f"frame of seed {seed}")
            ctx.frame_free(fid)
