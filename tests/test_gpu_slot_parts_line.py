"""The line up to which half-sweeps split their micro-images between CTAs: six items
per CTA.  View counts on both sides of it, of two parts' and of four parts' line,
and windows whose parts would hold fewer pixels than slots; a launch over several
frames whose views together lie on either side.  Every state field equals the CPU
oracle's bit for bit."""
import numpy as np
import pytest

from test_gpu_slot_parts import CTAS, _check, _frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("views,side", [(6 * CTAS, 12), (6 * CTAS - 1, 12), (3 * CTAS, 16), (3 * CTAS - 1, 16), (6 * CTAS - 1, 7)])
def test_views_on_both_sides_match_the_oracle(pfd, oracle, views, side):
    rs = np.random.RandomState(views)
    with pfd.Context(0) as ctx:
        fid, args, base = _frame(ctx, rs, views, 1, side, 3)
        P = pfd.PmParams(base=base, patch_size=5, max_iterations=1, top_k=1)
        orc = oracle.Oracle(*args)
        ctx.pm_init(fid, P, 3)
        st = orc.init(P, 3)
        for ph in (0, 1):
            ctx.pm_sweep(fid, P, 3, 0, ph)
            st = orc.sweep(P, 3, 0, ph, st)
            _check(ctx.download(fid), st, f"phase {ph}")
        ctx.frame_free(fid)


@pytest.mark.parametrize("last", [6 * CTAS - 1 - 2 * 880, 6 * CTAS - 2 * 880])
def test_frames_of_one_launch_on_both_sides(pfd, oracle, last):
    rs = np.random.RandomState(last)
    with pfd.Context(0) as ctx:
        made = [_frame(ctx, rs, c, 1, 12, 1) for c in (880, 880, last)]
        Ps = [pfd.PmParams(base=m[2], patch_size=5, max_iterations=1, top_k=1) for m in made]
        ctx.patchmatch_batch([m[0] for m in made], Ps, [7, 8, 9])
        for (fid, args, _), P, seed in zip(made, Ps, (7, 8, 9)):
            orc = oracle.Oracle(*args)
            st = orc.init(P, seed)
            for ph in (0, 1):
                st = orc.sweep(P, seed, 0, ph, st)
            _check(ctx.download(fid), st, f"frame of seed {seed}")
            ctx.frame_free(fid)
