"""The line from which a frame of a batch runs its own launches: four micro-images
per CTA of the sweep's grid.  The launches of the call tell which side ran, and
every frame's state equals the CPU oracle's bit for bit on both."""
import numpy as np
import pytest
import torch

from test_gpu_slot_parts import _check, _frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", [-1, 0])
def test_frames_on_both_sides_of_the_line(pfd, oracle, over):
    ctas = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    rs = np.random.RandomState(3)
    with pfd.Context(0) as ctx:
        made = [_frame(ctx, rs, c, r, 10, 3) for c, r in ((4 * ctas + over, 1), (20, 6), (5, 4))]
        Ps = [pfd.PmParams(base=m[2], patch_size=5, max_iterations=1, top_k=1) for m in made]
        before = ctx.launch_count()
        ctx.patchmatch_batch([m[0] for m in made], Ps, [7, 8, 9])
        # three initialisations; two half-sweeps of all frames, or two of the first and
        # two of the others
        assert ctx.launch_count() - before == (5 if over else 7)
        for (fid, args, _), P, seed in zip(made, Ps, (7, 8, 9)):
            orc = oracle.Oracle(*args)
            st = orc.init(P, seed)
            for ph in (0, 1):
                st = orc.sweep(P, seed, 0, ph, st)
            _check(ctx.download(fid), st, f"frame of seed {seed}")
            ctx.frame_free(fid)
