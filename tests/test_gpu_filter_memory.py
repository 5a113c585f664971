"""The filter's work area takes no device memory of its own: it lies in the frame's
idle state buffer and stored cost vectors.  Budgets that held a frame before a
filter hold it after one, the three-launch form runs under any of them, and what
the idle buffers carried is made anew by whoever needs it."""
import numpy as np
import pytest

from test_gpu_filter_resolve import BASE, _frame, _state

pytestmark = pytest.mark.gpu

FIELDS = ("plane", "cost", "disp", "sel")


def _equal(got, st):
    for nm, g in zip(FIELDS, got):
        o = st[nm]
        assert np.all((g == o) | (np.isnan(g) & np.isnan(o)) if g.dtype.kind == "f" else g == o), nm


def _create(ctx, fr, W, H):
    cen, keys, gray, ids, cnt = fr
    fid = ctx.frame_create(int(cen[:, 0].max() + W + 40), int(cen[:, 1].max() + H + 40), cen, keys, W, H, ids, cnt)
    ctx.frame_set_micro_images(fid, gray)
    return fid


@pytest.mark.parametrize("W,H,K,grid", [(2, 2, 1, (2, 1)), (3, 2, 2, (3, 1)), (16, 16, 6, (9, 6)), (32, 31, 32, (9, 6))])
def test_filter_needs_no_memory_beside_the_frame(pfd, oracle, W, H, K, grid):
    rs = np.random.RandomState(W + K)
    fr = _frame(rs, *grid, W, H, K)
    V, cfg = len(fr[0]), pfd.FilterCfg(max_triplet=32, use_selected_views_only=False)
    orc = oracle.Oracle(fr[2], fr[0], fr[3], fr[4])
    with pfd.Context(0) as probe:
        f = _create(probe, fr, W, H)
        frame = probe.bytes_in_use()
        probe.frame_free(f)
    # the frame, the reasons (a byte per pixel) and the counters
    own = V * W * H + 64
    with pfd.Context(0, hbm_budget=frame + own) as ctx:
        for rep in range(2):
            fid = _create(ctx, fr, W, H)
            st = _state(rs, V, W, H, K) if V * W * H > 100 else _small_state(rs, V * W * H)
            ctx.state_upload(fid, st["plane"], st["cost"], st["disp"], st["sel"])
            before = ctx.launch_count()
            reason, stats = ctx.filter(fid, cfg, BASE)
            assert ctx.launch_count() - before == 3
            o_reason, o_stats = oracle.filter_global(orc, cfg, BASE, st)
            assert np.array_equal(reason, o_reason)
            assert list(stats.values()) == [int(x) for x in o_stats]
            _equal(ctx.download(fid), st)
            assert ctx.bytes_in_use() == frame + own
            ctx.frame_free(fid)
            assert ctx.bytes_in_use() == 0


def _small_state(rs, n):
    plane = np.zeros((n, 4), np.float32)
    plane[:, 2] = 1
    plane[:, 3] = 1.0 + 0.2 * rs.randn(n)
    return dict(plane=plane, cost=np.abs(rs.randn(n)).astype(np.float32), disp=rs.rand(n, 4).astype(np.float32),
                sel=rs.randint(0, 4, n).astype(np.uint32))


def test_a_second_frame_fits_after_a_filter(pfd):
    rs = np.random.RandomState(3)
    fr = _frame(rs, 9, 6, 16, 16, 6)
    n = len(fr[0]) * 256
    with pfd.Context(0) as probe:
        _create(probe, fr, 16, 16)
        frame = probe.bytes_in_use()
    with pfd.Context(0, hbm_budget=2 * frame + n + 64) as ctx:
        a = _create(ctx, fr, 16, 16)
        st = _state(rs, len(fr[0]), 16, 16, 6)
        ctx.state_upload(a, st["plane"], st["cost"], st["disp"], st["sel"])
        ctx.filter(a, pfd.FilterCfg(), BASE)
        b = _create(ctx, fr, 16, 16)
        assert ctx.bytes_in_use() == 2 * frame + n + 64
        ctx.frame_free(a)
        ctx.frame_free(b)


def test_the_route_of_each_threshold(pfd):
    """-1 and above: three launches.  Below, and NaN: a rejected pixel's disparity is a
    usable one, and the wavefront runs, one launch per step of the 9x6 grid."""
    rs = np.random.RandomState(4)
    fr = _frame(rs, 9, 6, 16, 16, 6)
    with pfd.Context(0) as ctx:
        fid = _create(ctx, fr, 16, 16)
        for low, three in ((-1.0, True), (0.0, True), (-1.0001, False), (float("nan"), False)):
            st = _state(rs, len(fr[0]), 16, 16, 6)
            ctx.state_upload(fid, st["plane"], st["cost"], st["disp"], st["sel"])
            before = ctx.launch_count()
            ctx.filter(fid, pfd.FilterCfg(min_valid_disp=low), BASE)
            assert (ctx.launch_count() - before == 3) == three
            assert three or ctx.launch_count() - before >= 9


def test_sweeps_go_on_after_a_filter(pfd, oracle):
    """The stored cost vectors and the other state buffer are the filter's work area:
    the half-sweeps after it start from neither."""
    rs = np.random.RandomState(6)
    cen, keys, gray, ids, cnt = fr = _frame(rs, 9, 6, 16, 16, 6)
    P = pfd.PmParams(base=BASE, patch_size=7, max_iterations=1, top_k=3)
    orc = oracle.Oracle(gray, cen, ids, cnt)
    with pfd.Context(0) as ctx:
        fid = _create(ctx, fr, 16, 16)
        ctx.pm_init(fid, P, 5)
        st = orc.init(P, 5)
        for it in range(2):
            for ph in (0, 1):
                ctx.pm_sweep(fid, P, 5, it, ph)
                st = orc.sweep(P, 5, it, ph, st)
            ctx.filter(fid, pfd.FilterCfg(min_good_neighbors=1), BASE)
            oracle.filter_global(orc, pfd.FilterCfg(min_good_neighbors=1), BASE, st)
            _equal(ctx.download(fid), st)


@pytest.mark.parametrize("far,ok", [((0, 200_000_000), False), ((90_000, 1000), True), ((100_000, 100_000), True),
                                    ((-2**31, 2**31 - 1), True)])
def test_tile_keys_too_sparse_for_a_schedule_are_refused(pfd, far, ok):
    """As by the wavefront, whichever form runs: keys whose schedule would have more
    than 10^8 steps.  The last two pairs' bound says so, their schedules do not: with
    column weight 1 the far key is in step 200000, or in step -1."""
    rs = np.random.RandomState(7)
    cen, keys, gray, ids, cnt = _frame(rs, 3, 1, 16, 16, 2)
    keys = np.array([[0, 0], [1, 1], far], np.int32)
    ids[:] = -1
    ids[0, 0], ids[1, 0], cnt[:] = 1, 0, (1, 1, 0)
    with pfd.Context(0) as ctx:
        fid = _create(ctx, (cen, keys, gray, ids, cnt), 16, 16)
        st = _state(rs, 3, 16, 16, 2)
        ctx.state_upload(fid, st["plane"], st["cost"], st["disp"], st["sel"])
        for low in (0.0, -2.0):
            if ok and low < -1 and far[0] < 100_000:
                continue                                  # the wavefront of 9 10^7 steps is left out
            if ok:
                ctx.filter(fid, pfd.FilterCfg(min_valid_disp=low), BASE)
            else:
                with pytest.raises(pfd.PfdError, match="too sparse"):
                    ctx.filter(fid, pfd.FilterCfg(min_valid_disp=low), BASE)
