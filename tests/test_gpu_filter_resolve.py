"""The filter's three-launch form (pairs, masks to a fixed point, application) at
windows, neighbour counts and configurations where its packed tests and masks can
go wrong: the smallest and largest windows, mask words with a remainder, one and 32
views per pixel, none at all, spike thresholds around and below zero, long chains
of rejections, and a disparity threshold below -1, which runs as a wavefront.
Reasons, counters and the filtered state equal the CPU oracle's exactly."""
import numpy as np
import pytest

from scenes import value_texture

pytestmark = pytest.mark.gpu

BASE = 20.0


def _frame(rs, cols, rows, W, H, K):
    V = cols * rows
    gx, gy = np.meshgrid(np.arange(cols), np.arange(rows))
    keys = np.stack([gx.ravel(), gy.ravel()], 1).astype(np.int32)          # map order: row, then column
    cen = (keys * BASE + 40 + rs.uniform(-0.5, 0.5, (V, 2))).astype(np.float32)
    T = value_texture(H + 2 * rows + 8, W + 2 * cols + 8, int(rs.randint(1 << 20)), cell=4)
    gray = np.stack([T[y:y + H, x:x + W] for x, y in keys]).astype(np.uint8)
    ids = np.full((V, K), -1, np.int32)
    cnt = np.zeros(V, np.int32)
    for v in range(V):
        others = np.array([u for u in range(V) if u != v])
        near = others[np.argsort(np.hypot(*(cen[others] - cen[v]).T), kind="stable")][:K]
        ids[v, :len(near)] = near
        cnt[v] = len(near)
        if len(near) > 3 and v % 4 == 0:
            ids[v, 2] = -1
    cnt[V - 1] = 0
    return cen, keys, gray, ids, cnt


def _state(rs, V, W, H, K):
    n = V * W * H
    d = 1.0 + 0.2 * rs.randn(n)
    k = rs.permutation(n)
    d[k[:n // 10]] = rs.uniform(-2, 6, n // 10)
    d[k[n // 10:n // 10 + 3]] = (np.nan, np.inf, -1.0)
    plane = np.zeros((n, 4), np.float32)
    plane[:, 2] = 1
    plane[:, 3] = d
    cost = np.abs(rs.randn(n)).astype(np.float32) * 0.8
    cost[k[:4]] = (np.nan, np.inf, -0.5, 1.8)
    sel = rs.randint(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    sel[rs.rand(n) < 0.05] = 0
    return dict(plane=plane, cost=cost, disp=rs.rand(n, 4).astype(np.float32), sel=sel)


CASES = [
    (2, 2, 1, {}), (5, 3, 6, {}), (16, 16, 12, {}), (16, 16, 12, dict(min_good_neighbors=3, max_photo_err_u=0.3)),
    (17, 15, 8, dict(max_triplet=32, use_selected_views_only=False)), (15, 17, 32, dict(max_triplet=32)),
    (16, 16, 6, dict(max_triplet=0)), (16, 16, 6, dict(max_triplet=1, min_good_neighbors=1, spike_abs_diff=0.0)),
    (20, 20, 9, dict(spike_abs_diff=-1.0, spike_min_neighbors=1)), (32, 32, 6, dict(enable_cost_filter=False)),
    (31, 9, 7, dict(min_valid_disp=-1.0, min_good_neighbors=0)), (16, 16, 6, dict(min_valid_disp=-2.0)),
    (16, 16, 6, dict(min_valid_disp=0.5, enable_cycle_geo_filter=False, clear_selected_views_when_invalid=False)),
]


@pytest.mark.parametrize("W,H,K,kw", CASES)
def test_filter_equals_the_oracle(pfd, oracle, W, H, K, kw):
    rs = np.random.RandomState(W * 100 + H * 7 + K + len(kw))
    cols, rows = (9, 6)
    cen, keys, gray, ids, cnt = _frame(rs, cols, rows, W, H, K)
    V = len(cen)
    cfg = pfd.FilterCfg(**kw)
    orc = oracle.Oracle(gray, cen, ids, cnt)
    FW, FH = int(cen[:, 0].max() + W + 40), int(cen[:, 1].max() + H + 40)
    with pfd.Context(0) as ctx:
        fid = ctx.frame_create(FW, FH, cen, keys, W, H, ids, cnt)
        ctx.frame_set_micro_images(fid, gray)
        for rep in range(2):                              # the work area is reused
            st = _state(rs, V, W, H, K)
            ctx.state_upload(fid, st["plane"], st["cost"], st["disp"], st["sel"])
            reason, stats = ctx.filter(fid, cfg, BASE)
            after = ctx.download(fid)
            o_reason, o_stats = oracle.filter_global(orc, cfg, BASE, st)
            assert np.array_equal(reason, o_reason), f"{np.count_nonzero(reason != o_reason)} reasons differ"
            assert list(stats.values()) == [int(x) for x in o_stats]
            for nm, g in zip(("plane", "cost", "disp", "sel"), after):
                o = st[nm]
                assert np.all((g == o) | (np.isnan(g) & np.isnan(o)) if g.dtype.kind == "f" else g == o), nm
        ctx.frame_free(fid)


def test_filter_without_room_for_its_work_area(pfd, oracle):
    """An HBM budget that holds the frame but not the work area: the wavefront runs,
    with the same result."""
    rs = np.random.RandomState(5)
    cen, keys, gray, ids, cnt = _frame(rs, 9, 6, 16, 16, 6)
    orc = oracle.Oracle(gray, cen, ids, cnt)
    with pfd.Context(0) as probe:
        f = probe.frame_create(300, 260, cen, keys, 16, 16, ids, cnt)
        frame = probe.bytes_in_use()
        probe.frame_free(f)
    n = len(cen) * 256
    with pfd.Context(0, hbm_budget=frame + n + 4096) as ctx:
        fid = ctx.frame_create(300, 260, cen, keys, 16, 16, ids, cnt)
        ctx.frame_set_micro_images(fid, gray)
        st = _state(rs, len(cen), 16, 16, 6)
        ctx.state_upload(fid, st["plane"], st["cost"], st["disp"], st["sel"])
        reason, stats = ctx.filter(fid, pfd.FilterCfg(), BASE)
        o_reason, o_stats = oracle.filter_global(orc, pfd.FilterCfg(), BASE, st)
        assert np.array_equal(reason, o_reason)
        assert list(stats.values()) == [int(x) for x in o_stats]
        ctx.frame_free(fid)
