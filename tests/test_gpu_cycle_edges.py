"""The cycle check at the edges of its integer window sums and ordered tile sums:
windows of 2 to 32 (mirrored borders reach over the window), pixel counts that leave
a remainder in a warp, one and 32 views per pixel, none, infinite and invalid
disparities.  Maps, mask and statistics equal the CPU oracle's."""
import numpy as np
import pytest

from test_gpu_filter_resolve import BASE, _frame, _state

pytestmark = pytest.mark.gpu

CASES = [
    (2, 2, 1, {}), (3, 5, 4, {}), (5, 3, 6, dict(use_and=False)), (16, 16, 12, {}), (17, 15, 8, dict(max_triplet=32)),
    (15, 17, 32, dict(pixel_gate_enabled=True, gate_min_good_neighbors=1)), (20, 21, 9, dict(max_triplet=0)),
    (31, 9, 7, dict(clamp_geo=False, clamp_photo=False, max_triplet=1)), (32, 32, 6, dict(sobel_thresh=0.0, var_thresh=0.0)),
    (16, 16, 6, dict(pixel_gate_enabled=True, gate_use_clamped=True, gate_min_good_neighbors=0)),
]


@pytest.mark.parametrize("W,H,K,kw", CASES)
def test_cycle_check_equals_the_oracle(pfd, oracle, W, H, K, kw):
    rs = np.random.RandomState(W * 90 + H * 5 + K)
    cen, keys, gray, ids, cnt = _frame(rs, 9, 6, W, H, K)
    V = len(cen)
    cfg = pfd.CycleCfg(**kw)
    orc = oracle.Oracle(gray, cen, ids, cnt)
    st = _state(rs, V, W, H, K)
    FW, FH = int(cen[:, 0].max() + W + 40), int(cen[:, 1].max() + H + 40)
    with pfd.Context(0) as ctx:
        fid = ctx.frame_create(FW, FH, cen, keys, W, H, ids, cnt)
        ctx.frame_set_micro_images(fid, gray)
        ctx.state_upload(fid, st["plane"], st["cost"], st["disp"], st["sel"])
        stats, geo, pho, tm = ctx.cycle_check(fid, cfg, BASE)
        ctx.frame_free(fid)
    o_stats, o_geo, o_pho, o_tm = oracle.cycle_check(orc, cfg, BASE, st)
    assert np.array_equal(tm, o_tm)
    assert np.array_equal(geo, o_geo, equal_nan=True) and np.array_equal(pho, o_pho, equal_nan=True)
    for k, v in o_stats.items():
        assert stats[k] == v or (np.isnan(stats[k]) and np.isnan(v)), f"{k}: {stats[k]} != {v}"
