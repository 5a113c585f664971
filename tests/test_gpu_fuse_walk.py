"""The fusion's walk on bits (pm_fuse_resolve_kernel) where its masks and list
words can go wrong: windows whose pixel count leaves a remainder in a mask word,
lists of 1 to 128 entries, lists that name a micro-image twice or name the
micro-image itself, micro-images that are no reference, one, three or no consistent
entries asked for, tolerances that let nearly everything through (long chains of
masks).  Points, maps and counts equal the CPU oracle's exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BASE = 20.0

CASES = [
    # m, cols, rows, max_list, options
    (2, 5, 4, 3, {}), (5, 6, 5, 6, dict(min_consistent=1)), (16, 9, 6, 1, dict(min_consistent=1)),
    (16, 9, 7, 12, {}), (16, 9, 7, 12, dict(max_reproj_px=6.0, max_rel_vd=1.0, min_consistent=1)),
    (17, 8, 6, 33, dict(min_consistent=3)), (15, 12, 11, 128, dict(max_reproj_px=3.0, max_rel_vd=0.5)),
    (32, 5, 4, 8, {}), (21, 6, 5, 24, dict(min_consistent=0)), (16, 9, 7, 12, dict(self_and_twice=True)),
]


@pytest.mark.parametrize("m,cols,rows,max_list,opt", CASES)
def test_walk_equals_the_oracle(pfd, oracle, m, cols, rows, max_list, opt):
    opt = dict(opt)
    odd = opt.pop("self_and_twice", False)
    rs = np.random.RandomState(m * 100 + max_list + len(opt))
    V = cols * rows
    gx, gy = np.meshgrid(np.arange(cols), np.arange(rows))
    keys = np.stack([gx.ravel(), gy.ravel()], 1).astype(np.int32)
    cen = (keys * BASE + 30 + rs.uniform(-0.5, 0.5, (V, 2))).astype(np.float32)
    gray = rs.randint(0, 256, (V, m, m)).astype(np.uint8)
    lists = np.full((V, max_list), -1, np.int32)
    counts = np.zeros(V, np.int32)
    for v in range(V):
        others = np.array([u for u in range(V) if u != v])
        near = others[np.argsort(np.hypot(*(cen[others] - cen[v]).T), kind="stable")][:max_list]
        lists[v, :len(near)] = near
        counts[v] = len(near)
        if odd:
            lists[v, 3] = lists[v, 0]
            lists[v, 5] = v
    lists[rs.rand(*lists.shape) < 0.04] = -1
    is_ref = (rs.rand(V) > 0.1).astype(np.uint8)
    n = V * m * m
    d = 2.0 + 0.03 * rs.randn(n)
    k = rs.permutation(n)[:max(12, n // 12)]
    d[k] = rs.uniform(-1, 6, len(k))
    d[k[:3]] = (np.nan, np.inf, 0.0)
    plane = np.concatenate([rs.randn(n, 3), d[:, None]], 1).astype(np.float32)
    nb_ids = np.full((V, 1), -1, np.int32)
    nb_cnt = np.zeros(V, np.int32)
    FW, FH = int(cen[:, 0].max() + 40), int(cen[:, 1].max() + 40)
    orc = oracle.Oracle(gray, cen, nb_ids, nb_cnt)
    want = oracle.fuse_virtual_depth(orc, plane, lists, counts, is_ref, FW, FH, BASE, **opt)
    with pfd.Context(0) as ctx:
        fid = ctx.frame_create(FW, FH, cen, keys, m, m, nb_ids, nb_cnt)
        ctx.frame_set_micro_images(fid, gray)
        ctx.state_upload(fid, plane, np.zeros(n, np.float32), np.zeros((n, 4), np.float32), np.zeros(n, np.uint32))
        for rep in range(2):
            vd, cf, aif, pts = ctx.fuse_virtual_depth(fid, lists, counts, is_ref, BASE, **opt)
            assert len(pts) == len(want[3])
            assert np.array_equal(pts, want[3], equal_nan=True)
            assert np.array_equal(vd, want[0], equal_nan=True)
            assert np.array_equal(cf, want[1]) and np.array_equal(aif, want[2])
        ctx.frame_free(fid)
    if m >= 15:
        assert len(want[3]) > 0, "nothing fused: the case proves little"
