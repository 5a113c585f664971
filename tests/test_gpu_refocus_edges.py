"""The focal-stack render at the edges of its tiles and of its division: outputs of
one pixel, of one less and one more than a warp's and a CTA's pixels, the smallest
and largest windows, non-square ones, virtual depths far below and above the
scene's.  Every value equals the CPU oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mw,mh,out", [(2, 2, (1, 1)), (3, 5, (31, 7)), (16, 16, (33, 9)), (17, 15, (63, 15)),
                                       (32, 32, (65, 17)), (21, 20, (128, 33)), (5, 31, (97, 16))])
def test_refocus_edges(pfd, oracle, mw, mh, out):
    rs = np.random.RandomState(mw * 40 + mh)
    W, H, base = 240, 200, 21.0
    gx, gy = np.meshgrid(np.arange(8), np.arange(6))
    keys = np.stack([gx.ravel(), gy.ravel()], 1).astype(np.int32)
    cen = (keys * base + 34 + rs.uniform(-0.5, 0.5, (48, 2))).astype(np.float32)
    gray = rs.randint(0, 256, (48, mh, mw)).astype(np.uint8)
    raw = rs.randint(0, 256, (H, W)).astype(np.uint8)
    ids, cnt = np.full((48, 1), -1, np.int32), np.zeros(48, np.int32)
    vds = [1e-3, 0.4, 1.0, 1.7, 3.0, 7.77, 12.0, 40.0]
    orc = oracle.Oracle(gray, cen, ids, cnt)
    ref = oracle.refocus(orc, W, H, vds, out[0], out[1])
    with pfd.Context(0) as ctx:
        fid = ctx.frame_upload(raw, cen, keys, mw, mh, ids, cnt)
        ctx.frame_set_micro_images(fid, gray)
        got = ctx.refocus(fid, vds, out[0], out[1])
        ctx.frame_free(fid)
    bad = np.nonzero(got != ref)
    assert bad[0].size == 0, f"{bad[0].size} pixels differ, first {list(zip(*[b[:3] for b in bad]))}"
    if min(out) > 8:
        assert np.mean(ref > 0) > 0.2
