"""The similarity on row words: windows below, at and above the 16 and 32 lanes and
the 32-bit words it runs on, up to 64, square and not; lists equal the oracle's."""
import numpy as np
import pytest

from test_select_cpu import hex_array

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(2, 2), (7, 9), (16, 16), (15, 17), (32, 16), (31, 32), (33, 20), (40, 64), (64, 64)])
def test_lists_match_the_oracle(pfd, oracle, w, h):
    pitch = 23.2
    c, k = hex_array(14, 12, pitch)
    V = len(c)
    rs = np.random.RandomState(w * 100 + h)
    big = rs.randint(0, 256, (h + 24, w + 24)).astype(np.float64)
    for _ in range(3):
        big = (big + np.roll(big, 1, 0) + np.roll(big, 1, 1) + np.roll(big, (1, 1), (0, 1))) / 4
    big = (big - big.mean()) * 4 + 128
    imgs = np.stack([big[rs.randint(0, 24):, rs.randint(0, 24):][:h, :w] for _ in range(V)])
    imgs = np.clip(imgs + rs.randint(-40, 41, imgs.shape), 0, 255).astype(np.uint8)
    with pfd.Context(0) as ctx:
        ids, cnt = ctx.select_neighbors(c, k, 14, 12, pitch, imgs)
    oids, ocnt, _ = oracle.select_neighbors(c, k, 14, 12, pitch, images=imgs)
    assert np.array_equal(cnt, np.minimum(ocnt, 128)) and np.array_equal(ids, oids)
