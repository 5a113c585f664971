"""The fusion of frames with long lists, walked in bands of micro-images where the
work area would be large: it stays below 256 MB, or what a budget has left, and
the walk over the bands equals the CPU oracle's over the whole frame, with masks
that reach across bands."""
import ctypes

import numpy as np
import pytest

from test_gpu_fuse_walk import BASE, test_walk_equals_the_oracle as walk

pytestmark = pytest.mark.gpu

# m, cols, rows, max_list, options: in a context whose budget leaves nothing beside the
# frame, two bands (of 4 MB) or more
CASES = [
    (2, 50, 40, 128, dict(min_consistent=1)), (16, 16, 12, 128, {}), (16, 9, 7, 100, dict(self_and_twice=True)),
    (16, 16, 12, 128, dict(max_reproj_px=6.0, max_rel_vd=1.0, min_consistent=1)), (32, 8, 8, 33, dict(max_reproj_px=3.0)),
]


class _Tight:
    """The package with contexts of the smallest budget that holds their one frame."""

    def __init__(self, pfd, budget):
        self.pfd, self.budget = pfd, budget

    def Context(self, device):
        return self.pfd.Context(device, hbm_budget=self.budget)


@pytest.mark.parametrize("m,cols,rows,max_list,opt", CASES)
def test_bands_equal_the_oracle(pfd, oracle, m, cols, rows, max_list, opt):
    W, H = int((cols - 1) * BASE + 80), int((rows - 1) * BASE + 80)
    walk(_Tight(pfd, pfd.frame_bytes(W, H, cols * rows, m, 1)), oracle, m, cols, rows, max_list, opt)


def test_bands_of_a_large_frame_equal_the_oracle(pfd, oracle):
    walk(pfd, oracle, 16, 60, 60, 128, {})               # 270 MB in one band


class _Pool:
    """Bytes of device 0's default stream-ordered memory pool that are in use, and their peak."""

    def __init__(self):
        self.lib = ctypes.CDLL("libcuda.so.1")
        self.pool = ctypes.c_void_p()
        assert self.lib.cuDeviceGetDefaultMemPool(ctypes.byref(self.pool), 0) == 0

    def _get(self, attr):
        v = ctypes.c_uint64()
        assert self.lib.cuMemPoolGetAttribute(self.pool, attr, ctypes.byref(v)) == 0
        return v.value

    def start(self):
        zero = ctypes.c_uint64(0)
        assert self.lib.cuMemPoolSetAttribute(self.pool, 8, ctypes.byref(zero)) == 0        # USED_MEM_HIGH
        self.before = self._get(7)                                                          # USED_MEM_CURRENT

    def peak(self):
        return self._get(8) - self.before


@pytest.mark.parametrize("cols,rows,max_list,budget,most", [
    (30, 24, 12, 0, 256), (30, 24, 128, 1, 4), (100, 80, 128, 0, 256)])
def test_the_work_area_is_bounded(pfd, cols, rows, max_list, budget, most):
    rs = np.random.RandomState(max_list)
    m = 16
    V, n = cols * rows, cols * rows * 256
    gx, gy = np.meshgrid(np.arange(cols), np.arange(rows))
    keys = np.stack([gx.ravel(), gy.ravel()], 1).astype(np.int32)
    cen = (keys * BASE + 30).astype(np.float32)
    lists = ((np.arange(V)[:, None] + np.arange(1, max_list + 1)[None]) % V).astype(np.int32)
    counts = np.full(V, max_list, np.int32)
    plane = np.concatenate([rs.randn(n, 3), 2.0 + 0.03 * rs.randn(n, 1)], 1).astype(np.float32)
    FW, FH = int(cen[:, 0].max() + 40), int(cen[:, 1].max() + 40)
    pool = _Pool()
    with pfd.Context(0, hbm_budget=budget * pfd.frame_bytes(FW, FH, V, m, 1)) as ctx:
        fid = ctx.frame_create(FW, FH, cen, keys, m, m, np.full((V, 1), -1, np.int32), np.zeros(V, np.int32))
        ctx.frame_set_micro_images(fid, rs.randint(0, 256, (V, m, m)).astype(np.uint8))
        ctx.state_upload(fid, plane, np.zeros(n, np.float32), np.zeros((n, 4), np.float32), np.zeros(n, np.uint32))
        ctx.sync()
        pool.start()
        ctx.fuse_virtual_depth(fid, lists, counts, np.ones(V, np.uint8), BASE)
        ctx.sync()
        # the records and their flags, the maps, the list arrays, the points handed out
        own = 44 * n + 12 * FW * FH + 4 * V * max_list + 36 * n
        assert 44 * n < pool.peak() <= own + (most << 20) + (1 << 20)
        ctx.frame_free(fid)
