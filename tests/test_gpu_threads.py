"""Two threads, each with a context of its own, run the same kernels with shared
memory of different sizes at the same time: neither's launch depends on what the
other last asked for, and every result is the one of a thread alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BASE = 20.0


def _fuse_job(pfd, m, max_list, seed):
    rs = np.random.RandomState(seed)
    cols, rows = 5, 4
    V, n = cols * rows, cols * rows * m * m
    gx, gy = np.meshgrid(np.arange(cols), np.arange(rows))
    keys = np.stack([gx.ravel(), gy.ravel()], 1).astype(np.int32)
    cen = (keys * BASE + 30).astype(np.float32)
    lists = ((np.arange(V)[:, None] + np.arange(1, max_list + 1)[None]) % V).astype(np.int32)
    counts = np.full(V, max_list, np.int32)
    plane = np.concatenate([rs.randn(n, 3), 2.0 + 0.03 * rs.randn(n, 1)], 1).astype(np.float32)
    gray = rs.randint(0, 256, (V, m, m)).astype(np.uint8)
    FW, FH = int(cen[:, 0].max() + 40), int(cen[:, 1].max() + 40)
    ctx = pfd.Context(0)
    fid = ctx.frame_create(FW, FH, cen, keys, m, m, np.full((V, 1), -1, np.int32), np.zeros(V, np.int32))
    ctx.frame_set_micro_images(fid, gray)
    ctx.state_upload(fid, plane, np.zeros(n, np.float32), np.zeros((n, 4), np.float32), np.zeros(n, np.uint32))
    ref = np.ones(V, np.uint8)

    def run():
        for _ in range(40):                              # enqueued: the launches of both threads meet
            ctx.fuse_virtual_depth(fid, lists, counts, ref, BASE, download=False)
        return ctx.fuse_virtual_depth(fid, lists, counts, ref, BASE)
    return run


def _sweep_job(pfd, side, K, patch, seed):
    from test_gpu_slots import _grid
    rs = np.random.RandomState(seed)
    cen, keys, gray, ids, cnt = _grid(rs, 4, 4, side, side, K, side * 1.45)
    P = pfd.PmParams(base=side * 1.45, patch_size=patch, max_iterations=1, top_k=2)
    ctx = pfd.Context(0)
    fid = ctx.frame_create(int(cen[:, 0].max() + side + 40), int(cen[:, 1].max() + side + 40), cen, keys, side, side, ids, cnt)
    ctx.frame_set_micro_images(fid, gray)

    def run():
        for _ in range(10):
            ctx.patchmatch(fid, P, 7)
        reason, _ = ctx.filter(fid, pfd.FilterCfg(), side * 1.45)
        return (*ctx.download(fid), reason)
    return run


def _side_by_side(jobs, times):
    want = [j() for j in jobs]
    wrong = []

    def loop(job, ref):
        try:
            for _ in range(times):
                got = job()
                if not all(np.array_equal(a, b, equal_nan=np.asarray(a).dtype.kind == "f") for a, b in zip(got, ref)):
                    wrong.append("another result")
                    return
        except Exception as e:                            # noqa: BLE001 - reported below
            wrong.append(str(e))
    ts = [threading.Thread(target=loop, args=jr) for jr in zip(jobs, want)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong, wrong


def test_fusions_of_two_list_lengths(pfd):
    _side_by_side([_fuse_job(pfd, 4, 4, 1), _fuse_job(pfd, 8, 19, 2)], 25)


def test_matches_of_two_windows(pfd):
    _side_by_side([_sweep_job(pfd, 10, 2, 5, 1), _sweep_job(pfd, 20, 12, 9, 2)], 25)
