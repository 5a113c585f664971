"""The work a program has this engine do, as timed cases.

A case is one call sequence through the public entry points (include/pfd_abi.h,
bound by the package) on seeded synthetic frames with the shapes of the
repository's own configurations: 8-bit raw frames of 320x240 to 4080x3068,
hexagonal lens grids of 15 to 30 px pitch (micro-images of 10 to 21 px), 6 to 18
matching neighbours, bilateral NCC patches of 5 to 15 px, 1 to 5 PatchMatch
iterations.  What the caller gets back lands in page-locked host buffers that
the caller keeps, as a program that streams frames would hold them.

    listed()          the named cases
    draw(rng)         one more case of the same ranges
    prepare(case, s)  context, resident frame and buffers, from the seed alone
    run(state)        one pass; returns its outputs
    work(case)        bytes and operations the pass cannot do without
    exact(case, s)    the outputs in 64 bits, where they have such values
"""
import ctypes
import importlib
import math

import numpy as np
import torch

pfd = importlib.import_module("plenoptic-for-depth_b200")

BLURS = (0.6, 1.0, 1.4)          # sigma of the three interleaved lens types


def listed():
    return [
        # a region of interest at the lowest latency: launches and the copy back
        dict(name="match_tiny", kind="match", width=320, height=240, pitch=21.0, planes=3, nb=6, patch=9, iters=2),
        # the repository's small configuration: one preview frame
        dict(name="match_small", kind="match", width=1024, height=768, pitch=23.0, planes=4, nb=6, patch=11, iters=3),
        # the full sensor with three lens types, 12 neighbours and the 15 x 15 patch,
        # at the first iterations, where most hypotheses still differ
        dict(name="match_full", kind="match", width=4080, height=3068, pitch=23.2, planes=12, nb=12, patch=15, iters=3,
             types=3),
        # the ACMM matcher at its reference parameters (patch 5, 5 iterations)
        dict(name="match_acmm", kind="match", width=2048, height=1536, pitch=23.2, planes=8, nb=12, patch=5, iters=5,
             acmm=True, top_k=6, sigma_s=5.0, sigma_c=3.0),
        # an odd frame with large lenses, many neighbours, the blur channel and
        # the shifted moments
        dict(name="match_blur", kind="match", width=1531, height=1147, pitch=28.7, planes=9, nb=17, patch=13, iters=2,
             blur=True, shifted=True, types=3),
        # several cameras' frames of different sizes, lenses and parameters in one call
        dict(name="batch_mixed", kind="batch", count=5, width=701, height=523, pitch=17.3, planes=5, nb=9, patch=11,
             iters=2),
        # the request loop: frames submitted together, filtered, copied back
        dict(name="serve_mixed", kind="serve", count=4, width=640, height=487, pitch=19.1, planes=4, nb=8, patch=11,
             iters=1),
        # the consistency pass on a state that lies in host memory: cycle check,
        # filter, reprojection error, everything handed back
        dict(name="checks_mid", kind="checks", width=2048, height=1536, pitch=23.2, planes=8, nb=12),
        # the whole path on one preview frame: slice, choose neighbours, match,
        # check, filter, focal stack
        dict(name="frame_path", kind="path", width=1280, height=963, pitch=23.0, planes=6, nb=12, patch=11, iters=1,
             slices=12),
        # focal stack of the full sensor
        dict(name="stack_full", kind="stack", width=4080, height=3068, pitch=23.2, planes=12, nb=6, slices=16,
             out_w=2040, out_h=1534),
        # fused virtual-depth map, all-in-focus image and point cloud of a matched
        # frame, and its real depth
        dict(name="fuse_mid", kind="fuse", width=1536, height=1159, pitch=23.2, planes=6, nb=12),
        # a raw frame comes in: micro-images, matching neighbours, blur and richness
        # channels
        dict(name="ingest_full", kind="ingest", width=4080, height=3068, pitch=23.2, planes=12, nb=12),
    ]


# Widths of the drawn frames per kind: a drawn case costs no more than match_full.
_WIDTHS = {"match": (320, 2600), "batch": (400, 900), "serve": (400, 900), "checks": (500, 3000), "path": (500, 1700),
           "stack": (600, 4080), "fuse": (500, 1700), "ingest": (600, 4080)}


def draw(rng):
    kind = rng.choice(["match", "match", "match", "match", "batch", "serve", "checks", "path", "stack", "fuse", "ingest"])
    lo, hi = _WIDTHS[kind]
    w = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    h = int(w * rng.uniform(0.6, 0.8))
    c = dict(kind=kind, width=w, height=h, pitch=round(rng.uniform(15.0, 30.0), 1), planes=rng.randint(3, 12),
             nb=rng.randint(6, 18))
    if kind in ("match", "batch", "serve", "path"):
        c.update(patch=rng.choice([7, 9, 11, 13, 15]), iters=rng.randint(1, 3 if kind == "match" else 2))
    if kind == "match":
        c.update(types=rng.choice([1, 3]), blur=rng.random() < 0.25, shifted=rng.random() < 0.25)
        if rng.random() < 0.25:
            c.update(acmm=True, patch=5, iters=rng.randint(2, 5), top_k=6, sigma_s=5.0, sigma_c=3.0)
    if kind in ("batch", "serve"):
        c.update(count=rng.randint(2, 6))
    if kind == "path":
        c.update(slices=rng.randint(2, 16))
    if kind == "stack":
        f = rng.uniform(0.3, 0.6)
        c.update(slices=rng.randint(2, 16), out_w=max(16, int(w * f)), out_h=max(16, int(h * f)))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _workload(c, seed):
    types = c.get("types", 1)
    return pfd.make_workload(c["width"], c["height"], c["pitch"], c["planes"], seed=seed, max_nb=c["nb"],
                             n_lens_types=types, blur_sigma=BLURS if types == 3 else (0.0, 0.0, 0.0))


def _params(c):
    return pfd.PmParams(base=c["pitch"], max_iterations=c["iters"], patch_size=c["patch"], top_k=c.get("top_k", 5),
                        sigma_spatial=c.get("sigma_s", 3.0), sigma_color=c.get("sigma_c", 12.0))


def _several(c):
    """The frames of a batch or a stream: sizes, lenses and parameters around the case's."""
    out = []
    for i in range(c["count"]):
        s = 1.0 - 0.09 * i
        out.append(dict(c, width=int(c["width"] * s), height=int(c["height"] * s),
                        pitch=round(min(30.0, max(15.0, c["pitch"] * (1.0 + 0.07 * (i % 3)))), 1),
                        nb=max(6, c["nb"] - i % 3), patch=c["patch"] if i % 2 == 0 else max(7, c["patch"] - 2),
                        iters=1 + (c["iters"] - 1 + i) % max(1, c["iters"])))
    return out


class _Host:
    """Page-locked host arrays that outlive the pass (numpy views of torch tensors)."""

    def __init__(self):
        self.keep = []

    def empty(self, shape, dtype):
        t = torch.empty(tuple(int(x) for x in shape), dtype=dtype, pin_memory=True)
        self.keep.append(t)
        return t.numpy()

    def copy(self, a):
        t = torch.from_numpy(np.ascontiguousarray(a)).pin_memory()
        self.keep.append(t)
        return t.numpy()


def _p(a):
    return ctypes.c_void_p(a.ctypes.data)


def _ok(ctx, rc):
    if rc != pfd.PFD_OK:
        raise pfd.PfdError(rc, (ctx._L.pfd_last_error(ctx._h) or b"").decode())


def _state_buffers(host, n):
    return dict(plane=host.empty((n, 4), torch.float32), cost=host.empty((n,), torch.float32),
                disp=host.empty((n, 4), torch.float32), sel=host.empty((n,), torch.int32))


def _download(ctx, fid, o):
    _ok(ctx, ctx._L.pfd_download(ctx._h, fid, _p(o["plane"]), _p(o["cost"]), _p(o["disp"]), _p(o["sel"])))


def _scene_state(w, seed):
    """A matched frame's state from the scene's own depth: disparities with small
    errors and 8% outliers, normals near the axis, costs and selected views."""
    rs = np.random.RandomState(seed & 0x7FFFFFFF)
    mi, V = w.mi, w.centers.shape[0]
    vd = pfd.synth_vd_map(w.frame)
    o = pfd.window_origins(w.centers, mi).astype(np.int64)
    ys, xs = np.mgrid[0:mi, 0:mi]
    gt = vd[o[:, 1, None, None] + ys[None], o[:, 0, None, None] + xs[None]].reshape(-1)
    n = gt.size
    pitch = np.float32(w.frame.pitch)
    d = np.where(gt > 0, pitch / np.maximum(gt, np.float32(0.5)), np.float32(0.0)).astype(np.float32)
    d += rs.standard_normal(n).astype(np.float32) * np.float32(0.12)
    bad = rs.random_sample(n) < 0.08
    d[bad] = (rs.random_sample(int(bad.sum())) * pitch * 0.5).astype(np.float32)
    nx = rs.standard_normal(n).astype(np.float32) * np.float32(0.08)
    ny = rs.standard_normal(n).astype(np.float32) * np.float32(0.08)
    nz = np.sqrt(np.maximum(np.float32(0.2), 1 - nx * nx - ny * ny)).astype(np.float32)
    plane = np.stack([nx, ny, nz, d], axis=1)
    cost = np.abs(rs.standard_normal(n)).astype(np.float32) * np.float32(0.5)
    K = w.nb_ids.shape[1]
    sel = np.zeros(n, np.uint32)
    for _ in range(5):
        sel |= np.uint32(1) << rs.randint(0, K, n).astype(np.uint32)
    cnt = np.repeat(w.nb_counts.astype(np.uint32), mi * mi)
    sel &= ((np.uint64(1) << cnt.astype(np.uint64)) - np.uint64(1)).astype(np.uint32)
    disp = np.stack([d, d, np.full(n, pitch, np.float32), np.ones(n, np.float32)], axis=1).astype(np.float32)
    return plane, cost, disp, sel


class _State:
    def __init__(self, case, seed):
        self.c, self.seed, self.host = dict(case), int(seed), _Host()


# ---------------------------------------------------------------------------
# match: PatchMatch of one resident frame, its state copied back
# ---------------------------------------------------------------------------
def _prepare_match(S):
    c = S.c
    w = _workload(c, S.seed)
    S.ctx = pfd.Context()
    S.ctx.set_matcher(bool(c.get("acmm")))
    S.ctx.set_ncc_moments(bool(c.get("shifted")))
    S.fid = S.ctx.frame_upload(w.frame.raw, w.centers, w.tilekeys, w.mi, w.mi, w.nb_ids, w.nb_counts)
    if c.get("blur"):
        S.ctx.frame_compute_blur(S.fid, copy_back=False)
    S.params = _params(c)
    S.out = _state_buffers(S.host, w.centers.shape[0] * w.mi * w.mi)
    S.ctx.sync()


def _run_match(S):
    S.ctx.patchmatch(S.fid, S.params, S.seed)
    _download(S.ctx, S.fid, S.out)
    return S.out


# ---------------------------------------------------------------------------
# batch: PatchMatch of several resident frames in one call
# ---------------------------------------------------------------------------
def _prepare_batch(S):
    S.ctx = pfd.Context()
    S.fids, S.params, S.outs, S.seeds = [], [], [], []
    for i, c in enumerate(_several(S.c)):
        w = _workload(c, S.seed * 31 + i)
        S.fids.append(S.ctx.frame_upload(w.frame.raw, w.centers, w.tilekeys, w.mi, w.mi, w.nb_ids, w.nb_counts))
        S.params.append(_params(c))
        S.seeds.append(S.seed + i)
        S.outs.append(_state_buffers(S.host, w.centers.shape[0] * w.mi * w.mi))
    S.ctx.sync()


def _run_batch(S):
    S.ctx.patchmatch_batch(S.fids, S.params, S.seeds)
    for fid, o in zip(S.fids, S.outs):
        _download(S.ctx, fid, o)
    return S.outs


# ---------------------------------------------------------------------------
# serve: requests through the server's slots
# ---------------------------------------------------------------------------
def _prepare_serve(S):
    S.server = pfd.Server(slots=3)
    S.reqs = []
    for i, c in enumerate(_several(S.c)):
        S.reqs.append((_workload(c, S.seed * 31 + i), _params(c), S.seed + i, c["pitch"]))
    S.cfg = pfd.FilterCfg()


def _run_serve(S):
    tickets = [S.server.submit(w, p, seed, filter_cfg=S.cfg, baseline_unit=pitch) for w, p, seed, pitch in S.reqs]
    outs = []
    for t in tickets:
        plane, cost, disp, sel, _ms = S.server.wait(t)
        outs.append(dict(plane=plane, cost=cost, disp=disp, sel=sel.view(np.int32)))
    return outs


# ---------------------------------------------------------------------------
# checks: the consistency pass on an uploaded state
# ---------------------------------------------------------------------------
def _prepare_checks(S):
    c = S.c
    w = _workload(c, S.seed)
    S.ctx = pfd.Context()
    S.fid = S.ctx.frame_upload(w.frame.raw, w.centers, w.tilekeys, w.mi, w.mi, w.nb_ids, w.nb_counts)
    S.inp = [S.host.copy(a) for a in _scene_state(w, S.seed)]
    n = w.centers.shape[0] * w.mi * w.mi
    S.out = _state_buffers(S.host, n)
    S.geo, S.pho = S.host.empty((n,), torch.float32), S.host.empty((n,), torch.float32)
    S.tm, S.reason = S.host.empty((n,), torch.uint8), S.host.empty((n,), torch.uint8)
    S.err = S.host.empty((n,), torch.float32)
    S.fcfg, S.ccfg = pfd.FilterCfg().c(), pfd.CycleCfg().c()
    S.ctx.sync()


def _run_checks(S):
    ctx, L, unit = S.ctx, S.ctx._L, float(S.c["pitch"])
    ctx.state_upload(S.fid, *S.inp)
    stats = pfd.CycleStatsC()
    _ok(ctx, L.pfd_cycle_check(ctx._h, S.fid, ctypes.byref(S.ccfg), unit, ctypes.byref(stats), _p(S.geo), _p(S.pho),
                               _p(S.tm)))
    counts = np.zeros(8, np.int64)
    _ok(ctx, L.pfd_filter(ctx._h, S.fid, ctypes.byref(S.fcfg), unit, _p(S.reason), _p(counts)))
    _ok(ctx, L.pfd_reprojection_error(ctx._h, S.fid, ctypes.byref(S.fcfg), unit, _p(S.err)))
    _download(ctx, S.fid, S.out)
    return dict(state=S.out, geo=S.geo, pho=S.pho, mask=S.tm, reason=S.reason, err=S.err, counts=counts,
                stats=[float(getattr(stats, k)) for k in pfd.CYCLE_STATS])


# ---------------------------------------------------------------------------
# path: raw frame to filtered depth and focal stack
# ---------------------------------------------------------------------------
def _prepare_path(S):
    c = S.c
    w = _workload(c, S.seed)
    S.ctx = pfd.Context()
    S.fid = S.ctx.frame_create(c["width"], c["height"], w.centers, w.tilekeys, w.mi, w.mi, w.nb_ids, w.nb_counts)
    S.raw = S.host.copy(w.frame.raw)
    S.grid = (w.frame.n_cols, w.frame.n_rows)
    S.params = _params(c)
    S.out = _state_buffers(S.host, w.centers.shape[0] * w.mi * w.mi)
    S.size = (max(16, c["width"] // 2), max(16, c["height"] // 2))
    S.vds = np.linspace(2.0, 12.0, c["slices"]).astype(np.float32)
    S.stack = S.host.empty((c["slices"], S.size[1], S.size[0]), torch.float32)
    S.ccfg, S.fcfg = pfd.CycleCfg(), pfd.FilterCfg()
    S.ctx.sync()


def _run_path(S):
    ctx, unit = S.ctx, float(S.c["pitch"])
    ctx.frame_set_raw(S.fid, S.raw)
    ctx.frame_select_neighbors(S.fid, S.grid[0], S.grid[1], unit)
    ctx.patchmatch(S.fid, S.params, S.seed)
    ctx.cycle_check(S.fid, S.ccfg, unit, maps=False, stats=False)
    ctx.filter(S.fid, S.fcfg, unit, download=False)
    ctx.reprojection_error(S.fid, S.fcfg, unit, download=False)
    _ok(ctx, ctx._L.pfd_refocus(ctx._h, S.fid, _p(S.vds), len(S.vds), S.size[0], S.size[1], _p(S.stack)))
    _download(ctx, S.fid, S.out)
    stats = ctx.cycle_check_stats(S.fid)
    return dict(state=S.out, stack=S.stack, stats=[float(stats[k]) for k in pfd.CYCLE_STATS])


# ---------------------------------------------------------------------------
# stack: focal stack of a resident frame
# ---------------------------------------------------------------------------
def _prepare_stack(S):
    c = S.c
    w = _workload(c, S.seed)
    S.ctx = pfd.Context()
    S.fid = S.ctx.frame_upload(w.frame.raw, w.centers, w.tilekeys, w.mi, w.mi, w.nb_ids, w.nb_counts)
    S.vds = np.linspace(2.0, 12.0, c["slices"]).astype(np.float32)
    S.stack = S.host.empty((c["slices"], c["out_h"], c["out_w"]), torch.float32)
    S.ctx.sync()


def _run_stack(S):
    _ok(S.ctx, S.ctx._L.pfd_refocus(S.ctx._h, S.fid, _p(S.vds), len(S.vds), S.c["out_w"], S.c["out_h"], _p(S.stack)))
    return S.stack


def _exact_stack(c, seed):
    """The mean of the bilinear samples of every micro-image that sees the point,
    in 64 bits."""
    w = _workload(c, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m, V = w.mi, w.centers.shape[0]
    ow, oh = c["out_w"], c["out_h"]
    tiles = torch.from_numpy(w.gray).to(dev).double().reshape(V, m * m)
    cen = torch.from_numpy(w.centers).to(dev).double()
    sx, sy = c["width"] / ow, c["height"] / oh
    cm = (m - 1) * 0.5 + 1.0
    out = torch.empty((c["slices"], oh, ow), dtype=torch.float64)
    for s, vd in enumerate(np.linspace(2.0, 12.0, c["slices"]).astype(np.float32)):
        vd = float(vd)
        total = torch.zeros(oh * ow, dtype=torch.float64, device=dev)
        count = torch.zeros(oh * ow, dtype=torch.float64, device=dev)
        nx, ny = int(m * vd / sx) + 4, int(m * vd / sy) + 4
        step = max(1, 20_000_000 // (nx * ny))
        for a in range(0, V, step):
            p = cen[a:a + step]
            ox = torch.floor((p[:, 0] - cm * vd) / sx).long()[:, None] - 1 + torch.arange(nx, device=dev)[None]
            oy = torch.floor((p[:, 1] - cm * vd) / sy).long()[:, None] - 1 + torch.arange(ny, device=dev)[None]
            u = ((ox.double() + 0.5) * sx - 0.5 - p[:, :1]) / vd + cm
            v = ((oy.double() + 0.5) * sy - 0.5 - p[:, 1:]) / vd + cm
            oku = (ox >= 0) & (ox < ow) & (u >= 0) & (u <= m - 1)
            okv = (oy >= 0) & (oy < oh) & (v >= 0) & (v <= m - 1)
            ok = oku[:, None, :] & okv[:, :, None]
            x0, y0 = u.clamp(0, m - 1).floor().long(), v.clamp(0, m - 1).floor().long()
            fx, fy = (u.clamp(0, m - 1) - x0)[:, None, :], (v.clamp(0, m - 1) - y0)[:, :, None]
            x1, y1 = (x0 + 1).clamp(max=m - 1), (y0 + 1).clamp(max=m - 1)
            t = tiles[a:a + step]

            def at(y, x):
                i = (y[:, :, None] * m + x[:, None, :]).reshape(t.shape[0], -1)
                return t.gather(1, i).reshape(t.shape[0], ny, nx)
            val = (1 - fy) * ((1 - fx) * at(y0, x0) + fx * at(y0, x1)) + fy * ((1 - fx) * at(y1, x0) + fx * at(y1, x1))
            i = (oy[:, :, None] * ow + ox[:, None, :])[ok]
            total.index_add_(0, i, val[ok])
            count.index_add_(0, i, torch.ones_like(i, dtype=torch.float64))
        out[s] = torch.where(count > 0, total / count.clamp(min=1), torch.zeros_like(total)).reshape(oh, ow).cpu()
    return out


# ---------------------------------------------------------------------------
# fuse: virtual-depth fusion of a matched frame, and its real depth
# ---------------------------------------------------------------------------
def _prepare_fuse(S):
    c = S.c
    w = _workload(c, S.seed)
    S.ctx = pfd.Context()
    S.fid = S.ctx.frame_upload(w.frame.raw, w.centers, w.tilekeys, w.mi, w.mi, w.nb_ids, w.nb_counts)
    S.ctx.state_upload(S.fid, *_scene_state(w, S.seed))
    S.lists, S.counts = w.nb_ids, w.nb_counts
    S.is_ref = np.ones(w.centers.shape[0], np.uint8)
    S.model = np.array([0.011, 38.0, 120.0])
    n = w.centers.shape[0] * w.mi * w.mi
    H, W = c["height"], c["width"]
    S.fuse = pfd.FuseParamsC(float(c["pitch"]), 1.0, 1.0, 0.05, 2)
    S.vd, S.conf = S.host.empty((H, W), torch.float32), S.host.empty((H, W), torch.uint8)
    S.aif, S.depth = S.host.empty((H, W, 3), torch.uint8), S.host.empty((H, W), torch.float64)
    S.points = S.host.empty((n, 9), torch.float32)       # at most one point per micro-image pixel
    S.points.fill(0.0)
    S.ctx.sync()


def _run_fuse(S):
    ctx, L = S.ctx, S.ctx._L
    n = ctypes.c_longlong(0)
    _ok(ctx, L.pfd_fuse_virtual_depth(ctx._h, S.fid, ctypes.byref(S.fuse), _p(S.lists), _p(S.counts),
                                      S.lists.shape[1], _p(S.is_ref), None, _p(S.vd), _p(S.conf), _p(S.aif),
                                      _p(S.points), ctypes.byref(n)))
    _ok(ctx, L.pfd_vd_to_rd_map(ctx._h, _p(S.vd), S.vd.size, _p(S.model), _p(S.depth)))
    return dict(vd=S.vd, conf=S.conf, aif=S.aif, points=S.points, n=int(n.value), depth=S.depth)


# ---------------------------------------------------------------------------
# ingest: raw frame to micro-images, neighbours, blur and richness channels
# ---------------------------------------------------------------------------
def _prepare_ingest(S):
    c = S.c
    w = _workload(c, S.seed)
    S.ctx = pfd.Context()
    S.fid = S.ctx.frame_create(c["width"], c["height"], w.centers, w.tilekeys, w.mi, w.mi, w.nb_ids, w.nb_counts)
    S.raw = S.host.copy(w.frame.raw)
    S.grid = (w.frame.n_cols, w.frame.n_rows)
    V, m = w.centers.shape[0], w.mi
    S.ids, S.cnt = S.host.empty((V, c["nb"]), torch.int32), S.host.empty((V,), torch.int32)
    S.blur, S.sharp = S.host.empty((V, m, m), torch.uint8), S.host.empty((V,), torch.int32)
    S.rich, S.rich_n = S.host.empty((V, m, m), torch.uint8), S.host.empty((V,), torch.int32)
    S.ctx.sync()


def _run_ingest(S):
    ctx, L, c = S.ctx, S.ctx._L, S.c
    ctx.frame_set_raw(S.fid, S.raw)
    _ok(ctx, L.pfd_frame_select_neighbors(ctx._h, S.fid, S.grid[0], S.grid[1], float(c["pitch"]), c["nb"], _p(S.ids),
                                          _p(S.cnt)))
    _ok(ctx, L.pfd_frame_compute_blur(ctx._h, S.fid, _p(S.blur), _p(S.sharp)))
    _ok(ctx, L.pfd_frame_compute_richness(ctx._h, S.fid, None, _p(S.rich), _p(S.rich_n)))
    used = np.arange(c["nb"])[None] < S.cnt[:, None]
    return dict(ids=np.where(used, S.ids, -1), counts=S.cnt, blur=S.blur, sharp=S.sharp, rich=S.rich, rich_n=S.rich_n)


_PREPARE = {"match": _prepare_match, "batch": _prepare_batch, "serve": _prepare_serve, "checks": _prepare_checks,
            "path": _prepare_path, "stack": _prepare_stack, "fuse": _prepare_fuse, "ingest": _prepare_ingest}
_RUN = {"match": _run_match, "batch": _run_batch, "serve": _run_serve, "checks": _run_checks, "path": _run_path,
        "stack": _run_stack, "fuse": _run_fuse, "ingest": _run_ingest}


def prepare(case, seed):
    S = _State(case, seed)
    _PREPARE[case["kind"]](S)
    return S


def run(state):
    return _RUN[state.c["kind"]](state)


def exact(case, seed):
    # The PatchMatch is a random search over planes whose decisions hang on single
    # bits of the costs, and the checks and the fusion are chains of threshold
    # tests on it: their outputs have no 64-bit counterpart, nor have the lists and
    # bytes of the ingest.  The focal stack is a mean of samples.
    if case["kind"] == "stack" and case["slices"] * case["out_w"] * case["out_h"] <= 60_000_000:
        return _exact_stack(case, seed)
    return None


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _views(c):
    return max(1.0, c["width"] * c["height"] / (c["pitch"] * c["pitch"] * 0.8660254))


def _match_work(c):
    """Each micro-image read and each pixel's state (plane, cost, disp, views: 40
    bytes) written once.  Operations: 24 per NCC tap; half of the neighbours of a
    hypothesis hold its anchor and half of a patch lies in both windows; one
    hypothesis per pixel at the start, 8 per updated pixel and half-sweep, which
    is what is left when equal planes and unsampled views are not evaluated."""
    m = int(c["pitch"] * 0.7071)
    px = _views(c) * m * m
    side = min(c["patch"], m)
    nccs = px * c["nb"] * 0.5 * (1.0 + 8.0 * c["iters"])
    return px * 41.0, nccs * side * side * 0.5 * 24.0


def work(case):
    c = case
    m = int(c["pitch"] * 0.7071)
    px = _views(c) * m * m
    raw = float(c["width"] * c["height"])
    kind = c["kind"]
    if kind == "match":
        b, f = _match_work(c)
    elif kind in ("batch", "serve"):
        parts = [_match_work(x) for x in _several(c)]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind == "checks":
        # the state in and out, the maps (two floats, a mask byte, a reason byte and
        # one float); per pixel four neighbours with two bilinear reads and windows
        b, f = px * (40.0 + 40.0 + 14.0 + 1.0), px * 4.0 * 400.0
    elif kind == "path":
        b, f = _match_work(c)
        n_out = c["slices"] * (c["width"] // 2) * (c["height"] // 2)
        b, f = b + raw + n_out * 4.0, f + px * 4.0 * 400.0 + n_out * 30.0 * 20.0
    elif kind == "stack":
        n_out = float(c["slices"] * c["out_w"] * c["out_h"])
        # a lens covers ((m - 1) vd)^2 raw pixels: on average over vd 2 to 12 about 30
        # samples per output pixel, 20 operations each
        b, f = px + n_out * 4.0, n_out * 30.0 * 20.0
    elif kind == "fuse":
        b, f = px * 17.0 + raw * (4.0 + 1.0 + 3.0 + 4.0 + 8.0) + px * 0.3 * 36.0, px * c["nb"] * 60.0
    else:
        # raw in, tiles out, lists out; about 30 candidates' similarities per view over
        # two binarised windows at 8 shifts
        b, f = raw + px * 3.0 + _views(c) * (c["nb"] + 3.0) * 4.0, px * 30.0 * 8.0
    return {"bytes": float(b), "flops": float(f)}
