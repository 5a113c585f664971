"""The half-sweep kernel with pixel slots (pm_slots.cu) at the sizes where its
plan, its list of NCCs and its tap rectangles can go wrong: the smallest and
largest windows, odd and unequal sides, one and 32 neighbours, views with no or
missing neighbours, patches of 1 to 31, tap steps above 1, states with steep,
distant, negative, rejected and non-finite planes.  Every state field equals the
CPU oracle's bit for bit (the tolerance of every sweep test here)."""
import numpy as np
import pytest

from scenes import value_texture

pytestmark = pytest.mark.gpu


def _same(a, b):
    a = np.asarray(a)
    b = np.asarray(b)
    if a.dtype.kind == "f":
        return bool(np.all((a == b) | (np.isnan(a) & np.isnan(b))))
    return bool(np.array_equal(a, b))


def _grid(rs, cols, rows, W, H, K, base):
    """Lenses on a jittered grid seeing one texture at disparities around 1.5 px;
    random neighbour lists, some entries missing, one view without neighbours."""
    V = cols * rows
    gx, gy = np.meshgrid(np.arange(cols), np.arange(rows))
    keys = np.stack([gx.ravel(), gy.ravel()], 1).astype(np.int32)
    cen = (keys * base + 40 + rs.uniform(-0.5, 0.5, (V, 2))).astype(np.float32)
    T = value_texture(H + 4 * rows + 8, W + 4 * cols + 8, int(rs.randint(1 << 20)), cell=4)
    gray = np.stack([T[2 * y:2 * y + H, 2 * x:2 * x + W] for x, y in keys]).astype(np.uint8)
    gray = np.clip(gray.astype(int) + rs.randint(-3, 4, gray.shape), 0, 255).astype(np.uint8)
    ids = np.full((V, K), -1, np.int32)
    cnt = np.zeros(V, np.int32)
    for v in range(V):
        others = np.array([u for u in range(V) if u != v])
        d = np.hypot(*(cen[others] - cen[v]).T)
        near = others[np.argsort(d, kind="stable")][:K]
        n = len(near) if v % 5 else max(1, len(near) // 2)
        ids[v, :n] = near[:n]
        cnt[v] = n
        if n > 2 and v % 3 == 0:
            ids[v, 1] = -1
    cnt[V // 2] = 0
    return cen, keys, gray, ids, cnt


def _state(rs, V, W, H, K, base):
    n = V * W * H
    nrm = rs.randn(n, 3)
    nrm[:, 2] = np.abs(nrm[:, 2]) + 0.05
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    d = rs.uniform(0, base * 0.5, n)
    plane = np.concatenate([nrm, d[:, None]], 1).astype(np.float32)
    near = rs.rand(n) < 0.5                                   # plausible planes
    plane[near] = np.stack([0.02 * rs.randn(near.sum()), 0.02 * rs.randn(near.sum()), np.ones(near.sum()),
                            rs.uniform(1, 3, near.sum())], 1)
    k = rs.permutation(n)[:max(12, n // 50)]
    plane[k[0::6]] = (0, 0, 0, -1)                            # as the filter rejects a pixel
    plane[k[1::6], 2] = 1e-6                                  # nearly parallel to the axis
    plane[k[2::6], 3] = -5.0
    plane[k[3::6], 3] = 1e7
    plane[k[4::6], 3] = np.nan
    plane[k[5::6], 2] = -0.3
    cost = rs.uniform(0, 2, n).astype(np.float32)
    sel = rs.randint(0, 1 << min(K, 30), n).astype(np.uint32)
    disp = rs.uniform(0, 3, (n, 4)).astype(np.float32)
    return dict(plane=plane, cost=cost, disp=disp, sel=sel)


CASES = [
    # W, H, K, patch, step, mode
    (2, 2, 1, 3, 1, ""), (3, 5, 2, 1, 1, ""), (5, 3, 6, 15, 1, ""), (16, 16, 12, 15, 1, ""), (17, 15, 12, 9, 1, "shifted"),
    (15, 17, 16, 11, 1, "blur"), (16, 16, 17, 5, 1, "acmm"), (21, 20, 18, 13, 1, "blur shifted"),
    (20, 21, 12, 15, 2, ""), (16, 16, 6, 31, 3, "blur"), (32, 32, 12, 31, 1, ""), (32, 31, 32, 23, 1, "no init"),
    (24, 24, 32, 7, 1, "acmm blur, no init"), (31, 2, 5, 9, 2, "shifted"),
]


@pytest.mark.parametrize("W,H,K,patch,step,mode", CASES)
def test_slot_sweep_matches_the_oracle(pfd, oracle, W, H, K, patch, step, mode):
    rs = np.random.RandomState(W * 1000 + H * 31 + K)
    base = max(W, H) * 1.45
    cols, rows = (7, 5) if K > 16 else (4, 3)
    if W * H > 900:
        cols, rows = (6, 6) if K > 16 else (3, 3)
    cen, keys, gray, ids, cnt = _grid(rs, cols, rows, W, H, K, base)
    V = len(cen)
    blur = rs.randint(0, 256, gray.shape).astype(np.uint8) if "blur" in mode else None
    P = pfd.PmParams(base=base, patch_size=patch, radius_increment=step, max_iterations=1, top_k=min(5, K))
    orc = oracle.Oracle(gray, cen, ids, cnt, blur=blur, shifted="shifted" in mode, acmm="acmm" in mode)
    FW, FH = int(cen[:, 0].max() + W + 40), int(cen[:, 1].max() + H + 40)
    with pfd.Context(0) as ctx:
        ctx.set_ncc_moments("shifted" in mode)
        ctx.set_matcher("acmm" in mode)
        fid = ctx.frame_create(FW, FH, cen, keys, W, H, ids, cnt, blur)
        ctx.frame_set_micro_images(fid, gray)

        def check(st, what):
            for name, g in zip(("plane", "cost", "disp", "sel"), ctx.download(fid)):
                assert _same(g, st[name]), f"{what}: {name} differs at {np.count_nonzero(np.asarray(g) != st[name])}"

        # from an initialisation (stored cost vectors in use), where its plan fits
        if "no init" in mode:
            with pytest.raises(pfd.PfdError):
                ctx.pm_init(fid, P, 17)
        else:
            ctx.pm_init(fid, P, 17)
            st = orc.init(P, 17)
            check(st, "init")
            for ph in (0, 1):
                ctx.pm_sweep(fid, P, 17, 0, ph)
                st = orc.sweep(P, 17, 0, ph, st)
                check(st, f"sweep 0.{ph}")
        # from a state with every kind of plane (no stored vectors), a late iteration
        st = _state(rs, V, W, H, K, base)
        ctx.state_upload(fid, st["plane"], st["cost"], st["disp"], st["sel"])
        for ph in (1, 0):
            ctx.pm_sweep(fid, P, 18, 9, ph)
            st = orc.sweep(P, 18, 9, ph, st)
            check(st, f"uploaded state, phase {ph}")
        ctx.frame_free(fid)
