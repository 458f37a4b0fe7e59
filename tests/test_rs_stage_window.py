"""The staged projector (csrc/rs_stage.cuh) reads shared memory without bounds tests: every
footprint of a staged ray has to lie in its chunk's window. This restates the windows, the
chunking and the ray test in FP32 (numpy) and marches random tiles' rays by the kernel's
repeated additions (projection_ER_kernel.cuh:295-297) through them."""
import numpy as np
import pytest

f32 = np.float32


def _march(rng, n, nz, views_spread=True):
    """Random view, tile and detector; returns the number of staged rays checked."""
    fod = f32(rng.uniform(1.2, 3.0) * n)
    mag = f32(rng.uniform(1.3, 2.6))
    fdd = f32(fod * mag)
    nu, nv = int(rng.integers(n // 2, 2 * n)), int(rng.integers(max(8, nz // 2), 2 * nz + 8))
    du = f32(rng.uniform(0.6, 1.3) * mag * n / nu)
    uc, vc, xc, zc = f32(nu / 2 - 0.5), f32(nv / 2 - 0.5), f32(n / 2 - 0.5), f32(nz / 2 - 0.5)
    phi = rng.uniform(0, 2 * np.pi)
    al, be = f32(np.cos(phi)), f32(np.sin(phi))
    tu = 32
    u0, v0 = int(rng.integers(0, max(1, nu // tu))) * tu, int(rng.integers(0, max(1, nv // 8))) * 8
    u1, v1 = min(u0 + tu, nu) - 1, min(v0 + 8, nv) - 1
    cu = (f32(0.5) * f32(u0 + u1) - uc) * du
    cx, cy = al * fdd - cu * be, be * fdd + cu * al
    xm = abs(cx) >= abs(cy)
    up = (cx if xm else cy) > 0
    xs, ys = xc - fod * al, xc - fod * be
    ms, ts = (xs, ys) if xm else (ys, xs)
    st, sz, along = [], [], True
    for uu in (u0, u1):
        d = (f32(uu) - uc) * du
        dxr, dyr = al * fdd - d * be, be * fdd + d * al
        dm = dxr if xm else dyr
        along &= bool((dm if up else -dm) > f32(0.25) * fdd)
        st.append((dyr if xm else dxr) / dm)
        sz += [(f32(v0) - vc) * du / dm, (f32(v1) - vc) * du / dm]
    st, sz = (min(st), max(st)), (min(sz), max(sz))
    if not along:
        return 0
    # the rays: entry at the volume's box (any entry on the ray's line serves the purpose)
    u, v = np.meshgrid(np.arange(u0, u1 + 1), np.arange(v0, v1 + 1))
    uu, vv = (u.ravel().astype(f32) - uc) * du, (v.ravel().astype(f32) - vc) * du
    dx, dy = al * fdd - uu * be, be * fdd + uu * al
    inv = f32(1) / np.sqrt(dx * dx + dy * dy + vv * vv)
    S = np.stack([dx * inv, dy * inv, vv * inv]).astype(f32)
    o = np.array([xs, ys, zc], np.float64)[:, None]
    lim = np.array([n - 1, n - 1, nz - 1], np.float64)[:, None]
    with np.errstate(divide="ignore", invalid="ignore"):
        a, b = (0 - o) / S, (lim - o) / S
    l0, l1 = np.nanmax(np.minimum(a, b), 0), np.nanmin(np.maximum(a, b), 0)
    P = (o + l0 * S).astype(f32)
    cnt = np.where(l1 > l0, np.floor(l1 - l0), 0).astype(int)
    im, it = (0, 1) if xm else (1, 0)
    end = P + (cnt - 1).astype(f32) * S
    top = f32(n)

    def between(q):
        e = q[im] - ms
        ok = True
        for k, c, s in ((it, ts, st), (2, zc, sz)):
            x, y = e * f32(s[0]), e * f32(s[1])
            ok = ok & (q[k] >= c + np.minimum(x, y) - f32(0.05)) & (q[k] <= c + np.maximum(x, y) + f32(0.05))
        return ok

    sm = S[im] if up else -S[im]
    mn, mx = np.minimum(P[im], end[im]), np.maximum(P[im], end[im])
    ray = (cnt > 0) & (sm > f32(0.25)) & (mn >= f32(-1.5)) & (mx <= top + f32(0.5)) & between(P) & between(end)
    if not ray.any():
        return 0
    lo, hi = int(np.floor(mn[ray] - f32(0.15)).min()), int(np.floor(mx[ray] + f32(0.15)).max())
    big = f32(max(n, nz) + 2)
    pad = f32(0.1) + f32(3) * big * big * f32(2.98023224e-8)
    inv_s = f32(1) / np.abs(S[im])
    pos, rem = P.copy(), np.where(ray, cnt, 0)
    cur = lo if up else hi
    while cur <= hi if up else cur >= lo:
        C = min(int(rng.integers(1, 31)), hi - cur + 1 if up else cur - lo + 1)
        ma = cur if up else cur - C + 1
        e = np.array([ma - 0.15, ma + C + 0.15], f32) - ms
        win = []
        for c, s in ((ts, st), (zc, sz)):
            x = np.concatenate([e * f32(s[0]), e * f32(s[1])])
            win.append((int(np.floor(c + x.min() - pad)), int(np.floor(c + x.max() + pad)) + 1))
        plane0 = ma - 1 if up else ma
        edge = f32(ma + C if up else ma)
        dist = (edge - pos[im] if up else pos[im] - edge) - f32(0.1)
        k = np.where(dist > 0, np.minimum(rem, (dist * inv_s).astype(int) + 1), 0)
        rem = rem - k
        for j in range(int(k.max())):
            live = j < k
            f = np.floor(pos)[:, live].astype(int)
            assert f[im].min() >= plane0 and f[im].max() <= plane0 + C
            assert f[it].min() >= win[0][0] and f[it].max() + 1 <= win[0][1]
            assert f[2].min() >= win[1][0] and f[2].max() + 1 <= win[1][1]
            pos = np.where(live, pos + S, pos)
        cur += C if up else -C
    assert (rem == 0).all()  # nothing is left after the last chunk
    return int(ray.sum())


@pytest.mark.parametrize("n,nz,tiles", [(17, 9, 150), (64, 64, 60), (211, 173, 25), (512, 512, 10), (1024, 600, 4)])
def test_every_staged_footprint_lies_in_its_window(n, nz, tiles):
    rng = np.random.default_rng(n)
    staged = sum(_march(rng, n, nz) for _ in range(tiles))
    assert staged > 20 * tiles
