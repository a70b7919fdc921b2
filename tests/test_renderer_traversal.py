"""The renderer's traversal (ks_trace_rays_wide: the 4-wide view, conservative box tests, leaves checked
when a triangle is hit) against the reference-order binary traversal (ks_trace_rays) on the same
device, over trees of one leaf, a few and many nodes, duplicated and flat triangles, and rays with
zero components, finite and negative ranges, unnormalised directions.

Occlusion does not depend on the visiting order, so it is equal for every ray.  The closest hit is
equal bit for bit unless two triangles lie within rounding of each other on the ray; then the two
orders may keep different ones, whose distances agree within 8 ulp (the bound of the hit-id tests)
or, for hits whose computed distance lies before their leaf's entry, one part in 2^12."""
import numpy as np
import pytest

import scenes


def rays(v, idx, n, seed):
    rng = np.random.default_rng(seed)
    a = scenes.random_rays(v, n, seed)
    b = scenes.rays_at_triangles(v, idx, n, seed + 1)
    axis = scenes.random_rays(v, n, seed + 2)
    axis[:, 4:7] = 0.0
    axis[np.arange(n), 4 + rng.integers(0, 3, n)] = np.where(rng.random(n) < 0.5, 1.0, -1.0)
    axis[: n // 2, 0:3] = v[idx[rng.integers(0, len(idx), n // 2), 0]]  # from vertices: on the boxes' planes
    ranged = scenes.random_rays(v, n, seed + 3)
    ranged[:, 3] = rng.normal(size=n) * 0.2
    ranged[:, 7] = rng.random(n) * np.ptp(v) * 0.3
    scaled = scenes.random_rays(v, n, seed + 4)
    scaled[:, 4:7] *= rng.choice([1e-3, 37.0], size=(n, 1))
    scaled[: n // 2, 4] = -0.0
    return np.concatenate([a, b, axis, ranged, scaled]).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,n", [("one", 1), ("leaf", 4), ("small", 9), ("soup", 3000), ("flat", 0), ("copies", 400)])
@pytest.mark.parametrize("culling", [2, 0])
def test_wide_traversal_matches_binary(ctx, kind, n, culling):
    import keepsake_b200 as ks
    if kind == "flat":
        v, idx = scenes.degenerate_soup(2)
    else:
        v, idx = scenes.soup(n, seed=n, spread=1.0 if n < 10 else 6.0)
    if kind == "copies":
        v, idx = np.concatenate([v, v]), np.concatenate([idx, idx + len(v)])
    desc, keep = ks.triangle_soup_desc(v, idx)
    s = ks.Scene(ctx, desc, keep)
    s.build_bvh()
    r = rays(v, np.asarray(idx), 20000, 3)
    assert np.array_equal(s.trace(r, any_hit=True, culling=culling, wide=True)[0],
                          s.trace(r, any_hit=True, culling=culling)[0])
    tri, t, bary = s.trace(r, culling=culling, wide=True)
    tri0, t0, bary0 = s.trace(r, culling=culling)
    assert np.array_equal(tri == 0xFFFFFFFF, tri0 == 0xFFFFFFFF)
    same = tri == tri0
    assert np.array_equal(t[same], t0[same]) and np.array_equal(bary[same], bary0[same])
    off = np.abs(t[~same].astype(np.float64) - t0[~same]) / np.abs(t0[~same])
    assert (off <= 2.0 ** -12).all()
    if kind not in ("flat", "copies"):  # no coplanar or repeated triangles: ties are rare
        assert (~same).mean() < 1e-3 and (off <= 8 * 2.0 ** -23).all()
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("W,H", [(1, 1), (181, 181), (182, 182), (600, 400)])
@pytest.mark.parametrize("batch", [False, True])
def test_short_queues_render_the_same(ctx, W, H, batch):
    """Queues of up to 2^15 rays are traced by groups of lanes, longer ones by a lane per ray: a frame
    rendered whole equals, pixel by pixel, the same frame rendered in crops whose queues are shorter
    (181 x 181 is the largest square below the limit, 182 x 182 the first above it).  Both ways make the
    same tests, so the sums differ by the order of FP64 additions only."""
    import torch

    import keepsake_b200 as ks
    g = ks.Generated("icosphere", 3, level=5, sky=(128, 64), resolution=(W, H))
    s = ks.Scene(ctx, g.desc)
    s.build_bvh()
    cam = ks.camera_perspective(g.camera_to_world, g.vfov, g.aspect)
    size = dict(render_width=W, render_height=H, spp=1, bounces=6)

    def render(**crop):
        acc = torch.zeros((H, W, 3), dtype=torch.float64, device="cuda")
        wts = torch.zeros((H, W, 2), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        p = ks.SmallPTParams.make(**size, **crop)
        if batch:
            ks.batch_render(ctx, [(s, cam, p, acc.data_ptr(), wts.data_ptr())])
        else:
            s.render_device(cam, p, acc.data_ptr(), wts.data_ptr())
        return acc.cpu().numpy(), wts.cpu().numpy()

    acc, wts = render()
    rows = max(1, 8192 // W)
    acc_c, wts_c = np.zeros_like(acc), np.zeros_like(wts)
    for y in range(0, H, rows):
        a, w = render(crop_start_x=0, crop_start_y=y, crop_width=W, crop_height=min(rows, H - y))
        acc_c += a
        wts_c += w
    assert np.array_equal(wts, wts_c)
    assert np.allclose(acc, acc_c, rtol=1e-14, atol=0)
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("max_prims", [1, 4])
def test_hits_just_within_the_range(ctx, max_prims):
    """Rays that end within 8 ulp beyond a hit: flat triangles across the axes, so that their boxes are entered at
    the hit's distance, each in a plane of its own (no ties), among triangles that are passed by.  Axis rays
    from points with few bits meet the planes exactly; oblique ones start at 0, where the box test's
    padding by the origin vanishes."""
    import keepsake_b200 as ks
    rng = np.random.default_rng(5)
    n, m = 240, 4000
    axis, plane = np.arange(n) % 3, (1 + rng.permutation(n)).astype(np.float32) / 64
    v = rng.integers(-256, 257, (n, 3, 3)).astype(np.float32) / 64
    v[np.arange(n), :, axis] = plane[:, None]
    desc, keep = ks.triangle_soup_desc(v.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3))
    s = ks.Scene(ctx, desc, keep)
    s.build_bvh(max_prims=max_prims)
    r = np.zeros((2 * m, 8), np.float32)
    r[:m, 0:3] = rng.integers(-200, 200, (m, 3)) / 64 + 1 / 256
    k = rng.integers(0, 3, m)
    r[np.arange(m), k] = 0.0
    r[np.arange(m), 4 + k] = 1.0
    r[m:, 4:7] = np.abs(rng.normal(size=(m, 3))) + 1e-3
    r[:, 7] = np.inf
    tri0, t0, _ = s.trace(r)
    r = r[tri0 != 0xFFFFFFFF]
    t0 = t0[tri0 != 0xFFFFFFFF]
    assert len(r) > m // 2
    end = t0
    hits = []
    for ulp in range(0, 9):
        r[:, 7] = end
        tri, t, _ = s.trace(r)
        wtri, wt, _ = s.trace(r, wide=True)
        assert np.array_equal(tri, wtri) and np.array_equal(t[tri != 0xFFFFFFFF], wt[tri != 0xFFFFFFFF]), ulp
        assert np.array_equal(s.trace(r, any_hit=True)[0], s.trace(r, any_hit=True, wide=True)[0]), ulp
        end = np.nextafter(end, np.float32(np.inf))
        hits.append((tri != 0xFFFFFFFF).sum())
    assert hits[0] < hits[-1]  # the sweep crosses the ends that matter
    s.close()
