"""Subsurface walks cast their rays through the 4-wide view; in a scene whose tree is too deep for the
view, through the binary tree.  One scene (a closed subsurface sphere over a floor, beside a far chain of
triangles that makes the tree deep with 2 buckets) is built with options that give trees of different
shape and depth: every ray has the same closest hit in all of them, up to ties (fewer than one ray in
a thousand, see the hit-id tests: at 4 samples of some 20 rays a pixel, below 8 % of the pixels), so the images are
equal but for those pixels."""
import numpy as np
import pytest

import scenes


def sphere(center, radius, n=24):
    th, ph = np.meshgrid(np.linspace(0, np.pi, n + 1), np.linspace(0, 2 * np.pi, 2 * n + 1), indexing="ij")
    v = np.stack([np.sin(th) * np.cos(ph), np.cos(th), np.sin(th) * np.sin(ph)], -1).reshape(-1, 3)
    row = 2 * n + 1
    q = [(i * row + j, i * row + j + 1, (i + 1) * row + j, (i + 1) * row + j + 1) for i in range(n) for j in range(2 * n)]
    idx = [t for a, b, c, d in q for t in ((a, b, d), (a, d, c))]
    return (np.asarray(center) + radius * v).astype(np.float32), np.array(idx, np.uint32)


def scene(ks, depth_of_medium):
    plain, medium = ks.MaterialDesc(), ks.MaterialDesc()
    for m in (plain, medium):
        m.basecolor[:] = (0.6, 0.5, 0.4)
        m.roughness, m.ior, m.specular_r0_mul, m.diffuse_trans_fwd = 1.0, 1.5, 0.5, 0.5
    medium.has_subsurface = 1
    medium.ss_albedo[:] = (0.9, 0.7, 0.5)
    medium.ss_radius[:] = (depth_of_medium, 0.5 * depth_of_medium, 0.3 * depth_of_medium)
    medium.ss_anisotropy, medium.ss_ior = 0.2, 1.4
    ball = sphere((0.0, 0.0, 0.0), 0.5)
    floor = (np.array([[-3, -0.6, -3], [3, -0.6, -3], [3, -0.6, 3], [-3, -0.6, 3]], np.float32),
             np.array([[0, 2, 1], [0, 3, 2]], np.uint32))
    cv, ci = scenes.deep_chain(200, -100)
    cv[:, 1] += np.float32(1000.0)
    meshes = [(ball[0], ball[1], 1, dict(twosided=0)), (floor[0], floor[1], 0, dict(twosided=1)),
              (cv, ci, 0, dict(twosided=1))]
    desc, keep = ks.scene_desc(meshes, [plain, medium])
    light = (ks.LightDesc * 1)()
    light[0].type = 0
    light[0].color[:] = (3.0, 3.0, 3.0)
    light[0].vec[:] = (0.3, 1.0, 0.4)
    desc.lights = light
    desc.n_lights = 1
    return desc, [keep, light, ball, floor, cv, ci]


@pytest.mark.gpu
@pytest.mark.parametrize("depth_of_medium", [0.05, 0.5])
def test_walks_do_not_depend_on_the_tree(ctx, depth_of_medium):
    import keepsake_b200 as ks
    W, H, spp = 48, 40, 4
    desc, keep = scene(ks, depth_of_medium)
    s = ks.Scene(ctx, desc, keep)
    c2w = np.array([[1, 0, 0, 0.0], [0, 1, 0, 0.1], [0, 0, 1, 1.6], [0, 0, 0, 1]], np.float32)
    cam = ks.camera_perspective(c2w, 0.9, W / H)
    p = ks.SmallPTParams.make(render_width=W, render_height=H, spp=spp, bounces=5, clamp_indirect=0.0)
    depths, images = [], []
    for opts in (dict(buckets=16), dict(buckets=7, max_prims=1), dict(buckets=2)):
        s.build_bvh(**opts)
        depths.append(scenes.sbvh_depth(s.export_sbvh()["right"]))
        images.append(s.render(cam, p))
    s.close()
    assert depths[0] <= 64 < depths[2], depths  # the 4-wide view, and the binary tree
    a, w = images[0]
    assert a[H // 2 - 4:H // 2 + 4, W // 2 - 4:W // 2 + 4].sum() > 0
    for b, w2 in images[1:]:
        assert np.array_equal(w, w2)
        off = (np.abs(a - b) > 1e-9 * (np.abs(a) + np.abs(b))).any(-1)
        assert off.mean() < 0.08, off.mean()
        assert abs(a.sum() - b.sum()) < 0.02 * a.sum()
