"""Flat scenes whose trees are deep.  Beside a small room stands geometry that makes the tree deep with 2
buckets: nested clusters, each twice as far as the last (one binary level for every level of the 4-wide
view when that opens the largest child first: more levels than the stack holds, although the binary tree
has at most 64), or a chain (more than 64 binary levels: the exact traversal).  A step reads one whole
128-byte node either way.  Images equal those of an ordinary tree of the same scene but for ties (fewer
than one ray in a thousand, see the hit-id tests: at 4 samples of some 20 rays a pixel, below 8 % of the
pixels)."""
import numpy as np
import pytest

import scenes

W, H, SPP = 48, 36, 4


def clusters(n, seed=1):
    rng = np.random.default_rng(seed)
    v = []
    for k in range(30 - n, 30):  # up to 2^29: larger triangles overflow the shading's float32
        s = 2.0 ** k
        c = rng.uniform(-1, 1, (12, 1, 3)) * s * np.array([0.2, 0.45, 0.45]) + np.array([0.75 * s, -2, 0])
        v.append((c + rng.uniform(-0.03, 0.03, (12, 3, 3)) * s).reshape(-1, 3))
    v = np.concatenate(v).astype(np.float32)
    return v, np.arange(len(v), dtype=np.uint32).reshape(-1, 3)


def greedy_levels(tree):
    """Levels of the 4-wide view that opens the largest interior child until there are 4."""
    right, b = tree["right"], tree["bounds"].astype(np.float64)
    e = b[:, 3:] - b[:, :3]
    area = e[:, 0] * e[:, 1] + e[:, 1] * e[:, 2] + e[:, 2] * e[:, 0]
    levels, level = 0, [0]
    while level:
        levels += 1
        below = []
        for i in level:
            c = [i + 1, int(right[i])]
            while len(c) < 4:
                inner = [k for k in c if right[k] != 0]
                if not inner:
                    break
                k = max(inner, key=lambda k: area[k])
                c.remove(k)
                c += [k + 1, int(right[k])]
            below += [k for k in c if right[k] != 0]
        level = below
    return levels


def scene(ks, kind, opacity=False):
    g = ks.Generated("box_room", 0)
    meshes = [[m["vertices"].copy(), m["indices"], m["material"], dict(twosided=m["twosided"])] for m in g.meshes]
    for k in (5, 6):  # the boxes, off the floor: no face in the floor's plane
        meshes[k][0][:, 1] += np.float32(1e-3)
    mats = list(g.materials)
    if kind == "clusters":
        v, idx = clusters(45)
    else:
        v, idx = scenes.deep_chain(200, -100)
        v[:, 1] += np.float32(1000.0)
    meshes.append([v, idx, 0, dict(twosided=1)])
    keep = [g]
    if opacity:
        mats.append(ks.MaterialDesc((0.7, 0.6, 0.5), 0.8, 0.0, 1.5, 0.5, 0.0, 0.0, 0.5, (0, 0, 0), 0, 0, (0, 0, 0)))
        pane = np.array([[-0.8, 0.3, 0.7], [0.8, 0.3, 0.7], [0.8, 1.7, 0.7], [-0.8, 1.7, 0.7]], np.float32)
        meshes.append([pane, np.array([[0, 1, 2], [0, 2, 3]], np.uint32), len(mats) - 1,
                       dict(twosided=1, texcoords=np.array([[0, 0], [1, 0], [1, 1], [0, 1]], np.float32))])
    desc, alive = ks.scene_desc(meshes, mats, g.desc.contents.sky)
    if opacity:
        ys, xs = np.mgrid[0:16, 0:16]
        mask = (((xs // 4 + ys // 4) % 3) * 0.5).astype(np.float32)[..., None]
        alive += ks.attach_textures(desc, [(mask, False)], [ks.TextureBinding.make(len(mats) - 1, "opacity_map", 0, filter=0)])
    return g, desc, keep + alive


def params(ks, **kw):
    size = dict(render_width=W, render_height=H, spp=SPP, bounces=5, clamp_indirect=0.0)
    size.update(kw)
    return ks.SmallPTParams.make(**size)


def same_but_for_ties(a, b):
    (x, wx), (y, wy) = a, b
    assert np.array_equal(wx, wy)
    off = (np.abs(x - y) > 1e-9 * (np.abs(x) + np.abs(y))).any(-1)
    assert off.mean() < 0.08, off.mean()
    assert abs(x.sum() - y.sum()) < 0.02 * y.sum()


def build(ks, ctx, kind, opacity=False, **options):
    g, desc, keep = scene(ks, kind, opacity)
    s = ks.Scene(ctx, desc, keepalive=keep)
    s.build_bvh(**options)
    return s, ks.camera_perspective(g.camera_to_world, g.vfov, W / H)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["clusters", "chain"])
def test_the_trees_are_deep(ctx, kind):
    import keepsake_b200 as ks
    s, _ = build(ks, ctx, kind, buckets=2, max_prims=1)
    tree = s.export_sbvh()
    s.close()
    depth = scenes.sbvh_depth(tree["right"])
    if kind == "clusters":
        assert depth <= 64 and greedy_levels(tree) > 32
    else:
        assert depth > 64


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["clusters", "chain"])
@pytest.mark.parametrize("opacity", [False, True])
def test_images(ctx, kind, opacity):
    import keepsake_b200 as ks
    s, cam = build(ks, ctx, kind, opacity, buckets=2, max_prims=1)
    deep = s.render(cam, params(ks))
    s.build_bvh(buckets=16)
    ordinary = s.render(cam, params(ks))
    s.close()
    assert deep[0].sum() > 0
    same_but_for_ties(deep, ordinary)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["clusters", "chain"])
def test_a_step_reads_one_whole_node(ctx, kind):
    import keepsake_b200 as ks
    s, cam = build(ks, ctx, kind, buckets=2, max_prims=1)
    counts = []
    for k in range(24):  # one ray each
        s.render(cam, params(ks, spp=1, bounces=0, crop_start_x=2 * k, crop_start_y=k, crop_width=1, crop_height=1))
        assert s.stats().extension_rays == 1
        counts.append(s.stats().ext_nodes)
    s.close()
    assert max(counts) > 0 and all(c % 2 == 0 for c in counts), counts  # 64-byte units


@pytest.mark.gpu
@pytest.mark.parametrize("use_graph", [False, True])
def test_a_batch_with_deep_trees(ctx, use_graph):
    import torch

    import keepsake_b200 as ks
    made = [build(ks, ctx, kind, buckets=buckets, max_prims=1)
            for kind, buckets in (("chain", 2), ("clusters", 16), ("clusters", 2), ("chain", 2))]
    jobs, images = [], []
    for k, (s, cam) in enumerate(made):
        acc = torch.zeros((H, W, 3), dtype=torch.float64, device="cuda")
        wts = torch.zeros((H, W, 2), dtype=torch.float64, device="cuda")
        jobs.append((s, cam, params(ks, rng_seed=k), acc, wts))
    torch.cuda.synchronize()
    ks.batch_render(ctx, [(s, c, p, a.data_ptr(), w.data_ptr()) for s, c, p, a, w in jobs], use_graph=use_graph)
    images = [(a.cpu().numpy(), w.cpu().numpy()) for *_, a, w in jobs]
    for (s, cam, p, *_), (a, w) in zip(jobs, images):
        alone, weights = s.render(cam, p)
        # the same paths: sums differ by the order of their FP64 additions
        assert np.array_equal(w, weights) and np.allclose(a, alone, rtol=1e-12, atol=0)
    for s, _ in made:
        s.close()
