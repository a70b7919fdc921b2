"""Scenes with both simple materials (constant GGX principled ones) and general ones (other BSDFs,
textures): their hits go to two queues and two shading kernels.  The same scene with a constant
one-texel texture on every simple material (the same value, so the same image) has general materials
only and one queue; the two renders agree within the tolerance of same-seed renders by different
shading code (tests/test_render.py: relMSE 2e-3, median relative difference 1e-4), with equal weights.
So do guided renders (the guide reads the hits' common queue) and renders of instanced scenes."""
import numpy as np
import pytest

from imaging import composite, rel_mse


def room(ks, all_general, general):
    g = ks.Generated("box_room", 0)
    d = g.desc.contents
    textures, bindings = [], []
    for m in general:
        d.materials[m].bsdf, d.materials[m].specular = 1, 0.6
    if all_general:
        for m in range(d.n_materials):
            if m not in general:
                textures.append((np.array([[list(d.materials[m].basecolor)]], np.float32), False))
                bindings.append(ks.TextureBinding.make(m, "basecolor", len(textures) - 1, filter=0))
    keep = ks.attach_textures(g.desc, textures, bindings) if textures else None
    return g, keep


@pytest.mark.gpu
@pytest.mark.parametrize("general", [(5,), (0, 2, 5, 6)])
@pytest.mark.parametrize("batch", [False, True])
def test_split_hit_queues(ctx, general, batch):
    import torch

    import keepsake_b200 as ks
    W, H = 67, 45
    images = []
    for all_general in (False, True):
        g, keep = room(ks, all_general, general)
        s = ks.Scene(ctx, g.desc, keepalive=(g, keep))
        s.build_bvh()
        cam = ks.camera_perspective(g.camera_to_world, g.vfov, W / H)
        p = ks.SmallPTParams.make(render_width=W, render_height=H, spp=16, bounces=6, clamp_indirect=0.0)
        acc = torch.zeros((H, W, 3), dtype=torch.float64, device="cuda")
        wts = torch.zeros((H, W, 2), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        if batch:
            ks.batch_render(ctx, [(s, cam, p, acc.data_ptr(), wts.data_ptr())])
        else:
            s.render_device(cam, p, acc.data_ptr(), wts.data_ptr())
        images.append((acc.cpu().numpy(), wts.cpu().numpy()))
        s.close()
    (a, wa), (b, wb) = images
    assert np.array_equal(wa, wb) and (wa.sum(-1) == 16).all()
    x, y = composite(a, wa), composite(b, wb)
    assert rel_mse(x, y) < 2e-3
    assert np.median(np.abs(x - y) / (np.abs(y) + 1e-3)) < 1e-4


def agree(images):
    (a, wa), (b, wb) = images
    assert np.array_equal(wa, wb) and (wa.sum(-1) == 16).all()
    x, y = composite(a, wa), composite(b, wb)
    assert rel_mse(x, y) < 2e-3
    assert np.median(np.abs(x - y) / (np.abs(y) + 1e-3)) < 1e-4


@pytest.mark.gpu
def test_split_hit_queues_guided(ctx):
    import torch

    import keepsake_b200 as ks
    W, H = 67, 45
    images = []
    for all_general in (False, True):
        g, keep = room(ks, all_general, (0, 2, 5, 6))
        s = ks.Scene(ctx, g.desc, keepalive=(g, keep))
        s.build_bvh()
        cam = ks.camera_perspective(g.camera_to_world, g.vfov, W / H)
        p = ks.SmallPTParams.make(render_width=W, render_height=H, spp=16, bounces=6, clamp_indirect=0.0,
                                  spp_prog_interval=4)
        guide = ks.Guide(ctx, [-1.1, -0.1, -1.1, 1.1, 2.1, 1.1], seed=3)  # untrained and kept fixed
        acc = torch.zeros((H, W, 3), dtype=torch.float64, device="cuda")
        wts = torch.zeros((H, W, 2), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        s.render_guided_device(cam, p, guide, ks.GuideRenderOptions.make(train_passes=0, guide_from_pass=0),
                               acc.data_ptr(), wts.data_ptr())
        assert s.stats().guide_rows > 0
        images.append((acc.cpu().numpy(), wts.cpu().numpy()))
        guide.close()
        s.close()
    agree(images)


@pytest.mark.gpu
def test_split_hit_queues_instanced(ctx):
    import keepsake_b200 as ks
    W, H = 67, 45
    images = []
    for all_general in (False, True):
        g = ks.Generated("instanced", 5, sky=(64, 32), resolution=(W, H), prototypes=3, instances=24, frequency=6,
                         emitters=8)
        d = g.desc.contents
        plain = [m for m in range(d.n_materials) if not d.materials[m].has_emission]
        for m in plain[::2]:
            d.materials[m].bsdf, d.materials[m].specular = 1, 0.6
        textures, bindings = [], []
        if all_general:
            for m in range(d.n_materials):
                if m not in plain[::2]:
                    textures.append((np.array([[list(d.materials[m].basecolor)]], np.float32), False))
                    bindings.append(ks.TextureBinding.make(m, "basecolor", len(textures) - 1, filter=0))
        keep = ks.attach_textures(g.desc, textures, bindings) if textures else None
        s = ks.Scene(ctx, g.desc, keepalive=(g, keep))
        s.build_bvh()
        cam = ks.camera_perspective(g.camera_to_world, g.vfov, W / H)
        images.append(s.render(cam, ks.SmallPTParams.make(render_width=W, render_height=H, spp=16, bounces=6,
                                                          clamp_indirect=0.0)))
        s.close()
    agree(images)
