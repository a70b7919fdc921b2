"""Scenes with both simple materials (constant GGX principled ones) and general ones (other BSDFs,
textures): their hits go to two queues and two shading kernels.  The same scene with a constant
one-texel texture on every simple material (the same value, so the same image) has general materials
only and one queue; the two renders agree within the tolerance of same-seed renders by different
shading code (tests/test_render.py: relMSE 2e-3, median relative difference 1e-4), with equal weights."""
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
