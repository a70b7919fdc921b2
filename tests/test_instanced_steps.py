"""Closest-hit queries of instanced scenes: a warp takes one kind of traversal step at a time, so a ray pauses while
its neighbours step.  What a ray hits must not depend on its neighbours: crops of a frame, one pixel wide (few
lanes of a warp hold rays, of every kind of step) or ragged, equal the whole frame's pixels.  Paths of a pixel
draw the same samples in both; only the order of the pixel's FP64 sums may differ (spp terms: rtol 1e-12)."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("instances,prototypes", [(1, 1), (3, 2), (24, 4), (200, 8)])
def test_hits_do_not_depend_on_the_warp(ctx, instances, prototypes):
    import keepsake_b200 as ks
    W, H = 67, 41
    g = ks.Generated("instanced", 5, sky=(64, 32), resolution=(W, H), prototypes=prototypes, instances=instances,
                     frequency=6, emitters=8)
    s = ks.Scene(ctx, g.desc, keepalive=g)
    s.build_bvh()
    cam = ks.camera_perspective(g.camera_to_world, g.vfov, W / H)

    def render(**crop):
        return s.render(cam, ks.SmallPTParams.make(render_width=W, render_height=H, spp=4, bounces=6,
                                                   clamp_indirect=0.0, **crop))

    whole, weights = render()
    assert (weights.sum(-1) == 4).all()
    for x, y, w, h in ((0, 0, 1, 1), (33, 0, 1, H), (66, 40, 1, 1), (5, 7, 31, 3), (0, 20, W, 1)):
        a, n = render(crop_start_x=x, crop_start_y=y, crop_width=w, crop_height=h)
        got, count = (a, n) if a.shape == (h, w, 3) else (a[y:y + h, x:x + w], n[y:y + h, x:x + w])
        assert np.array_equal(count, weights[y:y + h, x:x + w]), (x, y)
        assert np.allclose(got, whole[y:y + h, x:x + w], rtol=1e-12, atol=0), (x, y)
    s.close()
