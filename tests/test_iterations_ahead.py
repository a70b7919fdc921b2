"""The render loop launches an iteration before it has read the last one's count.  What a caller can see of
that must not differ from reading each: the iteration limit is exact, the counts of rays are those of the
iterations that had paths, and the next pass starts from an empty queue.  The sizes lie on both sides of
the queue length (32768) from which rays are traced by another kernel, which the device then chooses."""
import numpy as np
import pytest

KS_ERR_WATCHDOG = 5


@pytest.mark.gpu
@pytest.mark.parametrize("width,height,spp,bounces", [(1, 1, 1, 0), (33, 31, 4, 8), (181, 181, 1, 3), (257, 129, 4, 8)])
def test_iteration_limit_is_exact(ctx, width, height, spp, bounces):
    import keepsake_b200 as ks
    g = ks.Generated("box_room", 0)
    cam = ks.camera_perspective(g.camera_to_world, g.vfov, width / height)
    s = ks.Scene(ctx, g.desc)
    s.build_bvh()
    p = ks.SmallPTParams.make(render_width=width, render_height=height, spp=spp, bounces=bounces, clamp_indirect=0.0)
    a, w = s.render(cam, p)
    want = s.stats()
    n = want.iterations
    assert 1 <= n <= bounces + 1 and (w.sum(-1) == spp).all()
    try:
        ctx.set_limits(wavefront_max_iterations=n)
        b, w2 = s.render(cam, p)
        got = s.stats()
        if n > 1:
            ctx.set_limits(wavefront_max_iterations=n - 1)
            with pytest.raises(ks.KsError) as e:
                s.render(cam, p)
            assert e.value.status == KS_ERR_WATCHDOG
    finally:
        ctx.set_limits()
    assert np.array_equal(a, b) and np.array_equal(w, w2)
    for k in ("iterations", "paths", "extension_rays", "shadow_rays"):
        assert getattr(got, k) == getattr(want, k), k
    # passes of one sample each: as many rays, and the same sums up to their order in 64 bits
    p.spp_prog_interval = 1
    c, w3 = s.render(cam, p)
    split = s.stats()
    assert np.array_equal(w, w3) and np.allclose(a, c, rtol=1e-12, atol=0)
    assert split.extension_rays == want.extension_rays and split.shadow_rays == want.shadow_rays
    assert n <= split.iterations <= n * spp
    s.close()
