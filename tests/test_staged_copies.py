"""Host arrays of the guide's entry points go through pinned memory in pieces, downloads above 1 MB and uploads
above 32 MB: what comes back is what was sent, whole and at sizes around the pieces' edges, and rows do not depend on how many are
sent together (each row of the network is computed by itself)."""
import numpy as np
import pytest

BOUND = [-1.0, -1.0, -1.0, 1.0, 1.0, 1.0]


@pytest.mark.gpu
def test_weights_round_trip(ctx):
    import keepsake_b200 as ks
    rng = np.random.default_rng(0)
    w = rng.standard_normal(ks.GUIDE_WEIGHTS).astype(np.float32)
    grid = rng.standard_normal((ks.GUIDE_LEVELS, ks.GUIDE_TABLE_SIZE, 2)).astype(np.float32)  # 64 MB: one part
    guide = ks.Guide(ctx, BOUND)
    guide.set_weights(w, grid)
    w1, grid1 = guide.get_weights()
    assert np.array_equal(w, w1) and np.array_equal(grid, grid1)
    guide.close()


@pytest.mark.gpu
# rows of 12 bytes up and 164 bytes down: below, at and above 1 MB either way, and above 64 MB down
@pytest.mark.parametrize("n", [1, 6393, 6394, 87381, 87382, 420001])
def test_rows_are_independent_of_their_number(ctx, n):
    import keepsake_b200 as ks
    rng = np.random.default_rng(n)
    pos = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    wo, normal = (rng.standard_normal((n, 3)).astype(np.float32) for _ in range(2))
    guide = ks.Guide(ctx, BOUND)
    whole = guide.infer(pos, wo, normal)
    at = sorted({0, n // 2, max(0, n - 128)})
    for k in at:
        part = guide.infer(pos[k:k + 128], wo[k:k + 128], normal[k:k + 128])
        assert np.array_equal(whole[k:k + 128], part)
    guide.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2796202, 2796203])  # rows of 12 bytes up: below and above 32 MB
def test_large_uploads(ctx, n):
    import keepsake_b200 as ks
    rng = np.random.default_rng(n)
    pos, wo, normal = (rng.standard_normal((n, 3), dtype=np.float32) for _ in range(3))
    guide = ks.Guide(ctx, BOUND)
    whole = guide.infer(pos, wo, normal)
    for k in (0, n // 2, n - 128):
        assert np.array_equal(whole[k:k + 128], guide.infer(pos[k:k + 128], wo[k:k + 128], normal[k:k + 128]))
    guide.close()


@pytest.mark.gpu
def test_pinned_arrays_go_straight(ctx):
    """Memory that the caller pinned takes no detour: 64 MB up or down in well below the time of pageable memory
    (about 2.4 times as long; through the stage both took the same)."""
    import time

    import torch

    import keepsake_b200 as ks
    guide = ks.Guide(ctx, BOUND)
    w, grid = guide.get_weights()
    pinned = torch.empty(grid.shape, dtype=torch.float32, pin_memory=True).numpy()
    pinned[:] = np.random.default_rng(1).standard_normal(grid.shape, dtype=np.float32)
    fn = ks.lib.ks_guide_get_weights

    def best(f):
        times = []
        for _ in range(8):
            t = time.perf_counter()
            f()
            times.append(time.perf_counter() - t)
        return min(times)

    up = [best(lambda a=a: guide.set_weights(w, a)) for a in (grid, pinned)]
    guide.set_weights(w, pinned)
    assert np.array_equal(guide.get_weights()[1], pinned)
    pinned[:] = 0.0
    down = [best(lambda a=a: ctx.check(fn(guide.handle, None, ks.ptr(a)), "get")) for a in (grid, pinned)]
    assert np.array_equal(grid, pinned) and pinned.any()
    guide.close()
    assert up[1] < 0.7 * up[0], up
    assert down[1] < 0.9 * down[0], down
