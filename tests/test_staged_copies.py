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
