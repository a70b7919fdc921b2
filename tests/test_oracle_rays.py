"""The CPU oracle loads on every machine, and its ray queries (the reference's SBVH, or the oracle's own
tree where that is not built) hit and miss as a search of all triangles in float64 says, at the distance
that the closest of the triangles has when each is a scene of its own.

Where two triangles lie within rounding of each other on a ray either may be kept: distances then agree
within 8 ulp (the bound of the hit-id tests).  The float64 search leaves out rays that pass a triangle's
edge at less than 1e-5 in barycentrics: there float32 may decide either way."""
import numpy as np
import pytest

import scenes

MISS = 0xFFFFFFFF


def rays(v, idx, n, seed):
    rng = np.random.default_rng(seed)
    axis = scenes.random_rays(v, n, seed + 2)
    axis[:, 4:7] = 0.0
    axis[np.arange(n), 4 + rng.integers(0, 3, n)] = np.where(rng.random(n) < 0.5, 1.0, -1.0)
    axis[: n // 2, 0:3] = v[idx[rng.integers(0, len(idx), n // 2), 0]]  # on the boxes' planes
    axis[: n // 4, 4:7][axis[: n // 4, 4:7] == 0] = -0.0
    ranged = scenes.random_rays(v, n, seed + 3)
    ranged[:, 7] = rng.random(n) * np.ptp(v) * 0.3
    return np.concatenate([scenes.random_rays(v, n, seed), scenes.rays_at_triangles(v, idx, n, seed + 1), axis,
                           ranged]).astype(np.float32)


def search(v, idx, r):
    """Whether some triangle is hit, in float64, and whether an edge or an end of the range is near."""
    o, d, lo, hi = r[:, None, 0:3].astype(np.float64), r[:, None, 4:7].astype(np.float64), r[:, 3:4], r[:, 7:8]
    p = v[idx].astype(np.float64)
    e1, e2 = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    with np.errstate(all="ignore"):
        q = np.cross(d, e2[None])
        det = (e1[None] * q).sum(-1)
        s = o - p[None, :, 0]
        b1 = (s * q).sum(-1) / det
        c = np.cross(s, e1[None])
        b2 = (d * c).sum(-1) / det
        t = (e2[None] * c).sum(-1) / det
        inside = np.minimum(np.minimum(b1, b2), 1 - b1 - b2)
        near = (np.abs(inside) < 1e-5) | (np.abs(det) < 1e-9)
        near |= (inside > 0) & ((np.abs(t - lo) < 1e-5) | (np.abs(t - hi) < 1e-5 * np.abs(t)))
        hit = (inside > 0) & (t > lo) & (t < hi)
    return hit.any(1), near.any(1)


@pytest.mark.parametrize("n", [1, 5, 700])
def test_oracle_rays_against_a_search(oracle, n):
    import keepsake_b200 as ks
    v, idx = scenes.soup(n, seed=n, spread=1.0 if n < 10 else 4.0)
    desc, keep = ks.triangle_soup_desc(v, idx)
    s = oracle.scene(desc, keep)
    r = rays(v, np.asarray(idx), 500, 7)
    hit, near = search(v, idx, r)
    tri, t, _ = s.trace(r)
    occluded, _, _ = s.trace(r, any_hit=True)
    assert np.array_equal((tri != MISS)[~near], hit[~near]) and np.array_equal(occluded[~near], hit[~near])
    assert near.mean() < 0.5 and (n == 1 or (hit & ~near).any())
    closest = np.full(len(r), np.inf)
    for k in range(n):
        one, alive = ks.triangle_soup_desc(v, idx[k:k + 1])
        found, dist, _ = oracle.scene(one, alive).trace(r)
        closest = np.where(found != MISS, np.minimum(closest, dist), closest)
    assert np.array_equal(np.isfinite(closest), tri != MISS) and np.array_equal(occluded, tri != MISS)
    got = tri != MISS
    assert (np.abs(t[got] - closest[got]) <= 8 * 2.0 ** -23 * closest[got]).all()
