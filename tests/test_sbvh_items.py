"""SBVH builder: nodes whose references are one work item, exactly one, or one and a bit (256 references per item,
see KS_BUILD_CHUNK), and bucket counts up to the lanes that evaluate a node's splits (16, the most that a build
takes: more are clamped), against an object-split builder in NumPy fp32 (alpha = 1: no node overlaps more than
the root's area, so none is split spatially).
Trees are equal: same nodes in depth-first order, bounds, axes, offsets and leaf contents."""
import numpy as np
import pytest

import scenes

F = np.float32


def area(lo, hi):
    e = (hi - lo).astype(F)
    return F(2) * (e[..., 0] * e[..., 1] + e[..., 1] * e[..., 2] + e[..., 0] * e[..., 2])


def best_bucket(lo, hi, bucket, buckets, trav_weight):
    node_area = area(lo.min(0), hi.max(0))
    best, best_cost = 0, None
    for i in range(buckets - 1):
        side = bucket <= i
        terms = []
        for m in (side, ~side):
            if m.any():
                terms.append(F(m.sum()) * area(lo[m].min(0), hi[m].max(0)))
            else:
                terms.append(F(0) * F(np.inf))  # an empty side: 0 x the area of an empty box
        with np.errstate(invalid="ignore"):
            cost = F(trav_weight) + (terms[0] + terms[1]) / node_area
        if best_cost is None or cost < best_cost:
            best, best_cost = i, cost
    return best, best_cost


def object_tree(v, idx, max_prims, buckets, trav_weight):
    lo, hi = v[idx].min(1), v[idx].max(1)
    center = F(0.5) * (lo + hi)
    out = dict(bounds=[], axis=[], right=[], prim_offset=[], prims=[])

    def emit(ids):
        me = len(out["axis"])
        blo, bhi = lo[ids].min(0), hi[ids].max(0)
        cmin, cmax = center[ids].min(0), center[ids].max(0)
        out["bounds"].append(np.concatenate([blo, bhi]))
        out["axis"].append(0)
        out["right"].append(0)
        out["prim_offset"].append(len(out["prims"]))
        ext = cmax - cmin
        d = int(np.argmax(ext))  # the first of the largest
        if len(ids) > 1 and ext[d] > 0:
            b = np.minimum(np.floor(F(buckets) * ((center[ids, d] - cmin[d]) / ext[d])), buckets - 1).astype(np.int64)
            k, cost = best_bucket(lo[ids], hi[ids], b, buckets, trav_weight)
            if not (len(ids) <= max_prims and F(len(ids)) <= cost):
                out["axis"][me] = d
                emit(ids[b <= k])
                out["right"][me] = len(out["axis"])
                emit(ids[b > k])
                return
        out["prims"] += ids.tolist()

    emit(np.arange(len(idx)))
    return {k: np.array(x) for k, x in out.items()}


def check(ctx, n, buckets, seed, **kw):
    import keepsake_b200 as ks
    v, i = scenes.soup(n, seed=seed)
    d, keep = ks.triangle_soup_desc(v, i)
    s = ks.Scene(ctx, d, keep)
    opts = dict(max_prims=4, trav_weight=1.0)
    opts.update(kw)
    s.build_bvh(buckets=buckets, alpha=1.0, **opts)
    got = s.export_sbvh()
    ref = object_tree(np.asarray(v, F).reshape(-1, 3), np.asarray(i).reshape(-1, 3).astype(np.int64), buckets=buckets, **opts)
    s.close()
    interior = ref["right"] != 0
    assert np.array_equal(got["right"], ref["right"])
    assert np.array_equal(got["prim_offset"], ref["prim_offset"])
    assert np.array_equal(got["axis"][interior], ref["axis"][interior])
    assert np.array_equal(got["bounds"], ref["bounds"].astype(F))
    ends = np.append(ref["prim_offset"][1:], len(ref["prims"]))
    for k in np.nonzero(~interior)[0]:
        a = slice(ref["prim_offset"][k], ends[k])
        assert np.array_equal(np.sort(got["prims"][a]), np.sort(ref["prims"][a]))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 512, 513, 3000])
@pytest.mark.parametrize("buckets", [2, 12, 16])
def test_object_splits(ctx, n, buckets):
    check(ctx, n, buckets, seed=n + buckets)


@pytest.mark.gpu
def test_more_buckets_than_lanes(ctx):
    import keepsake_b200 as ks
    v, i = scenes.soup(700, seed=9, spread=3.0, size=1.5)  # overlapping: spatial splits too
    d, keep = ks.triangle_soup_desc(v, i)
    s = ks.Scene(ctx, d, keep)
    trees = []
    for buckets in (16, 17, 40):
        s.build_bvh(buckets=buckets)
        trees.append(s.export_sbvh())
    s.close()
    for t in trees[1:]:
        assert all(np.array_equal(t[k], trees[0][k]) for k in ("bounds", "axis", "right", "prim_offset"))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [257, 1025])
def test_object_splits_leaves(ctx, n):
    check(ctx, n, 7, seed=n, max_prims=1)
    check(ctx, n, 7, seed=n, max_prims=8, trav_weight=10.0)
