"""The framework's work, as a program that uses it has it do: what is timed, over which sizes.

A case is a render of one kind of scene (or, for `train`, a training batch of the guiding network)
through the package's public entry points.  Scenes are the seeded procedural ones of this package
and the small hand-made ones of its tests; a seed changes the geometry, the materials and the
sampler's random numbers.  Sizes run from a thumbnail of a few thousand paths, where the time is
launches and round trips, to a full frame of tens of millions of paths, with odd resolutions,
single-sample passes and many-sample intervals, 36 to 1.3 million triangles, and the scene features
that select other kernels: textures and opacity maps, smooth normals, transmission, subsurface
walks, instances, several scenes in one batch, the learned guide.

Fields of a case: `kind` (what the program calls), `scene` and its sizes, `width`, `height`, `spp`,
`interval` (samples per pass) and `depth` (bounces).
"""
import math

import numpy as np
import torch

import keepsake_b200 as ks

GUIDE_ROWS_FLOPS = 3 * 2 * (4 * 64 * 64 + 48 * 64)  # forward, dX and dW of the network per row

# Mean number of closest-hit and shadow queries per camera path of each scene.
RAYS_PER_PATH = {"box": 4.9, "materials": 5.0, "subsurface": 4.5, "mesh": 2.4, "glossy": 2.5, "instanced": 2.6}


def listed():
    return [
        # A thumbnail into host buffers: the smallest call a viewer makes.
        dict(name="thumbnail", kind="host", scene="box", width=64, height=48, spp=4, interval=32, depth=8),
        # One sample per pixel of a small window at an odd size: an interactive preview's pass.
        dict(name="preview", kind="device", scene="mesh", level=6, sky=512, width=641, height=359, spp=1,
             interval=1, depth=12),
        # The box room at the size and samples of the benchmark's first configuration.
        dict(name="box_room", kind="device", scene="box", width=256, height=256, spp=64, interval=32, depth=8),
        # The benchmark's mesh and frame, two of its eight sample intervals: the largest render.
        dict(name="mesh_frame", kind="device", scene="mesh", level=8, sky=2048, width=1024, height=1024, spp=64,
             interval=32, depth=12),
        # Progressive passes of a glossy, partly occluded scene at 1080p, the image kept on the device.
        dict(name="glossy_passes", kind="progress", scene="glossy", level=7, sky=1024, width=1920, height=1080,
             spp=4, interval=1, depth=12),
        # Every material feature at once: textures, normal and opacity maps, smooth normals, glass,
        # a Beckmann lobe, a Gaussian pixel filter.
        dict(name="materials", kind="device", scene="materials", opacity=True, width=512, height=512, spp=16,
             interval=16, depth=8),
        # Random walks below the surface of one object.
        dict(name="subsurface", kind="device", scene="subsurface", width=256, height=256, spp=16, interval=16,
             depth=6),
        # Instances: the benchmark's 400 instances of 8 meshes at 1080p.
        dict(name="instanced", kind="device", scene="instanced", prototypes=8, instances=400, frequency=50,
             sky=1024, width=1920, height=1080, spp=4, interval=4, depth=16),
        # Passes that draw directions from a trained guide (kept fixed).
        dict(name="guided", kind="guided", scene="glossy", level=7, sky=1024, width=1280, height=720, spp=4,
             interval=1, depth=12),
        # One training batch of the guide: forward, loss, backward, gradients to the host.
        dict(name="guide_batch", kind="train", rows=131000),
        # Scenes of uneven size in one wavefront, as a dataset generator renders them.
        dict(name="batch", kind="batch", scene="mesh", jobs=8, frequency=100, sky=512, width=512, height=512,
             spp=8, interval=8, depth=12),
        # A scene that is new for every frame: upload, tree build, a short render, the image back.
        dict(name="new_scene", kind="new_scene", scene="mesh", level=7, sky=512, width=512, height=512, spp=4,
             interval=32, depth=12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["host", "device", "device", "progress", "materials", "subsurface", "instanced", "guided",
                       "train", "batch", "new_scene"])
    if what == "train":
        return dict(kind="train", rows=_log(rng, 4096, 262144))
    c = dict(kind=what)
    if what in ("materials", "subsurface"):
        c.update(kind=rng.choice(["host", "device"]), scene=what)
        if what == "materials":
            c["opacity"] = rng.random() < 0.5
    elif what == "instanced":
        c.update(kind="device", scene="instanced", prototypes=rng.randint(2, 8), instances=_log(rng, 24, 400),
                 frequency=_log(rng, 6, 50), sky=512)
    elif what == "guided":
        c.update(scene="glossy", level=rng.randint(5, 7), sky=512)
    elif what == "batch":
        c.update(scene="mesh", jobs=rng.randint(2, 12), frequency=_log(rng, 22, 200), sky=512)
    elif what == "new_scene":
        c.update(scene="mesh", level=rng.randint(4, 8), sky=rng.choice([256, 512, 1024]))
    else:
        c["scene"] = rng.choice(["box", "mesh", "mesh", "glossy"])
        if c["scene"] != "box":
            c.update(level=rng.randint(4, 8), sky=rng.choice([256, 512, 1024, 2048]))
    paths = _log(rng, 1 << 12, 1 << (22 if what in ("subsurface", "batch", "new_scene") else 24))
    c["spp"] = min(_log(rng, 1, 64), max(1, paths // 1024))
    pixels = max(1024, paths // c["spp"])
    if what == "batch":
        pixels = max(1024, pixels // c["jobs"])
    aspect = rng.choice([1.0, 4 / 3, 16 / 9])
    c["width"] = max(16, int(round(math.sqrt(pixels * aspect))))
    c["height"] = max(16, int(round(c["width"] / aspect)) + rng.randint(0, 1))
    c["interval"] = rng.choice([1, 4]) if c["kind"] in ("progress", "guided") else 32
    if c["kind"] in ("progress", "guided"):
        c["spp"] = min(c["spp"], 8 * c["interval"])
    c["depth"] = rng.choice([4, 6, 8, 12, 16])
    return c


# ---------------------------------------------------------------------------------------------
# Scenes
# ---------------------------------------------------------------------------------------------
_context = None


def _ctx():
    """The program's one context (device, stream, wavefront buffers)."""
    global _context
    if _context is None:
        _context = ks.Context(0)
    return _context


def _material(basecolor, roughness, metallic=0.0, **fields):
    m = ks.MaterialDesc(tuple(float(x) for x in basecolor), roughness, metallic, 1.5, 0.5, 0.0, 0.0, 0.5, (0, 0, 0),
                        0, 0, (0, 0, 0))
    for k, v in fields.items():
        if isinstance(v, tuple):
            getattr(m, k)[:] = v
        else:
            setattr(m, k, v)
    return m


def _sphere(center, radius, nu=48, nv=24):
    """A latitude-longitude sphere: vertices, indices, normals, texture coordinates."""
    ph, th = np.meshgrid(np.linspace(0, 2 * np.pi, nu + 1), np.linspace(0, np.pi, nv + 1))
    n = np.stack([np.sin(th) * np.cos(ph), np.cos(th), np.sin(th) * np.sin(ph)], -1).reshape(-1, 3)
    uv = np.stack([ph / (2 * np.pi), th / np.pi], -1).reshape(-1, 2)
    a = (np.arange(nv)[:, None] * (nu + 1) + np.arange(nu)[None, :]).reshape(-1)
    b = a + nu + 1
    idx = np.concatenate([np.stack([a, a + 1, b], -1), np.stack([a + 1, b + 1, b], -1)])
    v = np.asarray(center, np.float64) + radius * n
    p = v[idx]
    flat = np.linalg.norm(np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]), axis=1) > 1e-9  # the poles
    return v.astype(np.float32), idx[flat].astype(np.uint32), n.astype(np.float32), uv.astype(np.float32)


def _room(seed):
    g = ks.Generated("box_room", seed)
    meshes = [[m["vertices"].copy(), m["indices"], m["material"], dict(twosided=m["twosided"])] for m in g.meshes]
    for k in (5, 6):  # the boxes, off the floor: no face in the floor's plane
        meshes[k][0][:, 1] += np.float32(1e-3)
    return g, meshes, list(g.materials)


def _materials_scene(seed, opacity):
    g, meshes, mats = _room(seed)
    rng = np.random.default_rng(seed)
    ys, xs = np.mgrid[0:256, 0:256]
    checker = (((xs // 16) + (ys // 16)) % 2).astype(np.float32)[..., None]
    base = (checker * rng.uniform(90, 200, 3) + rng.uniform(20, 55, 3)).astype(np.uint8)
    rough = (rng.uniform(0.1, 0.9, (64, 64, 1)) * 65535).astype(np.uint16)
    n = np.stack([0.3 * np.sin(xs / 9.0), 0.3 * np.cos(ys / 7.0), np.ones_like(xs, float)], -1)
    n /= np.linalg.norm(n, axis=-1, keepdims=True)
    bump = (n * 0.5 + 0.5).astype(np.float32)
    mask = (((xs // 8) % 3 > 0) * 255).astype(np.uint8)[..., None]
    uv4 = np.array([[0, 0], [2, 0], [2, 2], [0, 2]], np.float32)
    for k in (0, 2):
        meshes[k][3]["texcoords"] = uv4
    first = len(mats)
    mats += [_material((0.95, 0.7, 0.35), 0.25, 1.0, microfacet=1),
             _material((1.0, 1.0, 1.0), 0.1, specular_trans=1.0, ior=1.5),
             _material(rng.uniform(0.3, 0.9, 3), 0.6, bsdf=1, specular=0.6),
             _material(rng.uniform(0.3, 0.9, 3), 0.5)]
    for k, (c, r) in enumerate([((-0.5, 0.32, 0.55), 0.3), ((0.4, 0.86, 0.35), 0.2), ((0.62, 0.16, 0.75), 0.14),
                                ((-0.1, 1.3, 0.2), 0.22)]):
        v, idx, nrm, uv = _sphere(c, r)
        meshes.append((v, idx, first + k, dict(twosided=0 if k == 1 else 1, normals=nrm, texcoords=uv)))
    bind = ks.TextureBinding.make
    bindings = [bind(meshes[0][2], "basecolor", 0, filter=1), bind(meshes[0][2], "normal_map", 2, filter=1, strength=0.7),
                bind(meshes[2][2], "roughness", 1, filter=2, cubic_kernel=2),
                bind(first, "roughness", 1, filter=1), bind(first + 2, "basecolor", 0, filter=0)]
    if opacity:
        bindings.append(bind(first + 3, "opacity_map", 3, filter=1, uv_scale=(2.0, 2.0)))
    desc, keep = ks.scene_desc(meshes, mats, g.desc.contents.sky)
    keep += [g] + ks.attach_textures(desc, [(base, True), (rough, False), (bump, False), (mask, False)], bindings)
    return g, desc, keep


def _subsurface_scene(seed):
    g, meshes, mats = _room(seed)
    rng = np.random.default_rng(seed)
    mats.append(_material((0.8, 0.7, 0.6), 0.5, has_subsurface=1, ss_albedo=tuple(rng.uniform(0.3, 0.9, 3)),
                          ss_radius=(0.3, 0.2, 0.1), ss_anisotropy=0.2, ss_ior=1.4))
    meshes[5][2], meshes[5][3]["twosided"] = len(mats) - 1, 0
    v, idx, nrm, uv = _sphere((0.4, 0.86, 0.35), 0.2)
    meshes.append((v, idx, len(mats) - 1, dict(twosided=0, normals=nrm)))
    desc, keep = ks.scene_desc(meshes, mats, g.desc.contents.sky)
    return g, desc, keep + [g]


def _describe(case, seed):
    """(generated scene that holds the camera, scene description, what must stay alive)."""
    s = case["scene"]
    res = (case["width"], case["height"])
    if s == "materials":
        return _materials_scene(seed, case["opacity"])
    if s == "subsurface":
        return _subsurface_scene(seed)
    if s == "box":
        g = ks.Generated("box_room", seed, resolution=res)
    elif s == "instanced":
        g = ks.Generated("instanced", seed, sky=(case["sky"], case["sky"] // 2), resolution=res,
                         prototypes=case["prototypes"], instances=case["instances"], frequency=case["frequency"])
    else:
        size = dict(frequency=case["frequency"]) if "frequency" in case else dict(level=case["level"])
        glossy = dict(roughness=(0.02, 0.2), occluder=True) if s == "glossy" else {}
        g = ks.Generated("icosphere", seed, sky=(case["sky"], case["sky"] // 2), resolution=res, **size, **glossy)
    return g, g.desc, g


def _camera(g, case):
    return ks.camera_perspective(g.camera_to_world, g.vfov, case["width"] / case["height"])


def _params(case, seed, **more):
    if case["scene"] == "materials":
        more.update(pixel_filter=1, pixel_filter_width=3.0)
    return ks.SmallPTParams.make(render_width=case["width"], render_height=case["height"], spp=case["spp"],
                                 bounces=case["depth"], rng_seed=seed & 0x3fffffff, spp_prog_interval=case["interval"],
                                 **more)


def _image(width, height):
    return (torch.zeros((height, width, 3), dtype=torch.float64, device="cuda"),
            torch.zeros((height, width, 2), dtype=torch.float64, device="cuda"))


def _guide_parameters(seed):
    """Weights of the layers' own scale and a table of features as a training of some hundred steps
    leaves them (a new guide's, of 1e-4, would give every point one mixture)."""
    rng = np.random.default_rng(seed)
    w = []
    for l, (rows, cols) in enumerate(ks.GUIDE_LAYERS):
        m = rng.uniform(-1, 1, (rows, cols)) * math.sqrt(6.0 / cols)
        if l == len(ks.GUIDE_LAYERS) - 1:
            m[ks.GUIDE_OUTPUTS:] = 0.0
        w.append(m.ravel())
    grid = rng.uniform(-0.5, 0.5, (ks.GUIDE_LEVELS, ks.GUIDE_TABLE_SIZE, 2)).astype(np.float32)
    return np.concatenate(w).astype(np.float32), grid


def _guide(seed, bound):
    guide = ks.Guide(_ctx(), bound, seed=1)
    guide.set_weights(*_guide_parameters(seed))
    return guide


_BOUND = [-1.5, -1.2, -1.5, 1.5, 1.8, 1.5]


def _train_rows(rows, seed):
    """Records as a render captures them: points on surfaces around the origin, directions over the
    sphere, mostly small targets with a few large ones, BSDF densities of rough materials."""
    rng = np.random.default_rng(seed)

    def directions():
        v = rng.normal(size=(rows, 3))
        return (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)

    pos = (directions() * rng.uniform(0.95, 1.05, (rows, 1))).astype(np.float32)
    target = rng.lognormal(-1.0, 1.2, rows).astype(np.float32)
    target[rng.random(rows) < 0.3] = 0.0
    return pos, directions(), directions(), directions(), target, rng.uniform(0.02, 0.6, rows).astype(np.float32)


# ---------------------------------------------------------------------------------------------
# The measured calls
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    st = dict(kind=kind)
    if kind == "train":
        st["guide"] = _guide(seed, _BOUND)
        st["rows"] = _train_rows(case["rows"], seed)
        return st
    if kind == "batch":
        st["jobs"], st["keep"] = [], []
        rng = np.random.default_rng(case["jobs"])
        for k in range(case["jobs"]):
            scale = float(rng.uniform(0.5, 1.0))
            job = dict(case, frequency=max(1, int(case["frequency"] * scale)),
                       width=max(16, int(case["width"] * (1.5 - scale))), height=max(16, int(case["height"] * (1.5 - scale))))
            g, desc, keep = _describe(job, seed * 1000 + k)
            scene = ks.Scene(_ctx(), desc, keepalive=keep)
            scene.build_bvh()
            st["jobs"].append((scene, _camera(g, job), _params(job, seed + k), *_image(job["width"], job["height"])))
        return st
    g, desc, keep = _describe(case, seed)
    st.update(desc=desc, keep=(g, keep), camera=_camera(g, case), params=_params(case, seed))
    if kind == "new_scene":
        return st
    st["scene"] = ks.Scene(_ctx(), desc, keepalive=keep)
    st["scene"].build_bvh()
    if kind != "host":
        st["image"] = _image(case["width"], case["height"])
    if kind == "guided":
        lo, hi = g.bound
        st["guide"] = _guide(seed, list(lo - 0.05) + list(hi + 0.05))
        st["options"] = ks.GuideRenderOptions.make(train_passes=0, guide_from_pass=0, min_roughness=0.05)
    return st


def run(state):
    kind = state["kind"]
    if kind == "train":
        pos, wo, normal, wi, target, pdf = state["rows"]
        return state["guide"].gradients(pos, wo, normal, wi, target, pdf)
    if kind == "host":
        return state["scene"].render(state["camera"], state["params"])
    if kind == "new_scene":
        scene = ks.Scene(_ctx(), state["desc"], keepalive=state["keep"])
        scene.build_bvh()
        image = scene.render(state["camera"], state["params"])
        scene.close()
        return image
    images = [(j[3], j[4]) for j in state["jobs"]] if kind == "batch" else [state["image"]]
    for acc, weights in images:
        acc.zero_()
        weights.zero_()
    torch.cuda.current_stream().synchronize()  # the renders run on the context's own stream
    if kind == "batch":
        ks.batch_render(_ctx(), [(s, c, p, a.data_ptr(), w.data_ptr()) for s, c, p, a, w in state["jobs"]])
        return images
    acc, weights = images[0]
    args = (state["camera"], state["params"])
    if kind == "device":
        state["scene"].render_device(*args, acc.data_ptr(), weights.data_ptr())
    elif kind == "progress":
        state["scene"].render_device_progress(*args, acc.data_ptr(), weights.data_ptr(), lambda spp: False)
    else:
        state["scene"].render_guided_device(*args, state["guide"], state["options"], acc.data_ptr(),
                                            weights.data_ptr())
    return acc, weights


def _triangles(case):
    s = case["scene"]
    if s in ("box", "subsurface"):
        return 36
    if s == "materials":
        return 9000
    if s == "instanced":
        return 20 * case["frequency"] ** 2 * case["prototypes"]
    return 20 * case["frequency"] ** 2 if "frequency" in case else 20 * 4 ** case["level"]


def work(case):
    """Bytes: the scene (36 B a triangle, 12 B a sky texel) read once, the image (40 B a pixel) written
    once.  Operations: a ray query descends a balanced binary tree (two boxes of 18 operations a
    level) to two triangles of 60, a path vertex shades with about 300."""
    if case["kind"] == "train":
        table = 4.0 * ks.GUIDE_LEVELS * ks.GUIDE_TABLE_SIZE * 2
        return {"bytes": 2 * table + 56.0 * case["rows"], "flops": float(GUIDE_ROWS_FLOPS) * case["rows"]}
    tris = _triangles(case)
    n = case.get("jobs", 1)
    paths = float(case["width"]) * case["height"] * case["spp"] * n
    rays = paths * RAYS_PER_PATH[case["scene"]]
    per_ray = 36.0 * max(1.0, math.log2(tris)) + 120.0 + 150.0
    flops = rays * per_ray
    if case["kind"] == "guided":
        flops += 0.5 * paths * GUIDE_ROWS_FLOPS / 3
    sky = case.get("sky", 0) ** 2 / 2
    return {"bytes": n * (36.0 * tris + 12.0 * sky + 40.0 * case["width"] * case["height"]), "flops": flops}


# ---------------------------------------------------------------------------------------------
# The training batch in 64 bits.  A render's value is an estimate over float32 decisions (which
# triangle, which lobe, which paths go on), so it has no value in 64 bits.
# ---------------------------------------------------------------------------------------------
def _corners(pos, level_res, table):
    """Table entries and trilinear weights of each level's cell; the cell and the weights are float32,
    as they decide which entries are meant."""
    lo, hi = (torch.tensor(_BOUND[k:k + 3], dtype=torch.float32, device=pos.device) for k in (0, 3))
    pn = ((pos - lo) * (1.0 / (hi - lo))).clamp(0, 1)
    for res in level_res:
        p = pn * float(res)
        cell = p.floor().clamp(max=float(res - 1))
        t, c = p - cell, cell.long()
        side = (res + 2) >> 1
        idx, weight = [], []
        for k in range(8):
            d = [(k >> a) & 1 for a in range(3)]
            x, y, z = (c[:, a] + d[a] for a in range(3))
            if side ** 3 * 8 <= table:
                inner = (x & 1) | ((y & 1) << 1) | ((z & 1) << 2)
                idx.append(((x >> 1) + side * ((y >> 1) + side * (z >> 1))) * 8 + inner)
            else:
                idx.append((x ^ (y * 2654435761) ^ (z * 805459861)) & (table - 1))
            w = [t[:, a] if d[a] else 1.0 - t[:, a] for a in range(3)]
            weight.append((w[0] * w[1]) * w[2])
        yield torch.stack(idx, 1), torch.stack(weight, 1).double()


def _harmonics(d):
    x, y, z = d.unbind(1)
    xx, yy, zz = x * x, y * y, z * z
    a, b, c, e = 0.48860251190291987, 1.0925484305920792, 0.59004358992664352, 0.45704579946446572
    return torch.stack([
        torch.full_like(x, 0.28209479177387814), -a * y, a * z, -a * x, b * x * y, -b * y * z,
        0.94617469575755997 * zz - 0.31539156525251999, -b * x * z, 0.54627421529603959 * (xx - yy),
        c * y * (-3.0 * xx + yy), 2.8906114426405538 * x * y * z, e * y * (1.0 - 5.0 * zz),
        0.3731763325901154 * z * (5.0 * zz - 3.0), e * x * (1.0 - 5.0 * zz), 1.4453057213202769 * z * (xx - yy),
        c * x * (-xx + 3.0 * yy)], 1)


def exact(case, seed):
    if case["kind"] != "train":
        return None
    dev = torch.device("cuda")
    w, grid = _guide_parameters(seed)
    # cells per axis: 16 to 2048 in a geometric row
    level_res = [math.floor(16.0 * math.exp(math.log(2048.0 / 16.0) / (ks.GUIDE_LEVELS - 1) * l) + 1e-9)
                 for l in range(ks.GUIDE_LEVELS)]
    pos, wo, normal, wi, target, pdf = (torch.from_numpy(a).to(dev) for a in _train_rows(case["rows"], seed))
    w = torch.from_numpy(w).to(dev).double().requires_grad_()
    grid = torch.from_numpy(grid).to(dev).double()
    unit = torch.nn.functional.normalize
    x = [(weight[..., None] * grid[l][idx]).sum(1)
         for l, (idx, weight) in enumerate(_corners(pos, level_res, ks.GUIDE_TABLE_SIZE))]
    x = torch.cat(x + [_harmonics(unit(wo.double())), _harmonics(unit(normal.double()))], 1)
    at = 0
    for l, (rows, cols) in enumerate(ks.GUIDE_LAYERS):
        x = x @ w[at:at + rows * cols].view(rows, cols).T
        at += rows * cols
        if l < len(ks.GUIDE_LAYERS) - 1:
            x = x.relu()
    lobes = x[:, :40].view(-1, 8, 5)
    mu, high, soft = unit(lobes[..., :3], dim=-1), math.log(1e4), torch.nn.functional.softplus
    kappa = torch.exp(-6.0 + soft(lobes[..., 3] + 6.0) - soft(lobes[..., 3] - high)).clamp(max=1e4)
    cos = (mu * unit(wi.double())[:, None]).sum(-1) - 1.0
    density = kappa / (2 * math.pi * -torch.expm1(-2.0 * kappa)) * torch.exp(kappa * cos.clamp(max=0.0))
    q = (lobes[..., 4].softmax(1) * density).sum(1)
    alpha = 0.8 * torch.sigmoid(x[:, 40])
    t = target.double() / case["rows"]
    m = alpha * q.detach() + (1.0 - alpha) * pdf.double()
    used = (t > 0) & (m > 1e-30) & (q > 1e-30)
    loss = -(t[used] * m[used].log()).sum()
    (loss - (t[used] * q[used].log()).sum()).backward()
    # the table's gradient is what is left of the batch after five layers of BF16 operands, 11 % from
    # this value at the start by design of the network's arithmetic: it is held to the start's instead
    return loss.item(), w.grad, None
