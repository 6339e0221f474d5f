"""What a program does with this framework, as timed cases.

frame    one animation frame through Context.frame: part transforms, tree
         build, primary / mirror / shadow rays, shading, into a device image
rays     closest hits of a ray batch on a tree that is already built, from
         host arrays (KDTreeCUDA.checkCollision) or device arrays
batch    many scenes with uneven ray batches in one launch (Batch)
resort   the reference's re-sampling SAH builder, then a render of its tree
forward  the split proposer's logits for recorded feature rows
grad     the proposer's gradients for a training batch

Scenes are the package's own generators (rigid parts, the 24,576-triangle
ground and spheres) and a clustered-triangle scene with walls made here on the
GPU, because the package's generator takes seconds on the host at 1M triangles.
"""
import math
import os

import numpy as np
import torch

import hulktracer_b200 as hk
from hulktracer_b200 import scenes

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(hk.__file__)), "weights", "proposer.bin")
MLP = (200, 256, 256, 256, 96)
MLP_MACS = sum(a * b for a, b in zip(MLP, MLP[1:]))
PART_TRIS, PART_VERTS = 3120, 1756   # mean of the three part shapes
_stream = []                         # the stream that every context of the program works on


def listed():
    return [
        # a preview of a toy scene: launches and latency; an image that does
        # not divide into ray tiles
        dict(name="frame_toy", kind="frame", scene="parts", parts=2, width=157, height=93, lights=1, variant="ropes",
             build="binned", exact_max=0, subtree_depth=8),
        # an interactive scene of the size that film-and-games test files have
        # (kitchen: 800x600, six lights), library defaults
        dict(name="frame_six_lights", kind="frame", scene="parts", parts=35, width=800, height=600, lights=6,
             variant="ropes", build="binned", exact_max=0, subtree_depth=8),
        # a small static scene rebuilt per frame with the API's default
        # traversal (ring short stack)
        dict(name="frame_24k_short", kind="frame", scene="spheres", width=512, height=512, lights=1,
             variant="shortstack", build="binned", exact_max=0, subtree_depth=8),
        # the benchmark's animated scene, builder layout as the tuner picks it
        dict(name="frame_200k", kind="frame", scene="parts", parts=64, width=1280, height=720, lights=1,
             variant="ropes", build="binned", exact_max=0, subtree_depth=0),
        # the same frames with the learned split proposer
        dict(name="frame_200k_learned", kind="frame", scene="parts", parts=64, width=1280, height=720, lights=1,
             variant="ropes", build="learned", exact_max=0, subtree_depth=0),
        # the same frames with the exact SAH on nodes of up to 1024 references
        dict(name="frame_200k_exact", kind="frame", scene="parts", parts=64, width=1280, height=720, lights=1,
             variant="ropes", build="binned", exact_max=1024, subtree_depth=0),
        # the largest frame: a million triangles, full HD, one mirror bounce
        dict(name="frame_1m_mirror", kind="frame", scene="rooms", tris=1000000, width=1920, height=1080, lights=1,
             variant="ropes", build="binned", exact_max=0, subtree_depth=0),
        # a picking / collision query from host arrays, a thousand rays
        dict(name="rays_host_1k", kind="rays", scene="spheres", rays=997, where="host", variant="shortstack"),
        # a light-transport batch: incoherent bounce rays on a static scene
        dict(name="rays_incoherent_1m", kind="rays", scene="rooms", tris=400000, rays=1000000, where="device",
             variant="ropes"),
        # a rendering service: scenes of very different sizes in one launch
        dict(name="batch_12", kind="batch", scenes=12, tris_lo=10000, tris_hi=300000, rays_lo=65536, rays_hi=524288,
             variant="ropes"),
        # the reference's alternative builder (--treeType=SAH) and a picture
        dict(name="resort_59k", kind="resort", scene="parts", parts=19, width=320, height=240, lights=1,
             variant="shortstack"),
        # one training batch of the split proposer: forward and backward
        dict(name="proposer_grad_4k", kind="grad", rows=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "rays", "rays", "batch", "resort", "forward", "grad"])
    variant = rng.choice(["ropes", "ropes", "ropes", "shortstack", "fullstack"])
    if kind == "frame":
        c = dict(kind=kind, scene=rng.choice(["parts", "parts", "rooms", "spheres"]), width=_log(rng, 96, 1600),
                 height=_log(rng, 64, 900), lights=rng.randint(1, 6), variant=variant,
                 build=rng.choice(["binned", "binned", "learned"]), exact_max=0,
                 subtree_depth=rng.choice([0, 8]))
        if c["width"] * c["height"] * c["lights"] > 1500000:
            c["lights"] = 1
        if c["build"] == "binned" and rng.random() < 0.25:
            c["exact_max"] = _log(rng, 32, 1024)
        if c["scene"] == "parts":
            c["parts"] = _log(rng, 1, 64)
        elif c["scene"] == "rooms":
            c["tris"] = _log(rng, 5000, 200000 if c["build"] == "learned" or c["exact_max"] else 800000)
        return c
    if kind == "rays":
        c = dict(kind=kind, scene=rng.choice(["rooms", "spheres"]), rays=_log(rng, 32, 1000000),
                 where=rng.choice(["host", "device"]), variant=variant)
        if c["scene"] == "rooms":
            c["tris"] = _log(rng, 5000, 400000)
        return c
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(2, 12), tris_lo=_log(rng, 2000, 20000),
                    tris_hi=_log(rng, 30000, 300000), rays_lo=_log(rng, 5000, 65536), rays_hi=_log(rng, 70000, 524288),
                    variant=variant)
    if kind == "resort":
        return dict(kind=kind, scene="parts", parts=_log(rng, 1, 19), width=_log(rng, 64, 320),
                    height=_log(rng, 64, 240), lights=1, variant=variant)
    return dict(kind=kind, rows=_log(rng, 33, 20000 if kind == "forward" else 8192))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _context(**config):
    if not _stream:
        _stream.append(torch.cuda.Stream())
    ctx = hk.Context(device=0, **config)
    ctx.set_stream(_stream[0].cuda_stream)
    return ctx


def _batch_sizes(case):
    """Triangles and rays of each scene: both spread evenly over their
    logarithms, the rays in another order than the triangles."""
    n = case["scenes"]

    def size(key, i):
        lo, hi = math.log(case[key + "_lo"]), math.log(case[key + "_hi"])
        return int(math.exp(lo + (hi - lo) * (i + 0.5) / n))
    return [(size("tris", i), size("rays", (i * 5 + 3) % n)) for i in range(n)]


def _weights(seed):
    """An untrained network (normal, variance 2 / fan-in, zero biases)."""
    rng = np.random.default_rng(seed)
    return np.concatenate([np.concatenate([rng.normal(0.0, math.sqrt(2.0 / a), a * b), np.zeros(b)])
                           for a, b in zip(MLP, MLP[1:])]).astype(np.float32)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rooms(ntris, seed, width, height):
    """Clustered small triangles of random orientation in a 100^3 box and 24
    walls of 2,048 triangles (scenes.static_large), made on the GPU."""
    g = _gen(seed)
    f = dict(device="cuda", dtype=torch.float64)
    centers = (torch.rand(200, 3, generator=g, **f) - 0.5) * 100.0
    sigma = 0.2 + 1.8 * torch.rand(200, generator=g, **f)
    of = torch.randint(0, 200, (ntris,), generator=g, device="cuda")
    c = centers[of] + torch.randn(ntris, 3, generator=g, **f) * sigma[of, None]
    e = torch.randn(ntris, 3, generator=g, **f)
    e = e / e.norm(dim=1, keepdim=True)
    h = torch.linalg.cross(e, torch.randn(ntris, 3, generator=g, **f))
    h = h / h.norm(dim=1, keepdim=True)
    l1 = 0.01 + 0.19 * torch.rand(ntris, 1, generator=g, **f)
    l2 = 0.01 + 0.19 * torch.rand(ntris, 1, generator=g, **f)
    a = 0.3 + 2.5 * torch.rand(ntris, 1, generator=g, **f)
    p = torch.stack([torch.zeros_like(c), e * l1, (e * a.cos() + h * a.sin()) * l2], 1)
    verts = [(p - p.mean(1, keepdim=True) + c[:, None]).reshape(-1, 3)]
    tris = [torch.arange(3 * ntris, device="cuda").reshape(-1, 3)]
    u = torch.linspace(-50.0, 50.0, 33, **f)
    gu, gw = torch.meshgrid(u, u, indexing="ij")
    i = torch.arange(32, device="cuda")
    q = (i[:, None] * 33 + i[None, :]).reshape(-1)
    quad = torch.cat([torch.stack([q, q + 33, q + 1], 1), torch.stack([q + 1, q + 33, q + 34], 1)])
    for k in range(24):
        w = torch.empty(33 * 33, 3, **f)
        w[:, k % 3] = -50.0 + 100.0 * ((k // 3) + 0.5) / 8.0
        w[:, (k + 1) % 3] = gu.reshape(-1)
        w[:, (k + 2) % 3] = gw.reshape(-1)
        verts.append(w)
        tris.append(quad + 3 * ntris + 33 * 33 * k)
    v, t = torch.cat(verts).float(), torch.cat(tris).int()
    V = torch.ones(v.shape[0], 4, device="cuda")
    V[:, :3] = v
    T = torch.zeros(t.shape[0], 4, dtype=torch.int32, device="cuda")
    T[:, :3] = t
    sc = scenes.Scene(V.cpu().numpy(), T.cpu().numpy().view(np.uint32),
                      np.stack([scenes.point_light((30.0, 80.0, 60.0))]),
                      scenes.look_at_camera((0.0, 10.0, 120.0), (0.0, 0.0, 0.0), 60.0, width, height), width, height)
    hsh = (np.arange(sc.ntris, dtype=np.uint64) * np.uint64(2654435761)) & np.uint64(0xFFFFFFFF)
    sc.extra["mirror"] = (hsh < np.uint64(int(0.3 * 2 ** 32))).astype(np.uint8)
    return sc


def _scene(case, seed):
    w, h = case.get("width", 512), case.get("height", 512)
    if case["scene"] == "parts":
        sc = scenes.animated_parts(seed=seed, width=w, height=h, n_parts=case["parts"])
    elif case["scene"] == "spheres":
        sc = scenes.static_small(seed=seed, width=w, height=h)
    else:
        sc = _rooms(case["tris"], seed, w, h)
    rng = np.random.default_rng(seed)
    lights = list(sc.lights)
    span = float(np.abs(sc.verts[:, :3]).max())
    while len(lights) < case.get("lights", 1):
        lights.append(scenes.point_light(rng.uniform(-1.5, 1.5, 3) * span + np.array([0.0, 2.0 * span, 0.0]),
                                         rng.uniform(0.1, 0.5, 3)))
    sc.lights = np.stack(lights)
    return sc


def _rays(V, T, cam, n, seed):
    """A quarter primary rays through random pixels, the rest leaving random
    triangle points in cosine-weighted directions (scenes.incoherent_rays)."""
    g = _gen(seed)
    f = dict(device="cuda", dtype=torch.float64)
    cam = torch.tensor(np.asarray(cam), **f)
    k = n // 4
    u, v = torch.rand(k, 1, generator=g, **f), torch.rand(k, 1, generator=g, **f)
    d = cam[3, :3] + cam[1, :3] * u + cam[2, :3] * v - cam[0, :3]
    d = d / d.norm(dim=1, keepdim=True)
    m = n - k
    V, T = torch.tensor(V, device="cuda").double(), torch.tensor(T.view(np.int32), device="cuda").long()
    p = V[T[torch.randint(0, T.shape[0], (m,), generator=g, device="cuda")][:, :3], :3]
    a, b = torch.rand(m, 1, generator=g, **f), torch.rand(m, 1, generator=g, **f)
    a, b = torch.where(a + b > 1, 1 - a, a), torch.where(a + b > 1, 1 - b, b)
    pos = p[:, 0] + (p[:, 1] - p[:, 0]) * a + (p[:, 2] - p[:, 0]) * b
    nrm = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
    up = torch.tensor([0.0, 1.0, 0.0], **f).expand(m, 3)
    nrm = torch.where(nrm.norm(dim=1, keepdim=True) > 1e-12, nrm, up)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    # cosine-weighted: a point on the unit sphere about the normal's tip
    s = torch.randn(m, 3, generator=g, **f)
    e = nrm * (1 + 1e-6) + s / s.norm(dim=1, keepdim=True)
    e = e / e.norm(dim=1, keepdim=True)
    e = torch.where(torch.rand(m, 1, generator=g, **f) < 0.5, e, -e)   # either face
    out = torch.zeros(n, 8, device="cuda")
    out[:k, :3], out[:k, 4:7] = cam[0, :3].float(), d.float()
    out[k:, :3], out[k:, 4:7] = (pos + e * 1e-3).float(), e.float()
    return out


def _features(n, seed):
    """Feature rows as the builder makes them (bin counts as fractions of the
    node's references, extents over the largest, depth, references / 1024)."""
    rng = np.random.default_rng(seed)
    X = np.zeros((n, 200), np.float32)
    cnt = np.exp(rng.uniform(np.log(33), np.log(1024), n)).astype(np.int64)
    w = rng.exponential(1.0, (n, 6, 32)) * (rng.random((n, 6, 32)) < 0.7) + 1e-3
    w /= w.sum(axis=2, keepdims=True)
    X[:, :192] = (np.floor(w * cnt[:, None, None]) / cnt[:, None, None]).reshape(n, 192)
    ext = rng.uniform(0.05, 1.0, (n, 3))
    X[:, 192:195] = ext / ext.max(axis=1, keepdims=True)
    X[:, 195] = rng.integers(4, 20, n) / 24.0
    X[:, 196] = cnt / 1024.0
    return X, rng.integers(0, 96, n).astype(np.int32)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("forward", "grad"):
        ctx = _context()
        if kind == "grad":
            ctx.mlp_set_params(_weights(seed))
        else:
            ctx.mlp_load(WEIGHTS)
        X, y = _features(case["rows"], seed)
        return dict(kind=kind, ctx=ctx, X=X, y=y)
    variant = hk.VARIANTS[case["variant"]]
    if kind == "batch":
        ctx = _context()
        batch = hk.engine.Batch(ctx)
        rays, offsets = [], [0]
        for i, (nt, nr) in enumerate(_batch_sizes(case)):
            sc = _rooms(nt, seed * 1000 + i, 256, 256)
            batch.add_scene(sc.verts, sc.tris)
            rays.append(_rays(sc.verts, sc.tris, sc.camera, nr, seed * 1000 + i))
            offsets.append(offsets[-1] + nr)
        rays = torch.cat(rays)
        hits = torch.zeros(rays.shape[0], 2, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        return dict(kind=kind, ctx=ctx, batch=batch, rays=rays, offsets=np.array(offsets, np.uint32), hits=hits,
                    variant=variant)
    sc = _scene(case, seed)
    if kind == "rays":
        tree = hk.engine.KDTreeCUDA(_context())
        tree.buildKDTree(sc)
        rays = _rays(sc.verts, sc.tris, sc.camera, case["rays"], seed)
        if case["where"] == "host":
            return dict(kind=kind, tree=tree, rays=rays.cpu().numpy(), variant=variant)
        hits = torch.zeros(case["rays"], 2, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        return dict(kind=kind, tree=tree, rays=rays, hits=hits, variant=variant)
    image = torch.zeros(sc.width * sc.height, dtype=torch.int32, device="cuda")
    ctx = _context(exact_max=case.get("exact_max", 0))
    ctx.upload(sc.verts, sc.tris)
    state = dict(kind=kind, ctx=ctx, cam=sc.camera, lights=sc.lights, w=sc.width, h=sc.height, image=image,
                 variant=variant)
    frame = 1 + seed % 59
    if kind == "resort":
        ctx.set_parts(sc.part_of_vertex, sc.part_center.shape[0])
        ctx.transform(scenes.part_matrices(sc, frame))
        torch.cuda.synchronize()
        return state
    state["mode"] = hk.BUILD_LEARNED if case["build"] == "learned" else hk.BUILD_BINNED
    if case["build"] == "learned":
        ctx.mlp_load(WEIGHTS)
    ctx.set_build_layout(32, case["subtree_depth"])
    state["mats"] = None
    if sc.part_of_vertex is not None:
        ctx.set_parts(sc.part_of_vertex, sc.part_center.shape[0])
        state["mats"] = scenes.part_matrices(sc, frame)
    if "mirror" in sc.extra:
        ctx.set_mirrors(sc.extra["mirror"])
        ctx.set_frame_shading(hk.SHADE_MIRROR)
    # an animation is running: the frame before this one has been rendered
    before = None if state["mats"] is None else scenes.part_matrices(sc, frame - 1)
    torch.cuda.synchronize()
    ctx.frame(before, sc.camera, sc.lights, sc.width, sc.height, image.data_ptr(), state["mode"], variant)
    ctx.synchronize()
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "frame":
        state["ctx"].frame(state["mats"], state["cam"], state["lights"], state["w"], state["h"],
                           state["image"].data_ptr(), state["mode"], state["variant"])
        return state["image"]
    if kind == "rays":
        if "hits" not in state:
            hits = state["tree"].checkCollision(state["rays"], state["variant"])
            return {"t": hits["t"], "tri": hits["tri"]}
        state["tree"].ctx.trace_device(state["rays"].data_ptr(), state["rays"].shape[0], state["hits"].data_ptr(),
                                       state["variant"])
        return {"t": state["hits"][:, 0].view(torch.float32), "tri": state["hits"][:, 1]}
    if kind == "batch":
        state["batch"].trace_device(state["rays"].data_ptr(), state["offsets"], state["hits"].data_ptr(),
                                    state["variant"])
        return {"t": state["hits"][:, 0].view(torch.float32), "tri": state["hits"][:, 1]}
    if kind == "resort":
        stats = state["ctx"].build(hk.BUILD_SAH_RESORT)
        state["ctx"].render_device(state["cam"], state["lights"], state["w"], state["h"], state["image"].data_ptr(),
                                   state["variant"])
        return {"image": state["image"], "nodes": stats["nodes"], "refs": stats["refs"], "depth": stats["depth"]}
    if kind == "forward":
        return state["ctx"].mlp_forward(state["X"])
    grads, loss = state["ctx"].mlp_grad(state["X"], state["y"])
    return {"grads": grads, "loss": loss}


def _size(case):
    """(vertices, triangles) of a scene."""
    if case["scene"] == "parts":
        return case["parts"] * PART_VERTS, case["parts"] * PART_TRIS
    if case["scene"] == "spheres":
        return 13473, 24576
    return 3 * case["tris"] + 24 * 1089, case["tris"] + 24 * 2048


def work(case):
    kind = case["kind"]
    if kind in ("forward", "grad"):
        n, params = case["rows"], MLP_MACS + 256 * 3 + 96
        if kind == "forward":
            return {"bytes": 4 * (n * 296 + params), "flops": 2.0 * MLP_MACS * n}
        # weight gradients of every layer, input gradients of all but the first
        return {"bytes": 4 * (n * 201 + 2 * params), "flops": 2.0 * n * (3 * MLP_MACS - 200 * 256)}
    if kind == "batch":
        nt, nr = (sum(x) for x in zip(*_batch_sizes(case)))
        return {"bytes": 64 * nt + 40 * nr, "flops": 0}
    nv, nt = _size(case)
    if kind == "rays":
        # a ray in, a hit out; of the scene what the rays can touch
        return {"bytes": 40 * case["rays"] + min(64 * nt, 1000 * case["rays"]), "flops": 0}
    # vertices (and the part of each when it moves), triangles, the image
    return {"bytes": nv * (20 if case["scene"] == "parts" else 16) + nt * 16 + 4 * case["width"] * case["height"],
            "flops": 0}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _exact_hits(sc, rays):
    """Closest hits by testing every triangle (front and back faces, t >= 0)."""
    V = torch.tensor(sc.verts[:, :3], device="cuda").double()
    T = torch.tensor(sc.tris.view(np.int32), device="cuda").long()
    p, e0, e1 = V[T[:, 0]], V[T[:, 1]] - V[T[:, 0]], V[T[:, 2]] - V[T[:, 0]]
    n = torch.linalg.cross(e0, e1)
    e00, e01, e11 = (e0 * e0).sum(1), (e0 * e1).sum(1), (e1 * e1).sum(1)
    det = e00 * e11 - e01 * e01
    inf = torch.tensor(math.inf, device="cuda", dtype=torch.float64)
    best = []
    step = max(1, 20000000 // T.shape[0])
    for r in rays.double().split(step):
        o, d = r[:, :3], r[:, 4:7]
        t = ((p * n).sum(1) - o @ n.T) / (d @ n.T)
        c0 = o @ e0.T + t * (d @ e0.T) - (p * e0).sum(1)
        c1 = o @ e1.T + t * (d @ e1.T) - (p * e1).sum(1)
        a, b = (e11 * c0 - e01 * c1) / det, (e00 * c1 - e01 * c0) / det
        ok = (t >= 0) & (a >= 0) & (b >= 0) & (a + b <= 1)
        best.append(torch.where(ok, t, inf).min(1).values)
    return torch.cat(best)


def exact(case, seed):
    kind = case["kind"]
    if kind == "rays":
        if case["rays"] * _size(case)[1] > 2e10:
            return None
        sc = _scene(case, seed)
        return {"t": _exact_hits(sc, _rays(sc.verts, sc.tris, sc.camera, case["rays"], seed)).cpu(), "tri": None}
    if kind not in ("forward", "grad"):
        return None   # whole numbers (images), or too many rays
    X, y = _features(case["rows"], seed)
    params = _weights(seed) if kind == "grad" else np.fromfile(WEIGHTS, np.uint8)[28:].view(np.float32)
    P = torch.from_numpy(params.copy()).double().cuda().requires_grad_(kind == "grad")
    h, at = torch.from_numpy(X).double().cuda(), 0
    for i, (a, b) in enumerate(zip(MLP, MLP[1:])):
        h = h @ P[at:at + a * b].view(a, b) + P[at + a * b:at + a * b + b]
        at += a * b + b
        if i < 3:
            h = h.relu()
    if kind == "forward":
        return h.cpu()
    loss = torch.nn.functional.cross_entropy(h, torch.from_numpy(y).long().cuda())
    loss.backward()
    return {"grads": P.grad.cpu(), "loss": loss.detach().cpu()}
