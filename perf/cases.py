"""Workloads of the ray pipeline as a program that uses the library runs them.

Four families, each through the public binding:

* rays    a batch of rays against a built scene (`Context.collide_device`, or
          `Context.collide` with host arrays): picking, occlusion queries, the
          ray microbenchmark;
* build   a scene that changed: (upload,) LBVH build, and the first rays
          against the new tree, which are the part of the tree a caller sees;
* frame   a whole frame: `render_setup` (clears the film), `render`, and the
          film read back; one scene or a batch of scenes;
* adjoint one optimisation step of the differentiable estimator: new
          parameters, frozen directions, forward with loss, backward.

Scenes come from the library's own seeded generators (their configurations 0
to 5 are the ones the benchmark and the tests use); rays are drawn here.
"""
import math

import numpy as np
import torch

import woodenpbrengine_gb300 as W

DEV = "cuda"


def listed():
    return [
        # mouse picking / physics probes: a thousand rays against a small scene of spheres and a ground quad
        {"name": "rays_pick_1k", "kind": "rays", "config": 0, "level": 0, "rays": 1000, "mode": "closest", "mix": "aimed",
         "host": False},
        # line-of-sight queries of a frame's worth of agents: any-hit segments over a mid-size mesh
        {"name": "rays_occlusion_100k", "kind": "rays", "config": 1, "level": 6, "rays": 100003, "mode": "any",
         "mix": "segments", "host": False},
        # an engine that keeps its rays in host memory: the whole call, copies included
        {"name": "rays_host_300k", "kind": "rays", "config": 1, "level": 7, "rays": 300001, "mode": "closest",
         "mix": "benchmark", "host": True},
        # the LBVH microbenchmark: half coherent camera rays, half incoherent surface rays, 1.31 M triangles
        {"name": "rays_large_8m", "kind": "rays", "config": 1, "level": 8, "rays": 8388608, "mode": "closest",
         "mix": "benchmark", "host": False},
        # a level change: a small scene with an environment map is uploaded and built, then first probed
        {"name": "scene_load_5k", "kind": "build", "config": 2, "level": 4, "upload": True, "rays": 4096},
        # the build of the microbenchmark's mesh, and the first rays against it
        {"name": "build_1m", "kind": "build", "config": 1, "level": 8, "upload": False, "rays": 65536},
        # preview of the plain scene
        {"name": "frame_preview_256", "kind": "frame", "config": 0, "level": 0, "width": 256, "height": 256, "spp": 4,
         "spectral": False},
        # the full frame: mesh, spheres, glass and environment light at 1080p
        {"name": "frame_full_1080p", "kind": "frame", "config": 2, "level": 8, "width": 1920, "height": 1080, "spp": 16,
         "spectral": False},
        # the same scene kind in the 64-bin spectral mode, at an odd film size
        {"name": "frame_spectral_1001", "kind": "frame", "config": 2, "level": 6, "width": 1001, "height": 563, "spp": 8,
         "spectral": True},
        # textured metal: MIP-mapped lookups at every hit
        {"name": "frame_textured_1080p", "kind": "frame", "config": 5, "level": 0, "width": 1920, "height": 1080, "spp": 16,
         "spectral": False},
        # thumbnails of many uneven scenes in one batch
        {"name": "frame_batch_12", "kind": "batch", "set": 3, "scenes": 12, "film": 512, "prims": 50000, "spp": 4},
        # inverse rendering: one optimisation step over 98,944 parameters
        {"name": "adjoint_step_512", "kind": "adjoint", "width": 512, "height": 512, "spp": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "rays", "build", "frame", "frame", "batch", "adjoint"])
    if kind == "rays":
        config = rng.choice([0, 1, 1])
        host = rng.random() < 0.25
        mode = rng.choice(["closest", "any"])
        return {"kind": kind, "config": config, "level": rng.randint(3, 8) if config == 1 else 0,
                "rays": _log_int(rng, 500, 1000000 if host else 4000000), "mode": mode,
                "mix": rng.choice(["aimed", "segments"] if config == 0 else ["aimed", "segments", "benchmark"]), "host": host}
    if kind == "build":
        config = rng.choice([0, 1, 2])
        return {"kind": kind, "config": config, "level": rng.randint(2, 8 if config == 1 else 6) if config else 0,
                "upload": config != 1, "rays": _log_int(rng, 1000, 65536)}
    if kind == "frame":
        config = rng.choice([0, 2, 5])
        w, h = _log_int(rng, 120, 1500), _log_int(rng, 90, 1000)
        spectral = rng.random() < 0.3
        return {"kind": kind, "config": config, "level": rng.randint(4, 7) if config == 2 else 0, "width": w, "height": h,
                "spp": rng.choice([1, 2, 4, 6, 8] if spectral else [1, 3, 4, 8, 16]), "spectral": spectral}
    if kind == "batch":
        return {"kind": kind, "set": rng.randint(1, 99), "scenes": rng.randint(2, 12), "film": _log_int(rng, 100, 512), "prims": _log_int(rng, 10000, 50000),
                "spp": rng.choice([1, 2, 4])}
    return {"kind": kind, "width": _log_int(rng, 60, 512), "height": _log_int(rng, 60, 512), "spp": rng.choice([1, 2, 5, 8, 16])}


# ---- inputs -------------------------------------------------------------------


def _mesh(desc):
    """(positions (V, 3), indices (T, 3)) of a scene's triangles on the device."""
    d = desc.contents
    pos = np.ctypeslib.as_array(d.positions, shape=(d.n_vertices, 3)).astype(np.float32)
    idx = np.ctypeslib.as_array(d.indices, shape=(d.n_triangles, 3)).astype(np.int64)
    return torch.from_numpy(pos).to(DEV), torch.from_numpy(idx).to(DEV)


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _surface(mesh, n, gen):
    """Area-weighted surface points moved 1e-4 along the outward normal, and the normals."""
    pos, idx = mesh
    a, b, c = pos[idx[:, 0]], pos[idx[:, 1]], pos[idx[:, 2]]
    cdf = torch.linalg.cross(b - a, c - a).norm(dim=1).double().cumsum(0)
    u = torch.rand(n, generator=gen, device=DEV, dtype=torch.float64) * cdf[-1]
    t = torch.searchsorted(cdf, u).clamp_(max=idx.shape[0] - 1)
    a, b, c = a[t], b[t], c[t]
    s = torch.rand(n, 1, generator=gen, device=DEV).sqrt()
    r = torch.rand(n, 1, generator=gen, device=DEV)
    p = a * (1 - s) + b * (s * r) + c * (s - s * r)
    nrm = _unit(torch.linalg.cross(b - a, c - a))
    nrm = torch.where((nrm * p).sum(1, keepdim=True) < 0, -nrm, nrm)
    return p + 1e-4 * nrm, nrm


def _camera_rays(n, gen, radius):
    """n rays of a pinhole at a random side of the scene, in film order."""
    side = max(1, math.isqrt(n))
    i = torch.arange(n, device=DEV)
    x, y = (i % side).float(), torch.div(i, side, rounding_mode="floor").float()
    eye = _unit(torch.randn(1, 3, generator=gen, device=DEV)) * radius
    f = -_unit(eye)
    up = torch.tensor([[0.0, 1.0, 0.0]], device=DEV)
    r = _unit(torch.linalg.cross(f, up))
    q = torch.linalg.cross(r, f)
    s = 2 * math.tan(math.radians(22.5)) / side
    d = f + r * ((x + 0.5 - side / 2) * s)[:, None] + q * ((y + 0.5 - n / side / 2) * s)[:, None]
    return eye.expand(n, 3), _unit(d)


def _rays(desc, config, n, mix, seed):
    """(n, 8) rays: origin, 0, direction, tmax."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    out = torch.zeros(n, 8, device=DEV)
    out[:, 7] = math.inf
    extent = 10.0 if config in (0, 2) else 1.0

    def rand(k, half):
        return (torch.rand(k, 3, generator=gen, device=DEV) * 2 - 1) * half

    if mix == "aimed":  # from around the scene towards points in it
        o = _unit(torch.randn(n, 3, generator=gen, device=DEV)) * (2.5 * extent)
        out[:, 0:3], out[:, 4:7] = o, _unit(rand(n, 0.9 * extent) - o)
    elif mix == "segments":  # from a surface (or inside a sphere scene) to a point, no further than it
        if config == 1:
            o, _ = _surface(_mesh(desc), n, gen)
        else:
            o = rand(n, extent)
        to = rand(n, 2.0 * extent) - o
        out[:, 0:3], out[:, 4:7], out[:, 7] = o, _unit(to), to.norm(dim=1)
    else:  # half camera rays, half cosine-distributed rays off the surface
        k = n // 2
        out[:k, 0:3], out[:k, 4:7] = _camera_rays(k, gen, 2.4 * extent)
        o, nrm = _surface(_mesh(desc), n - k, gen)
        d = _unit(nrm + _unit(torch.randn(n - k, 3, generator=gen, device=DEV)))
        out[k:, 0:3], out[k:, 4:7] = o, d
    return out


def _scene(case, seed, res=(64, 64)):
    return W.SceneGen(case["config"], seed & 0xFFFFFF, res, level=case.get("level", 0))


def _context(torch_stream):
    ctx = W.Context(torch.cuda.current_device())
    if torch_stream:  # device tensors are produced and consumed on torch's stream
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    return ctx


def _adjoint_params(desc):
    d = desc.contents
    mat = np.zeros((d.n_materials, 10), np.float32)
    for i in range(d.n_materials):
        m = d.materials[i]
        mat[i] = [m.alpha_x, *m.R, *m.eta_t, *m.k]
    e = d.envmap.contents
    env = np.ctypeslib.as_array(e.rgb, shape=(e.height * e.width * 3,)).astype(np.float32)
    return torch.from_numpy(mat.reshape(-1)).to(DEV), torch.from_numpy(env).to(DEV)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "seed": seed & 0xFFFFFF}
    if kind == "rays":
        g = _scene(case, seed)
        s["ctx"] = ctx = _context(not case["host"])
        ctx.upload(g.desc)
        ctx.build()
        rays = _rays(g.desc, case["config"], case["rays"], case["mix"], seed)
        if case["host"]:
            s["rays"] = rays.cpu().numpy()
        else:
            s["rays"], s["hits"] = rays, torch.empty(case["rays"], 4, device=DEV)
    elif kind == "build":
        s["scene"] = _scene(case, seed)
        s["ctx"] = ctx = _context(True)
        ctx.upload(s["scene"].desc)
        s["rays"] = _rays(s["scene"].desc, case["config"], case["rays"], "aimed", seed)
        s["hits"] = torch.empty(case["rays"], 4, device=DEV)
    elif kind == "frame":
        g = _scene(case, seed, (case["width"], case["height"]))
        s["ctx"] = ctx = _context(False)
        if case["spectral"]:
            ctx.set_spectrum(W.SPECTRUM_SAMPLED64)
        ctx.upload(g.desc)
        ctx.build()
    elif kind == "batch":
        s["batch"] = b = W.Batch(torch.cuda.current_device())
        for k in range(case["scenes"]):  # the set fixes the film sizes, the seed the samples
            g = W.SceneGen(3, case["set"], (case["film"], case["prims"]), level=k)
            b.add(g.desc)
            g.close()
        b.build()
    else:
        res = (case["width"], case["height"])
        start = W.SceneGen(4, seed & 0xFFFFFF, res, level=1 + (seed & 0xFFFF))
        goal = W.SceneGen(4, seed & 0xFFFFFF, res, level=2 + (seed & 0xFFFF))
        s["ctx"] = ctx = _context(True)
        ctx.upload(goal.desc)
        ctx.build()
        n_mat, n_env = ctx.adjoint_setup(case["spp"], seed=s["seed"])
        s["target"] = torch.empty(res[0] * res[1] * 3, device=DEV)
        ctx.adjoint_forward_device(None, s["target"].data_ptr())
        s["mat"], s["env"] = _adjoint_params(start.desc)
        s["grad_mat"], s["grad_env"] = torch.empty(n_mat, device=DEV), torch.empty(n_env, device=DEV)
    return s


# ---- one pass -----------------------------------------------------------------


def _hits(h, mode):
    if mode == "any":  # occlusion only: whether the segment hits
        return {"occluded": torch.isfinite(h[:, 0]) if isinstance(h, torch.Tensor) else np.isfinite(h[:, 0])}
    ids = h[:, 1].view(torch.int32) if isinstance(h, torch.Tensor) else np.ascontiguousarray(h[:, 1]).view(np.int32)
    return {"t": h[:, 0], "prim": ids, "bary": h[:, 2:4]}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "rays":
        mode = W.TRACE_ANY if case["mode"] == "any" else W.TRACE_CLOSEST
        if case["host"]:
            return _hits(s["ctx"].collide(s["rays"], mode), case["mode"])
        s["ctx"].collide_device(s["rays"].data_ptr(), case["rays"], s["hits"].data_ptr(), mode)
        return _hits(s["hits"], case["mode"])
    if kind == "build":
        ctx = s["ctx"]
        if case["upload"]:
            ctx.upload(s["scene"].desc)
        ctx.build()
        ctx.collide_device(s["rays"].data_ptr(), case["rays"], s["hits"].data_ptr())
        return {**_hits(s["hits"], "closest"), "tree": ctx.bvh_info()}
    if kind == "frame":
        ctx = s["ctx"]
        ctx.render_setup(case["spp"], seed=s["seed"])
        ctx.render()
        L, w = ctx.film(case["width"], case["height"])
        return {"L": L, "w": w}
    if kind == "batch":
        b = s["batch"]
        b.render_setup(case["spp"], seed=s["seed"])
        b.render()
        return [b.film(k) for k in range(case["scenes"])]
    ctx = s["ctx"]
    ctx.adjoint_set_params_device(s["mat"].data_ptr(), s["env"].data_ptr())
    ctx.adjoint_freeze()
    loss = ctx.adjoint_forward_device(s["target"].data_ptr())
    ctx.adjoint_backward_device(s["grad_mat"].data_ptr(), s["grad_env"].data_ptr())
    return {"loss": loss, "grad_mat": s["grad_mat"], "grad_env": s["grad_env"]}


# ---- what a pass cannot do without --------------------------------------------


def _prims(case):
    mesh = 20 * 4 ** case["level"]
    return {0: 67, 1: mesh, 2: mesh + 256, 5: 67}[case["config"]]


def _ray_flops(prims):
    """A near-first descent tests two boxes a level (24 flops each) and a few primitives (40 flops each)."""
    return 48 * math.log2(max(prims, 2)) + 160


def work(case):
    kind = case["kind"]
    if kind == "rays":
        prims = _prims(case)
        return {"bytes": 48 * case["rays"] + 36 * prims, "flops": case["rays"] * _ray_flops(prims)}
    if kind == "build":
        # vertices and indices in, node and primitive records out; a comparison sort and a box union per primitive
        prims = _prims(case)
        return {"bytes": (18 + 64 + 48) * prims + 48 * case["rays"],
                "flops": prims * (60 + 2 * math.log2(max(prims, 2))) + case["rays"] * _ray_flops(prims)}
    if kind == "frame":
        prims, n = _prims(case), case["width"] * case["height"]
        per = 400 + (64 * 60 if case["spectral"] else 0) + 2 * _ray_flops(prims)
        return {"bytes": 16 * n + 84 * prims, "flops": n * case["spp"] * per}
    if kind == "batch":  # films of half the cap on average
        n = case["scenes"] * (0.6 * case["film"]) ** 2
        return {"bytes": 16 * n + 84 * case["scenes"] * 20000, "flops": n * case["spp"] * (400 + 2 * _ray_flops(20000))}
    n = case["width"] * case["height"]
    return {"bytes": n * 28 + 98944 * 8, "flops": n * case["spp"] * (1600 + 2 * _ray_flops(66))}


# ---- references in 64 bits ----------------------------------------------------


def _exact_hits(desc, rays, chunk=1 << 22):
    """Closest hits by testing every primitive, in float64: (t, (b1, b2))."""
    d = desc.contents
    o, v, tmax = rays[:, 0:3].double(), rays[:, 4:7].double(), rays[:, 7].double()
    n = o.shape[0]
    best = torch.full((n,), math.inf, dtype=torch.float64, device=DEV)
    bary = torch.zeros(n, 2, dtype=torch.float64, device=DEV)
    for i in range(d.n_spheres):
        m = torch.tensor(list(d.spheres[i].world_to_object.m), dtype=torch.float64, device=DEV).reshape(4, 4)
        oo, dd = o @ m[:3, :3].T + m[:3, 3], v @ m[:3, :3].T
        a, b, c = (dd * dd).sum(1), 2 * (dd * oo).sum(1), (oo * oo).sum(1) - float(d.spheres[i].radius) ** 2
        disc = b * b - 4 * a * c
        root = disc.clamp(min=0).sqrt()
        t0, t1 = (-b - root) / (2 * a), (-b + root) / (2 * a)
        t = torch.where(t0 <= 0, t1, t0)
        best = torch.where((disc >= 0) & (t1 > 0) & (t < tmax) & (t < best), t, best)
    if d.n_triangles:
        pos, idx = _mesh(desc)
        pos = pos.double()
        p0, e1, e2 = pos[idx[:, 0]], pos[idx[:, 1]] - pos[idx[:, 0]], pos[idx[:, 2]] - pos[idx[:, 0]]
        step = max(1, chunk // idx.shape[0])
        for at in range(0, n, step):
            r, q = o[at:at + step, None], v[at:at + step, None]
            h = torch.linalg.cross(q.expand(-1, idx.shape[0], 3), e2[None].expand(r.shape[0], -1, 3))
            det = (e1[None] * h).sum(2)
            s = r - p0[None]
            u = (s * h).sum(2) / det
            k = torch.linalg.cross(s, e1[None].expand(r.shape[0], -1, 3))
            w = (q * k).sum(2) / det
            t = (e2[None] * k).sum(2) / det
            ok = (det != 0) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0) & (t < tmax[at:at + step, None])
            t = torch.where(ok, t, math.inf)
            tt, j = t.min(1)
            near = tt < best[at:at + step]
            uv = torch.stack([u.gather(1, j[:, None])[:, 0], w.gather(1, j[:, None])[:, 0]], 1)
            bary[at:at + step] = torch.where(near[:, None], uv, bary[at:at + step])
            best[at:at + step] = torch.where(near, tt, best[at:at + step])
    return best, bary


def _philox(c0, c1, c2, k0, k1):
    """Philox-4x32-10 of the counters (c0, c1, c2, 0): the first two output words."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [np.asarray(x, np.uint64) * np.ones_like(np.asarray(c0, np.uint64)) for x in (c0, c1, c2, 0)]
    for r in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        x, y = np.uint64((k0 + r * 0x9E3779B9) & 0xFFFFFFFF), np.uint64((k1 + r * 0xBB67AE85) & 0xFFFFFFFF)
        c = [(b >> np.uint64(32)) ^ c[1] ^ x, b & m32, (a >> np.uint64(32)) ^ c[3] ^ y, a & m32]
    return c[0], c[1]


def _mitchell(x):
    """Mitchell-Netravali filter (B = C = 1/3) of radius 2, without its normalisation over the plane."""
    x = np.abs(x)
    far = ((-7 / 3 * x + 12) * x - 20) * x + 32 / 3
    return np.where(x > 1, far, (7 * x - 12) * x * x + 16 / 3) / 6


def _exact_weights(width, height, spp, seed):
    """Film weights: the filter summed over every pass's camera samples, within 32 x 32 tiles."""
    pix = np.arange(width * height, dtype=np.uint64)
    px, py = (pix % np.uint64(width)).astype(np.int64), (pix // np.uint64(width)).astype(np.int64)
    nx = max(d for d in range(1, spp + 1) if d * d <= spp and spp % d == 0)
    offset = (_philox(pix, 0xFFFFFFFF, 0, seed, 0)[0] % np.uint64(spp)).astype(np.int64)
    w = np.zeros(width * height)
    for p in range(spp):
        a, b = _philox(pix, p, 0, seed, 0)
        k = (p + offset) % spp
        fx = px + (k % nx + (a >> np.uint64(8)).astype(np.float64) * 2.0 ** -24) / nx
        fy = py + (k // nx + (b >> np.uint64(8)).astype(np.float64) * 2.0 ** -24) / (spp // nx)
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                x, y = px + dx, py + dy
                ok = (x >= px // 32 * 32) & (x < np.minimum(px // 32 * 32 + 32, width))
                ok &= (y >= py // 32 * 32) & (y < np.minimum(py // 32 * 32 + 32, height))
                ok &= (np.abs(x - fx + 0.5) <= 2) & (np.abs(y - fy + 0.5) <= 2)
                np.add.at(w, (y * width + x)[ok], (_mitchell(x - fx) * _mitchell(y - fy))[ok])
    return w.reshape(height, width)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("rays", "build") and case.get("mode") != "any" and case["rays"] * _prims(case) <= 3e8:
        g = _scene(case, seed)
        rays = _rays(g.desc, case["config"], case["rays"], case.get("mix", "aimed"), seed)
        t, bary = _exact_hits(g.desc, rays)
        out = {"t": t, "prim": None, "bary": bary}
        return out if kind == "rays" else {**out, "tree": None}
    if kind == "frame" and case["width"] * case["height"] * case["spp"] <= 1 << 21:
        return {"L": None, "w": _exact_weights(case["width"], case["height"], case["spp"], seed & 0xFFFFFF)}
    return None
