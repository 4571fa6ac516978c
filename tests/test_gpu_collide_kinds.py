"""Collide batches against the oracle over the kernels a batch can take: scenes
of triangles only, of spheres and a quad, and of both; batches of one ray a warp
up to full warps, with and without rays left for the warps to fetch, in input
order and (2^19 rays and more) in ray order; bounded and unbounded rays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def random_rays(n, extent, seed):
    rng = np.random.default_rng(seed)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = rng.uniform(-1.5 * extent, 1.5 * extent, (n, 3))
    d = rng.uniform(-extent, extent, (n, 3)) - rays[:, :3]
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = np.where(rng.random(n) < 0.3, rng.uniform(0.1, extent, n), np.inf)
    return rays


@pytest.mark.parametrize("config,level,extent", [(1, 3, 1.2), (0, 0, 12.0), (2, 4, 12.0)])
@pytest.mark.parametrize("n", [1, 33, 2433, 5000, 77825, 155649, (1 << 19) + 7])
def test_scene_kinds(W, O, ctx, config, level, extent, n):
    g = W.SceneGen(config, 11, (64, 64), level=level)
    ctx.set_quirks(0)
    ctx.set_traversal(W.TRAVERSAL_BINARY)
    ctx.upload(g.desc)
    ctx.build()
    rays = random_rays(n, extent, n)
    hg, ag = ctx.collide(rays), ctx.collide(rays, mode=W.TRACE_ANY)
    at = np.arange(n) if n <= 5000 else np.random.default_rng(1).choice(n, 20000, replace=False)
    ho = O.OracleScene(g.desc).trace(rays[at], mode=0)  # of the unbounded rays
    beyond = ~(ho[:, 0] < rays[at, 7])
    ho[beyond] = np.array([np.inf, 0, 0, 0], np.float32)
    ho.view(np.uint32)[beyond, 1] = 0xFFFFFFFF
    assert np.array_equal(hg[at].view(np.uint32), ho.view(np.uint32))
    assert np.array_equal(np.isfinite(ag[:, 0]), np.isfinite(hg[:, 0]))
    ctx.check_device_errors()


@pytest.mark.parametrize("row", [0, 1, 2])
def test_bounds_that_hold_a_nan(W, row):
    # a finite transform that overflows to inf - inf gives one sphere's bounds,
    # and those of nodes above it, a NaN: boxes are still decided as the
    # statistics kernel decides them, over the same leaves (the sphere itself
    # is where no ray meets it: its hits would lie outside such a box)
    g = W.SceneGen(2, 3, (32, 32), level=2)
    s = g.desc.contents.spheres[5]
    s.radius = 2.0
    for c, v in enumerate([3e38, -3e38, 0.0, 0.0]):
        s.object_to_world.m[4 * row + c] = v
    s.world_to_object.m[3] = 1e6
    rays = random_rays(20000, 12.0, 5)
    with W.Context(0) as c:
        c.upload(g.desc)
        c.build()
        assert np.isnan(c.bvh_export()["node_bounds"]).any()
        c.set_traversal(W.TRAVERSAL_BINARY_FULL_LEAVES)
        hits = c.collide(rays)
        want, _ = c.collide(rays, stats=True)
        c.check_device_errors()
    assert np.array_equal(hits.view(np.uint32), want.view(np.uint32))
