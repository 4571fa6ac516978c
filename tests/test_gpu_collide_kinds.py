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
