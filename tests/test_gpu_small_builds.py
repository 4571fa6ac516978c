"""Builds around the sizes where the build changes its kernels (one-block order
and scans, one-launch SAH start) against the oracle: the tree, its order and
its bounds; both sort orders; primitives that share one code; and one context
built at alternating sizes."""
import zlib

import numpy as np
import pytest
from scenes import cluster_desc, mesh_desc
from test_gpu_bvh import compare_build

pytestmark = pytest.mark.gpu


def soup(n, seed):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1, 1, (n, 1, 3)) ** 3
    tris = (c + rng.normal(0, 0.02, (n, 3, 3))).astype(np.float32)
    return mesh_desc(tris.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32))


@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 255, 1023, 1025, 4095, 4096, 4097, 8191, 8192, 8193, 16385])
@pytest.mark.parametrize("full", [False, True])
def test_sizes(W, O, ctx, n, full):
    d, keep = soup(n, n)
    compare_build(W, O, ctx, d, W.Q_FULL_MORTON_SORT if full else 0)
    ctx.set_quirks(0)


@pytest.mark.parametrize("k", [40, 4000, 8000])
def test_one_code(W, O, ctx, k):
    d, keep = cluster_desc(k)
    compare_build(W, O, ctx, d)


def test_alternating_sizes(W, O, ctx):
    for n in (9000, 60, 5000, 2, 20000, 700):
        d, keep = soup(n, n + 1)
        compare_build(W, O, ctx, d)


@pytest.mark.parametrize("config,level,seed,row,crc", [
    (0, 0, 0, 0, 0xc608f3e0), (0, 0, 2, 1, 0xd7fe3ee3), (2, 2, 3, 0, 0x41cf4e4a), (2, 4, 3, 2, 0x04ab9671),
    (3, 1, 0, 0, 0xc4966775), (3, 1, 2, 1, 0x5b5a3afc), (3, 1, 4, 2, 0x093bb4f1), (3, 1, 5, 0, 0x1ea60681),
])
def test_bounds_that_hold_a_nan(W, config, level, seed, row, crc):
    # one sphere's finite transform overflows to inf - inf; the trees of such
    # scenes follow from how the NaN travels, and stay as they were
    g = W.SceneGen(config, seed, (64, 20000), level=level)
    s = g.desc.contents.spheres[5]
    s.radius = 2.0
    s.world_to_object.m[3] = 1e6
    for c, v in enumerate([3e38, -3e38, 0.0, 0.0]):
        s.object_to_world.m[4 * row + c] = v
    with W.Context(0) as c:
        c.upload(g.desc)
        c.build()
        e = c.bvh_export()
    assert np.isnan(e["node_bounds"]).any()
    assert zlib.crc32(e["nodes"].tobytes() + e["node_bounds"].tobytes()) == crc
