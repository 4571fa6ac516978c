"""Builds around the sizes where the build changes its kernels (one-block order
and scans, one-launch SAH start) against the oracle: the tree, its order and
its bounds; both sort orders; primitives that share one code; and one context
built at alternating sizes."""
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
