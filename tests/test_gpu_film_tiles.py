"""The film gather against the oracle at film sizes where its tiles can go
wrong: narrower than a tile, one pixel more than tiles and half tiles, both
block heights, several passes; and films that hold non-finite samples (the
tested walk)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res", [(1, 1), (3, 40), (31, 17), (32, 16), (33, 33), (65, 49), (700, 5), (1000, 700)])
def test_film_sizes(W, O, ctx, res):
    g = W.SceneGen(0, 6, res)
    ctx.set_quirks(0)
    ctx.upload(g.desc)
    ctx.build()
    spp = 1 if res[0] * res[1] > 100000 else 3
    ctx.render_setup(spp, seed=8)
    ctx.render()
    L, w = ctx.film(*res)
    Lo, wo = O.OracleScene(g.desc).render(res[0], res[1], spp, 8)
    assert np.array_equal(w.view(np.uint32), wo.view(np.uint32))
    # (NaN payloads differ between device and host)
    assert np.all((L.view(np.uint32) == Lo.view(np.uint32)) | (np.isnan(L) & np.isnan(Lo)))


def test_non_finite_samples(W, O, ctx):
    # an environment map with infinite and NaN texels: their samples and no
    # others become non-finite pixels
    g = W.SceneGen(2, 1, (70, 50), level=3)
    e = g.desc.contents.envmap.contents
    rgb = np.ctypeslib.as_array(e.rgb, shape=(e.height, e.width, 3))
    keep = rgb.copy()
    rgb[e.height // 3:e.height // 3 + 40, ::3] = np.inf
    rgb[e.height // 3:e.height // 3 + 40, 1::3, 1] = np.nan
    try:
        ctx.set_quirks(0)
        ctx.upload(g.desc)
        ctx.build()
        ctx.render_setup(2, seed=3)
        ctx.render()
        L, w = ctx.film(70, 50)
        Lo, wo = O.OracleScene(g.desc).render(70, 50, 2, 3)
        assert not np.isfinite(L).all() and np.isfinite(L).any()
        assert np.array_equal(w.view(np.uint32), wo.view(np.uint32))
        assert np.all((L.view(np.uint32) == Lo.view(np.uint32)) | (np.isnan(L) & np.isnan(Lo)))
    finally:
        rgb[:] = keep
