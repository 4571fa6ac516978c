"""The 64-bin film gather against the oracle at film sizes where its blocks can
go wrong (a film tile's width, four rows, two pixels a thread): narrower and
one pixel more than those, odd heights, one and several passes; and a film that
holds non-finite samples (the tested walk)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _film(W, O, ctx, g, res, spp, seed):
    ctx.set_quirks(0)
    ctx.set_spectrum(W.SPECTRUM_SAMPLED64)
    try:
        ctx.upload(g.desc)
        ctx.build()
        ctx.render_setup(spp, seed=seed)
        ctx.render()
        L, w = ctx.film(*res)
    finally:
        ctx.set_spectrum(W.SPECTRUM_RGB)
    Lo, wo = O.OracleScene(g.desc).render_spectral(res[0], res[1], spp, seed)
    assert np.array_equal(w.view(np.uint32), wo.view(np.uint32))
    # (NaN payloads differ between device and host)
    assert np.all((L.view(np.uint32) == Lo.view(np.uint32)) | (np.isnan(L) & np.isnan(Lo)))
    return L


@pytest.mark.parametrize("res", [(1, 1), (2, 5), (31, 33), (32, 4), (33, 3), (65, 37), (300, 2)])
@pytest.mark.parametrize("spp", [1, 2, 4])
def test_film_sizes(W, O, ctx, res, spp):
    _film(W, O, ctx, W.SceneGen(0, 6, res), res, spp, 8)


@pytest.mark.parametrize("spp", [1, 2])
def test_non_finite_samples(W, O, ctx, spp):
    g = W.SceneGen(2, 1, (70, 50), level=3)
    e = g.desc.contents.envmap.contents
    rgb = np.ctypeslib.as_array(e.rgb, shape=(e.height, e.width, 3))
    keep = rgb.copy()
    rgb[e.height // 3:e.height // 3 + 40, ::3] = np.inf
    rgb[e.height // 3:e.height // 3 + 40, 1::3, 1] = np.nan
    try:
        L = _film(W, O, ctx, g, (70, 50), spp, 3)
        assert not np.isfinite(L).all() and np.isfinite(L).any()
    finally:
        rgb[:] = keep


def test_more_rows_than_a_grid_dimension_of_blocks(W, O, ctx):
    # 4 pixel rows a block: more than 65,535 rows of blocks
    _film(W, O, ctx, W.SceneGen(0, 6, (1, 262150)), (1, 262150), 1, 8)
