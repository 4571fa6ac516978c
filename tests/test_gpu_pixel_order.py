"""The material order of large films (tiles of 8,192 pixels) against the
oracle: whole tiles, one pixel more and one less than whole tiles, scenes of
spheres and triangles and of textured metals, RGB and Sampled64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res", [(512, 256), (43691, 3), (46421, 3)])
@pytest.mark.parametrize("config,spectral", [(0, False), (5, False), (0, True)])
def test_films(W, O, ctx, res, config, spectral):
    assert res[0] * res[1] >= 1 << 17 and res[0] * res[1] % 8192 in (0, 1, 8191)
    g = W.SceneGen(config, 2, res)
    ctx.set_quirks(0)
    ctx.set_spectrum(W.SPECTRUM_SAMPLED64 if spectral else W.SPECTRUM_RGB)
    try:
        ctx.upload(g.desc)
        ctx.build()
        ctx.render_setup(1, seed=6)
        ctx.render()
        L, w = ctx.film(*res)
    finally:
        ctx.set_spectrum(W.SPECTRUM_RGB)
    o = O.OracleScene(g.desc)
    Lo, wo = (o.render_spectral if spectral else o.render)(res[0], res[1], 1, 6)
    assert np.array_equal(w, wo)
    # (NaN payloads differ between device and host)
    assert np.all((L.view(np.uint32) == Lo.view(np.uint32)) | (np.isnan(L) & np.isnan(Lo)))
    ctx.check_device_errors()
