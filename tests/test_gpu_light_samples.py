"""The fused passes with and without the environment light's sampled radiance
(they leave out draws that cannot contribute): films against the oracle, RGB and
Sampled64, on a scene with an environment light only and one with both kinds of
light."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(a, b):
    return np.all((a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b)))


@pytest.mark.parametrize("config,level", [(2, 3), (4, 1)])
@pytest.mark.parametrize("quirks", [0, 2])
@pytest.mark.parametrize("spectral", [False, True])
def test_films(W, O, config, level, quirks, spectral):
    assert quirks in (0, W.Q_ENV_LI_SAMPLE_FIX)
    res, spp = (48, 40), 3
    g = W.SceneGen(config, 5, res, level=level)
    with W.Context(0) as ctx:
        ctx.set_quirks(quirks)
        if spectral:
            ctx.set_spectrum(W.SPECTRUM_SAMPLED64)
        ctx.upload(g.desc)
        ctx.build()
        ctx.render_setup(spp, seed=9)
        ctx.render()
        L, w = ctx.film(*res)
        ctx.check_device_errors()
    o = O.OracleScene(g.desc, quirks)
    Lo, wo = (o.render_spectral if spectral else o.render)(res[0], res[1], spp, 9)
    assert same(w, wo) and same(L, Lo)
    assert (L > 0).any()
