"""Film reads on both sides of the size from which the film is split on the
device: against the oracle, and either array alone."""
import numpy as np
import pytest

from woodenpbrengine_gb300 import lib, _fp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res", [(1, 1), (96, 128), (12289, 1), (200, 150)])
def test_film_read(W, O, ctx, res):
    g = W.SceneGen(0, 3, res)
    ctx.set_quirks(0)
    ctx.upload(g.desc)
    ctx.build()
    ctx.render_setup(2, seed=5)
    ctx.render()
    Lo, wo = O.OracleScene(g.desc).render(res[0], res[1], 2, 5)
    n = res[0] * res[1]
    for _ in range(2):
        L, w = ctx.film(*res)
        assert np.array_equal(w, wo)
        # (NaN payloads differ between device and host)
        assert np.all((L.view(np.uint32) == Lo.view(np.uint32)) | (np.isnan(L) & np.isnan(Lo)))
    only_L, only_w = np.full(n * 3 + 1, -7, np.float32), np.full(n + 1, -7, np.float32)
    assert lib().wpbr_film_read(ctx._h, _fp(only_L), None) == 0
    assert lib().wpbr_film_read(ctx._h, None, _fp(only_w)) == 0
    assert only_L[-1] == -7 and only_w[-1] == -7
    assert np.array_equal(only_L[:-1].view(np.uint32), L.reshape(-1).view(np.uint32))
    assert np.array_equal(only_w[:-1], w.reshape(-1))
