"""Texture lookups against the oracle at texture sizes where the walks can go
wrong: the smallest, long rows and columns, even and odd widths (the elliptical
walk takes a row's texels in pairs), and texels that are not finite (texels
outside the ellipse must not enter a sum)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RES = (96, 64)


@pytest.mark.parametrize("size", [(4, 4), (5, 4), (4, 9), (7, 6), (5, 64), (64, 5), (255, 130)])
@pytest.mark.parametrize("odd_texels", [False, True])
def test_texture_sizes(W, O, ctx, size, odd_texels):
    g = W.SceneGen(5, 0, RES)
    d = g.desc.contents
    rng = np.random.default_rng(5)
    texs = (type(d.textures[0]) * d.n_textures)()
    keep = []
    for i in range(d.n_textures):
        # roughness textures: log-uniform like the scene's own
        rgb = rng.uniform(0.2, 3.0, (size[1], size[0], 3)) if i % 2 == 0 else 10 ** rng.uniform(-5, -2, (size[1], size[0], 3))
        rgb = np.ascontiguousarray(rgb, np.float32)
        if odd_texels:
            rgb.reshape(-1, 3)[::7] = [np.inf, np.nan, 1.0]
        keep.append(rgb)
        texs[i].width, texs[i].height = size
        texs[i].rgb = rgb.ctypes.data_as(type(texs[i].rgb))
    d2 = type(d).from_buffer_copy(d)
    d2.textures = C.cast(texs, type(d.textures))
    ctx.set_quirks(0)
    ctx.upload(C.pointer(d2))
    ctx.build()
    ctx.render_setup(2, seed=4)
    ctx.render()
    L, w = ctx.film(*RES)
    Lo, wo = O.OracleScene(C.pointer(d2)).render(RES[0], RES[1], 2, 4)
    assert np.array_equal(w, wo)
    # (NaN payloads differ between device and host)
    assert np.all((L.view(np.uint32) == Lo.view(np.uint32)) | (np.isnan(L) & np.isnan(Lo)))
    assert np.isfinite(L).any()


@pytest.mark.parametrize("size", [(4, 4), (7, 6), (255, 130)])
@pytest.mark.parametrize("res,spectral", [((728, 728), False), ((1031, 1031), True)])
def test_both_builds_of_the_spawn(W, size, res, spectral):
    # single passes take the wide build, groups of more than 2^22 pixels in
    # flight (8 passes, Sampled64 4 and 3 x 2^20) the compact one: the same film,
    # over finite texels and some that are not
    spp = 4 if spectral else 8
    g = W.SceneGen(5, 0, res)
    d = g.desc.contents
    rng = np.random.default_rng(6)
    texs = (type(d.textures[0]) * d.n_textures)()
    keep = []
    for i in range(d.n_textures):
        rgb = np.ascontiguousarray(10 ** rng.uniform(-5, 0.5, (size[1], size[0], 3)), np.float32)
        if i >= 2:
            rgb.reshape(-1, 3)[::7] = [np.inf, np.nan, 1.0]
        keep.append(rgb)
        texs[i].width, texs[i].height = size
        texs[i].rgb = rgb.ctypes.data_as(type(texs[i].rgb))
    d2 = type(d).from_buffer_copy(d)
    d2.textures = C.cast(texs, type(d.textures))
    with W.Context(0) as c:
        if spectral:
            c.set_spectrum(W.SPECTRUM_SAMPLED64)
        c.upload(C.pointer(d2))
        c.build()
        c.render_setup(spp, seed=4)
        c.render()
        group = c.film(*res)
        c.render_setup(spp, seed=4)
        for p in range(spp):
            c.render_pass(p)
        single = c.film(*res)
        c.check_device_errors()
    for a, b in zip(group, single):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert np.isfinite(group[0]).any()
