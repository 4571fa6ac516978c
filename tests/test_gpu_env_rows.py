"""The environment map's sampling distribution against the oracle at the sizes
where its chunked row sums can go wrong: rows and columns shorter than a
block, of one chunk, of one value more and of several chunks; black maps and
maps with a black row; both index rules."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(2, 2), (3, 5), (130, 7), (2048, 2), (2049, 3), (4100, 2), (5, 2500)])
@pytest.mark.parametrize("fill", ["random", "black_row", "black"])
@pytest.mark.parametrize("quirk", [False, True])
def test_distribution(W, O, ctx, size, fill, quirk):
    w, h = size
    if quirk and h > w:
        pytest.skip("the reference's index rule writes past its array on maps higher than wide")
    rng = np.random.default_rng(w * 7 + h)
    rgb = np.exp(rng.normal(0, 2, (h, w, 3))).astype(np.float32)
    if fill == "black_row":
        rgb[: max(1, h // 2)] = 0.0
    elif fill == "black":
        rgb[:] = 0.0
    g = W.SceneGen(4, 0, (8, 8), level=1)
    e = g.desc.contents.envmap.contents
    keep = (e.width, e.height, e.rgb)
    flags = W.Q_ENV_DISTRIB_INDEX_BUG if quirk else 0
    e.width, e.height, e.rgb = w, h, rgb.ctypes.data_as(C.POINTER(C.c_float))
    try:
        ctx.set_quirks(flags)
        ctx.upload(g.desc)
        got = ctx.env_distribution(w, h)
        ref = O.OracleScene(g.desc, flags).env_distribution(w, h)
        for a, b in zip(got, ref):
            assert np.array_equal(np.asarray(a).view(np.uint32), np.asarray(b, np.float32).view(np.uint32))
    finally:
        e.width, e.height, e.rgb = keep
        ctx.set_quirks(0)
