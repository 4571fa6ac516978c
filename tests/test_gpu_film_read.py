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


def test_reads_leave_a_running_frame_alone(W):
    # reads on a second stream while a frame still renders on the first give
    # whatever has arrived, and the frame ends as it would have alone
    torch = pytest.importorskip("torch")
    res, spp = (1001, 563), 64
    g = W.SceneGen(2, 3, res, level=5)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with W.Context(0) as c:
        c.upload(g.desc)
        c.build()
        c.render_setup(spp, seed=5)
        c.render()
        want = [x.view(np.uint32) for x in c.film(*res)]
        c.set_stream(a.cuda_stream)
        c.render_setup(spp, seed=5)
        c.render()
        c.set_stream(b.cuda_stream)
        for _ in range(3):
            c.film(*res)
            c.tonemap(*res)
        torch.cuda.synchronize()
        got = [x.view(np.uint32) for x in c.film(*res)]
        c.check_device_errors()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("spectral", [False, True])
def test_read_without_device_memory(W, spectral):
    res = (200, 150)
    g = W.SceneGen(0, 3, res)
    with W.Context(0) as c:
        if spectral:
            c.set_spectrum(W.SPECTRUM_SAMPLED64)
        c.upload(g.desc)
        c.build()
        c.render_setup(2, seed=5)
        c.render()
        W.debug_fail_allocations(0)
        try:
            got = c.film(*res)
        finally:
            W.debug_fail_allocations(-1)
        want = c.film(*res)
        assert np.array_equal(got[0].view(np.uint32), want[0].view(np.uint32)) and np.array_equal(got[1], want[1])
