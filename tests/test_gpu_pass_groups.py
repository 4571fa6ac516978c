"""wpbr_render in pass groups against the same passes rendered one at a time
(wpbr_render_pass): identical films, over whole and ragged groups, films below
and above the material-sorting size, RGB and Sampled64, on the legacy default
stream (which cannot be captured) and without memory for the group's state."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def frame(W, ctx, res, spp, one_by_one=False):
    ctx.render_setup(spp, seed=3, stream=1)
    if one_by_one:
        for p in range(spp):
            ctx.render_pass(p)
    else:
        ctx.render()
    L, w = ctx.film(*res)
    ctx.check_device_errors()
    return L.view(np.uint32), w.view(np.uint32)


def context(W, config, res, spectral):
    g = W.SceneGen(config, 2, res, level=3)
    ctx = W.Context(0)
    if spectral:
        ctx.set_spectrum(W.SPECTRUM_SAMPLED64)
    ctx.upload(g.desc)
    ctx.build()
    return ctx


@pytest.mark.parametrize("config,res,spp,spectral", [
    (0, (33, 17), 1, False), (0, (33, 17), 9, False), (2, (420, 333), 8, False), (5, (420, 333), 11, False),
    (2, (41, 27), 5, True), (2, (420, 333), 7, True)])
def test_groups_match_single_passes(W, config, res, spp, spectral):
    with context(W, config, res, spectral) as ctx:
        one = frame(W, ctx, res, spp, one_by_one=True)
        for again in range(2):  # the second frame reuses the graphs
            got = frame(W, ctx, res, spp)
            assert np.array_equal(got[0], one[0]) and np.array_equal(got[1], one[1]), again
        shorter = frame(W, ctx, res, max(1, spp - 1))
        assert np.array_equal(shorter[0], frame(W, ctx, res, max(1, spp - 1), one_by_one=True)[0])


@pytest.mark.parametrize("spectral", [False, True])
def test_groups_without_capture_or_memory(W, spectral):
    res, spp = (130, 70), 6
    with context(W, 2, res, spectral) as ctx:
        one = frame(W, ctx, res, spp, one_by_one=True)
        W.debug_fail_allocations(0)  # no room for the group: one pass at a time
        try:
            ctx.render_setup(spp, seed=3, stream=1)
            if not spectral:
                ctx.render()
        finally:
            W.debug_fail_allocations(-1)
        if not spectral:
            assert np.array_equal(ctx.film(*res)[0].view(np.uint32), one[0])
        ctx.set_stream(None)
        got = frame(W, ctx, res, spp)
        assert np.array_equal(got[0], one[0]) and np.array_equal(got[1], one[1])


@pytest.mark.parametrize("spectral", [False, True])
def test_each_group_allocation_may_fail(W, spectral):
    # whichever of the group's buffers cannot be had, the frame renders one
    # pass at a time in the buffers of render_setup, which stay usable
    res, spp = (70, 41), 5
    for budget in range(5):
        with context(W, 2, res, spectral) as ctx:
            ctx.render_setup(spp, seed=3, stream=1)
            W.debug_fail_allocations(budget)
            try:
                ctx.render()
            finally:
                W.debug_fail_allocations(-1)
            got = [a.view(np.uint32) for a in ctx.film(*res)]
            one = frame(W, ctx, res, spp, one_by_one=True)
            assert np.array_equal(got[0], one[0]) and np.array_equal(got[1], one[1]), budget
