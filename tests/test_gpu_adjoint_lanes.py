"""The differentiable estimator with several passes in flight: the image of the
fused render at equal parameters (bit-identical films), gradients that do not
depend on how many passes run side by side, over pass counts around the number
in flight, without memory for more than one, and on the legacy stream."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grads(W, ctx, res, spp, target):
    nm, ne = ctx.adjoint_setup(spp, seed=2)
    img, loss = ctx.adjoint_forward(*res, target)
    gm, ge = ctx.adjoint_backward()
    ctx.check_device_errors()
    return img, loss, gm, ge


@pytest.mark.parametrize("res,spp", [((24, 17), 1), ((24, 17), 9), ((40, 33), 16), ((300, 280), 5), ((760, 700), 2)])
def test_passes_in_flight(W, res, spp):
    g = W.SceneGen(4, 0, res, level=1)
    rng = np.random.default_rng(spp)
    target = rng.uniform(0, 2, (res[1], res[0], 3)).astype(np.float32)
    with W.Context(0) as ctx:
        ctx.upload(g.desc)
        ctx.build()
        img, loss, gm, ge = grads(W, ctx, res, spp, target)
        W.debug_fail_allocations(0)  # no room for more than one pass
        try:
            one = grads(W, ctx, res, spp, target)
        finally:
            W.debug_fail_allocations(-1)
        ctx.set_stream(None)
        legacy = grads(W, ctx, res, spp, target)
    with W.Context(0) as ctx:  # from the start without room
        ctx.upload(g.desc)
        ctx.build()
        ctx.adjoint_setup(spp, seed=2)
        W.debug_fail_allocations(0)
        try:
            alone = grads(W, ctx, res, spp, target)
        finally:
            W.debug_fail_allocations(-1)
    for other in (one, legacy, alone):
        # the image is summed in pass order: equal bits; the gradients are
        # float sums in any order over n samples: 2 sqrt(n) 2^-24 of their norm
        assert np.array_equal(other[0].view(np.uint32), img.view(np.uint32))
        tol = 2 * np.sqrt(res[0] * res[1] * spp) * 2.0 ** -24
        for a, b in ((other[2], gm), (other[3], ge)):
            assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b) + 1e-30
        assert abs(other[1] - loss) <= 1e-12 * abs(loss)
