"""The order in which backward_views adds to one voxel's albedo gradient.

Float atomics round, so a voxel that fills much of several views gets a sum
that depends on their order; it has to be about the order of one call per view
(the views' order).  Here one voxel fills every view and all its terms in a view
are equal, so that the order inside a view changes nothing: 720 x 720 terms of
1.3 from the first view, then terms of 0.004 from the 15 others, which
leave the sum as it is from 2^17 on (half a unit in the last place is 2^-7
there), a fifth of the first view's sum.  A view has 2025 tiles, more than twice
the blocks a GPU of 152 SMs holds, so the second view's terms come when more
than half of the first's are in: the result equals one call per view exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDE, VIEWS = 720, 16


def test_albedo_of_a_voxel_that_fills_every_view(vt, ctx):
    mats = np.zeros((40, 40, 40), np.uint8)
    mats[20, 20, 20] = 7
    w = vt.World(ctx, (40, 40, 40))
    w.upload_dense(mats)
    cam = vt.Camera(pos=(20.5, 20.5, 19.7), fov=0.9, width=SIDE, height=SIDE).as_uniform_data()
    n = SIDE * SIDE
    hits, image, first, rest = ctx.alloc(n * 16), ctx.alloc(n * 12), ctx.alloc(n * 12), ctx.alloc(n * 12)
    vt.render(ctx, w, cam, vt.default_params(rays=vt.RAYS_PRIMARY, shade=vt.SHADE_NONE), hits)
    ctx.sync()
    cell = 20 + 40 * (20 + 40 * 20)
    assert np.all(hits.download(np.zeros(n, vt.HIT_DTYPE))["voxel"] == cell)
    sh = vt.Shading(ctx, w, np.full((256, 3), 0.5, np.float32), np.ones(40 ** 3, np.float32), (0.2, 0.3, -0.9))
    try:
        sh.forward(cam, hits, image)
        ctx.sync()
        c = image.download(np.zeros((n, 3), np.float32))
        assert np.all(c == c[0])
        shade = float(c[0, 0]) / 0.5
        first.upload(np.zeros((n, 3), np.float32))
        rest.upload(c - np.float32(0.004 / (6 * 0.5 * shade)))   # a term is 6 * 0.5 * shade * (image - target)
        targets = [first] + [rest] * (VIEWS - 1)
        sh.zero_grad()
        for t in targets:
            sh.backward(cam, hits, t)
        want = sh.grads()["albedo"]
        assert want[cell] > 2.0 ** 18 and np.count_nonzero(want) == 1
        sh.zero_grad()
        sh.backward_views([cam] * VIEWS, [hits] * VIEWS, targets)
        got = sh.grads()["albedo"]
        assert np.array_equal(got, want), (got[cell], want[cell])
    finally:
        sh.close()
        w.close()
        for b in (hits, image, first, rest):
            b.free()
