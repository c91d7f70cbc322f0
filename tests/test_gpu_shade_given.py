"""Shading with a given shadow term (vt_shade_forward's d_vis_in) has a kernel of
its own: its images are the tracing kernel's for the traced term, and a mix of
the all-lit and the all-dark image for any other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(1, 1), (16, 16), (17, 33), (251, 130)])
def test_given_shadow_term(vt, ctx, W, H):
    d = vt.gen_desc((90, 70, 80), scale=0.5, seed=21, trees=15, caves=True)
    w = vt.World(ctx, (90, 70, 80))
    w.generate(d)
    rng = np.random.default_rng(W)
    n = W * H
    cam = vt.gen_camera(d, 1, W, H)
    hits, rgb, vis = ctx.alloc(n * 16), ctx.alloc(n * 12), ctx.alloc(n)
    vt.render(ctx, w, cam, vt.default_params(rays=vt.RAYS_PRIMARY, shade=vt.SHADE_NONE), hits)
    sh = vt.Shading(ctx, w, rng.uniform(0.1, 0.9, (256, 3)).astype(np.float32),
                    rng.uniform(0.5, 1.5, 90 * 70 * 80).astype(np.float32), (0.5, 0.7, 0.2))

    def image(term):
        vis.upload(term)
        sh.forward(cam, hits, rgb, vis_in=vis)
        ctx.sync()
        return rgb.download(np.full((n, 3), -1.0, np.float32))

    try:
        sh.forward(cam, hits, rgb, vis_out=vis)
        ctx.sync()
        traced = rgb.download(np.zeros((n, 3), np.float32))
        assert np.array_equal(image(vis.download(np.zeros(n, np.uint8))), traced)
        lit, dark = image(np.ones(n, np.uint8)), image(np.zeros(n, np.uint8))
        some = rng.choice(np.array([0, 1, 255], np.uint8), n)
        assert np.array_equal(image(some), np.where((some != 0)[:, None], lit, dark))
        if n > 1000:
            assert np.any(lit != dark) and np.any(traced != lit)
    finally:
        sh.close()
        w.close()
        for b in (hits, rgb, vis):
            b.free()
