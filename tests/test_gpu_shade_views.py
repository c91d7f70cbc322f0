"""The shading kernels' launch shapes: several tiles per backward block (ragged
right edges, more views than one launch holds) against single views, and the
general kernels (long step limits, sun directions with a reciprocal out of the
forward walk's range) against the frame kernel's shadow flags.

Gradients are float sums in another order.  A sum of n terms taken in any
order is within (n - 1) 2^-24 of the sum of their magnitudes; the atomics of
these frames add at most 2^13 partial sums of 2^8 terms, so two orders agree
within 2^14 * 2^-24 = 2^-10 of the magnitudes in the worst case and near its
square root in practice: 2^-17 of the magnitudes is the bar, the magnitudes
bounded below by the largest element of the group."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(vt, ctx):
    d = vt.gen_desc((150, 90, 130), scale=0.6, seed=51, trees=40, caves=True)
    w = vt.World(ctx, (150, 90, 130))
    w.generate(d)
    rng = np.random.default_rng(51)
    pal = rng.uniform(0.1, 0.9, (256, 3)).astype(np.float32)
    alb = rng.uniform(0.5, 1.5, 150 * 90 * 130).astype(np.float32)
    yield d, w, pal, alb
    w.close()


def hits_of(vt, ctx, w, cams):
    p = vt.default_params(rays=vt.RAYS_PRIMARY, shade=vt.SHADE_NONE)
    out = []
    for cam in cams:
        out.append(ctx.alloc(cam.width * cam.height * 16))
        vt.render(ctx, w, cam, p, out[-1])
    ctx.sync()
    return out


@pytest.mark.parametrize("views,size", [(17, (361, 339)), (3, (1040, 700)), (2, (16, 16)), (5, (65, 3))])
def test_views_equal_single_views(vt, ctx, scene, views, size):
    d, w, pal, alb = scene
    cams = [vt.gen_camera(d, v, size[0] - (v % 2), size[1]) for v in range(views)]
    hits = hits_of(vt, ctx, w, cams)
    sh = vt.Shading(ctx, w, pal, alb, vt.gen_sun(3))
    rng = np.random.default_rng(views)
    tgts = [ctx.alloc(c.width * c.height * 12) for c in cams]
    for t, c in zip(tgts, cams):
        t.upload(rng.uniform(0, 1, c.width * c.height * 3).astype(np.float32))
    many, one = ([ctx.alloc(c.width * c.height * 12) for c in cams] for _ in range(2))
    try:
        sh.forward_views(cams, hits, many)
        for c, h, o in zip(cams, hits, one):
            sh.forward(c, h, o)
        for c, a, b in zip(cams, many, one):
            n = c.width * c.height * 3
            assert np.array_equal(a.download(np.zeros(n, np.float32)), b.download(np.ones(n, np.float32)))
        sh.zero_grad()
        sh.backward_views(cams, hits, tgts)
        got = sh.grads()
        sh.zero_grad()
        for c, h, t in zip(cams, hits, tgts):
            sh.backward(c, h, t)
        want = sh.grads()
        for k in ("loss", "palette", "sun", "albedo"):
            a, b = np.atleast_1d(np.asarray(got[k], np.float64)), np.atleast_1d(np.asarray(want[k], np.float64))
            assert np.abs(a - b).max() <= 2.0 ** -17 * max(np.abs(b).max(), 1e-30), k
            assert np.array_equal(a == 0, b == 0), k
    finally:
        sh.close()
        for b in hits + tgts + many + one:
            b.free()


@pytest.mark.parametrize("sun,steps", [((0.6, 0.5, 0.3), 512), ((0.6, 0.5, 0.3), 1025), ((0.6, 0.5, 1e-33), 512),
                                       ((0.6, 0.5, 0.0), 512), ((1e18, 8e17, -2e17), 512), ((0.3, 0.9, 1e-20), 2000)])
def test_shadow_term_equals_the_frame_kernels(vt, ctx, scene, sun, steps):
    d, w, pal, alb = scene
    cam = vt.gen_camera(d, 4, 211, 97)
    hits = ctx.alloc(211 * 97 * 16)
    vt.render(ctx, w, cam, vt.default_params(rays=vt.RAYS_PRIMARY | vt.RAYS_SHADOW, sun_dir=sun,
                                             shadow_max_steps=steps), hits)
    rec = hits.download(np.zeros(211 * 97, vt.HIT_DTYPE))
    sh = vt.Shading(ctx, w, pal, alb, sun, shadow_max_steps=steps)
    rgb, vis = ctx.alloc(211 * 97 * 12), ctx.alloc(211 * 97)
    try:
        sh.forward(cam, hits, rgb, vis_out=vis)
        ctx.sync()
        lit = vis.download(np.zeros(211 * 97, np.uint8))
        hit = (rec["flags"] & vt.HIT_PRIMARY) != 0
        assert np.array_equal(lit != 0, hit & ((rec["flags"] & vt.HIT_SHADOWED) == 0))
        assert hit.sum() > 5000
    finally:
        sh.close()
        for b in (hits, rgb, vis):
            b.free()


def test_backward_on_concurrent_streams(vt, ctx, scene):
    """Twenty backward calls over four streams, more than the context's
    accumulator regions, into accumulators of their own: each equals the first
    (sums in 64 bits: only the float atomics of the albedo vary)."""
    d, w, pal, alb = scene
    cam = vt.gen_camera(d, 2, 333, 211)
    (hits,) = hits_of(vt, ctx, w, [cam])
    tgt = ctx.alloc(333 * 211 * 12)
    tgt.upload(np.random.default_rng(1).uniform(0, 1, 333 * 211 * 3).astype(np.float32))
    streams = [ctx.stream() for _ in range(4)]
    all_sh = [vt.Shading(ctx, w, pal, alb, vt.gen_sun(3)) for _ in range(20)]
    try:
        for i, sh in enumerate(all_sh):
            sh.backward(cam, hits, tgt, stream=streams[i % 4])
        for s in streams:
            ctx.sync(s)
        want = all_sh[0].grads()
        assert want["loss"] > 0
        for sh in all_sh[1:]:
            got = sh.grads()
            for k in ("loss", "palette", "sun"):
                a, b = np.asarray(got[k], np.float64), np.asarray(want[k], np.float64)
                assert np.abs(a - b).max() <= 2.0 ** -20 * np.abs(b).max(), k
    finally:
        for sh in all_sh:
            sh.close()
        hits.free()
        tgt.free()
        for s in streams:
            ctx.lib.vt_stream_destroy(ctx.handle, s)
