"""vt_render_host with bounce rays into pinned memory: the frame is rendered in
device memory and copied; where that memory cannot be had, the kernels write
into the host's.  Both equal vt_render's records."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(17, 5), (333, 211), (1283, 721)])
def test_pinned_bounce_frames_equal_device_frames(vt, W, H):
    d = vt.gen_desc((128, 96, 128), seed=11, trees=10, caves=True)
    p = vt.default_params(rays=vt.RAYS_PRIMARY | vt.RAYS_SHADOW | vt.RAYS_BOUNCE, seed=4, sun_dir=vt.gen_sun(11))
    with vt.Context(0) as ctx:
        w = vt.World(ctx, (128, 96, 128))
        w.generate(d)
        cam = vt.gen_camera(d, 2, W, H)
        buf = ctx.alloc(W * H * 16)
        pin = vt.PinnedBuffer(ctx, W * H, vt.HIT_DTYPE)
        try:
            vt.render(ctx, w, cam, p, buf)      # (also makes the screen table and the bounce queue)
            want = buf.download(np.zeros(W * H, vt.HIT_DTYPE))
            assert np.any(want["flags"] & vt.HIT_BOUNCE)
            for fails in (True, False):
                made = vt.alloc_counts()[0]
                pin.array[:] = np.zeros(1, vt.HIT_DTYPE)
                vt.fail_alloc(1 if fails else 0)
                try:
                    vt.render_host(ctx, w, cam, p, pin.array)
                finally:
                    vt.fail_alloc(0)
                assert np.array_equal(pin.array, want), fails
                assert vt.alloc_counts()[0] == made + (0 if fails else 1)
        finally:
            pin.free()
            buf.free()
            w.close()
