"""Cameras whose cell the frame kernel takes from the host (near, one cell
inside the grid) and those next to that rule's edges: on integer planes, at the
margin, just past it, in the grid's outermost cells and far outside, with sun
directions of every octant.  Records against the oracle's, batch included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (61, 45, 70)


@pytest.fixture(scope="module")
def scene(vt, ctx):
    d = vt.gen_desc(DIMS, scale=0.25, seed=91, trees=6, caves=True)
    mats = vt.gen_world(d)
    w = vt.World(ctx, DIMS)
    w.upload_dense(mats)
    yield mats, w
    w.close()


@pytest.mark.parametrize("pos", [(1.0, 40.0, 1.0), (60.0, 44.0, 69.0), (0.999, 40.5, 30.0), (60.001, 40.0, 35.5),
                                 (30.0, 40.0, 35.0), (0.0, 44.999, 70.0), (30.5, 20.5, 35.5), (-20.0, 60.0, 90.0),
                                 (30.0, 300000.0, 35.0)])
def test_camera_positions(vt, ctx, oracle, scene, pos):
    mats, w = scene
    yaw = float(np.arctan2(30 - pos[0], 35 - pos[2]))
    pitch = float(np.clip(np.arctan2(10 - pos[1], max(1.0, np.hypot(30 - pos[0], 35 - pos[2]))), -1.55, 1.55))
    fov = 1.1 if abs(pos[1]) < 1000 else 2e-4
    cam = vt.Camera(pos=pos, yaw=yaw, pitch=pitch, fov=fov, width=83, height=47).as_uniform_data()
    ow = oracle.OracleWorld(mats)
    for octant in range(8):
        sun = [(-1.0 if octant >> i & 1 else 1.0) * v for i, v in enumerate((0.5, 0.7, 0.3))]
        p = vt.default_params(rays=vt.RAYS_PRIMARY | vt.RAYS_SHADOW, sun_dir=sun, max_steps=400, shadow_max_steps=300)
        got = vt.render_host(ctx, w, cam, p)
        want, _ = oracle.render(ow, vt.default_palette(), cam, p, threads=4)
        for f in ("voxel", "face", "material", "flags"):
            assert np.array_equal(got[f], want[f]), (octant, f)
        assert np.array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32)), octant
        buf = ctx.alloc(83 * 47 * 16)
        batch = vt.Batch(ctx, [(w, cam, buf)], p)
        batch.launch()
        ctx.sync()
        assert np.array_equal(buf.download(np.zeros(83 * 47, vt.HIT_DTYPE)), got)
        batch.close()
        buf.free()
