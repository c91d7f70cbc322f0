"""Step limits around kChunkSteps (1024): above it frames, batches, ray lists
and bounce rays run kernels with chunk jumps, at or below it kernels without.
Both must write the oracle's records."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sparse(vt, ctx):
    """1500 voxels long, nearly empty: rays of more than 1024 crossings."""
    rng = np.random.default_rng(41)
    mats = np.zeros((70, 40, 1500), np.uint8)
    mats[:, 0, ::3] = 2
    i = rng.integers(0, mats.size, 400)
    mats.reshape(-1)[i] = rng.integers(1, 255, 400)
    w = vt.World(ctx, (1500, 40, 70))
    w.upload_dense(mats)
    yield mats, w
    w.close()


@pytest.mark.parametrize("steps", [1023, 1024, 1025, 5000])
def test_rays_and_frames_at_the_limit(vt, ctx, oracle, sparse, steps):
    mats, w = sparse
    rng = np.random.default_rng(steps)
    o = np.stack([rng.choice([0.5, 1499.5], 4000), rng.uniform(1, 40, 4000), rng.uniform(0, 70, 4000)], 1)
    d = np.stack([np.where(o[:, 0] < 700, 1.0, -1.0), rng.normal(0, 0.01, 4000), rng.normal(0, 0.02, 4000)], 1)
    o, d = np.ascontiguousarray(o, np.float32), np.ascontiguousarray(d, np.float32)
    ow = oracle.OracleWorld(mats)
    got, ref = vt.trace_rays(ctx, w, o, d, steps), oracle.trace_rays(ow, o, d, steps)
    for f in ("voxel", "face", "material", "flags"):
        assert np.array_equal(got[f], ref[f]), f
    assert np.array_equal(got["t"].view(np.uint32), ref["t"].view(np.uint32))
    cam = vt.Camera(pos=(2.5, 30.2, 35.1), yaw=np.pi / 2, pitch=-0.02, fov=0.3, width=97, height=61).as_uniform_data()
    for rays in (vt.RAYS_SHADOW, vt.RAYS_SHADOW | vt.RAYS_BOUNCE):
        p = vt.default_params(rays=vt.RAYS_PRIMARY | rays, max_steps=steps, shadow_max_steps=steps,
                              bounce_max_steps=steps, seed=5, sun_dir=(0.9, 0.01, 0.05))
        frame = vt.render_host(ctx, w, cam, p)
        want, _ = oracle.render(ow, vt.default_palette(), cam, p, threads=4)
        for f in ("voxel", "face", "material", "flags"):
            assert np.array_equal(frame[f], want[f]), (rays, f)
        assert np.array_equal(frame["t"].view(np.uint32), want["t"].view(np.uint32))
        buf = ctx.alloc(cam.width * cam.height * 16)
        batch = vt.Batch(ctx, [(w, cam, buf)], p)
        batch.launch()
        ctx.sync()
        assert np.array_equal(buf.download(np.zeros(cam.width * cam.height, vt.HIT_DTYPE)), frame)
        batch.close()
        buf.free()
