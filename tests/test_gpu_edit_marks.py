"""Device-side edits whose distance updates are cut down (x pass in the edit's
block, z pass only over column groups the y pass changed, chunk passes only
when a coarse bit changed, one or three launches by grid size): after
every edit the distances equal a fresh upload's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same_as_fresh(vt, ctx, w, dims):
    mats = w.download_dense()
    f = vt.World(ctx, dims)
    try:
        f.upload_dense(mats)
        for a, b in zip(w.distances(), f.distances()):
            assert np.array_equal(a, b), np.flatnonzero(a != b)[:5]
    finally:
        f.close()


# the last has more chunks than the one-launch chunk passes take
@pytest.mark.parametrize("dims", [(150, 70, 140), (33, 200, 35), (700, 64, 3072)])
def test_edits_against_fresh_uploads(vt, ctx, dims):
    X, Y, Z = dims
    rng = np.random.default_rng(X)
    mats = np.zeros((Z, Y, X), np.uint8)
    mats[:, :3, :] = 1
    i = rng.integers(0, mats.size, 40)
    mats.reshape(-1)[i] = 2
    w = vt.World(ctx, dims)
    try:
        w.upload_dense(mats)
        assert w.info().chunks[0] * w.info().chunks[1] * w.info().chunks[2] > (4096 if X == 700 else 0)
        spots = [(X / 2, Z / 2), (0.6, 0.6), (X - 0.6, Z - 0.7), (X / 3, Z - 1.3)]
        for k, (x, z) in enumerate(spots if X < 700 else spots[:2]):
            down = vt.Camera(pos=(x, Y - 0.5, z), yaw=0.0, pitch=-np.pi / 2, fov=1.0, width=16, height=16).as_uniform_data()
            for mode in (7, 7, 0, 9, 0, 0):      # towers, and holes to the bottom layer
                w.edit(down, 1000, mode)
            same_as_fresh(vt, ctx, w, dims)
        # a voxel alone high in an empty chunk: its coarse bit rises and falls
        lift = next(c for c in range(Y - 1, 3, -1) if c % 32 > 4)
        w.set(X // 2, lift, Z // 2, 5)
        same_as_fresh(vt, ctx, w, dims)
        side = vt.Camera(pos=(X / 2 - 10.2, lift + 0.5, Z // 2 + 0.5), yaw=np.pi / 2, pitch=0.0, fov=1.0, width=16,
                         height=16).as_uniform_data()
        for mode in (6, 0, 0):
            w.edit(side, 1000, mode)
            same_as_fresh(vt, ctx, w, dims)
    finally:
        w.close()
