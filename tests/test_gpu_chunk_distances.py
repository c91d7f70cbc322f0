"""Chunk distances against three one-sided numpy passes, on both sides of the
grid size (4096 chunks) up to which one launch computes them, after an upload
and after device-side edits that set and clear a coarse bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CAP = 15


def chunk_distances(occ):
    """occ: bool [CZ, CY, CX] -> uint8 [8, chunks]."""
    out = []
    for octant in range(8):
        f = np.where(occ, 0, CAP + 1)
        for axis in range(3):                # x, y, z
            ax, fwd = 2 - axis, (octant >> axis) & 1
            g = f if fwd else np.flip(f, ax)
            best = g.copy()
            for d in range(1, min(CAP, g.shape[ax] - 1) + 1):
                ahead = np.full_like(g, CAP + 1)
                dst, src = [slice(None)] * 3, [slice(None)] * 3
                dst[ax], src[ax] = slice(0, -d), slice(d, None)
                ahead[tuple(dst)] = g[tuple(src)]
                best = np.minimum(best, np.maximum(d, ahead))
            f = best if fwd else np.flip(best, ax)
        out.append(f.reshape(-1))
    return np.array(out, np.uint8)


@pytest.mark.parametrize("chunks", [(1, 1, 1), (2, 7, 3), (20, 3, 17), (16, 1, 256), (16, 16, 16), (17, 1, 241)])
def test_chunk_distances(vt, ctx, chunks):
    CX, CY, CZ = chunks
    rng = np.random.default_rng(CX * CY * CZ)
    occ = np.zeros((CZ, CY, CX), bool)
    for _ in range(3):
        occ[rng.integers(CZ), rng.integers(CY), rng.integers(CX)] = True
    mats = np.zeros((32 * CZ, 32 * CY, 32 * CX), np.uint8)
    for z, y, x in np.argwhere(occ):
        mats[32 * z + 7, 32 * y + 30, 32 * x + 21] = 3
    w = vt.World(ctx, (32 * CX, 32 * CY, 32 * CZ))
    try:
        w.upload_dense(mats)
        assert np.array_equal(w.distances()[1], chunk_distances(occ))
        z, y, x = np.argwhere(occ)[0]
        top = y + np.flatnonzero(occ[z, y:, x])[-1]
        down = vt.Camera(pos=(32 * x + 21.5, 32 * CY - 0.25, 32 * z + 7.5), yaw=0.0, pitch=-np.pi / 2, fov=1.0,
                         width=16, height=16).as_uniform_data()
        if top + 1 == CY:                    # the chunk's lone voxel away
            w.edit(down, 1000, 0)
            occ[z, top, x] = False
        else:                                # one voxel on it in its chunk, the next in the chunk above
            w.edit(down, 1000, 9)
            w.edit(down, 1000, 9)
            occ[z, top + 1, x] = True
        assert np.array_equal(w.distances()[1], chunk_distances(occ))
    finally:
        w.close()
