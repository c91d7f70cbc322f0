"""The entity boxes of the reference frame (map.glsl:172-201) where its shadow
rays meet or nearly meet them: flat ground under the five boxes, seen from
close, pixel for pixel against the CPU restatement."""
import numpy as np
import pytest

import refworld

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pos,yaw,pitch", [((253.5, 30.0, 250.0), 0.4, -1.2), ((240.0, 26.0, 244.0), 0.7, -0.35),
                                           ((262.0, 40.0, 266.0), 3.8, -0.8), ((250.5, 21.5, 258.5), 0.0, -1.5)])
def test_ground_under_the_boxes(vt, ctx, oracle, pos, yaw, pitch):
    mats = np.zeros((320, 64, 320), np.uint8)      # [z, y, x]
    mats[180:320, 12:20, 180:320] = 1
    rng = np.random.default_rng(7)
    chunks, data = refworld.build_map(mats, np.zeros(256, np.uint32))
    atlas = refworld.build_atlas(refworld.random_models(rng, 1, full=True))
    bm = vt.Brickmap(ctx)
    try:
        bm.upload(chunks, data)
        bm.set_atlas(atlas, 1)
        cam = vt.Camera(pos=pos, yaw=yaw, pitch=pitch, fov=1.2, width=120, height=90).as_uniform_data()
        got, want = bm.render(cam), oracle.render_reference(oracle.OracleRefWorld(chunks, data, atlas), cam)
        for f in ("normal", "illumination"):
            assert np.array_equal(got[f], want[f]), f
        assert np.array_equal(got["position"].view(np.uint32), want["position"].view(np.uint32))
        for f in ("albedo", "color"):
            g, w = (np.ascontiguousarray(r[f]).view(np.uint8).astype(int) for r in (got, want))
            assert np.abs(g - w).max() <= 1, f
        # flat ground shadows nothing: what is dark is dark by a box
        hit = got["position"][:, 0] >= 0
        dark = hit & (got["illumination"] >> 24 == 0)
        assert hit.sum() > 2000 and 10 < dark.sum() < hit.sum()
    finally:
        bm.close()
