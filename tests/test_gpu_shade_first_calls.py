"""A context's first backward calls, from its creation on and past its eight
accumulator regions, in device memory that held other values: every call's sums
are the same.  A context makes four allocations (status word, counters with the
regions, queue counters, pinned status word)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_first_backward_calls_of_a_context(vt, ctx):
    d = vt.gen_desc((64, 64, 64), scale=0.5, seed=31)
    rng = np.random.default_rng(31)
    pal = rng.uniform(0.1, 0.9, (256, 3)).astype(np.float32)
    tgt = rng.uniform(0, 1, 64 * 48 * 3).astype(np.float32)
    dirty = [ctx.alloc(size) for size in (4096, 51200, 65536, 1 << 21) for _ in range(8)]
    for b in dirty:
        b.upload(np.full(b.nbytes, 0x5A, np.uint8))
    for b in dirty:
        b.free()
    made = vt.alloc_counts()[0]
    with vt.Context(0) as c:
        assert vt.alloc_counts()[0] - made == 4
        w = vt.World(c, (64, 64, 64))
        w.generate(d)
        cam = vt.gen_camera(d, 0, 64, 48)
        hits, target, stream = c.alloc(64 * 48 * 16), c.alloc(64 * 48 * 12), c.stream()
        target.upload(tgt)
        vt.render(c, w, cam, vt.default_params(rays=vt.RAYS_PRIMARY, shade=vt.SHADE_NONE), hits, stream)
        c.sync(stream)
        sh = vt.Shading(c, w, pal, None, (0.5, 0.7, 0.2))
        try:
            got = []
            for _ in range(19):
                sh.zero_grad()
                sh.backward(cam, hits, target, stream=stream)
                c.sync(stream)
                got.append(sh.grads())
            assert got[0]["loss"] > 0 and np.any(got[0]["palette"])
            for g in got[1:]:
                for k in ("loss", "palette", "sun"):
                    a, b = np.asarray(g[k], np.float64), np.asarray(got[0][k], np.float64)
                    assert np.abs(a - b).max() <= 2.0 ** -20 * np.abs(b).max(), k
        finally:
            sh.close()
            w.close()
            c.lib.vt_stream_destroy(c.handle, stream)
            hits.free()
            target.free()
