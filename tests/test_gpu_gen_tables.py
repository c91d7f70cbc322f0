"""Scene generation on the device at the edges of its two kernels' ranges
(noise just coarse enough for the lattice tables, and finer: the cell-by-cell
kernel) and where the 32-bit noise often cannot decide (thresholds and
terrain levels on values the noise takes exactly), against the host generator
byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(vt, ctx, d):
    want = vt.gen_world(d)
    w = vt.World(ctx, tuple(d.dims))
    try:
        w.generate(d)
        got = w.download_dense()
        assert np.array_equal(got, want), np.argwhere(got != want)[:5]
    finally:
        w.close()
    return want


@pytest.mark.parametrize("period,octaves,cave_period", [
    (64.0, 4, 24.0), (16.0, 1, 6.0), (4.1, 4, 3.3), (4.0, 4, 24.0),    # tables up to their largest sides
    (3.9, 4, 24.0), (64.0, 8, 24.0), (64.0, 16, 24.0),                 # heights too fine for tables
    (64.0, 4, 1.1), (64.0, 4, 1.0), (64.0, 4, 0.37), (300.0, 2, 5.0),  # caves too fine; very coarse heights
])
def test_noise_scales(vt, ctx, period, octaves, cave_period):
    d = vt.gen_desc((70, 66, 97), scale=0.5, seed=int(period * 10) + octaves, trees=30, caves=True)
    d.period, d.octaves, d.cave_period = period, octaves, cave_period
    assert len(np.unique(check(vt, ctx, d))) > 3


@pytest.mark.parametrize("base,amplitude,threshold", [
    (30.0, 0.0, 0.6), (30.0, 1e-6, 0.0), (30.0, 24.0, -2.0), (30.0, 24.0, 2.0), (-5.0, 3.0, 0.1),
    (1e7, 24.0, 0.3), (30.0, 1e9, 0.3), (30.0, -20.0, float("nan")),
])
def test_levels_the_short_noise_cannot_decide(vt, ctx, base, amplitude, threshold):
    d = vt.gen_desc((40, 60, 33), scale=0.5, seed=77, trees=12, caves=True)
    d.base_height, d.amplitude, d.cave_threshold = base, amplitude, threshold
    check(vt, ctx, d)


def test_cells_next_to_the_cave_threshold(vt, ctx):
    """The threshold set to the noise of a cell (to the last bit, and one float
    up and down): the cells around it are within the 32-bit error."""
    d = vt.gen_desc((64, 64, 64), scale=0.5, seed=5, caves=True)
    for t in (0.05, 0.1, 0.15):
        for step in (-np.inf, None, np.inf):
            d.cave_threshold = t if step is None else float(np.nextafter(np.float32(t), np.float32(step)))
            check(vt, ctx, d)
