"""Cells and columns that the device generator's 32-bit noise cannot decide, so
that its 64-bit fallback does, against the host generator byte for byte: cave
thresholds set to the noise of a solid cell (the nearest float and its
neighbours), base heights that put a column's terrain on a whole number; and
worlds near the largest side, where the 32-bit positions are least exact.

The margin inside which a cell is undecided is 16 units of 2^-24 in the two
octaves' sum (1.5 times the noise) and 4 of the threshold; a column's is
(8 + octaves) units times the amplitude and 4 of the terrain's value.  Both
choices land within half a unit of the float chosen: far inside."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent
SRC = HERE / "host" / "noise_host.cpp"
OUT = HERE / "host" / "_build" / "libnoise_host.so"
U = 2.0 ** -24


@pytest.fixture(scope="module")
def noise(vt):
    if not OUT.exists() or SRC.stat().st_mtime > OUT.stat().st_mtime:
        OUT.parent.mkdir(exist_ok=True)
        subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", str(SRC), "-o", str(OUT)],
                       check=True)
    lib = C.CDLL(str(OUT))
    lib.nh_cave.restype = lib.nh_terrain.restype = C.c_double
    lib.nh_height.restype = C.c_int
    return lib


def check(vt, w, d):
    want = vt.gen_world(d)
    w.generate(d)
    got = w.download_dense()
    assert np.array_equal(got, want), np.argwhere(got != want)[:5]
    return want


def around(x):
    f = np.float32(x)
    return [float(v) for v in (np.nextafter(f, np.float32(-np.inf)), f, np.nextafter(f, np.float32(np.inf)))]


def test_thresholds_at_the_noise_of_solid_cells(vt, ctx, noise):
    d = vt.gen_desc((40, 48, 37), scale=0.5, seed=5, caves=True)
    rng = np.random.default_rng(5)
    w = vt.World(ctx, (40, 48, 37))
    try:
        chosen = 0
        while chosen < 24:
            x, z = int(rng.integers(0, 40)), int(rng.integers(0, 37))
            h = noise.nh_height(C.byref(d), x, z)
            if h < 3:
                continue
            y = int(rng.integers(1, h))
            v = noise.nh_cave(C.byref(d), x, y, z)
            carved = set()
            for t in around(v):
                assert abs(1.5 * (v - t)) <= 16 * U + 4 * U * abs(1.5 * t)
                d.cave_threshold = t
                carved.add(bool(check(vt, w, d)[z, y, x] == 0))
            assert carved == {False, True}   # one float decides the cell
            chosen += 1
    finally:
        w.close()


def test_columns_on_whole_heights(vt, ctx, noise):
    d = vt.gen_desc((40, 48, 37), scale=0.5, seed=6, trees=4)
    rng = np.random.default_rng(6)
    w = vt.World(ctx, (40, 48, 37))
    try:
        for _ in range(24):
            x, z = int(rng.integers(0, 40)), int(rng.integers(0, 37))
            rise = float(np.float32(d.amplitude)) * noise.nh_terrain(C.byref(d), x, z)
            heights = set()
            for base in around(20.0 - rise):
                value = base + rise
                assert abs(value - 20.0) <= abs(d.amplitude) * (8 + d.octaves) * U + 4 * U * abs(value)
                d.base_height = base
                heights.add(noise.nh_height(C.byref(d), x, z))
                check(vt, w, d)
            assert heights == {19, 20}
    finally:
        w.close()


@pytest.mark.parametrize("dims,octaves,period,cave_period", [
    ((8190, 40, 33), 8, 900.0, 7.3), ((33, 40, 8191), 16, 70000.0, 3.7), ((4100, 40, 300), 4, 4.3, 5.9),
])
def test_long_worlds(vt, ctx, dims, octaves, period, cave_period):
    d = vt.gen_desc(dims, scale=0.4, seed=octaves, trees=300, caves=True)
    d.octaves, d.period, d.cave_period = octaves, period, cave_period
    w = vt.World(ctx, dims)
    try:
        assert len(np.unique(check(vt, w, d))) > 4
    finally:
        w.close()
