"""Every walk ends and reads inside its world, whatever the camera or the hit
records hold: the frame's pixel compiled as host C++ (host/walk_ends.cpp) under
a limit of walk steps far above what any ray of these worlds takes, its world
reads checked.  What the records say is compared with the unit-step oracle."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from test_host_trace import HERE, cuda_include, ht  # noqa: F401

SRC = HERE / "host" / "walk_ends.cpp"
OUT = HERE / "host" / "_build" / "libwalk_ends.so"
DIMS = (64, 70, 61)
LIMIT = 100000


@pytest.fixture(scope="module")
def we(ht):  # noqa: F811
    deps = [SRC, HERE.parent / "include" / "vt.h"] + sorted((HERE.parent / "unnamed-voxel-tracer_gb300" / "csrc").glob("*.cuh")) + \
        sorted((HERE.parent / "unnamed-voxel-tracer_gb300" / "csrc").glob("*.h"))
    if not OUT.exists() or any(d.stat().st_mtime > OUT.stat().st_mtime for d in deps):
        OUT.parent.mkdir(exist_ok=True)
        subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I", cuda_include(),
                        str(SRC), "-o", str(OUT)], check=True)
    return C.CDLL(str(OUT))


def with_distances(ht, mats):  # noqa: F811
    """Dims, voxels and distance fields of a world."""
    dims = mats.shape[::-1]
    nch = int(np.prod([(d + 31) // 32 for d in dims]))
    brick, chunk = np.zeros(8 * nch * 512, np.uint8), np.zeros(8 * nch, np.uint8)
    dims = (C.c_int32 * 3)(*dims)
    ht.ht_distances.argtypes = [C.POINTER(C.c_int32), C.c_void_p, C.c_void_p, C.c_void_p]
    ht.ht_distances(dims, mats.ctypes.data, brick.ctypes.data, chunk.ctypes.data)
    return dims, mats, brick, chunk


@pytest.fixture(scope="module")
def world(ht, vtlib):  # noqa: F811
    """A small cave world."""
    return with_distances(ht, vtlib.gen_world(vtlib.gen_desc(DIMS, scale=0.5, seed=7, trees=12, caves=True)))


SUN = (0.4, 0.8, -0.3)


def trace_frame(we, world, pos, view, tan_half_fov, W, H, max_steps, limit):
    """Per pixel of a frame's primary and shadow rays {how the walks ended, the record's flags}."""
    out = np.zeros((H * W, 2), np.uint8)
    we.we_frame.argtypes = [C.POINTER(C.c_int32)] + [C.c_void_p] * 5 + [C.c_float] + [C.c_int32] * 2 + [C.c_void_p, C.c_int32, C.c_int64, C.c_void_p]
    p, sun = np.array(pos, np.float32), np.array(SUN, np.float32)
    dims, mats, brick, chunk = world
    we.we_frame(dims, mats.ctypes.data, brick.ctypes.data, chunk.ctypes.data, p.ctypes.data, view.ctypes.data,
                tan_half_fov, W, H, sun.ctypes.data, max_steps, limit, out.ctypes.data)
    return out


@pytest.mark.parametrize("pos", [(30.5, 55.5, 30.5), (-40.0, 60.0, -30.0), (3e5, 2e5, 4e5)])
@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e-19, 1e-22, 3e-23, 1e-23, 1e-25, 1e-30, 1e-38, 1e-44, 0.0, 1e15, 1e19,
                                   1e25, 1e38])
def test_frames_of_scaled_views(we, oracle, vtlib, world, pos, scale):
    """A view whose rows are so small (or large) that a direction's squared
    length leaves the float range: components of the normalised direction are
    infinite, NaN, or all zero (replaced by 0.001)."""
    W, H = 24, 17
    cam = vtlib.Camera(pos=pos, yaw=0.7, pitch=-0.5, fov=1.3, width=W, height=H).as_uniform_data()
    with np.errstate(over="ignore", under="ignore"):
        view = (np.array(list(cam.view), np.float32) * np.float32(scale)).astype(np.float32)
    cam.view = (C.c_float * 16)(*view)
    out = trace_frame(we, world, pos, view, cam.tan_half_fov, W, H, 512, LIMIT)
    assert np.all(out[:, 0] == 0), (np.bincount(out[:, 0]), "pixels that ended, did not end, read out of range")
    params = vtlib.default_params(rays=vtlib.RAYS_PRIMARY | vtlib.RAYS_SHADOW, shade=vtlib.SHADE_NONE, sun_dir=SUN)
    ref, _ = oracle.render(oracle.OracleWorld(world[1]), vtlib.default_palette(), cam, params, threads=4)
    assert np.array_equal(out[:, 1], ref["flags"])
    if scale == 1.0 and pos[0] == 30.5:
        assert np.count_nonzero(out[:, 1]) > 100 and np.any(out[:, 1] & vtlib.HIT_SHADOWED)


@pytest.mark.parametrize("exponent", [12, 19, 19.95, 20.1, 21, 24, 30, 36, 42, 46, 60])
def test_frames_of_far_cameras(we, oracle, vtlib, world, exponent):
    """Cameras at 2^exponent cells on a diagonal, looking at the world: on both
    sides of the bound of near origins, and where plane times run together."""
    W, H = 31, 29
    away = np.array([0.6, 0.62, 0.5])
    pos = np.float32(np.array(DIMS) / 2 + away / np.linalg.norm(away) * 2.0 ** exponent)
    f = (np.array(DIMS) / 2 - pos.astype(np.float64))
    f /= np.linalg.norm(f)
    r = np.cross([0.0, 1.0, 0.0], f)
    r /= np.linalg.norm(r)
    view = np.zeros((4, 4), np.float32)
    view[0, :3], view[1, :3], view[2, :3] = r, np.cross(f, r), f
    cam = vtlib.Camera(pos=pos, fov=1.0, width=W, height=H).as_uniform_data()
    cam.view = (C.c_float * 16)(*view.reshape(-1))
    cam.tan_half_fov = min(1.0, 60.0 * 2.0 ** -exponent)
    out = trace_frame(we, world, pos, view.reshape(-1), cam.tan_half_fov, W, H, 512, LIMIT)
    assert np.all(out[:, 0] == 0), np.bincount(out[:, 0])
    params = vtlib.default_params(rays=vtlib.RAYS_PRIMARY | vtlib.RAYS_SHADOW, shade=vtlib.SHADE_NONE, sun_dir=SUN)
    ref, _ = oracle.render(oracle.OracleWorld(world[1]), vtlib.default_palette(), cam, params, threads=4)
    assert np.array_equal(out[:, 1], ref["flags"])
    if exponent < 20:
        assert np.count_nonzero(out[:, 1]) > 100


@pytest.mark.parametrize("sun", [(0.6, 0.5, 0.3), (-0.6, -0.5, -0.3), (0.3, -0.9, 0.0), (-1e12, 2e12, 5e11)])
def test_shadow_rays_from_any_point(we, world, sun):
    """Points the shading kernels make from hit records that no frame of this
    world wrote (any t): far away on the line into the world, infinite, NaN."""
    dims, mats, brick, chunk = world
    rng = np.random.default_rng(3)
    n = 20000
    d = np.array(sun, np.float64)
    d[d == 0] = 0.001
    d /= np.linalg.norm(d)
    inside = rng.uniform([0, 0, 0], DIMS, (n, 3))
    back = np.where(rng.random(n) < 0.2, 0.0, 2.0 ** rng.uniform(-3, 40, n))
    o = (inside - d * back[:, None]).astype(np.float32)
    o[::50, 0] = np.inf
    o[1::50, 1] = -np.inf
    o[2::50] = np.nan
    o[3::50, 2] = np.float32(3e38)
    o[4::50] = np.sign(-d).astype(np.float32) * np.float32(1e30)
    s = np.array(sun, np.float32)
    out = np.zeros((n, 3, 2), np.uint8)
    we.we_shadow.argtypes = [C.POINTER(C.c_int32)] + [C.c_void_p] * 5 + [C.c_int64, C.c_int32, C.c_int64, C.c_void_p]
    we.we_shadow(dims, mats.ctypes.data, brick.ctypes.data, chunk.ctypes.data, s.ctypes.data, o.ctypes.data, n, 512,
                 LIMIT, out.ctypes.data)
    assert np.all(out[:, :, 0] == 0), [np.bincount(out[:, k, 0]) for k in range(3)]
    assert np.array_equal(out[:, 0, 1], out[:, 2, 1]) and np.array_equal(out[:, 1, 1], out[:, 2, 1])
    assert 1000 < np.count_nonzero(out[:, 2, 1]) < n - 1000


@pytest.mark.parametrize("max_steps", [620, 1024, 1025])
def test_open_space_takes_few_jumps(we, ht, vtlib, max_steps):  # noqa: F811
    """Rays through 594 empty cells of a grid of 2 x 2 x 19 chunks: two jumps out
    of boxes of empty chunks (nine of the brick distances' 66 cells), whatever
    the step limit."""
    open_world = with_distances(ht, np.zeros((600, 64, 64), np.uint8))
    pos = (32.5, 32.5, 5.5)
    cam = vtlib.Camera(pos=pos, fov=0.05, width=8, height=8).as_uniform_data()
    view = np.array(list(cam.view), np.float32)
    out = trace_frame(we, open_world, pos, view, cam.tan_half_fov, 8, 8, max_steps, 3)
    assert np.all(out == 0), np.bincount(out[:, 0])
