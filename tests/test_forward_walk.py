"""The forward walk (trace_p.cuh, FwdWalk: the production traversal of ordinary
rays) compiled as host C++ against the unit-step oracle, bit for bit: worlds of
every padding, step limits around the crossing counts, origins on planes,
outside and far from the grid, exact diagonal ties, and rays it hands to the
general walk."""
import ctypes as C

import numpy as np
import pytest

from test_host_trace import ht, random_rays  # noqa: F401


def trace(ht, mats, o, d, steps):
    ht.ht_world_new.restype = C.c_void_p
    ht.ht_world_new.argtypes = [C.POINTER(C.c_int32), C.c_void_p]
    ht.ht_world_free.argtypes = [C.c_void_p]
    ht.ht_trace_mt.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int64, C.c_int32, C.c_void_p, C.c_int32]
    Z, Y, X = mats.shape
    hw = ht.ht_world_new((C.c_int32 * 3)(X, Y, Z), mats.ctypes.data)
    try:
        out = []
        for s in steps:
            r = np.zeros((o.shape[0], 4), np.uint32)
            ht.ht_trace_mt(hw, o.ctypes.data, d.ctypes.data, o.shape[0], s, r.ctypes.data, 4)
            out.append(r)
        return out
    finally:
        ht.ht_world_free(hw)


def check(ht, oracle, mats, o, d, steps):
    w = oracle.OracleWorld(mats)
    hits = 0
    for s, got in zip(steps, trace(ht, mats, o, d, steps)):
        ref = oracle.trace_rays(w, o, d, s)
        hit = ref["face"] != 0xFF
        bad = np.flatnonzero((got[:, 0] != ref["voxel"]) | (got[:, 1] != ref["t"].view(np.uint32)) |
                             (got[:, 2] != ref["material"]) | ((got[:, 3] & 0xFF) != ref["face"]))
        assert bad.size == 0, (s, bad[:5], o[bad[:3]], d[bad[:3]], got[bad[:3]], ref[bad[:3]])
        hits += int(hit.sum())
    return hits


@pytest.mark.parametrize("dims,seed", [((64, 64, 64), 1), ((90, 70, 101), 2), ((33, 7, 1), 3), ((5, 130, 66), 4)])
def test_random_rays_and_step_limits(ht, oracle, vtlib, dims, seed):
    mats = vtlib.gen_world(vtlib.gen_desc(dims, scale=min(1.0, dims[1] / 128), seed=seed, trees=10, caves=True))
    rng = np.random.default_rng(seed)
    mats[rng.random(mats.shape) < 0.002] = 9
    o, d = random_rays(rng, dims, 20000)
    assert check(ht, oracle, mats, o, d, (-1, 0, 1, 2, 3, 7, 40, 150, 1 << 20, 2 ** 31 - 1)) > 500


def test_long_empty_boxes_and_chunk_jumps(ht, oracle):
    """A nearly empty world longer than the brick distances' cap: chunk jumps
    and capped brick jumps, and the empty padding past every side."""
    rng = np.random.default_rng(5)
    mats = np.zeros((129, 33, 601), np.uint8)
    i = rng.integers(0, mats.size, 60)
    mats.reshape(-1)[i] = rng.integers(1, 255, 60)
    o, d = random_rays(rng, (601, 33, 129), 30000)
    d[::3, 1] *= 0.02
    aim = np.stack(np.unravel_index(rng.choice(i, 10000), mats.shape)[::-1], 1) + rng.uniform(0, 1, (10000, 3))
    d[1::3] = (aim - o[1::3]).astype(np.float32)
    assert check(ht, oracle, mats, o, np.ascontiguousarray(d), (3, 90, 100000)) > 5000


def test_ties_on_planes_and_diagonals(ht, oracle):
    """Integer and half-integer origins with directions of equal components:
    plane times tie on two and three axes at once."""
    rng = np.random.default_rng(6)
    mats = (rng.random((40, 44, 37)) < 0.03).astype(np.uint8) * 3
    n = 20000
    o = rng.integers(0, 80, (n, 3)) / 2.0
    d = rng.choice([-1.0, -0.5, 0.0, 0.5, 1.0, 2.0], (n, 3))
    d[np.all(d == 0, axis=1)] = 1.0
    o, d = np.ascontiguousarray(o, np.float32), np.ascontiguousarray(d, np.float32)
    assert check(ht, oracle, mats, o, d, (1, 6, 5000)) > 5000


def test_far_origins_and_extreme_directions(ht, oracle, vtlib):
    """Origins to 2^22 away, on both sides of the 2^20 bound, and direction
    components whose reciprocals leave the ordinary range."""
    dims = (96, 64, 80)
    mats = vtlib.gen_world(vtlib.gen_desc(dims, scale=0.5, seed=9, trees=15, caves=True))
    rng = np.random.default_rng(8)
    n = 12000
    target = rng.uniform([0, 0, 0], dims, (n, 3))
    away = rng.normal(size=(n, 3))
    away /= np.linalg.norm(away, axis=1, keepdims=True)
    far = 2.0 ** rng.uniform(0, 22, n)
    o = target + away * far[:, None]
    d = -away * (10.0 ** rng.uniform(-3, 3, n))[:, None]
    wild = rng.random((n, 3)) < 0.05
    d = np.where(wild, np.sign(d) * rng.choice([0.0, 1e-38, 1e-31, 1e-29, 1e29, 1e31, 1e38], (n, 3)), d)
    o, d = np.ascontiguousarray(o, np.float32), np.ascontiguousarray(d, np.float32)
    assert check(ht, oracle, mats, o, d, (30, 1 << 20)) > 5000
