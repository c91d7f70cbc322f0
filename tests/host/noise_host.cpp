// Test-only: the generator's 64-bit noise (gen_noise.cuh) at single points, from
// which the tests choose thresholds and levels that the device's 32-bit noise
// cannot decide.
#include <stdint.h>

#include "../../unnamed-voxel-tracer_gb300/csrc/gen_noise.cuh"

using namespace vt::gen;

extern "C" double nh_cave(const vt_gen_desc* d, int x, int y, int z) {
    return fbm3(stream_seed(d->seed, kCaves), (double)x, (double)y, (double)z, 1.0 / (double)d->cave_period);
}

extern "C" double nh_terrain(const vt_gen_desc* d, int x, int z) {
    return fbm2(stream_seed(d->seed, kTerrain), (double)x, (double)z, 1.0 / (double)d->period, d->octaves);
}

extern "C" int nh_height(const vt_gen_desc* d, int x, int z) { return height_at(d, x, z); }
