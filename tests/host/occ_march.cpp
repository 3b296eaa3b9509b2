// occ_box_steps: the samples that it passes lie in the box. Rays through octants of 8 to 256 voxels, for a map
// at `offset` metres from the world's origin and a camera `back` metres behind the octant, the samples
// accumulated as the raycast does. Prints the rays, the samples passed and those of them outside the box.
#include "cuda_host.hpp"

#include "../../supereight2_gb300/csrc/occ_march.cuh"

#include <cstdlib>
#include <random>

using namespace se_gpu;

int main(int argc, char** argv)
{
    if (argc != 5)
        return 2;
    const float res = strtof(argv[1], nullptr), offset = strtof(argv[2], nullptr), back = strtof(argv[3], nullptr);
    const bool rotated = atoi(argv[4]) != 0;
    std::mt19937 rng(3);
    std::normal_distribution<float> normal;
    std::uniform_real_distribution<float> unit(0.0f, 1.0f);
    OccDevice m = {};
    m.size = 1024;
    m.res = res;
    m.dim = 1024 * res;
    const float c = rotated ? cosf(0.7f) : 1.0f, s = rotated ? sinf(0.7f) : 0.0f;
    const float R[9] = {c, -s, 0, s, c, 0, 0, 0, 1};
    std::copy(R, R + 9, m.T_MW.R);
    const F3 at = f3(offset, -0.37f * offset, 0.11f * offset); // the map's origin in the world
    const F3 rt = rot(m.T_MW, at);
    m.T_MW.t[0] = -rt.x;
    m.T_MW.t[1] = -rt.y;
    m.T_MW.t[2] = -rt.z;
    const float step = res / 2;
    long rays = 0, passed = 0, outside = 0;
    while (rays < 20000) {
        // a camera that looks at a point of the map
        F3 d = f3(normal(rng), normal(rng), normal(rng));
        if (rng() % 4 == 0)
            d.y *= 1e-3f;
        d = normalized(d);
        const F3 p_M = f3(unit(rng) * m.dim, unit(rng) * m.dim, unit(rng) * m.dim);
        const F3 p_W = f3((c * p_M.x + s * p_M.y) + at.x, (c * p_M.y - s * p_M.x) + at.y, p_M.z + at.z);
        const F3 o = sub(p_W, mul(back, d));
        const OccRes r = occ_res(m, o);
        float t = back;
        const F3 v = occ_sample_voxel(r, occ_to_map(m, r, add(o, mul(t, d))));
        if (!(v.x >= 0 && v.x < m.size && v.y >= 0 && v.y < m.size && v.z >= 0 && v.z < m.size))
            continue;
        ++rays;
        const int side = 8 << (rng() % 6), mask = ~(side - 1);
        const int bx = (int) v.x & mask, by = (int) v.y & mask, bz = (int) v.z & mask;
        const F3 dv = mul(rot(m.T_MW, d), r.inv);
        for (int n = occ_box_steps(r, bx, by, bz, side, v, dv, step); n > 0; --n) {
            t += step;
            const F3 q = occ_sample_voxel(r, occ_to_map(m, r, add(o, mul(t, d))));
            ++passed;
            outside += (((int) q.x ^ bx) & mask) || (((int) q.y ^ by) & mask) || (((int) q.z ^ bz) & mask);
        }
    }
    printf("%ld %ld %ld\n", rays, passed, outside);
    return 0;
}
