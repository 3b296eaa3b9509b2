// occ_march.cuh — the sample positions of an occupancy ray: from the world to voxels, and how many of them
// are certain to lie in one octant.
#pragma once

#include "occupancy.cuh"

namespace se_gpu {

// A map's resolution and transform, and the bounds of occ_box_steps, for the rays of a launch.
struct OccRes {
    float res, inv;
    int translation; // T_MW is a translation
    float off, less; // voxels, steps
};

constexpr int kOccSkipMax = 256;

// The rays start at o. With u = 2^-24 and k the largest row sum of |R| (at least 1), a component of o + t d is off
// by u (2 t + |o|), of T_MW p by another u k (4 (t + |o|) + 3 |t_MW|), and the division by res by u dim: in all
// less than 8 u k (t + |o| + |t_MW| + dim) / res voxels, where t is less than sqrt(3) (dim + |T_MW o|) inside the
// map. A step t + step is off by u t. off: four times the first for two samples, and a quarter
// voxel for the rounding of occ_box_steps' own sums; less: kOccSkipMax times the second, and one step.
inline OccRes occ_res(const OccDevice& m, F3 o)
{
    OccRes r = {m.res, 1.0f / m.res, 1, 0.0f, 0.0f};
    float k = 1.0f, t_MW = 0.0f;
    for (int i = 0; i < 9; ++i)
        if (m.T_MW.R[i] != ((i % 4 == 0) ? 1.0f : 0.0f))
            r.translation = 0;
    for (int i = 0; i < 3; ++i) {
        k = fmaxf(k, fabsf(m.T_MW.R[3 * i]) + fabsf(m.T_MW.R[3 * i + 1]) + fabsf(m.T_MW.R[3 * i + 2]));
        t_MW = fmaxf(t_MW, fabsf(m.T_MW.t[i]));
    }
    const F3 o_M = apply(m.T_MW, o);
    const float o_max = fmaxf(fmaxf(fabsf(o.x), fabsf(o.y)), fabsf(o.z));
    const float t = 2.0f * (m.dim + fmaxf(fmaxf(fabsf(o_M.x), fabsf(o_M.y)), fabsf(o_M.z)));
    r.off = 0.25f + 0x1p-19f * k * (t + o_max + t_MW + m.dim) * r.inv;
    r.less = 1.0f + (float) kOccSkipMax * 0x1p-24f * t * (2.0f * r.inv);
    return r;
}

// x / res, correctly rounded, from the reciprocal and one residual (div_res in se_gpu_internal.cuh)
__device__ __forceinline__ float occ_div_res(const OccRes& r, float x)
{
    if (!(fabsf(x) >= 0x1p-100f && fabsf(x) < 0x1p100f))
        return x / r.res;
    const float q = x * r.inv;
    return fmaf(fmaf(-q, r.res, x), r.inv, q);
}

__device__ __forceinline__ bool occ_in_map(const OccDevice& m, F3 p)
{
    return p.x >= 0.0f && p.x < m.dim && p.y >= 0.0f && p.y < m.dim && p.z >= 0.0f && p.z < m.dim;
}

// The same for a sample of the march: a coordinate below 2^-100 or beyond 2^100 may come out an ulp off,
// which neither its voxel nor its place in a cell (less half a voxel) can tell.
__device__ __forceinline__ F3 occ_sample_voxel(const OccRes& r, F3 p)
{
    const F3 q = f3(p.x * r.inv, p.y * r.inv, p.z * r.inv);
    return f3(fmaf(fmaf(-q.x, r.res, p.x), r.inv, q.x), fmaf(fmaf(-q.y, r.res, p.y), r.inv, q.y),
              fmaf(fmaf(-q.z, r.res, p.z), r.inv, q.z));
}

// T_MW p; translation: T_MW's rotation is exactly the identity (the products by 1 and 0 change nothing
// but the sign of a zero).
__device__ __forceinline__ F3 occ_to_map(const OccDevice& m, const OccRes& r, F3 p)
{
    if (r.translation)
        return f3(p.x + m.T_MW.t[0], p.y + m.T_MW.t[1], p.z + m.T_MW.t[2]);
    return apply(m.T_MW, p);
}

__device__ __forceinline__ F3 occ_voxel_f(const OccRes& r, F3 p_M)
{
    return f3(occ_div_res(r, p_M.x), occ_div_res(r, p_M.y), occ_div_res(r, p_M.z));
}

__device__ __forceinline__ F3 occ_to_voxel_f(const OccDevice& m, const OccRes& r, F3 p_W)
{
    return occ_voxel_f(r, apply(m.T_MW, p_W));
}

// The samples t + step, t + 2 step, ... (at most kOccSkipMax of them) of a ray that are certain to lie in the
// leaf octant's box (side voxels from bx, by, bz on), from the voxel position v of sample t and the ray's
// direction dv in voxels per unit of t: the distance to the box's faces less the bounds of OccRes. (A quarter
// voxel and a step alone do for a map at the world's origin; at 2 cm and 100 km from it samples outside the
// box were passed.)
__device__ __forceinline__ int occ_box_steps(const OccRes& r, int bx, int by, int bz, int side, F3 v, F3 dv, float step)
{
    const float size = (float) side;
    const float rx = dv.x > 0.0f ? (float) bx + size - v.x : v.x - (float) bx;
    const float ry = dv.y > 0.0f ? (float) by + size - v.y : v.y - (float) by;
    const float rz = dv.z > 0.0f ? (float) bz + size - v.z : v.z - (float) bz;
    const float lim = fminf(fminf((rx - r.off) / fabsf(dv.x), (ry - r.off) / fabsf(dv.y)), (rz - r.off) / fabsf(dv.z));
    const float n = fminf(lim / step, (float) kOccSkipMax) - r.less;
    return n > 0.0f ? (int) n : 0; // also 0 for a NaN
}

} // namespace se_gpu
