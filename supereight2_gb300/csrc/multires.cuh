// multires.cuh — voxel access for multi-resolution TSDF maps (Map<Data<TSDF>, Res::Multi, 8>).
//
// Each block keeps the reference's voxel pyramid (BlockMultiRes, block.hpp:66-166): scale 0
// holds 8^3 voxels at offset 0, scale 1 4^3 at 512, scale 2 2^3 at 576, scale 3 one at 584,
// each x + n*y + n^2*z. Every entry stores the data and the past data used by delta
// down-propagation, side by side so that one 16-byte (FP32) or 8-byte (FP16) access moves both:
//   SE_GPU_STORAGE_F32: float4 {tsdf, weight, past tsdf, past weight}
//   SE_GPU_STORAGE_F16: uint2  {f16x_pack(tsdf, weight), f16x_pack(past tsdf, past weight)}
// A block's current scale is the one it integrates at; reads "at the block's data" use it.
#pragma once

#include "se_gpu_internal.cuh"

namespace se_gpu {

__host__ __device__ __forceinline__ int mr_scale_offset(int scale)
{
    return scale == 0 ? 0 : scale == 1 ? 512 : scale == 2 ? 576 : 584;
}

// BlockMultiRes::getVoxelIdx (block_impl.hpp:80-91) from offsets within the block.
__device__ __forceinline__ int mr_index(int ox, int oy, int oz, int scale)
{
    const int n = kBlockSize >> scale;
    return mr_scale_offset(scale) + (ox >> scale) + n * (oy >> scale) + n * n * (oz >> scale);
}

struct MrVoxel {
    float tsdf, weight, past_tsdf, past_weight;
};

template <int S>
__device__ __forceinline__ MrVoxel mr_load(const MapDevice& m, int blk, int i)
{
    MrVoxel v;
    if (S == SE_GPU_STORAGE_F32) {
        const float4 d = reinterpret_cast<const float4*>(m.voxels)[(size_t) blk * kMrVoxels + i];
        v.tsdf = d.x;
        v.weight = d.y;
        v.past_tsdf = d.z;
        v.past_weight = d.w;
    }
    else {
        const uint2 d = reinterpret_cast<const uint2*>(m.voxels)[(size_t) blk * kMrVoxels + i];
        f16x_unpack(d.x, v.tsdf, v.weight);
        f16x_unpack(d.y, v.past_tsdf, v.past_weight);
    }
    return v;
}

// Data half only (tsdf, weight).
template <int S>
__device__ __forceinline__ void mr_load_data(const MapDevice& m, int blk, int i, float& t, float& w)
{
    if (S == SE_GPU_STORAGE_F32) {
        const float2 d = reinterpret_cast<const float2*>(m.voxels)[2 * ((size_t) blk * kMrVoxels + i)];
        t = d.x;
        w = d.y;
    }
    else {
        f16x_unpack(reinterpret_cast<const uint32_t*>(m.voxels)[2 * ((size_t) blk * kMrVoxels + i)], t, w);
    }
}

template <int S>
__device__ __forceinline__ void mr_store(const MapDevice& m, int blk, int i, const MrVoxel& v)
{
    if (S == SE_GPU_STORAGE_F32) {
        reinterpret_cast<float4*>(m.voxels)[(size_t) blk * kMrVoxels + i] =
            make_float4(v.tsdf, v.weight, v.past_tsdf, v.past_weight);
    }
    else {
        reinterpret_cast<uint2*>(m.voxels)[(size_t) blk * kMrVoxels + i] =
            make_uint2(f16x_pack(v.tsdf, v.weight), f16x_pack(v.past_tsdf, v.past_weight));
    }
}

__device__ __forceinline__ int mr_block_of(const MapDevice& m, int vx, int vy, int vz)
{
    return __ldg(&m.block_index[((size_t) (vz >> 3) << (2 * m.log2_bps)) | ((size_t) (vy >> 3) << m.log2_bps)
                                | (size_t) (vx >> 3)]);
}

// The block last looked up by a thread, with its current scale (-1 before its first update or where
// nothing is allocated).
struct MrCache {
    int bx, by, bz;
    int idx, cur;
};

__device__ __forceinline__ void mr_lookup(const MapDevice& m, MrCache& c, int vx, int vy, int vz)
{
    const int bx = vx >> 3, by = vy >> 3, bz = vz >> 3;
    if (bx != c.bx || by != c.by || bz != c.bz) {
        c.bx = bx;
        c.by = by;
        c.bz = bz;
        c.idx = mr_block_of(m, vx, vy, vz);
        c.cur = c.idx < 0 ? -1 : (int) m.block_scale[2 * (size_t) c.idx];
    }
}

// visitor::getData multi-res (visitor_impl.hpp:704-717): the data at the block's current scale, or the default
// data (tsdf 1, weight 0) where no block is allocated. A block that has never been integrated holds the default
// data.
template <int S>
__device__ __forceinline__ void mr_get_data(const MapDevice& m, MrCache& c, int vx, int vy, int vz, float& t, float& w)
{
    mr_lookup(m, c, vx, vy, vz);
    t = 1.0f;
    w = 0.0f;
    if (c.cur >= 0)
        mr_load_data<S>(m, c.idx, mr_index(vx & 7, vy & 7, vz & 7, c.cur), t, w);
}

// visitor::getInterp multi-res (visitor_impl.hpp:906-972) with detail::get_neighbours
// (:398-697). From max(current scale of the query's block, desired scale) upwards, a scale is
// skipped when a block its neighbourhood touches is unallocated or integrates at a coarser
// scale; a base outside the AABB or an invalid neighbour ends the query. The 8 corners' block
// lookups, scales and voxels are each in flight together (one corner after another was a chain of 24
// loads); where they lie in the query's own block there is nothing to look up.
template <int S>
__device__ __forceinline__ bool mr_interp(const MapDevice& m, MrCache& c, F3 vf, int desired_scale, float& out,
                                          int* returned_scale)
{
    mr_lookup(m, c, (int) vf.x, (int) vf.y, (int) vf.z);
    if (c.idx < 0)
        return false;
    const int init = c.cur > desired_scale ? c.cur : desired_scale;
#pragma unroll 1
    for (int scale = init; scale <= kMaxBlockScale; ++scale) {
        const int stride = 1 << scale;
        const float inv = __int_as_float((127 - scale) << 23); // 1 / stride
        const F3 bf = f3(inv * vf.x - 0.5f, inv * vf.y - 0.5f, inv * vf.z - 0.5f);
        const int b0 = stride * (int) bf.x, b1 = stride * (int) bf.y, b2 = stride * (int) bf.z;
        if (b0 < m.aabb[0] || b1 < m.aabb[1] || b2 < m.aabb[2] || b0 > m.aabb[3] || b1 > m.aabb[4] || b2 > m.aabb[5])
            return false;
        if (b0 < 0 || b1 < 0 || b2 < 0 || b0 + stride >= m.size || b1 + stride >= m.size || b2 + stride >= m.size)
            continue;
        float f[8], w[8];
        const bool own = (b0 >> 3) == c.bx && (b1 >> 3) == c.by && (b2 >> 3) == c.bz && (b0 & 7) + stride < 8
            && (b1 & 7) + stride < 8 && (b2 & 7) + stride < 8;
        if (own) { // its current scale is at most `scale` by construction
            const int side = kBlockSize >> scale, at = mr_index(b0 & 7, b1 & 7, b2 & 7, scale);
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                f[n] = 1.0f;
                w[n] = 0.0f;
                if (c.cur >= 0)
                    mr_load_data<S>(m, c.idx, at + (n & 1) + side * ((n >> 1) & 1) + side * side * (n >> 2), f[n], w[n]);
            }
        }
        else {
            int b[8], cur[8];
            bool ok = true;
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                b[n] = mr_block_of(m, b0 + ((n & 1) ? stride : 0), b1 + ((n & 2) ? stride : 0), b2 + ((n & 4) ? stride : 0));
                ok = ok && b[n] >= 0;
            }
            if (!ok)
                continue;
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                cur[n] = (int) m.block_scale[2 * (size_t) b[n]];
                ok = ok && cur[n] <= scale;
            }
            if (!ok)
                continue;
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                // a block never integrated (current scale -1) holds the default data
                f[n] = 1.0f;
                w[n] = 0.0f;
                if (cur[n] >= 0)
                    mr_load_data<S>(m, b[n],
                                    mr_index((b0 + ((n & 1) ? stride : 0)) & 7, (b1 + ((n & 2) ? stride : 0)) & 7,
                                             (b2 + ((n & 4) ? stride : 0)) & 7, scale),
                                    f[n], w[n]);
            }
        }
        bool valid = true;
#pragma unroll
        for (int n = 0; n < 8; ++n)
            valid = valid && w[n] != 0.0f;
        if (!valid)
            return false;
        if (returned_scale)
            *returned_scale = scale;
        const F3 t = f3(bf.x - floorf(bf.x), bf.y - floorf(bf.y), bf.z - floorf(bf.z));
        const F3 tc = f3(1.0f - t.x, 1.0f - t.y, 1.0f - t.z);
        out = ((f[0] * tc.x + f[1] * t.x) * tc.y + (f[2] * tc.x + f[3] * t.x) * t.y) * tc.z
            + ((f[4] * tc.x + f[5] * t.x) * tc.y + (f[6] * tc.x + f[7] * t.x) * t.y) * t.z;
        return true;
    }
    return false;
}

template <int S>
__device__ __forceinline__ bool mr_interp(const MapDevice& m, F3 vf, int desired_scale, float& out, int* returned_scale)
{
    MrCache c{-1, -1, -1, -1, -1};
    return mr_interp<S>(m, c, vf, desired_scale, out, returned_scale);
}

// The 32 gradient samples (visitor_impl.hpp:1332-1412): per axis a selector of
// {base-1, base, base+1, base+2} strides (clamped to the map), packed x | y << 2 | z << 4.
__host__ __device__ constexpr int grad_sel(int i)
{
    constexpr unsigned char t[32] = {0x14, 0x18, 0x24, 0x28, 0x11, 0x21, 0x05, 0x15, 0x25, 0x35, 0x09,
                                     0x19, 0x29, 0x39, 0x1d, 0x2d, 0x12, 0x22, 0x06, 0x16, 0x26, 0x36,
                                     0x0a, 0x1a, 0x2a, 0x3a, 0x1e, 0x2e, 0x17, 0x1b, 0x27, 0x2b};
    return t[i];
}

// grad_sel for the loop below.
static __constant__ unsigned char kGradSel[32] = {
    0x14, 0x18, 0x24, 0x28, 0x11, 0x21, 0x05, 0x15, 0x25, 0x35, 0x09, 0x19, 0x29, 0x39, 0x1d, 0x2d,
    0x12, 0x22, 0x06, 0x16, 0x26, 0x36, 0x0a, 0x1a, 0x2a, 0x3a, 0x1e, 0x2e, 0x17, 0x1b, 0x27, 0x2b};

// mr_grad from scale 2 or coarser up. The samples span up to 3 blocks per axis at scale 2 and 4 at scale 3:
// each has its own lookup, 8 at a time in flight. A 174x133 pass with most of the room at these scales:
// one sample after another 138 us, all 32 unrolled 131, groups of 8 in a loop 124 (the kernel's first pass
// over its code is a good part of such a call). The same loop for scales 0 and 1 would lose there: 1280x960
// 441 -> 488 us without the block table, 457 with it.
template <int S>
__device__ __noinline__ bool mr_grad_coarse(const MapDevice& m, F3 vf, int from, F3& g)
{
    const int q = mr_block_of(m, (int) vf.x, (int) vf.y, (int) vf.z);
    if (q < 0)
        return false;
    const int top = m.size - 1;
#pragma unroll 1
    for (int scale = from; scale <= kMaxBlockScale; ++scale) {
        const int stride = 1 << scale;
        const float inv = 1.0f / (float) stride;
        const F3 sv = f3(inv * vf.x - 0.5f, inv * vf.y - 0.5f, inv * vf.z - 0.5f);
        const F3 fac = f3(sv.x - floorf(sv.x), sv.y - floorf(sv.y), sv.z - floorf(sv.z));
        const int base[3] = {stride * (int) sv.x, stride * (int) sv.y, stride * (int) sv.z};
        // finest_octant(base, scale): a TSDF node holds no data, so only a block goes on
        const int hint = mr_block_of(m, base[0], base[1], base[2]);
        if (hint < 0)
            continue;
        float v[32];
        bool ok = true;
        const int off = mr_scale_offset(scale), sh = 3 - scale;
#pragma unroll 1
        for (int i0 = 0; i0 < 32 && ok; i0 += 8) {
            int b[8], cur[8], at[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int code = kGradSel[i0 + i];
                const int x = min(max(base[0] + ((code & 3) - 1) * stride, 0), top);
                const int y = min(max(base[1] + (((code >> 2) & 3) - 1) * stride, 0), top);
                const int z = min(max(base[2] + ((code >> 4) - 1) * stride, 0), top);
                b[i] = mr_block_of(m, x, y, z);
                at[i] = off + ((x & 7) >> scale) + (((y & 7) >> scale) << sh) + (((z & 7) >> scale) << (2 * sh));
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                cur[i] = b[i] < 0 ? -1 : (int) m.block_scale[2 * (size_t) b[i]];
                ok = ok && cur[i] >= 0 && cur[i] <= scale;
            }
            if (!ok)
                break;
            float t[8], w[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                mr_load_data<S>(m, b[i], at[i], t[i], w[i]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                ok = ok && w[i] != 0.0f;
                v[i0 + i] = t[i];
            }
        }
        if (!ok)
            continue;
        const float rx = 1.0f - fac.x, ry = 1.0f - fac.y, rz = 1.0f - fac.z;
        const float gx = (((v[19] - v[0]) * rx + (v[28] - v[7]) * fac.x) * ry
                          + ((v[23] - v[1]) * rx + (v[29] - v[11]) * fac.x) * fac.y) * rz
            + (((v[20] - v[2]) * rx + (v[30] - v[8]) * fac.x) * ry
               + ((v[24] - v[3]) * rx + (v[31] - v[12]) * fac.x) * fac.y) * fac.z;
        const float gy = (((v[11] - v[4]) * rx + (v[23] - v[16]) * fac.x) * ry
                          + ((v[14] - v[7]) * rx + (v[26] - v[19]) * fac.x) * fac.y) * rz
            + (((v[12] - v[5]) * rx + (v[24] - v[17]) * fac.x) * ry
               + ((v[15] - v[8]) * rx + (v[27] - v[20]) * fac.x) * fac.y) * fac.z;
        const float gz = (((v[8] - v[6]) * rx + (v[20] - v[18]) * fac.x) * ry
                          + ((v[12] - v[10]) * rx + (v[24] - v[22]) * fac.x) * fac.y) * rz
            + (((v[9] - v[7]) * rx + (v[21] - v[19]) * fac.x) * ry
               + ((v[13] - v[11]) * rx + (v[25] - v[23]) * fac.x) * fac.y) * fac.z;
        const float sf = (float) stride;
        g = f3((0.5f * gx) / sf, (0.5f * gy) / sf, (0.5f * gz) / sf);
        return true;
    }
    return false;
}

// visitor::getFieldGrad multi-res with desired scale 0 (visitor_impl.hpp:1257-1497): the
// central-difference gradient at the first scale, from the block's current one up, whose 32
// samples are all valid and stored at exactly that scale; in voxel units (the caller divides
// by the resolution). The samples of scales 0 and 1 span at most 8 voxels: the at most 2 x 2 x 2 blocks
// are looked up once into bt (this thread's 8 entries, bt[k * bs]; -1 where a block has no data at the
// scale), then the 32 loads are in flight together. Coarser scales look each sample's block up.
template <int S>
__device__ __forceinline__ bool mr_grad(const MapDevice& m, MrCache& c, F3 vf, F3& g, int* bt, int bs)
{
    mr_lookup(m, c, (int) vf.x, (int) vf.y, (int) vf.z);
    if (c.idx < 0)
        return false;
    const int init = c.cur > 0 ? c.cur : 0;
    const int top = m.size - 1;
#pragma unroll 1
    for (int scale = init; scale <= 1; ++scale) {
        const int stride = 1 << scale;
        const float inv = __int_as_float((127 - scale) << 23); // 1 / stride
        const F3 sv = f3(inv * vf.x - 0.5f, inv * vf.y - 0.5f, inv * vf.z - 0.5f);
        const F3 fac = f3(sv.x - floorf(sv.x), sv.y - floorf(sv.y), sv.z - floorf(sv.z));
        const int base[3] = {stride * (int) sv.x, stride * (int) sv.y, stride * (int) sv.z};
        int sel[3][4];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            sel[i][0] = max(base[i] - stride, 0);
            sel[i][1] = max(base[i], 0);
            sel[i][2] = min(base[i] + stride, top);
            sel[i][3] = min(base[i] + 2 * stride, top);
        }
        // finest_octant(base, scale): a TSDF node holds no data, so only a block goes on
        if (mr_block_of(m, base[0], base[1], base[2]) < 0)
            continue;
        float v[32];
        bool ok = true;
        {
            int lo[3], two[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                lo[a] = sel[a][0] >> 3;
                two[a] = (sel[a][3] >> 3) != lo[a];
            }
            int blk[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int ox = k & 1, oy = (k >> 1) & 1, oz = k >> 2;
                blk[k] = -1;
                if ((!ox || two[0]) && (!oy || two[1]) && (!oz || two[2]))
                    blk[k] = mr_block_of(m, 8 * (lo[0] + ox), 8 * (lo[1] + oy), 8 * (lo[2] + oz));
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int cur = blk[k] < 0 ? -1 : (int) m.block_scale[2 * (size_t) blk[k]];
                bt[k * bs] = cur >= 0 && cur <= scale ? blk[k] : -1;
            }
            const int off = mr_scale_offset(scale), sh = 3 - scale, mask = kBlockSize - 1;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const int code = grad_sel(i);
                const int x = sel[0][code & 3], y = sel[1][(code >> 2) & 3], z = sel[2][(code >> 4) & 3];
                const int b = bt[(((x >> 3) - lo[0]) | (((y >> 3) - lo[1]) << 1) | (((z >> 3) - lo[2]) << 2)) * bs];
                float t = 1.0f, w = 0.0f;
                if (b >= 0)
                    mr_load_data<S>(m, b,
                                    off + ((x & mask) >> scale) + (((y & mask) >> scale) << sh) + (((z & mask) >> scale) << (2 * sh)),
                                    t, w);
                ok = ok && w != 0.0f;
                v[i] = t;
            }
        }
        if (!ok)
            continue;
        const float rx = 1.0f - fac.x, ry = 1.0f - fac.y, rz = 1.0f - fac.z;
        const float gx = (((v[19] - v[0]) * rx + (v[28] - v[7]) * fac.x) * ry
                          + ((v[23] - v[1]) * rx + (v[29] - v[11]) * fac.x) * fac.y) * rz
            + (((v[20] - v[2]) * rx + (v[30] - v[8]) * fac.x) * ry
               + ((v[24] - v[3]) * rx + (v[31] - v[12]) * fac.x) * fac.y) * fac.z;
        const float gy = (((v[11] - v[4]) * rx + (v[23] - v[16]) * fac.x) * ry
                          + ((v[14] - v[7]) * rx + (v[26] - v[19]) * fac.x) * fac.y) * rz
            + (((v[12] - v[5]) * rx + (v[24] - v[17]) * fac.x) * ry
               + ((v[15] - v[8]) * rx + (v[27] - v[20]) * fac.x) * fac.y) * fac.z;
        const float gz = (((v[8] - v[6]) * rx + (v[20] - v[18]) * fac.x) * ry
                          + ((v[12] - v[10]) * rx + (v[24] - v[22]) * fac.x) * fac.y) * rz
            + (((v[9] - v[7]) * rx + (v[21] - v[19]) * fac.x) * ry
               + ((v[13] - v[11]) * rx + (v[25] - v[23]) * fac.x) * fac.y) * fac.z;
        g = f3((0.5f * gx) * inv, (0.5f * gy) * inv, (0.5f * gz) * inv);
        return true;
    }
    return mr_grad_coarse<S>(m, vf, init > 2 ? init : 2, g);
}

} // namespace se_gpu
