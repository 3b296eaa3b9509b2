// occupancy.cu — multi-resolution occupancy maps (Map<Data<Occupancy>, Res::Multi, 8>): the
// map's pools (creation, destruction, checks, downloads) and the raycast over the octree
// (raycaster_impl.hpp:32-452). Integration lives in occ_integrate.cu.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "occ_march.cuh"
#include "occupancy.cuh"
#include "pipeline.cuh"
#include "profile.cuh"

namespace se_gpu {

// ----------------------------------------------------------------- queries / raycast --

// The occupancy raycast gives each ray eight lanes of a warp. A ray's samples, its interpolations and
// its walk over the octree form one serial chain, and the rays of a view differ in length by a factor
// of ten, so with a lane to a ray the launch lasts as long as its longest rays, at 3 warps in flight
// per SM. Eight lanes take eight successive samples, the eight corners of an interpolation, a
// quarter of the gradient's samples each, or six octant sizes of the walk, and agree by a ballot on
// where the serial algorithm would have stopped; every ray's arithmetic is the serial one's.
// Measured on GB300 (320x240 view of the room at 2 cm / 160x120 view over 40 m at 0.4 m): one lane to
// a ray with the reference's nested loops 8.8-12 / 6.1 ms (rays that leave a loop at different samples
// are not brought together again), one lane to a ray in a common loop 1.5 / 0.68 ms.
constexpr int kOccCtaThreads = 128; // 16 rays: 4 x 4 pixels, a warp 2 x 2
constexpr int kOccPathLevels = 10;  // levels 4..13: nodes of 16^3 to 8192^3 voxels

// A lane's place in the octree. Successive lookups lie in the same leaf octant or next to it, so each
// starts from what the last one found instead of from the root:
//   - the box of the last leaf lookup (the answer is the same for every voxel in it), with
//     its block's scales or its node's data;
//   - the nodes on the path to the last voxel descended to, one per level, in shared memory
//     (path[L * kOccCtaThreads], this thread's column): a lookup restarts at the deepest node that
//     the two voxels share, found by the highest bit in which their coordinates differ.
// Every answer is the root descent's.
struct OccCursor {
    int* path;
    uint64_t* near; // a whole warp's leaves, see occ_seek_warp
    int px, py, pz; // the voxel of the path (masked to the map)
    int low;        // path entries of levels low..log2_size are valid
    int slot;       // fetcher::leaf's answer inside the box (bx, by, bz) / mask: a slot, or -1
    int bx, by, bz, mask;
    int cur, fin;   // a block's current and finest allocated scale
    OccD nd;        // a leaf node's data (default for -1)
};

__device__ __forceinline__ int& occ_path(const OccCursor& c, int level) { return c.path[(level - 4) * kOccCtaThreads]; }

__device__ __forceinline__ void occ_cursor_init(OccCursor& c, const OccDevice& m, int* path, uint64_t* near)
{
    c.path = path;
    c.near = near;
    c.px = c.py = c.pz = 0;
    c.low = m.log2_size;
    occ_path(c, m.log2_size) = 0;
    c.slot = -1;
    c.bx = c.by = c.bz = -1; // masked coordinates are never negative: the first lookup misses
    c.mask = -1;
    c.cur = c.fin = 0;
    c.nd = occ_default();
}

__device__ __forceinline__ bool occ_no_children(const OccDevice& m, int n)
{
    const int4* ch = reinterpret_cast<const int4*>(m.node_child + 8 * (size_t) n);
    const int4 a = ch[0], b = ch[1];
    return (a.x & a.y & a.z & a.w & b.x & b.y & b.z & b.w) == -1; // every slot is -1
}

// fetcher::finest_octant (fetcher_impl.hpp:69-94) down to level `stop` (>= 3) as a slot: the octant
// of size 2^stop on the voxel's path, the block above it, the deepest node when it has no children,
// or -1. level: the size of the box around the voxel that shares the answer, as a power of two.
__device__ __forceinline__ int occ_descend(const OccDevice& m, OccCursor& c, int x, int y, int z, int stop, int& level)
{
    const int mk = m.size - 1;
    x &= mk;
    y &= mk;
    z &= mk;
    const int diff = (x ^ c.px) | (y ^ c.py) | (z ^ c.pz);
    int L = max(c.low, 32 - __clz(diff));
    if (L <= stop) { // the path holds the octant itself (stop > 3: blocks are not on the path)
        level = stop;
        return occ_path(c, stop);
    }
    int n = occ_path(c, L);
    int slot;
    for (;;) {
        const int s = L - 1;
        const int ch = m.node_child[8 * (size_t) n + (((x >> s) & 1) | (((y >> s) & 1) << 1) | (((z >> s) & 1) << 2))];
        if (ch == -1) {
            const bool leaf = occ_no_children(m, n);
            slot = leaf ? n : -1;
            level = leaf ? L : s;
            break;
        }
        if (slot_is_block(ch)) {
            slot = ch;
            level = s;
            break;
        }
        n = ch;
        L = s;
        if (L >= 4)
            occ_path(c, L) = n;
        if (L == stop) {
            slot = n;
            level = L;
            break;
        }
    }
    c.px = x;
    c.py = y;
    c.pz = z;
    c.low = max(L, 4);
    return slot;
}

// fetcher::leaf through the cursor: afterwards the cursor describes the leaf at the voxel.
__device__ __forceinline__ int occ_seek(const OccDevice& m, OccCursor& c, int x, int y, int z)
{
    const int mk = m.size - 1;
    const int xm = x & mk, ym = y & mk, zm = z & mk;
    if ((((xm ^ c.bx) | (ym ^ c.by) | (zm ^ c.bz)) & c.mask) == 0)
        return c.slot;
    int level;
    const int slot = occ_descend(m, c, xm, ym, zm, 3, level);
    c.slot = slot;
    c.mask = ~((1 << level) - 1);
    c.bx = xm & c.mask;
    c.by = ym & c.mask;
    c.bz = zm & c.mask;
    c.nd = occ_default();
    if (slot_is_block(slot)) {
        const OccBlockState& st = m.block_state[slot_block(slot)];
        c.cur = st.current_scale;
        c.fin = st.finest;
    }
    else if (slot != -1) {
        c.nd = node_data(m, slot);
    }
    return slot;
}

// A voxel's index in its block at scale s.
__device__ __forceinline__ int blk_voxel_idx(int x, int y, int z, int s) { return occ_voxel_idx(x & 7, y & 7, z & 7, s); }

// visitor::getMaxData (visitor_impl.hpp:815-835)
__device__ OccD occ_max_data(const OccDevice& m, OccCursor& c, int x, int y, int z, int scale_desired)
{
    int level;
    const int slot = occ_descend(m, c, x, y, z, max(scale_desired, 3), level);
    if (slot == -1)
        return occ_default();
    if (slot_is_block(slot)) {
        const int b = slot_block(slot);
        const OccBlockState& st = m.block_state[b];
        const int so = max(scale_desired, st.current_scale);
        return blk_max(m, b, st.finest, so)[blk_voxel_idx(x, y, z, so)];
    }
    return m.node_max[slot];
}

// visitor::getData(octree, voxel): a block's data at its current scale, a leaf node's data
__device__ __forceinline__ OccD occ_get_data_voxel(const OccDevice& m, OccCursor& c, int x, int y, int z)
{
    const int slot = occ_seek(m, c, x, y, z);
    if (slot_is_block(slot))
        return blk_mean(m, slot_block(slot), c.cur)[blk_voxel_idx(x, y, z, c.cur)];
    return c.nd;
}

constexpr unsigned kOccWarp = 0xffffffffu;

// 2^-scale: dividing by an octant's size, a power of two, is the same as multiplying by this (exact).
__device__ __forceinline__ float occ_inv_size(int scale) { return __int_as_float((127 - scale) << 23); }

// The votes of this lane's group of eight (every lane of the warp takes part).
__device__ __forceinline__ unsigned occ_votes(bool b) { return (__ballot_sync(kOccWarp, b) >> (threadIdx.x & 24)) & 0xffu; }

// The value that lane k of this lane's group holds.
__device__ __forceinline__ float occ_from(float v, int k) { return __shfl_sync(kOccWarp, v, (threadIdx.x & 24) | (k & 7)); }

// The same over the kLanes lanes that sample a ray, a group or the whole warp.
template <int kLanes>
__device__ __forceinline__ unsigned occ_sample_votes(bool b)
{
    return kLanes == 32 ? __ballot_sync(kOccWarp, b) : occ_votes(b);
}
template <int kLanes>
__device__ __forceinline__ float occ_sample_from(float v, int k)
{
    return kLanes == 32 ? __shfl_sync(kOccWarp, v, k & 31) : occ_from(v, k);
}

// The data of a voxel at `scale` (BlockMultiRes::data or a leaf node's): false where nothing is
// allocated or the block's current scale is coarser.
__device__ __forceinline__ bool occ_data_at(const OccDevice& m, OccCursor& c, int x, int y, int z, int scale, OccD& d)
{
    const int slot = occ_seek(m, c, x, y, z);
    if (slot == -1 || (slot_is_block(slot) && c.cur > scale))
        return false;
    d = c.nd;
    if (slot_is_block(slot))
        d = scale < c.fin ? m.block_state[slot_block(slot)].init_data
                          : blk_mean(m, slot_block(slot), scale)[blk_voxel_idx(x, y, z, scale)];
    return true;
}

// ---- lookups of a warp that has one ray
//
// Each lane has a sample of its own, so lanes' lookups differ in length; left to themselves the lanes part
// and the rest of the turn runs lane by lane. Here the warp stays together: every lane calls, those with
// `run` set look up. The leaves found last are kept for the warp, one for each of the block coordinates'
// low two bits on each axis (a turn's samples and their cells span at most four blocks an axis); a descent
// is one to four dependent loads. An entry is one 64-bit word (lanes store and load it whole): the block
// coordinates (10 bits an axis), the slot (28 bits and whether it is a block), and a block's scales or a
// node's level. A slot beyond its field is not kept.
constexpr int kOccNear = 64;
constexpr uint64_t kOccNearEmpty = ~0ull; // no entry: a slot is less

// The leaf at a voxel (masked to the map) for the lanes with `need` set, from level L of the path down: its
// slot, and level | current scale << 4 | finest << 8 | (the path's new lowest level, 0: not walked) << 12. A
// function of its own, for the code's size: its callers are many and its rays few.
static __device__ __noinline__ int2 occ_find_warp(const OccDevice& m, uint64_t* near, int* path, int xm, int ym, int zm, int L,
                                                  bool need)
{
    const uint32_t tag = (uint32_t) (xm >> 3) | ((uint32_t) (ym >> 3) << 10) | ((uint32_t) (zm >> 3) << 20);
    volatile uint64_t* entry = near + (((xm >> 3) & 3) | (((ym >> 3) & 3) << 2) | (((zm >> 3) & 3) << 4));
    int slot = -1, level = 3, scales = 0, low = 0;
    bool go = need;
    if (need) {
        const uint64_t e = *entry;
        if ((uint32_t) (e >> 34) == tag && e != kOccNearEmpty) {
            go = false;
            slot = (int) ((e >> 5) & 0xfffffffu);
            if (e & 1u) {
                slot = -2 - slot;
                scales = (int) (e >> 1) & 15; // current | finest << 2
            }
            else {
                level = (int) (e >> 1) & 15;
            }
        }
    }
    if (__any_sync(kOccWarp, go)) {
        const bool walk = go;
        int n = walk ? path[(L - 4) * kOccCtaThreads] : 0;
        while (__any_sync(kOccWarp, go)) {
            if (go) {
                const int s = L - 1;
                const int ch =
                    m.node_child[8 * (size_t) n + (((xm >> s) & 1) | (((ym >> s) & 1) << 1) | (((zm >> s) & 1) << 2))];
                if (ch == -1) {
                    const bool leaf = occ_no_children(m, n);
                    slot = leaf ? n : -1;
                    level = leaf ? L : s;
                    go = false;
                }
                else if (slot_is_block(ch)) {
                    slot = ch;
                    level = s;
                    go = false;
                }
                else {
                    n = ch;
                    L = s;
                    path[(L - 4) * kOccCtaThreads] = n;
                }
            }
        }
        if (walk)
            low = L;
        if (walk && slot != -1) {
            uint64_t e = (uint64_t) (level << 1);
            int idx = slot;
            if (slot_is_block(slot)) {
                idx = slot_block(slot);
                const OccBlockState& st = m.block_state[idx];
                scales = st.current_scale | st.finest << 2;
                e = (uint64_t) (scales << 1 | 1);
            }
            if (idx < 0xfffffff)
                *entry = e | ((uint64_t) tag << 34) | ((uint64_t) idx << 5);
        }
    }
    __syncwarp();
    return make_int2(slot, level | (scales & 3) << 4 | (scales >> 2) << 8 | low << 12);
}

__device__ __forceinline__ int occ_seek_warp(const OccDevice& m, OccCursor& c, int x, int y, int z, bool run)
{
    const int mk = m.size - 1;
    const int xm = x & mk, ym = y & mk, zm = z & mk;
    const bool miss = run && (((xm ^ c.bx) | (ym ^ c.by) | (zm ^ c.bz)) & c.mask) != 0;
    if (!__any_sync(kOccWarp, miss))
        return c.slot;
    const int2 f = occ_find_warp(m, c.near, c.path, xm, ym, zm,
                                 max(c.low, 32 - __clz((xm ^ c.px) | (ym ^ c.py) | (zm ^ c.pz))), miss);
    if (miss) {
        const int slot = f.x;
        if (f.y >> 12) {
            c.px = xm;
            c.py = ym;
            c.pz = zm;
            c.low = f.y >> 12;
        }
        if (slot_is_block(slot)) {
            c.cur = (f.y >> 4) & 3;
            c.fin = (f.y >> 8) & 3;
        }
        c.slot = slot;
        c.mask = ~((1 << (f.y & 15)) - 1);
        c.bx = xm & c.mask;
        c.by = ym & c.mask;
        c.bz = zm & c.mask;
        c.nd = occ_default();
        if (slot >= 0)
            c.nd = node_data(m, slot);
    }
    __syncwarp();
    return c.slot;
}

// visitor::getInterp multi-res with get_neighbours on an occupancy octree (leaf nodes take part), desired
// scale 0, lane k of a group taking corner k; called by the whole warp, for the groups with `run` set.
// aabb: the map's seven box words, in shared memory. The sums pair up as the serial expression's, so
// every lane of the group gets its value.
template <bool kWarp>
__device__ __forceinline__ bool occ_interp(const OccDevice& m, OccCursor& c, const int* aabb, F3 vf, bool run, float& out,
                                           int& returned_scale)
{
    const int k = threadIdx.x & 7;
    int q = -1;
    if constexpr (kWarp)
        q = occ_seek_warp(m, c, (int) vf.x, (int) vf.y, (int) vf.z, run);
    else if (run)
        q = occ_seek(m, c, (int) vf.x, (int) vf.y, (int) vf.z);
    const bool q_block = slot_is_block(q);
    int scale = q_block ? c.cur : 0;
    run = run && q != -1;
    bool ok = false;
    while (__any_sync(kOccWarp, run)) {
        bool skip = false, fail = false, have = true;
        OccD e = occ_default();
        F3 t = f3(0.0f, 0.0f, 0.0f);
        if (run) {
            const int stride = 1 << scale;
            const float inv = occ_inv_size(scale);
            const F3 bf = f3(inv * vf.x - 0.5f, inv * vf.y - 0.5f, inv * vf.z - 0.5f);
            const int b0 = stride * (int) bf.x, b1 = stride * (int) bf.y, b2 = stride * (int) bf.z;
            t = f3(bf.x - floorf(bf.x), bf.y - floorf(bf.y), bf.z - floorf(bf.z));
            if (aabb[6] || b0 < aabb[0] || b1 < aabb[1] || b2 < aabb[2] || b0 > aabb[3] || b1 > aabb[4] || b2 > aabb[5])
                fail = true;
            else if (b0 + stride >= m.size || b1 + stride >= m.size || b2 + stride >= m.size || b0 < 0 || b1 < 0 || b2 < 0)
                skip = true;
            else {
                const int x = b0 + ((k & 1) ? stride : 0), y = b1 + ((k & 2) ? stride : 0), z = b2 + ((k & 4) ? stride : 0);
                if constexpr (kWarp) // run is the warp's: one ray
                    occ_seek_warp(m, c, x, y, z, true);
                have = occ_data_at(m, c, x, y, z, scale, e);
            }
        }
        const bool all_have = occ_votes(have) == 0xffu, all_valid = occ_votes(occ_valid(e)) == 0xffu;
        // ((f0 tcx + f1 tx) tcy + (f2 tcx + f3 tx) ty) tcz + (...) tz
        float s = occ_field(e) * ((k & 1) ? t.x : 1.0f - t.x);
        s = s + __shfl_xor_sync(kOccWarp, s, 1);
        s = s * ((k & 2) ? t.y : 1.0f - t.y);
        s = s + __shfl_xor_sync(kOccWarp, s, 2);
        s = s * ((k & 4) ? t.z : 1.0f - t.z);
        s = s + __shfl_xor_sync(kOccWarp, s, 4);
        if (run) {
            if (fail) {
                run = false;
            }
            else if (skip || !all_have) {
                run = ++scale <= kOccMaxScale;
            }
            else {
                run = false;
                if (all_valid) {
                    ok = true;
                    out = s;
                    returned_scale = q_block ? scale : (31 - __clz(m.node_coord[q].w));
                }
            }
        }
    }
    return ok;
}

// The 32 gradient samples in the reference's order: per axis a selector of {base - stride, base,
// base + stride, base + 2 stride}, packed x | y << 2 | z << 4.
static __constant__ unsigned char kOccGradSel[32] = {
    0x14, 0x18, 0x24, 0x28, 0x11, 0x21, 0x05, 0x15, 0x25, 0x35, 0x09, 0x19, 0x29, 0x39, 0x1d, 0x2d,
    0x12, 0x22, 0x06, 0x16, 0x26, 0x36, 0x0a, 0x1a, 0x2a, 0x3a, 0x1e, 0x2e, 0x17, 0x1b, 0x27, 0x2b};

// That selector's coordinate, clamped to the map.
__device__ __forceinline__ int occ_grad_coord(int base, int sel, int stride, int top)
{
    const int x = base + (sel - 1) * stride;
    return sel < 2 ? max(x, 0) : min(x, top);
}

// visitor::getFieldGrad multi-res, desired scale 0 (visitor_impl.hpp:1257-1497), occupancy; lane k of a
// group takes samples k, k + 8, k + 16, k + 24, whose values meet in the ray's 32 words of shared memory.
// Called by the whole warp, for the groups with `run` set.
__device__ __forceinline__ bool occ_grad(const OccDevice& m, OccCursor& c, F3 vf, bool run, float* v, F3& g)
{
    const int k = threadIdx.x & 7;
    bool ok = false;
    g = f3(0.0f, 0.0f, 0.0f);
    int scale = 0;
    if (run) {
        // finest_octant(voxel, 0) is the leaf at the voxel
        const int q = occ_seek(m, c, (int) vf.x, (int) vf.y, (int) vf.z);
        if (slot_is_block(q)) {
            scale = c.cur > 0 ? c.cur : 0;
        }
        else {
            run = false;
            ok = q != -1 && occ_valid(c.nd); // a constant octant: gradient 0
        }
    }
    const int top = m.size - 1;
    while (__any_sync(kOccWarp, run)) {
        bool have = false, flat = false;
        F3 fac = f3(0.0f, 0.0f, 0.0f);
        if (run) {
            const int stride = 1 << scale;
            const float inv = occ_inv_size(scale);
            const F3 sv = f3(inv * vf.x - 0.5f, inv * vf.y - 0.5f, inv * vf.z - 0.5f);
            fac = f3(sv.x - floorf(sv.x), sv.y - floorf(sv.y), sv.z - floorf(sv.z));
            const int b0 = stride * (int) sv.x, b1 = stride * (int) sv.y, b2 = stride * (int) sv.z;
            const int oct = occ_seek(m, c, b0, b1, b2); // finest_octant: a scale up to 3 gives the leaf
            if (slot_is_block(oct)) {
                have = true;
#pragma unroll 1
                for (int i = k; i < 32; i += 8) {
                    const int code = kOccGradSel[i];
                    OccD d = occ_default();
                    have = occ_data_at(m, c, occ_grad_coord(b0, code & 3, stride, top),
                                       occ_grad_coord(b1, (code >> 2) & 3, stride, top),
                                       occ_grad_coord(b2, (code >> 4) & 3, stride, top), scale, d)
                        && occ_valid(d) && have;
                    v[i] = occ_field(d);
                }
            }
            else {
                flat = oct != -1 && occ_valid(c.nd);
            }
        }
        __syncwarp();
        const bool all = occ_votes(have) == 0xffu;
        if (run) {
            if (flat) {
                ok = true;
                run = false;
            }
            else if (!all) {
                run = ++scale <= kOccMaxScale;
            }
            else {
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
                const float inv = occ_inv_size(scale);
                g = f3((0.5f * gx) * inv, (0.5f * gy) * inv, (0.5f * gz) * inv);
                ok = true;
                run = false;
            }
        }
        __syncwarp(); // the values are read before the next scale's are written
    }
    return ok;
}

// Whether occ_interp has a value at vf, each lane with `run` set for its own point. The blocks of a cell's
// corners (one, or two along an axis the cell crosses a block's face on) are looked up into `tab` (the
// lane's 8 words of shared memory, kOccCtaThreads apart): a block and whether its initial data holds at the
// scale, or -1 / -2 for a leaf node with / without valid data: from the warp's leaves where all eight are
// there, otherwise one after another. The corners' weights then load together.
__device__ __forceinline__ bool occ_interp_exists(const OccDevice& m, OccCursor& c, const int* aabb, F3 vf, bool run, int* tab)
{
    const int q = occ_seek_warp(m, c, (int) vf.x, (int) vf.y, (int) vf.z, run);
    run = run && q != -1;
    int scale = slot_is_block(q) ? c.cur : 0;
    bool ok = false;
    while (__any_sync(kOccWarp, run)) {
        const int stride = 1 << scale;
        int b0 = 0, b1 = 0, b2 = 0;
        bool have = false;
        if (run) {
            const float inv = occ_inv_size(scale);
            b0 = stride * (int) (inv * vf.x - 0.5f);
            b1 = stride * (int) (inv * vf.y - 0.5f);
            b2 = stride * (int) (inv * vf.z - 0.5f);
            if (aabb[6] || b0 < aabb[0] || b1 < aabb[1] || b2 < aabb[2] || b0 > aabb[3] || b1 > aabb[4] || b2 > aabb[5])
                run = false;
            else
                have = !(b0 + stride >= m.size || b1 + stride >= m.size || b2 + stride >= m.size || b0 < 0 || b1 < 0 || b2 < 0);
        }
        const int two = ((b0 & 7) + stride > 7 ? 1 : 0) | ((b1 & 7) + stride > 7 ? 2 : 0) | ((b2 & 7) + stride > 7 ? 4 : 0);
        // the warp's leaves first, the corners' entries read together
        bool known = have;
        if (have) {
            const uint32_t x0 = b0 >> 3, x1 = (b0 + stride) >> 3, y0 = b1 >> 3, y1 = (b1 + stride) >> 3, z0 = b2 >> 3,
                           z1 = (b2 + stride) >> 3;
            bool fine = true;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const uint32_t x = (k & 1) ? x1 : x0, y = (k & 2) ? y1 : y0, z = (k & 4) ? z1 : z0;
                const uint64_t e = *(volatile uint64_t*) (c.near + ((x & 3) | ((y & 3) << 2) | ((z & 3) << 4)));
                const uint32_t low = (uint32_t) e;
                known = known && (uint32_t) (e >> 34) == (x | (y << 10) | (z << 20)) && (low & 1u) && e != kOccNearEmpty;
                fine = fine && (int) (low >> 1 & 3u) <= scale;
                tab[k * kOccCtaThreads] = (int) ((e >> 5) & 0xfffffffu) << 1 | (scale < (int) (low >> 3 & 3u) ? 1 : 0);
            }
            if (known)
                have = fine;
        }
        const bool seek = have && !known;
        if (__any_sync(kOccWarp, seek)) {
#pragma unroll 1
            for (int k = 0; k < 8; ++k) {
                const bool look = seek && have && (k & ~two) == 0;
                if (!__any_sync(kOccWarp, look))
                    continue;
                const int slot = occ_seek_warp(m, c, b0 + ((k & 1) ? stride : 0), b1 + ((k & 2) ? stride : 0),
                                               b2 + ((k & 4) ? stride : 0), look);
                if (look) {
                    have = slot != -1 && !(slot_is_block(slot) && c.cur > scale);
                    tab[k * kOccCtaThreads] = slot_is_block(slot) ? (slot_block(slot) << 1) | (scale < c.fin ? 1 : 0)
                                                                  : (occ_valid(c.nd) ? -1 : -2);
                }
            }
        }
        bool valid = true;
        if (have) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int e = tab[(k & two) * kOccCtaThreads];
                float w = e == -1 ? 1.0f : 0.0f;
                if (e >= 0) {
                    const OccD* d = (e & 1) ? &m.block_state[e >> 1].init_data
                                            : blk_mean(m, e >> 1, scale)
                            + blk_voxel_idx(b0 + ((k & 1) ? stride : 0), b1 + ((k & 2) ? stride : 0), b2 + ((k & 4) ? stride : 0),
                                            scale);
                    w = d->weight;
                }
                valid = valid && w != 0.0f;
            }
        }
        if (run) {
            ok = have && valid;
            run = !have && ++scale <= kOccMaxScale;
        }
        __syncwarp();
    }
    return ok;
}

// compute_map_intersection (raycaster_impl.hpp:85-173)
__device__ float occ_map_intersection(const OccDevice& m, F3 pos_W, F3 dir_W, float t_far, bool& valid)
{
    const F3 p = apply(m.T_MW, pos_W), dr = rot(m.T_MW, dir_W);
    const float pm[3] = {p.x, p.y, p.z}, dm[3] = {dr.x, dr.y, dr.z};
    const float mx = m.dim;
    bool inside = true;
    int quadrant[3];
    float cand[3] = {0.0f, 0.0f, 0.0f}, maxT[3];
    for (int i = 0; i < 3; ++i) {
        if (pm[i] < 0.0f) {
            quadrant[i] = 1;
            cand[i] = 0.0f;
            inside = false;
        }
        else if (pm[i] > mx) {
            quadrant[i] = 0;
            cand[i] = mx;
            inside = false;
        }
        else {
            quadrant[i] = 2;
        }
    }
    if (inside)
        return 0.0f;
    for (int i = 0; i < 3; ++i)
        maxT[i] = (quadrant[i] != 2 && dm[i] != 0.0f) ? (cand[i] - pm[i]) / dm[i] : -1.0f;
    int which = 0;
    for (int i = 1; i < 3; ++i)
        if (maxT[which] < maxT[i])
            which = i;
    if (maxT[which] < 0.0f) {
        valid = false;
        return 0.0f;
    }
    float hit[3];
    for (int i = 0; i < 3; ++i) {
        if (which != i) {
            hit[i] = pm[i] + maxT[which] * dm[i];
            if (hit[i] < 0.0f || hit[i] > mx) {
                valid = false;
                return 0.0f;
            }
        }
        else {
            hit[i] = cand[i];
        }
    }
    const F3 dh = f3(hit[0] - pm[0], hit[1] - pm[1], hit[2] - pm[2]);
    const float t = sqrtf(dot(dh, dh));
    if (t_far < t) {
        valid = false;
        return 0.0f;
    }
    return t;
}

// advance_ray (raycaster_impl.hpp:189-338): through the octants on the ray, to finer ones where the
// maximum field is above -0.2 (unknown or occupied) and back to coarser ones over free space. Lane k of
// a group evaluates the octant of scale max_scale - k (down to 2) around the ray's place, so that the
// whole way down or up at that place is one ballot. Called by the whole warp; valid: this group's ray
// is under way.
__device__ __forceinline__ void occ_advance_ray(const OccDevice& m, OccCursor& cu, const OccRes& r, F3 o, F3 d, float& t,
                                                float& t_far, int max_scale, bool& valid)
{
    const float voxel_dim = m.res;
    int scale = max_scale;
    float v_add = 0.0f;
    const float v = 1.0f / voxel_dim * t;
    float v_far = 1.0f / voxel_dim * t_far;
    F3 oc = f3(-1.0f, -1.0f, -1.0f);
    const F3 o_M = apply(m.T_MW, o);
    if (occ_in_map(m, o_M))
        oc = occ_voxel_f(r, o_M);
    const float sz = (float) m.size, inv_sz = occ_inv_size(m.log2_size);
    const float dv[3] = {d.x, d.y, d.z};
    const float ocv[3] = {oc.x, oc.y, oc.z};
    // 1 / |d|: times an octant's size it is the correctly rounded size / |d| (a size is a power of two),
    // unless the quotient leaves the normal range, which the test of |d| below keeps it from
    float inv_d[3], vmap[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float dvm = sz / fabsf(dv[i]);
        const float frac = ocv[i] * inv_sz;
        inv_d[i] = 1.0f / fabsf(dv[i]);
        vmap[i] = dv[i] < 0 ? frac * dvm : (1 - frac) * dvm;
    }
    v_far = fminf(fminf(fminf(vmap[0], vmap[1]), vmap[2]) + v, v_far);
    t_far = voxel_dim * v_far;
    F3 rc = oc;
    int guard = 0;
    bool busy = valid;
    const int my_scale = max_scale - (int) (threadIdx.x & 7);
    while (__any_sync(kOccWarp, busy)) {
        bool solid = false;
        if (busy && my_scale >= 2)
            solid = occ_field(occ_max_data(m, cu, (int) rc.x, (int) rc.y, (int) rc.z, my_scale)) > -0.2f;
        const unsigned at = occ_votes(solid); // bit k: the octant of scale max_scale - k
        if (busy) {
            if ((at >> (max_scale - scale)) & 1u) {
                while (scale > 2 && ((at >> (max_scale - scale)) & 1u))
                    scale -= 1;
            }
            else {
                while (scale < max_scale && !((at >> (max_scale - scale - 1)) & 1u))
                    scale += 1;
            }
            if (!((v + v_add) < v_far && guard < (1 << 22))) {
                valid = false;
                busy = false;
            }
            else if (scale <= 2) {
                t = voxel_dim * (v + v_add - 4);
                busy = false;
            }
            else {
                ++guard;
                const int node_size = 1 << scale;
                const float inv_size = occ_inv_size(scale);
                const float rcv[3] = {rc.x, rc.y, rc.z};
                float Vmax[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const int curr = node_size * (int) (floorf(rcv[i]) * inv_size);
                    const float frac = (rcv[i] - (float) curr) * inv_size;
                    const float dV = (float) node_size * inv_d[i];
                    Vmax[i] = dv[i] < 0 ? frac * dV : (1 - frac) * dV;
                    if (fabsf(dv[i]) < 1.0e-6f)
                        Vmax[i] = __int_as_float(0x7f800000);
                }
                const float Vmin = fminf(fminf(Vmax[0], Vmax[1]), Vmax[2]);
                v_add = (float) ((double) v_add + ((double) Vmin + 0.01));
                rc = add(mul(v + v_add, d), oc);
            }
        }
    }
}

// raycast<Occupancy> (raycaster_impl.hpp:352-452) with find_valid_point (:32-70), called by the whole
// warp (active: this group has a ray). A turn of the loop takes eight samples of every ray that is not
// done: it looks for a point with data (find, for the reason `why`), or marches from such a point through
// free space to the surface. The first sample that the serial loop would act on (data found, data lost,
// a field above -0.2, the end of the ray) is taken up, the ones before it only move the ray on, the ones
// after it are dropped. Where a search falls in a leaf octant without data (an unallocated octant, an
// unobserved node) the samples that are certain to stay in it are passed without a lookup.
//
// Along the edge of what has been seen a ray meets hundreds of points whose interpolation has no value (up
// to 269 in a view of the room). After kOccTries of them in a row it is put aside (`susp`, with the state
// that the search needs), and RESUME takes it up: a ray has a warp, a turn 32 samples, and each lane looks
// for itself whether its sample has a value.
struct OccSuspended {
    float t, t_far, value_tt, t_ptt;
    int bits; // why | has_tt << 2 | (scale_tt + 1) << 3
};
constexpr int kOccTries = 2;
template <bool RESUME>
__device__ __forceinline__ bool occ_raycast(const OccDevice& m, OccCursor& c, const OccRes& r, const int* aabb, F3 o, F3 d,
                                            float t_far, bool active, int* tab, OccSuspended& susp, bool& suspended, F3& hit,
                                            int& scale_out)
{
    constexpr int kLanes = RESUME ? 32 : 8; // the samples of a turn
    const int lane = threadIdx.x & (kLanes - 1);
    bool valid = active;
    float t = 0.0f;
    suspended = false;
    if constexpr (RESUME) {
        t = susp.t;
        t_far = susp.t_far;
    }
    else {
        if (active)
            t = occ_map_intersection(m, o, d, t_far, valid);
        const int max_scale = min(7, m.log2_size - 1);
        occ_advance_ray(m, c, r, o, d, t, t_far, max_scale, valid);
    }
    const float step = m.res / 2;
    const F3 dv = mul(rot(m.T_MW, d), r.inv); // voxels per unit of t, for the box skips only
    float value_t = 0.0f, value_tt = 0.0f;
    bool has_tt = false;
    float t_pt = 0.0f, t_ptt = 0.0f; // the samples of value_t and value_tt
    int scale_tt = 0;
    enum { kFind, kMarch, kDone };
    enum { kWhyFirst, kWhyNoData, kWhyNoInterp };
    int mode = valid ? kFind : kDone, why = kWhyFirst;
    bool found = false;
    hit = f3(0.0f, 0.0f, 0.0f);
    bool want = false; // the sample at t waits for its interpolation
    float value = 0.0f;
    int failed = 0; // interpolations that the search made in a row without a value
    if constexpr (RESUME) {
        why = susp.bits & 3;
        has_tt = (susp.bits >> 2) & 1;
        scale_tt = (susp.bits >> 3) - 1;
        value_tt = susp.value_tt;
        t_ptt = susp.t_ptt;
        failed = kOccTries;
    }
    for (;;) {
        const bool take = mode != kDone && !want, find = mode == kFind;
        float tk = t; // sample `lane`, its steps accumulated one by one
#pragma unroll
        for (int j = 0; j < kLanes - 1; ++j)
            if (j < lane)
                tk += step;
        // the samples that the loops would reach: the first is not tested again
        const bool there = lane == 0 || (find ? tk <= t_far : tk < t_far);
        bool has = false;
        int pass = 0; // samples certain to lie in the same octant without data
        float fk = 0.0f;
        const F3 p_M = occ_to_map(m, r, add(o, mul(tk, d)));
        // the march's Map::getData has no bounds check (Safe::Off)
        const bool look = take && there && (!find || occ_in_map(m, p_M));
        const F3 vk = occ_sample_voxel(r, p_M);
        if constexpr (RESUME)
            occ_seek_warp(m, c, (int) vk.x, (int) vk.y, (int) vk.z, look);
        if (look) {
            const OccD data = occ_get_data_voxel(m, c, (int) vk.x, (int) vk.y, (int) vk.z);
            has = occ_valid(data);
            fk = occ_field(data);
            if (find && !has && lane == kLanes - 1 && !slot_is_block(c.slot))
                pass = occ_box_steps(r, c.bx, c.by, c.bz, ~c.mask + 1, vk, dv, step);
        }
        if constexpr (RESUME) {
            const bool probe = find && has && failed >= kOccTries;
            if (__any_sync(kOccWarp, probe)) {
                const bool exists = occ_interp_exists(m, c, aabb, vk, probe, tab);
                if (probe)
                    has = exists;
            }
        }
        const unsigned events = occ_sample_votes<kLanes>(take && there && (find ? has : !has || fk > -0.2f));
        const unsigned gone = occ_sample_votes<kLanes>(!there), data_bits = occ_sample_votes<kLanes>(has);
        const int e = events ? __ffs(events) - 1 : kLanes - 1; // the sample to act on, or the last one
        const float t_e = occ_sample_from<kLanes>(tk, e), f_e = occ_sample_from<kLanes>(fk, e);
        const float t_b = occ_sample_from<kLanes>(tk, e - 1), f_b = occ_sample_from<kLanes>(fk, e - 1);
        pass = __shfl_sync(kOccWarp, pass, threadIdx.x | (kLanes - 1));
        if (take) {
            if (events) {
                t = t_e;
                value = f_e;
                if (!find && e > 0) {
                    value_t = value_tt = f_b;
                    t_pt = t_ptt = t_b;
                    has_tt = true;
                }
                if (find || ((data_bits >> e) & 1u)) {
                    want = true;
                }
                else {
                    t += step;
                    mode = kFind;
                    why = kWhyNoData;
                }
            }
            else if (gone) {
                mode = kDone; // a march ends behind a free sample: no hit
                if (find) {
                    has_tt = false;
                    found = why == kWhyNoData; // reported as a hit at the origin
                }
                else {
                    has_tt = false;
                }
            }
            else {
                t = t_e;
                if (find) {
                    for (; pass > 0 && t <= t_far; --pass)
                        t += step;
                    if (t <= t_far)
                        t += step;
                    if (!(t <= t_far)) {
                        mode = kDone;
                        has_tt = false;
                        found = why == kWhyNoData;
                    }
                }
                else {
                    value_t = value_tt = f_e;
                    t_pt = t_ptt = t_e;
                    has_tt = true;
                    t += step;
                    if (!(t < t_far))
                        mode = kDone;
                }
            }
        }
        // an interpolation is made for every ray that waits for one, when half of the rays under way do:
        // the others go on sampling until then
        const unsigned waiting = __ballot_sync(kOccWarp, want), alive = __ballot_sync(kOccWarp, mode != kDone);
        if (alive == 0u)
            break;
        if (2 * __popc(waiting) < __popc(alive))
            continue;
        int sc = scale_tt;
        const F3 v = occ_sample_voxel(r, occ_to_map(m, r, add(o, mul(t, d))));
        const bool ok = occ_interp<RESUME>(m, c, aabb, v, want, value, sc);
        if (!want)
            continue;
        want = false;
        if (mode == kFind) {
            if (!RESUME) // a ray once put aside looks ahead from then on
                failed = ok ? 0 : failed + 1;
            if (ok) {
                t_pt = t;
                value_t = value;
                t += step;
                // a search inside the march goes on unless the point is already behind the surface (the
                // end of the first search behind it is no hit either way: has_tt is false)
                const bool go = why == kWhyFirst ? value_t <= 0.0f : !(value_t > 0.0f);
                mode = go && t < t_far ? kMarch : kDone;
            }
            else {
                t += step;
                if (!(t <= t_far)) {
                    mode = kDone;
                    has_tt = false;
                    found = why == kWhyNoData;
                }
                else if (!RESUME && failed >= kOccTries) {
                    suspended = true;
                    mode = kDone;
                }
            }
        }
        else if (!ok) {
            has_tt = false;
            t += step;
            mode = kFind;
            why = kWhyNoInterp;
        }
        else {
            value_tt = value;
            has_tt = true;
            t_ptt = t;
            scale_tt = sc;
            if (value_tt > 0.0f) {
                mode = kDone;
            }
            else {
                value_t = value_tt;
                t_pt = t_ptt;
                t += step;
                if (!(t < t_far))
                    mode = kDone;
            }
        }
    }
    if (suspended) {
        susp = OccSuspended{t, t_far, value_tt, t_ptt, why | (has_tt ? 4 : 0) | ((scale_tt + 1) << 3)};
        return false;
    }
    if (found) {
        scale_out = 0;
        return true;
    }
    if (has_tt && value_tt > 0.0f && value_t < 0.0f) {
        const F3 dd = sub(add(o, mul(t_ptt, d)), add(o, mul(t_pt, d)));
        t = t - sqrtf(dot(dd, dd)) * (value_tt - 0.0f) / (value_tt - value_t);
        hit = add(o, mul(d, t));
        scale_out = scale_tt;
        return true;
    }
    return false;
}

// raycaster::raycast_volume for occupancy maps, in three launches: the rays, four to a warp; the rays put
// aside (RESUME), a warp for a ray; the normals. In between a pixel's outputs hold its ray's state, marked in
// the normal's x by a value that is none (kOccHitMark: a hit without its normal; kOccSuspendedMark).
//
// Why: rays along the edge of what has been seen take 50 to 120 turns of the loop, the others 7, and lie
// together. Four to a warp, 1 % of the warps were most of the time, with the rest of the GPU idle, and all
// of them waited for instructions (2 stall cycles an issue with 65 KB of code in one kernel, 0.3 to 0.6
// now). A view of a room,
// 2 cm, with its integration: 320x240 820 us as one kernel, 744 with the rays put aside, 704 with the normals
// apart too; a 160x120 view after eight LiDAR scans 577, 590 and 567. (8 CTAs an SM for the rays: 640x480 1411
// to 1392 us, with the 72 registers they would take 7.)
constexpr float kOccSuspendedMark = 2.0f, kOccHitMark = 3.0f;

// The pixel of a CTA's warp and group in a grid of occ_tiles: 4 x 4 pixels a CTA, the rows of CTAs along y and,
// past the 65,535 of a grid's y (262,140 pixels), along z.
__device__ __forceinline__ void occ_pixel_of(int warp, int ray, int& x, int& y)
{
    x = blockIdx.x * 4 + (warp & 1) * 2 + (ray & 1);
    y = (blockIdx.z * gridDim.y + blockIdx.y) * 4 + (warp >> 1) * 2 + (ray >> 1);
}
static dim3 occ_tiles(int w, int h)
{
    const unsigned rows = ((unsigned) h + 3) / 4, y = std::min(rows, 65535u);
    return dim3(((unsigned) w + 3) / 4, y, (rows + y - 1) / y);
}

template <bool RESUME>
__global__ void __launch_bounds__(kOccCtaThreads, RESUME ? 5 : 8)
    occ_raycast_kernel(const __grid_constant__ OccDevice m, OccRes r, Pinhole s, Tf T_WS, float* __restrict__ pts,
                       float* __restrict__ nrm, int8_t* __restrict__ scale)
{
    grid_dep_wait();
    __shared__ int sh_path[kOccPathLevels * kOccCtaThreads];
    __shared__ int sh_tab[RESUME ? 8 * kOccCtaThreads : 1];
    __shared__ uint64_t sh_near[RESUME ? kOccNear * (kOccCtaThreads / 32) : 1];
    __shared__ int sh_aabb[7];
    if (threadIdx.x < 7)
        sh_aabb[threadIdx.x] = m.aabb[threadIdx.x];
    __syncthreads();
    const int warp = threadIdx.x >> 5, ray = (threadIdx.x >> 3) & 3, lane = threadIdx.x & 7;
    int x, y;
    if constexpr (RESUME) {
        const size_t i = (size_t) blockIdx.x * (kOccCtaThreads / 32) + warp;
        if (i >= (size_t) s.w * s.h || nrm[3 * i] != kOccSuspendedMark)
            return;
        x = (int) (i % s.w);
        y = (int) (i / s.w);
    }
    else {
        occ_pixel_of(warp, ray, x, y);
    }
    const bool in_image = x < s.w && y < s.h; // rays past the edge stay for the warp's votes
    OccCursor c;
    occ_cursor_init(c, m, sh_path + threadIdx.x, RESUME ? sh_near + kOccNear * warp : nullptr);
    if constexpr (RESUME) {
        for (int k = threadIdx.x & 31; k < kOccNear; k += 32)
            c.near[k] = kOccNearEmpty;
        __syncwarp();
    }
    const size_t idx = (size_t) x + (size_t) y * s.w;
    const F3 ray_S = back_project(s, (float) x, (float) y);
    const F3 nS = normalized(ray_S);
    const F3 dir_W = rot(T_WS, nS);
    const F3 origin = f3(T_WS.t[0], T_WS.t[1], T_WS.t[2]);
    F3 hit, p = f3(0.0f, 0.0f, 0.0f), n = f3(0.0f, 0.0f, 0.0f);
    int sc = 0;
    OccSuspended susp;
    bool suspended;
    if constexpr (RESUME)
        susp = OccSuspended{pts[3 * idx], pts[3 * idx + 1], pts[3 * idx + 2], nrm[3 * idx + 1],
                            __float_as_int(nrm[3 * idx + 2])};
    const bool is_hit = occ_raycast<RESUME>(m, c, r, sh_aabb, origin, dir_W, s.far_plane / nS.z, in_image,
                                            RESUME ? sh_tab + threadIdx.x : nullptr, susp, suspended, hit, sc);
    if (is_hit) {
        p = hit;
        n.x = kOccHitMark;
    }
    else {
        sc = 0;
    }
    if (suspended) {
        p = f3(susp.t, susp.t_far, susp.value_tt);
        n = f3(kOccSuspendedMark, susp.t_ptt, __int_as_float(susp.bits));
    }
    __syncwarp(); // every lane has read the ray's state
    if (!in_image || (RESUME && ray != 0))
        return;
    if (lane < 3)
        pts[3 * idx + lane] = lane == 0 ? p.x : lane == 1 ? p.y : p.z;
    else if (lane < 6)
        nrm[3 * idx + lane - 3] = lane == 3 ? n.x : lane == 4 ? n.y : n.z;
    else if (lane == 6 && scale)
        scale[idx] = (int8_t) sc;
}

// The normals at the hits, which occ_raycast_kernel has marked.
__global__ void __launch_bounds__(kOccCtaThreads) occ_normal_kernel(const __grid_constant__ OccDevice m, OccRes r, int w, int h,
                                                                    const float* __restrict__ pts, float* __restrict__ nrm)
{
    grid_dep_wait();
    __shared__ int sh_path[kOccPathLevels * kOccCtaThreads];
    __shared__ float sh_grad[kOccCtaThreads / 8][33];
    const int warp = threadIdx.x >> 5, ray = (threadIdx.x >> 3) & 3, lane = threadIdx.x & 7;
    int x, y;
    occ_pixel_of(warp, ray, x, y);
    const size_t idx = (size_t) x + (size_t) y * w;
    const bool is_hit = x < w && y < h && nrm[3 * idx] == kOccHitMark;
    if (!__any_sync(kOccWarp, is_hit))
        return;
    OccCursor c;
    occ_cursor_init(c, m, sh_path + threadIdx.x, nullptr);
    F3 hit = f3(0.0f, 0.0f, 0.0f), g, n = f3(0.0f, 0.0f, 0.0f);
    if (is_hit)
        hit = f3(pts[3 * idx], pts[3 * idx + 1], pts[3 * idx + 2]);
    if (occ_grad(m, c, occ_to_voxel_f(m, r, hit), is_hit, sh_grad[threadIdx.x >> 3], g)) {
        g = f3(g.x / m.res, g.y / m.res, g.z / m.res);
        const float nn = sqrtf(dot(g, g));
        n = nn > 0.0f ? f3(-(g.x / nn), -(g.y / nn), -(g.z / nn)) : f3(-g.x, -g.y, -g.z);
    }
    if (is_hit && lane < 3)
        nrm[3 * idx + lane] = lane == 0 ? n.x : lane == 1 ? n.y : n.z;
}

se_gpu_status occ_raycast_volume(const se_gpu_occ_map* om, const se_gpu_pinhole& sensor, const float* T_WS16,
                                 float* pts, float* nrm, int8_t* scale, cudaStream_t stream)
{
    const Pinhole s = make_pinhole(sensor);
    const dim3 grid = occ_tiles(s.w, s.h);
    const Tf T_WS = tf_from16(T_WS16);
    const OccRes r = occ_res(om->dev, f3(T_WS.t[0], T_WS.t[1], T_WS.t[2]));
    ProfScope ps(kProfRaycast, stream);
    launch_chained(occ_raycast_kernel<false>, grid, kOccCtaThreads, stream, om->dev, r, s, T_WS, pts, nrm, scale);
    constexpr int kWarps = kOccCtaThreads / 32;
    const unsigned warps_ctas = (unsigned) (((size_t) s.w * s.h + kWarps - 1) / kWarps);
    launch_chained(occ_raycast_kernel<true>, warps_ctas, kOccCtaThreads, stream, om->dev, r, s,
                   T_WS, pts, nrm, scale);
    launch_chained(occ_normal_kernel, grid, kOccCtaThreads, stream, om->dev, r, s.w, s.h, pts, nrm);
    SE_CUDA_TRY(cudaGetLastError());
    return SE_GPU_OK;
}

} // namespace se_gpu

using namespace se_gpu;

namespace se_gpu {

se_gpu_status occ_map_create(const se_gpu_map_config* cfg, const se_gpu_occupancy_config* occ, int size,
                             se_gpu_occ_map** out)
{
    se_gpu_occ_map* om = new se_gpu_occ_map();
    std::memset(&om->dev, 0, sizeof(om->dev));
    om->scratch = OccScratch();
    OccDevice& m = om->dev;
    m.size = size;
    m.log2_size = 0;
    while ((1 << m.log2_size) < size)
        ++m.log2_size;
    m.block_depth = m.log2_size - 3;
    m.res = cfg->res;
    m.dim = (float) size * cfg->res;
    if (cfg->has_T_MW) {
        m.T_MW = tf_from16(cfg->T_MW);
    }
    else {
        for (int i = 0; i < 9; ++i)
            m.T_MW.R[i] = (i % 4 == 0) ? 1.0f : 0.0f;
        m.T_MW.t[0] = cfg->dim[0] / 2.0f;
        m.T_MW.t[1] = cfg->dim[1] / 2.0f;
        m.T_MW.t[2] = cfg->dim[2] / 2.0f;
    }
    m.T_WM = inverse_iso(m.T_MW);
    se_gpu_occupancy_config c;
    if (occ) {
        c = *occ;
    }
    else {
        c.k_sigma = 0.052f;
        c.sigma_min_factor = 1.5f;
        c.sigma_max_factor = 6.0f;
        c.k_tau = 0.026f;
        c.tau_min_factor = 6.0f;
        c.tau_max_factor = 16.0f;
        c.log_odd_min = (float) -5.015;
        c.log_odd_max = (float) 5.015;
        c.fs_integr_scale = 1;
    }
    m.cfg.k_sigma = c.k_sigma;
    m.cfg.sigma_min_factor = c.sigma_min_factor;
    m.cfg.sigma_max_factor = c.sigma_max_factor;
    m.cfg.k_tau = c.k_tau;
    m.cfg.tau_min_factor = c.tau_min_factor;
    m.cfg.tau_max_factor = c.tau_max_factor;
    m.cfg.log_odd_min = c.log_odd_min;
    m.cfg.log_odd_max = c.log_odd_max;
    m.cfg.fs_integr_scale = c.fs_integr_scale;
    // FieldData<Occupancy>::Config::max_weight keeps its default (data_field.hpp:67): the YAML
    // reader does not recompute it from a configured log_odd_min
    m.cfg.max_weight = std::floor(std::fabs(-100.0f / (0.97f * (float) -5.015)));
    m.block_capacity = (int) cfg->max_blocks;
    // nodes per block stay below 0.3 in the tests' scenes; half the block capacity leaves margin
    m.node_capacity = (int) (cfg->max_blocks / 2 + 4096);
    auto fail = [&](cudaError_t e, const char* what) {
        se_gpu_status st = cuda_status(e, what);
        occ_map_destroy(om);
        return st;
    };
    cudaError_t e;
    const size_t nc = (size_t) m.node_capacity, bc = (size_t) m.block_capacity;
    if ((e = cudaMalloc(&m.node_coord, nc * sizeof(int4))) != cudaSuccess) return fail(e, "cudaMalloc(nodes)");
    if ((e = cudaMalloc(&m.node_parent, nc * sizeof(int))) != cudaSuccess) return fail(e, "cudaMalloc(nodes)");
    if ((e = cudaMalloc(&m.node_child, nc * 8 * sizeof(int))) != cudaSuccess) return fail(e, "cudaMalloc(nodes)");
    if ((e = cudaMalloc(&m.node_min, nc * sizeof(OccD))) != cudaSuccess) return fail(e, "cudaMalloc(nodes)");
    if ((e = cudaMalloc(&m.node_max, nc * sizeof(OccD))) != cudaSuccess) return fail(e, "cudaMalloc(nodes)");
    if ((e = cudaMalloc(&m.node_mark, nc * sizeof(int))) != cudaSuccess) return fail(e, "cudaMalloc(nodes)");
    if ((e = cudaMalloc(&m.node_ts, nc * sizeof(int))) != cudaSuccess) return fail(e, "cudaMalloc(nodes)");
    if ((e = cudaMalloc(&m.block_coord, bc * 3 * sizeof(int))) != cudaSuccess) return fail(e, "cudaMalloc(blocks)");
    if ((e = cudaMalloc(&m.block_state, bc * sizeof(OccBlockState))) != cudaSuccess) return fail(e, "cudaMalloc(blocks)");
    if ((e = cudaMalloc(&m.block_mean, bc * 585 * sizeof(OccD))) != cudaSuccess) return fail(e, "cudaMalloc(blocks)");
    if ((e = cudaMalloc(&m.block_min, bc * 585 * sizeof(OccD))) != cudaSuccess) return fail(e, "cudaMalloc(blocks)");
    if ((e = cudaMalloc(&m.block_max, bc * 585 * sizeof(OccD))) != cudaSuccess) return fail(e, "cudaMalloc(blocks)");
    if ((e = cudaMalloc(&m.block_buffer, bc * 512 * sizeof(OccD))) != cudaSuccess) return fail(e, "cudaMalloc(blocks)");
    if ((e = cudaMalloc(&m.block_ts, bc * sizeof(int))) != cudaSuccess) return fail(e, "cudaMalloc(blocks)");
    if ((e = cudaMalloc(&m.aabb, 8 * sizeof(int))) != cudaSuccess) return fail(e, "cudaMalloc(aabb)");
    if ((e = cudaMalloc(&m.counters, kOccCounters * sizeof(int))) != cudaSuccess) return fail(e, "cudaMalloc(counters)");
    {
        const int aabb[8] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN, 1, 0};
        if ((e = cudaMemcpy(m.aabb, aabb, sizeof(aabb), cudaMemcpyHostToDevice)) != cudaSuccess) return fail(e, "aabb");
        if ((e = cudaMemset(m.counters, 0, kOccCounters * sizeof(int))) != cudaSuccess) return fail(e, "counters");
        // the root: node 0
        const int one = 1;
        if ((e = cudaMemcpy(m.counters + kOccNodes, &one, sizeof(int), cudaMemcpyHostToDevice)) != cudaSuccess)
            return fail(e, "counters");
        const int4 rc = make_int4(0, 0, 0, size);
        const int minus1[8] = {-1, -1, -1, -1, -1, -1, -1, -1};
        const int rp = -1;
        const OccD def = occ_default();
        if ((e = cudaMemcpy(m.node_coord, &rc, sizeof(rc), cudaMemcpyHostToDevice)) != cudaSuccess) return fail(e, "root");
        if ((e = cudaMemcpy(m.node_parent, &rp, sizeof(int), cudaMemcpyHostToDevice)) != cudaSuccess) return fail(e, "root");
        if ((e = cudaMemcpy(m.node_child, minus1, sizeof(minus1), cudaMemcpyHostToDevice)) != cudaSuccess) return fail(e, "root");
        if ((e = cudaMemcpy(m.node_min, &def, sizeof(def), cudaMemcpyHostToDevice)) != cudaSuccess) return fail(e, "root");
        if ((e = cudaMemcpy(m.node_max, &def, sizeof(def), cudaMemcpyHostToDevice)) != cudaSuccess) return fail(e, "root");
        if ((e = cudaMemcpy(m.node_mark, &rp, sizeof(int), cudaMemcpyHostToDevice)) != cudaSuccess) return fail(e, "root");
        if ((e = cudaMemcpy(m.node_ts, &rp, sizeof(int), cudaMemcpyHostToDevice)) != cudaSuccess) return fail(e, "root");
    }
    if ((e = cudaDeviceSynchronize()) != cudaSuccess) return fail(e, "cudaDeviceSynchronize");
    *out = om;
    return SE_GPU_OK;
}

void occ_map_destroy(se_gpu_occ_map* om)
{
    if (!om)
        return;
    OccDevice& m = om->dev;
    cudaFree(m.node_coord);
    cudaFree(m.node_parent);
    cudaFree(m.node_child);
    cudaFree(m.node_min);
    cudaFree(m.node_max);
    cudaFree(m.node_mark);
    cudaFree(m.node_ts);
    cudaFree(m.block_coord);
    cudaFree(m.block_state);
    cudaFree(m.block_mean);
    cudaFree(m.block_min);
    cudaFree(m.block_max);
    cudaFree(m.block_buffer);
    cudaFree(m.block_ts);
    cudaFree(m.aabb);
    cudaFree(m.counters);
    occ_scratch_free(om);
    ri_scratch_free(om->ri);
    delete om;
}

} // namespace se_gpu

namespace se_gpu {

se_gpu_status occ_check(se_gpu_occ_map* om)
{
    int err = 0;
    SE_CUDA_TRY(cudaMemcpy(&err, om->dev.counters + kOccError, sizeof(int), cudaMemcpyDeviceToHost));
    if (!err)
        return SE_GPU_OK;
    SE_CUDA_TRY(cudaMemset(om->dev.counters + kOccError, 0, sizeof(int)));
    if (err & kOccErrBlockPool) {
        set_last_error("occupancy block pool of %d blocks is full", om->dev.block_capacity);
        return SE_GPU_ERR_POOL_FULL;
    }
    if (err & kOccErrNodePool) {
        set_last_error("occupancy node pool of %d nodes is full", om->dev.node_capacity);
        return SE_GPU_ERR_POOL_FULL;
    }
    if (err & kOccErrTimeout) {
        set_last_error("a grid barrier of the persistent batch launch waited past its limit; the frame is incomplete");
        return SE_GPU_ERR_CUDA;
    }
    set_last_error("an occupancy work list overflowed");
    return SE_GPU_ERR_POOL_FULL;
}

se_gpu_status occ_aabb(const se_gpu_occ_map* om, int32_t mn[3], int32_t mx[3], int* empty)
{
    int a[8];
    SE_CUDA_TRY(cudaMemcpy(a, om->dev.aabb, sizeof(a), cudaMemcpyDeviceToHost));
    *empty = a[6];
    for (int i = 0; i < 3; ++i) {
        mn[i] = a[6] ? 0 : a[i];
        mx[i] = a[6] ? 0 : a[3 + i];
    }
    return SE_GPU_OK;
}

} // namespace se_gpu

static se_gpu_status occ_args(const se_gpu_map* map, const char* fn)
{
    if (!map) {
        set_last_error("%s: null map", fn);
        return SE_GPU_ERR_BAD_ARG;
    }
    if (!map->occ) {
        set_last_error("%s: not an occupancy map", fn);
        return SE_GPU_ERR_NOT_SUPPORTED;
    }
    return SE_GPU_OK;
}

extern "C" {

se_gpu_status se_gpu_map_occupancy_stats(se_gpu_map* map, int64_t stats[4])
{
    se_gpu_status st = occ_args(map, "se_gpu_map_occupancy_stats");
    if (st != SE_GPU_OK)
        return st;
    SE_CUDA_TRY(cudaStreamSynchronize(map->last_stream));
    int c[kOccCounters];
    SE_CUDA_TRY(cudaMemcpy(c, map->occ->dev.counters, sizeof(c), cudaMemcpyDeviceToHost));
    stats[0] = c[kOccBlockListN];
    stats[1] = c[kOccNodeListN];
    stats[2] = c[kOccFreedN];
    stats[3] = c[kOccPruned];
    return SE_GPU_OK;
}

se_gpu_status se_gpu_map_download_occupancy(const se_gpu_map* map, int64_t capacity, int32_t* coords, int32_t* scales,
                                            int64_t* counts, float* mean, float* min_data, float* max_data,
                                            int64_t* count)
{
    se_gpu_status st = occ_args(map, "se_gpu_map_download_occupancy");
    if (st != SE_GPU_OK)
        return st;
    if (capacity < 0) {
        set_last_error("se_gpu_map_download_occupancy: negative capacity");
        return SE_GPU_ERR_BAD_ARG;
    }
    SE_CUDA_TRY(cudaStreamSynchronize(map->last_stream));
    const OccDevice& m = map->occ->dev;
    int nb = 0;
    SE_CUDA_TRY(cudaMemcpy(&nb, m.counters + kOccBlocks, sizeof(int), cudaMemcpyDeviceToHost));
    nb = nb < m.block_capacity ? nb : m.block_capacity;
    std::vector<OccBlockState> states((size_t) nb);
    std::vector<int> bc((size_t) nb * 3);
    if (nb) {
        SE_CUDA_TRY(cudaMemcpy(states.data(), m.block_state, (size_t) nb * sizeof(OccBlockState), cudaMemcpyDeviceToHost));
        SE_CUDA_TRY(cudaMemcpy(bc.data(), m.block_coord, (size_t) nb * 3 * sizeof(int), cudaMemcpyDeviceToHost));
    }
    int64_t live = 0;
    for (int b = 0; b < nb; ++b)
        live += states[(size_t) b].live ? 1 : 0;
    if (count)
        *count = live;
    const bool want_data = mean || min_data || max_data;
    std::vector<OccD> hm, hn, hx;
    if (want_data && nb) {
        hm.resize((size_t) nb * 585);
        hn.resize((size_t) nb * 585);
        hx.resize((size_t) nb * 585);
        SE_CUDA_TRY(cudaMemcpy(hm.data(), m.block_mean, hm.size() * sizeof(OccD), cudaMemcpyDeviceToHost));
        SE_CUDA_TRY(cudaMemcpy(hn.data(), m.block_min, hn.size() * sizeof(OccD), cudaMemcpyDeviceToHost));
        SE_CUDA_TRY(cudaMemcpy(hx.data(), m.block_max, hx.size() * sizeof(OccD), cudaMemcpyDeviceToHost));
    }
    int64_t k = 0;
    for (int b = 0; b < nb && k < capacity; ++b) {
        const OccBlockState& s = states[(size_t) b];
        if (!s.live)
            continue;
        if (coords)
            for (int a = 0; a < 3; ++a)
                coords[3 * k + a] = bc[(size_t) b * 3 + a];
        if (scales) {
            scales[3 * k] = s.current_scale;
            scales[3 * k + 1] = s.min_scale;
            scales[3 * k + 2] = s.buffer_scale;
        }
        if (counts) {
            counts[4 * k] = (int64_t) s.curr_integr;
            counts[4 * k + 1] = (int64_t) s.curr_obs;
            counts[4 * k + 2] = (int64_t) s.buf_integr;
            counts[4 * k + 3] = (int64_t) s.buf_obs;
        }
        if (want_data) {
            for (int sc = 0; sc <= kOccMaxScale; ++sc) {
                const int nv = (8 >> sc) * (8 >> sc) * (8 >> sc);
                for (int v = 0; v < nv; ++v) {
                    const size_t src = (size_t) b * 585 + occ_scale_offset(sc) + v;
                    const size_t o = ((size_t) k * 585 + occ_scale_offset(sc) + v) * 3;
                    const OccD e = sc < s.finest ? s.init_data : hm[src];
                    const OccD mn = sc < s.finest ? s.init_data : (sc == s.finest ? hm[src] : hn[src]);
                    const OccD mx = sc < s.finest ? s.init_data : (sc == s.finest ? hm[src] : hx[src]);
                    const OccD* ds[3] = {&e, &mn, &mx};
                    float* outs[3] = {mean, min_data, max_data};
                    for (int q = 0; q < 3; ++q) {
                        if (!outs[q])
                            continue;
                        outs[q][o] = ds[q]->occ;
                        outs[q][o + 1] = ds[q]->weight;
                        outs[q][o + 2] = ds[q]->observed ? 1.0f : 0.0f;
                    }
                }
            }
        }
        ++k;
    }
    return SE_GPU_OK;
}

se_gpu_status se_gpu_map_download_nodes(const se_gpu_map* map, int64_t capacity, int32_t* coords, float* min_data,
                                        float* max_data, int32_t* leaf, int64_t* count)
{
    se_gpu_status st = occ_args(map, "se_gpu_map_download_nodes");
    if (st != SE_GPU_OK)
        return st;
    SE_CUDA_TRY(cudaStreamSynchronize(map->last_stream));
    const OccDevice& m = map->occ->dev;
    int nn = 0;
    SE_CUDA_TRY(cudaMemcpy(&nn, m.counters + kOccNodes, sizeof(int), cudaMemcpyDeviceToHost));
    nn = nn < m.node_capacity ? nn : m.node_capacity;
    std::vector<int4> nc((size_t) nn);
    std::vector<int> ch((size_t) nn * 8);
    std::vector<OccD> nmin((size_t) nn), nmax((size_t) nn);
    SE_CUDA_TRY(cudaMemcpy(nc.data(), m.node_coord, (size_t) nn * sizeof(int4), cudaMemcpyDeviceToHost));
    SE_CUDA_TRY(cudaMemcpy(ch.data(), m.node_child, (size_t) nn * 8 * sizeof(int), cudaMemcpyDeviceToHost));
    SE_CUDA_TRY(cudaMemcpy(nmin.data(), m.node_min, (size_t) nn * sizeof(OccD), cudaMemcpyDeviceToHost));
    SE_CUDA_TRY(cudaMemcpy(nmax.data(), m.node_max, (size_t) nn * sizeof(OccD), cudaMemcpyDeviceToHost));
    std::vector<int> stack{0};
    int64_t k = 0;
    while (!stack.empty()) {
        const int n = stack.back();
        stack.pop_back();
        if (k < capacity) {
            if (coords) {
                coords[4 * k] = nc[(size_t) n].x;
                coords[4 * k + 1] = nc[(size_t) n].y;
                coords[4 * k + 2] = nc[(size_t) n].z;
                coords[4 * k + 3] = nc[(size_t) n].w;
            }
            const OccD* ds[2] = {&nmin[(size_t) n], &nmax[(size_t) n]};
            float* outs[2] = {min_data, max_data};
            for (int q = 0; q < 2; ++q) {
                if (!outs[q])
                    continue;
                outs[q][3 * k] = ds[q]->occ;
                outs[q][3 * k + 1] = ds[q]->weight;
                outs[q][3 * k + 2] = ds[q]->observed ? 1.0f : 0.0f;
            }
            if (leaf) {
                bool is_leaf = true;
                for (int i = 0; i < 8; ++i)
                    is_leaf = is_leaf && ch[(size_t) n * 8 + i] == -1;
                leaf[k] = is_leaf ? 1 : 0;
            }
        }
        ++k;
        for (int i = 7; i >= 0; --i) {
            const int c = ch[(size_t) n * 8 + i];
            if (c >= 0)
                stack.push_back(c);
        }
    }
    if (count)
        *count = k;
    return SE_GPU_OK;
}

} // extern "C"
