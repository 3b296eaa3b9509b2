// occ_propagate.cuh — node propagation of the occupancy map: the propagation sets of each depth and their
// nodes' minimum and maximum data, by groups of eight lanes.
#pragma once

#include <cfloat>

#include "occupancy.cuh"

namespace se_gpu {

// 0.95 * -100 of the reference's tests, which is -95 in double.
constexpr float kOccFreeField = -95.0f;
static_assert(0.95 * -100.0 == (double) kOccFreeField);

__device__ __forceinline__ int occ_node_depth(const OccDevice& m, int n)
{
    return m.log2_size - (31 - __clz(m.node_coord[n].w));
}

// Insert node n into the propagation set of its depth (std::set semantics: once per frame).
__device__ __forceinline__ void occ_set_insert(const OccDevice& m, int* sets, int n, int frame_id)
{
    if (n < 0)
        return;
    if (atomicExch(&m.node_mark[n], frame_id) == frame_id)
        return;
    const int d = occ_node_depth(m, n);
    const int k = atomicAdd(&m.counters[kOccSetN + d], 1);
    if (k < m.node_capacity)
        sets[(size_t) d * m.node_capacity + k] = n;
    else
        atomicOr(&m.counters[kOccError], kOccErrList);
}

// The reduction of 8 children to their parent's minimum (or maximum) data (multires_ofusion_core_impl.hpp:
// 14-85): the first child with the least (greatest) field, observed if all 8 are; child 0 where no field
// beats the bound. A group of 8 lanes holds a child each; the lane with the result returns true, with the
// data in d; none where no child is valid.
__device__ __forceinline__ bool occ_up_best8(const OccD& c, bool want_min, int lane, OccD& d)
{
    const unsigned group = 0xffu << (lane & 24);
    const bool valid = occ_valid(c);
    const unsigned nv = __ballot_sync(0xffffffffu, valid) & group;
    const unsigned no = __ballot_sync(0xffffffffu, valid && c.observed) & group;
    const float bound = want_min ? FLT_MAX : -FLT_MAX;
    float best = valid ? occ_field(c) : bound;
    const bool cand = want_min ? best < bound : best > bound; // a NaN is none
    best = cand ? best : bound;
    int at = cand ? (lane & 7) : 8;
    for (int o = 1; o < 8; o <<= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oa = __shfl_xor_sync(0xffffffffu, at, o);
        if ((want_min ? ob < best : ob > best) || (ob == best && oa < at)) {
            best = ob;
            at = oa;
        }
    }
    d = c;
    d.observed = no == group ? 1 : 0;
    return nv != 0 && (lane & 7) == (at & 7); // none beat the bound: child 0
}

// updater::propagate_to_parent_node (multires_ofusion_core_impl.hpp:88-117) by a group of 8 lanes, a child
// each (all 32 lanes call it; n < 0: an idle group). A child's data are three dependent loads, which one
// thread for a node did eight times in turn. The node's maximum is returned to the group.
__device__ OccD occ_propagate_node(const OccDevice& m, int n, int timestamp, int lane)
{
    OccD cmin = occ_default(), cmax = occ_default(), mx = occ_default();
    if (n >= 0) {
        const int c = m.node_child[8 * (size_t) n + (lane & 7)];
        mx = m.node_max[n];
        if (c != -1) {
            if (slot_is_block(c)) {
                const int b = slot_block(c);
                const int fin = m.block_state[b].finest;
                cmin = blk_min(m, b, fin, kOccMaxScale)[0];
                cmax = blk_max(m, b, fin, kOccMaxScale)[0];
            }
            else {
                cmin = m.node_min[c];
                cmax = m.node_max[c];
            }
        }
        if ((lane & 7) == 0)
            m.node_ts[n] = timestamp;
    }
    OccD d;
    if (occ_up_best8(cmin, true, lane, d) && n >= 0)
        m.node_min[n] = d;
    const bool mine = occ_up_best8(cmax, false, lane, d);
    if (mine && n >= 0)
        m.node_max[n] = d;
    const unsigned who = (__ballot_sync(0xffffffffu, mine) >> (lane & 24)) & 0xffu;
    const int src = (lane & 24) + (who ? __ffs(who) - 1 : 0);
    const float occ = __shfl_sync(0xffffffffu, d.occ, src), weight = __shfl_sync(0xffffffffu, d.weight, src);
    const int observed = __shfl_sync(0xffffffffu, d.observed, src);
    if (who)
        mx = OccD{occ, weight, observed};
    return mx;
}

// Octree::deleteChildren: detach the subtree; its blocks stop being live
__device__ void occ_delete_children(const OccDevice& m, int n)
{
    int stack[64];
    int sp = 0;
    stack[sp++] = n;
    while (sp > 0) {
        const int q = stack[--sp];
        for (int i = 0; i < 8; ++i) {
            const int c = m.node_child[8 * (size_t) q + i];
            if (c == -1)
                continue;
            if (slot_is_block(c))
                m.block_state[slot_block(c)].live = 0;
            else if (sp < 64)
                stack[sp++] = c;
            else
                atomicOr(&m.counters[kOccError], kOccErrList);
            m.node_child[8 * (size_t) q + i] = -1;
        }
    }
}

// Up to 4 nodes of a map's propagation set at one depth, first and on, by a warp: 8 lanes a node.
__device__ __forceinline__ void occ_propagate_set(const OccJob& J, int depth, int first, int total, int lane)
{
    const OccDevice& m = J.m;
    const OccDyn& D = *J.dyn;
    const int idx = first + (lane >> 3);
    int node = idx < total ? J.sets[(size_t) depth * m.node_capacity + idx] : -1;
    int parent = -1;
    if (node >= 0) {
        parent = m.node_parent[node];
        if (m.node_ts[node] == D.timestamp || parent < 0)
            node = -1;
    }
    __syncwarp(); // a node's eight lanes have read its time stamp, which occ_propagate_node sets
    const OccD nd = occ_propagate_node(m, node, D.timestamp, lane);
    if (node >= 0 && (lane & 7) == 0) {
        occ_set_insert(m, J.sets, parent, D.frame_id);
        if (nd.observed && occ_field(nd) <= kOccFreeField) {
            occ_delete_children(m, node);
            atomicAdd(&m.counters[kOccPruned], 1);
        }
    }
    __syncwarp();
}

} // namespace se_gpu
