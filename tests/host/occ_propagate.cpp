// occ_propagate_set on a small tree of 32^3 voxels, against the children's minimum and maximum taken one
// after another. Prints the nodes compared and those that differ.
#include "cuda_host.hpp"

#include "../../supereight2_gb300/csrc/occ_propagate.cuh"

#include <random>

using namespace se_gpu;

namespace {

constexpr int kNodes = 9, kBlocks = 64, kFrame = 7, kTime = 5;

struct Tree {
    std::vector<int4> coord = std::vector<int4>(kNodes);
    std::vector<int> parent = std::vector<int>(kNodes, -1), child = std::vector<int>(8 * kNodes, -1),
                     mark = std::vector<int>(kNodes, -1), ts = std::vector<int>(kNodes, -1),
                     counters = std::vector<int>(kOccCounters), sets = std::vector<int>(3 * kNodes);
    std::vector<OccD> node_min = std::vector<OccD>(kNodes), node_max = std::vector<OccD>(kNodes),
                      mean = std::vector<OccD>(kBlocks * 585), bmin = mean, bmax = mean;
    std::vector<OccBlockState> state = std::vector<OccBlockState>(kBlocks);
    OccJob job = {};
    OccDyn dyn = {};

    explicit Tree(unsigned seed)
    {
        std::mt19937 rng(seed);
        const auto data = [&] { return OccD{(float) (int) (rng() % 9) - 4.0f, (float) (rng() % 4), (int) (rng() % 2)}; };
        coord[0] = {0, 0, 0, 32};
        for (int n = 1; n < kNodes; ++n) {
            coord[n] = {16 * ((n - 1) & 1), 16 * (((n - 1) >> 1) & 1), 16 * ((n - 1) >> 2), 16};
            parent[n] = 0;
            child[n - 1] = n;
            node_min[n] = data();
            node_max[n] = data();
            sets[kNodes + n - 1] = n;
            for (int i = 0; i < 8; ++i) {
                const int b = 8 * (n - 1) + i;
                state[b].finest = rng() % 4;
                state[b].live = 1;
                for (int s = 0; s <= kOccMaxScale; ++s)
                    mean[b * 585 + occ_scale_offset(s)] = data();
                bmin[b * 585 + 584] = data();
                bmax[b * 585 + 584] = data();
                if (n == 4 || rng() % 8) // (node 4 is free space: its children go)
                    child[8 * n + i] = -2 - b;
                if (n == 4)
                    bmax[b * 585 + 584] = mean[b * 585 + 584] = {-50.0f, 3.0f, 1};
            }
        }
        ts[3] = kTime; // done before
        counters[kOccSetN + 1] = kNodes - 1;
        OccDevice& m = job.m;
        m.size = 32;
        m.log2_size = 5;
        m.node_capacity = kNodes;
        m.node_coord = coord.data();
        m.node_parent = parent.data();
        m.node_child = child.data();
        m.node_min = node_min.data();
        m.node_max = node_max.data();
        m.node_mark = mark.data();
        m.node_ts = ts.data();
        m.block_state = state.data();
        m.block_mean = mean.data();
        m.block_min = bmin.data();
        m.block_max = bmax.data();
        m.counters = counters.data();
        job.sets = sets.data();
        dyn.frame_id = kFrame;
        dyn.timestamp = kTime;
        job.dyn = &dyn;
    }
};

void best_of(const OccD* c, bool want_min, OccD& d)
{
    float best = want_min ? FLT_MAX : -FLT_MAX;
    int at = 0, valid = 0, observed = 0;
    for (int i = 0; i < 8; ++i)
        if (occ_valid(c[i])) {
            ++valid;
            observed += c[i].observed;
            if (want_min ? occ_field(c[i]) < best : occ_field(c[i]) > best) {
                best = occ_field(c[i]);
                at = i;
            }
        }
    if (valid) {
        d = c[at];
        d.observed = observed == 8;
    }
}

// One node after another, one child after another.
void serial(Tree& t)
{
    const OccDevice& m = t.job.m;
    for (int n = 1; n < kNodes; ++n) {
        if (t.ts[n] == kTime)
            continue;
        t.ts[n] = kTime;
        OccD lo[8], hi[8];
        for (int i = 0; i < 8; ++i) {
            lo[i] = hi[i] = occ_default();
            const int c = t.child[8 * n + i];
            if (c != -1) {
                lo[i] = blk_min(m, slot_block(c), t.state[slot_block(c)].finest, kOccMaxScale)[0];
                hi[i] = blk_max(m, slot_block(c), t.state[slot_block(c)].finest, kOccMaxScale)[0];
            }
        }
        best_of(lo, true, t.node_min[n]);
        best_of(hi, false, t.node_max[n]);
        t.mark[0] = kFrame;
        t.counters[kOccSetN] = 1;
        t.sets[0] = 0;
        if (t.node_max[n].observed && occ_field(t.node_max[n]) <= kOccFreeField) {
            t.counters[kOccPruned]++;
            for (int i = 0; i < 8; ++i) {
                if (t.child[8 * n + i] != -1)
                    t.state[slot_block(t.child[8 * n + i])].live = 0;
                t.child[8 * n + i] = -1;
            }
        }
    }
}

bool same(const OccD& a, const OccD& b) { return a.occ == b.occ && a.weight == b.weight && a.observed == b.observed; }

} // namespace

int main()
{
    int n = 0, differ = 0, pruned = 0;
    for (unsigned seed = 0; seed < 20; ++seed) {
        Tree warp(seed), ref(seed);
        for (int first = 0; first < kNodes - 1; first += 4)
            HostWarp::run(seed & 1, [&](int lane) { occ_propagate_set(warp.job, 1, first, kNodes - 1, lane); });
        serial(ref);
        for (int k = 1; k < kNodes; ++k, ++n)
            differ += !same(warp.node_min[k], ref.node_min[k]) || !same(warp.node_max[k], ref.node_max[k]);
        differ += warp.child != ref.child || warp.ts != ref.ts || warp.mark != ref.mark || warp.sets != ref.sets
            || warp.counters != ref.counters;
        for (int b = 0; b < kBlocks; ++b)
            differ += warp.state[b].live != ref.state[b].live;
        pruned += ref.counters[kOccPruned];
    }
    printf("%d %d %d\n", n, pruned, differ);
    return 0;
}
