// ri_update_voxel against the division that it stands for, over the weights that a block takes on: integers,
// and the ceil(sum) / count that a block has after it went to a coarser scale. Prints the number of updates
// and of wrong ones.
#include "cuda_host.hpp"

#include "../../supereight2_gb300/csrc/ray_voxel.cuh"

#include <random>

using namespace se_gpu;

int main()
{
    float inv[kRiInv];
    for (int i = 0; i < kRiInv; ++i)
        inv[i] = 1.0f / (float) i;
    std::mt19937 rng(1);
    std::uniform_real_distribution<float> log_odds(-5.015f, 5.015f);
    long n = 0, wrong = 0;
    for (const float max_weight : {20.0f, 1.0f, 7.5f, 100.0f})
        for (int count = 1; count <= 8; ++count)
            for (int sum = 0; sum <= 40 * count; ++sum)
                for (int r = 0; r < 8; ++r) {
                    OccFieldConfig c = {};
                    c.max_weight = max_weight;
                    OccD d = {log_odds(rng), (float) sum / (float) count, 0};
                    for (int k = 0; k < 8; ++k) {
                        const float sample = k & 1 ? -5.015f : log_odds(rng);
                        const float w = d.weight < max_weight ? d.weight + 1.0f : d.weight;
                        const float occ = (d.occ * (w - 1.0f) + sample) / w;
                        ri_update_voxel(d, sample, c, inv);
                        ++n;
                        wrong += d.weight != w || __float_as_uint(d.occ) != __float_as_uint(occ) || d.observed != 1;
                    }
                }
    printf("%ld %ld\n", n, wrong);
    return 0;
}
