// ray_voxel.cuh — the ray batches' update of one voxel.
#pragma once

#include "occupancy.cuh"

namespace se_gpu {

// inv: 1 / w for the integer weights w < kRiInv, correctly rounded: the quotient by such a w from it and one
// residual is the correctly rounded one (Markstein's theorem, as div_res in se_gpu_internal.cuh).
constexpr int kRiInv = 32;

// The mean of a sample's log-odds into a voxel (multires_ofusion_core_impl.hpp:46-77). The weights are integers
// until a block becomes coarser; ri_propagate_to_scale then leaves ceil(sum) / count, which stays with the
// block when it becomes finer again. Such weights divide.
__device__ __forceinline__ void ri_update_voxel(OccD& d, float sample, const OccFieldConfig& c, const float* inv)
{
    if (d.weight < c.max_weight)
        d.weight = d.weight + 1.0f;
    const float w = d.weight, x = d.occ * (w - 1.0f) + sample;
    const int wi = w < (float) kRiInv ? (int) w : 0;
    if (wi >= 1 && (float) wi == w && fabsf(x) >= 0x1p-100f && fabsf(x) < 0x1p100f) {
        const float i = inv[wi], q = x * i;
        d.occ = fmaf(fmaf(-q, w, x), i, q);
    }
    else {
        d.occ = x / w;
    }
    d.observed = 1;
}

} // namespace se_gpu
