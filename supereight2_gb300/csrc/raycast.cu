// raycast.cu — se::raycaster::raycast_volume for single-res TSDF maps, and the batched
// Map::getFieldInterp / Map::getFieldGrad queries.
//
// One thread per pixel (an 8 x 4 pixel tile per warp for coherent block lookups):
//   1. first allocated block on the ray (VoxelBlockRayIterator,
//      voxel_block_ray_iterator_impl.hpp:19-249): a level DDA over the occupancy pyramid from
//      cells of 4^3 blocks down to blocks, with the reference traversal's plane parameters and
//      child choices (first_block in raycast_core.cuh);
//   2. the TSDF march of raycast<TSDF> (raycaster_impl.hpp:456-533): voxel fetches through the
//      dense block index with a one-block cache, trilinear interpolation near the surface
//      (visitor_impl.hpp:976-1024) and the linear zero-crossing estimate;
//   3. the surface normal from the 32-sample central-difference gradient
//      (visitor_impl.hpp:1094-1251, map_impl.hpp:236-262), its 32 loads issued together.
// The gradient's block table lives in shared memory; the register cap of 9 CTAs per SM (a few
// spilled words) is faster than the 5 CTAs that 92 registers allow.
// Sample loops are deliberately not unrolled: one copy of the fetch path keeps the kernel
// inside the instruction cache.
#include <cmath>

#include "pipeline.cuh"
#include "profile.cuh"
#include "raycast_core.cuh"

namespace se_gpu {

__global__ void raycast_prep_kernel(const float* pose12, RaycastParams host_p, MapDevice m, RaycastParams* out)
{
    grid_dep_wait();
    RaycastParams p = host_p;
    if (pose12 != nullptr)
        p.T_WS = tf_from12(pose12);
    set_raycast_origin(m, p);
    *out = p;
}

// The pixel of a thread, TILE 0: each warp takes 8 x 4 pixels (a CTA 16 x 8); TILE 1: 16 x 2 (a CTA 32 x 4).
template <int TILE>
__device__ __forceinline__ bool raycast_pixel(const Pinhole& s, int& x, int& y)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int kWx = TILE == 0 ? 8 : 16, kWy = 32 / kWx; // warp tile
    x = blockIdx.x * (2 * kWx) + (warp & 1) * kWx + (lane % kWx);
    y = blockIdx.y * (2 * kWy) + (warp >> 1) * kWy + (lane / kWx);
    return x < s.w && y < s.h;
}

// Single-res maps: the whole raycast. Multi-res maps: the points and scales, and in the normals' x whether
// the pixel has a hit (1 or 0, the other components 0) for raycast_normal_kernel.
//
// The multi-res gradient is a kernel of its own because the code of both together does not stay in the
// SM's instruction caches (9.3 stall cycles per issue went to instruction fetch, against 1.3 for the
// single-res kernel): a 1280x960 pass of integration and raycast 501 us as one kernel, 441 as two. The
// single-res kernel loses by the split (640x480, FP16: 149 against 151 us; 320x240: 68 against 70).
template <int S, bool MR, int TILE>
__global__ void __launch_bounds__(128, MR ? 10 : 9) raycast_kernel(MapDevice m, Pinhole s, const RaycastParams* __restrict__ P,
                                                                float* __restrict__ pts, float* __restrict__ nrm,
                                                                int8_t* __restrict__ scale)
{
    grid_dep_wait();
    // per-thread scratch in shared memory (column threadIdx.x): the gradient's block table
    __shared__ int sh_bt[MR ? 1 : 8 * 128];
    int x, y;
    if (!raycast_pixel<TILE>(s, x, y))
        return;
    const RaycastParams rp = *P;
    const size_t idx = (size_t) x + (size_t) y * s.w;
    const F3 ray_S = back_project(s, (float) x, (float) y);
    const F3 nS = normalized(ray_S);
    const F3 dir_W = rot(rp.T_WS, nS);
    const F3 origin = f3(rp.T_WS.t[0], rp.T_WS.t[1], rp.T_WS.t[2]);
    const float t_near = s.near_plane / nS.z;
    const float t_far = s.far_plane / nS.z;
    RayCache<MR> c;
    F3 hit;
    F3 n = f3(0.0f, 0.0f, 0.0f);
    F3 p = f3(0.0f, 0.0f, 0.0f);
    int hit_scale = 0;
    if (raycast_tsdf<S, MR>(m, rp, c, origin, dir_W, t_near, t_far, hit, hit_scale)) {
        p = hit;
        if constexpr (MR) {
            n.x = 1.0f;
        }
        else {
            F3 g;
            if (field_grad_batched<S>(m, c.c, hit, g, sh_bt + threadIdx.x, 128))
                n = normalized(g);
        }
    }
    pts[3 * idx + 0] = p.x;
    pts[3 * idx + 1] = p.y;
    pts[3 * idx + 2] = p.z;
    nrm[3 * idx + 0] = n.x;
    nrm[3 * idx + 1] = n.y;
    nrm[3 * idx + 2] = n.z;
    if (scale)
        scale[idx] = (int8_t) hit_scale;
}

// The normals at a multi-res raycast's hits.
template <int S>
__global__ void __launch_bounds__(128, 6) raycast_normal_kernel(MapDevice m, Pinhole s, const float* __restrict__ pts,
                                                             float* __restrict__ nrm)
{
    grid_dep_wait();
    __shared__ int sh_bt[8 * 128]; // the gradients' block tables, column threadIdx.x
    int x, y;
    if (!raycast_pixel<0>(s, x, y))
        return;
    const size_t idx = (size_t) x + (size_t) y * s.w;
    if (nrm[3 * idx] == 0.0f)
        return;
    const F3 hit = f3(pts[3 * idx], pts[3 * idx + 1], pts[3 * idx + 2]);
    MrCache c{-1, -1, -1, -1, -1};
    F3 g, n = f3(0.0f, 0.0f, 0.0f);
    if (mr_field_grad<S>(m, c, hit, g, sh_bt + threadIdx.x, 128))
        n = normalized(g);
    nrm[3 * idx + 0] = n.x;
    nrm[3 * idx + 1] = n.y;
    nrm[3 * idx + 2] = n.z;
}

// The batched field queries, a thread per point. A gradient's 32 samples are in flight together, as in
// the raycast.
template <int S, bool MR, bool GRAD>
__global__ void __launch_bounds__(128) field_query_kernel(MapDevice m, int n, const float* __restrict__ pts,
                                                          float* __restrict__ out, int* __restrict__ valid,
                                                          uint8_t* __restrict__ valid8)
{
    __shared__ int sh_bt[GRAD ? 8 * 128 : 1];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const F3 p = f3(pts[3 * (size_t) i], pts[3 * (size_t) i + 1], pts[3 * (size_t) i + 2]);
    RayCache<MR> c;
    bool ok;
    if constexpr (GRAD) {
        F3 g = f3(0.0f, 0.0f, 0.0f);
        if constexpr (MR)
            ok = mr_field_grad<S>(m, c.c, p, g, sh_bt + threadIdx.x, 128);
        else
            ok = field_grad_batched<S>(m, c.c, p, g, sh_bt + threadIdx.x, 128);
        out[3 * (size_t) i] = ok ? g.x : 0.0f;
        out[3 * (size_t) i + 1] = ok ? g.y : 0.0f;
        out[3 * (size_t) i + 2] = ok ? g.z : 0.0f;
    }
    else {
        float v = 0.0f;
        if constexpr (MR)
            ok = mr_field_interp<S>(m, p, v, nullptr);
        else
            ok = field_interp<S>(m, p, v);
        out[i] = ok ? v : 0.0f;
    }
    if (valid8)
        valid8[i] = ok ? 1 : 0;
    if (valid)
        valid[i] = ok ? 1 : 0;
}

} // namespace se_gpu

using namespace se_gpu;

namespace se_gpu {

se_gpu_status enqueue_raycast(const se_gpu_map* map, const se_gpu_pinhole& sensor, const float* T_WS_host16,
                              const float* pose12_dev, float* pts_dev, float* nrm_dev, int8_t* scale_dev,
                              cudaStream_t stream)
{
    const MapDevice& m = map->dev;
    const Pinhole s = make_pinhole(sensor);
    RaycastParams rp;
    for (int i = 0; i < 9; ++i)
        rp.T_WS.R[i] = (i % 4 == 0) ? 1.0f : 0.0f;
    rp.T_WS.t[0] = rp.T_WS.t[1] = rp.T_WS.t[2] = 0.0f;
    if (T_WS_host16)
        rp.T_WS = tf_from16(T_WS_host16);
    rp.scaling = (float) m.size * m.res;
    rp.eps = std::exp2((float) (-std::log2((double) m.size)));
    rp.min_scale = 23 - m.log2_bps;
    // (a launch of its own also keeps the raycast's CTAs off the SMs until the update is done: scheduled
    // in its tail they pile up on the SMs that are free first, 320x240 67 -> 77 us)
    launch_chained(raycast_prep_kernel, 1, 1, stream, T_WS_host16 ? nullptr : pose12_dev, rp, m, map->rparams);
    const int tile = map->tiles.raycast_tile;
    const dim3 grid = tile == 0 ? dim3((s.w + 15) / 16, (s.h + 7) / 8) : dim3((s.w + 31) / 32, (s.h + 3) / 4);
    ProfScope ps(kProfRaycast, stream);
    const bool mr = m.res_type == SE_GPU_RES_MULTI;
    if (map->tune)
        SE_CUDA_TRY(cudaEventRecord(map->tune->ev[2], stream));
#define SE_RAYCAST_LAUNCH(S_, MR_)                                                                                  \
    do {                                                                                                            \
        if (tile == 0)                                                                                              \
            launch_chained(raycast_kernel<S_, MR_, 0>, grid, 128, stream, m, s, map->rparams, pts_dev, nrm_dev,     \
                           scale_dev);                                                                              \
        else                                                                                                        \
            launch_chained(raycast_kernel<S_, MR_, 1>, grid, 128, stream, m, s, map->rparams, pts_dev, nrm_dev,     \
                           scale_dev);                                                                              \
        if (MR_)                                                                                                    \
            launch_chained(raycast_normal_kernel<S_>, dim3((s.w + 15) / 16, (s.h + 7) / 8), 128, stream, m, s,      \
                           pts_dev, nrm_dev);                                                                       \
    } while (0)
    if (m.storage == SE_GPU_STORAGE_F32 && !mr)
        SE_RAYCAST_LAUNCH(SE_GPU_STORAGE_F32, false);
    else if (!mr)
        SE_RAYCAST_LAUNCH(SE_GPU_STORAGE_F16, false);
    else if (m.storage == SE_GPU_STORAGE_F32)
        SE_RAYCAST_LAUNCH(SE_GPU_STORAGE_F32, true);
    else
        SE_RAYCAST_LAUNCH(SE_GPU_STORAGE_F16, true);
#undef SE_RAYCAST_LAUNCH
    if (map->tune)
        SE_CUDA_TRY(cudaEventRecord(map->tune->ev[3], stream));
    SE_CUDA_TRY(cudaGetLastError());
    return SE_GPU_OK;
}

} // namespace se_gpu

extern "C" se_gpu_status se_gpu_raycast(const se_gpu_map* map, const se_gpu_pinhole* sensor, const float T_WS[16],
                                        float* pts_dev, float* nrm_dev, int8_t* scale_dev, void* stream_p)
{
    if (!map || !sensor || !T_WS || !pts_dev || !nrm_dev || sensor->width <= 0 || sensor->height <= 0) {
        set_last_error("se_gpu_raycast: invalid argument");
        return SE_GPU_ERR_BAD_ARG;
    }
    cudaStream_t stream = (cudaStream_t) stream_p;
    const_cast<se_gpu_map*>(map)->last_stream = stream;
    if (map->occ)
        return occ_raycast_volume(map->occ, *sensor, T_WS, pts_dev, nrm_dev, scale_dev, stream);
    return enqueue_raycast(map, *sensor, T_WS, nullptr, pts_dev, nrm_dev, scale_dev, stream);
}

static se_gpu_status field_query(const se_gpu_map* map, int64_t n, const float* pts, float* out, int* valid,
                                 uint8_t* valid8, void* stream_p, int grad)
{
    if (!map || n < 0 || n > (1ll << 31) - 1 || (n > 0 && (!pts || !out))) {
        set_last_error("se_gpu_map_field_%s: invalid argument", grad ? "grad" : "interp");
        return SE_GPU_ERR_BAD_ARG;
    }
    if (map->occ) {
        set_last_error("se_gpu_map_field_%s: TSDF maps only", grad ? "grad" : "interp");
        return SE_GPU_ERR_NOT_SUPPORTED;
    }
    if (n == 0)
        return SE_GPU_OK;
    cudaStream_t stream = (cudaStream_t) stream_p;
    const unsigned blocks = (unsigned) ((n + 127) / 128);
    const bool mr = map->dev.res_type == SE_GPU_RES_MULTI;
#define SE_QUERY_LAUNCH(S_, MR_)                                                                                     \
    do {                                                                                                            \
        if (grad)                                                                                                   \
            field_query_kernel<S_, MR_, true><<<blocks, 128, 0, stream>>>(map->dev, (int) n, pts, out, valid, valid8); \
        else                                                                                                        \
            field_query_kernel<S_, MR_, false><<<blocks, 128, 0, stream>>>(map->dev, (int) n, pts, out, valid, valid8); \
    } while (0)
    if (map->dev.storage == SE_GPU_STORAGE_F32 && !mr)
        SE_QUERY_LAUNCH(SE_GPU_STORAGE_F32, false);
    else if (!mr)
        SE_QUERY_LAUNCH(SE_GPU_STORAGE_F16, false);
    else if (map->dev.storage == SE_GPU_STORAGE_F32)
        SE_QUERY_LAUNCH(SE_GPU_STORAGE_F32, true);
    else
        SE_QUERY_LAUNCH(SE_GPU_STORAGE_F16, true);
#undef SE_QUERY_LAUNCH
    SE_CUDA_TRY(cudaGetLastError());
    return SE_GPU_OK;
}

extern "C" se_gpu_status se_gpu_map_field_interp(const se_gpu_map* map, int64_t n, const float* pts, float* values,
                                                 int* valid, void* stream)
{
    return field_query(map, n, pts, values, valid, nullptr, stream, 0);
}

extern "C" se_gpu_status se_gpu_map_field_grad(const se_gpu_map* map, int64_t n, const float* pts, float* grads,
                                               int* valid, void* stream)
{
    return field_query(map, n, pts, grads, valid, nullptr, stream, 1);
}

extern "C" se_gpu_status se_gpu_map_field_query(const se_gpu_map* map, int64_t n, const float* pts, int grad, float* out,
                                                uint8_t* valid, void* stream)
{
    return field_query(map, n, pts, out, nullptr, valid, stream, grad != 0);
}
