// voxelize.cu — GPU ShadowVox voxelizer (ShadowVoxSystem::OnUpdate inner
// loops, Sources/World/Systems/ShadowVoxSystem.cpp:137-177, SetVolumeAt :82-94).
//
// One launch applies a level of instances whose writes commute: instances of
// one op store the same bit value, and instances of different ops in one level
// touch different cells (the host orders the others into later levels). Bits
// are combined with atomicOr / atomicAnd on the 64-bit brick words.
#include <algorithm>

#include "voxel_tile.cuh"

namespace vxl {

// Every block takes an equal run of the level's tiles: one search for the job
// of its first tile, then it walks on.
__global__ void __launch_bounds__(kVoxThreads, 12) k_voxelize(GridView g, unsigned long long* words,
                                                          const VoxJob* __restrict__ jobs,
                                                          const uint64_t* __restrict__ first,
                                                          const DevModel* __restrict__ models, int job0, int job1,
                                                          int32_t* aabb) {
    __shared__ VoxTileShared sh;
    const uint64_t base = first[job0], n = first[job1] - base;
    uint64_t k = base + n * blockIdx.x / gridDim.x;
    const uint64_t end = base + n * (blockIdx.x + 1ull) / gridDim.x;
    if (k >= end) return;
    int lo = job0, hi = job1 - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (first[mid] <= k)
            lo = mid;
        else
            hi = mid - 1;
    }
    voxel_tile_init(sh);
    while (k < end) {
        while (first[lo + 1] <= k) lo++;
        const VoxJob& J = jobs[lo];
        const DevModel M = models[J.model];
        const uint64_t stop = first[lo + 1] < end ? first[lo + 1] : end;
        VoxTileAt at(M, (uint32_t)(k - first[lo]));
        for (; k < stop; k++, at.next())
            voxel_tile(g, words, J.m, M, at, J.op != 0, aabb ? aabb + 6 * (size_t)J.index : nullptr, sh);
    }
}

vxl_status launch_voxelize_level(vxl_grid* g, const VoxJob* d_jobs, const uint64_t* d_first, const DevModel* d_models,
                                 int job0, int job1, uint64_t ntiles, int32_t* d_aabb, cudaStream_t s) {
    if (ntiles == 0) return VXL_OK;
    // 12 blocks of 4 warps are what an SM's registers hold (40 a thread: 48 of
    // its 64 warps); runs of several tiles per block spare the searches
    const unsigned blocks = (unsigned)std::min<uint64_t>(ntiles, (uint64_t)g->ctx->sm_count * 12);
    k_voxelize<<<blocks, kVoxThreads, 0, s>>>(view_of(g), (unsigned long long*)g->words, d_jobs, d_first, d_models, job0,
                                              job1, d_aabb);
    g->ctx->launches++;
    VXL_TRY_CUDA(cudaGetLastError());
    return VXL_OK;
}

}  // namespace vxl
