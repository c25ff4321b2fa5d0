// The voxelizer's host side (csrc/vxl_api.cpp) on a CUDA runtime of this file's
// own: copies wait in a queue until something synchronises, as a GPU's do, and
// the n-th call after the tables' upload fails. Prints, per n, the status of
// the call and how many copies its return left waiting.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

#include "vxl_internal.h"

static std::vector<std::function<void()>> queue_;
static int after_upload = -1, fail_at = -1;  // calls since the upload; the one that fails
static bool failing() { return after_upload >= 0 && ++after_upload == fail_at; }
static void drain() {
    for (auto& f : queue_) f();
    queue_.clear();
}
static cudaError_t plain(void** p, size_t n) {
    *p = std::calloc(1, n);
    return cudaSuccess;
}

extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return plain(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return plain(p, n); }
cudaError_t cudaFree(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { return std::memset(p, v, n), cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "made by the test"; }
const char* cudaGetErrorName(cudaError_t) { return "test"; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    return *s = cudaStreamCaptureStatusNone, cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t)1, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (failing()) return cudaErrorUnknown;
    if (after_upload < 0) after_upload = 0;
    queue_.push_back([=] { std::memcpy(d, s, n); });
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return failing() ? cudaErrorUnknown : cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) {
    if (failing()) return cudaErrorUnknown;
    return drain(), cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return drain(), cudaSuccess; }
}

namespace vxl {
void trace_layout_dims(vxl_grid* g) { g->tl_nwords = 0; }
vxl_status launch_build_tile_mask(vxl_grid*, cudaStream_t) {
    return failing() ? fail(VXL_ERR_CUDA, "tile mask") : VXL_OK;
}
vxl_status launch_voxelize_level(vxl_grid*, const VoxJob*, const uint64_t*, const DevModel*, int, int, uint64_t,
                                 int32_t*, cudaStream_t) {
    return failing() ? fail(VXL_ERR_CUDA, "level") : VXL_OK;
}
}  // namespace vxl

int main() {
    vxl_ctx* ctx = nullptr;
    vxl_grid* grid = nullptr;
    if (vxl_ctx_create(0, &ctx) || vxl_grid_create(ctx, 32, 32, 32, &grid)) return 1;
    const uint8_t voxel = 20;
    const vxl_model model{&voxel, 1, 1, 1};
    float m[16] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, 0.5f, 0.5f, 0.5f, 1};
    int32_t region[6];
    for (fail_at = 0; fail_at <= 5; fail_at++) {
        after_upload = -1;
        const vxl_status st = vxl_vox_destroyed(ctx, grid, &model, m, region, nullptr);
        std::printf("%d %d %zu\n", fail_at, (int)st, queue_.size());
    }
    return 0;
}
