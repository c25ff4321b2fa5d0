// The voxelizer's host side (csrc/vxl_api.cpp) on a CUDA runtime of this file's
// own: copies wait in a queue until something synchronises, as a GPU's do.
// Without arguments the n-th call after the tables' upload fails; prints, per
// n, the status of the call and how many copies its return left waiting. With
// the name of a list and its length: orders that list, checks the order, and
// prints its levels and the fastest of three calls in ms.
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <random>
#include <string>
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
static std::vector<int> levels_;  // first job of each level launched
static const VoxJob* jobs_;
vxl_status launch_voxelize_level(vxl_grid*, const VoxJob* jobs, const uint64_t*, const DevModel*, int job0, int,
                                 uint64_t, int32_t*, cudaStream_t) {
    levels_.push_back(job0);
    jobs_ = jobs;
    return failing() ? fail(VXL_ERR_CUDA, "level") : VXL_OK;
}
}  // namespace vxl

// Cells of a model of one voxel by axis-aligned placements: bounds of the image in the reference's arithmetic.
static void cells(const float* m, const vxl_model& M, int* lo, int* hi) {
    const int last[3] = {M.sx - 1, M.sy - 1, M.sz - 1};
    for (int a = 0; a < 3; a++) {
        lo[a] = (int)(m[12 + a] * 10.0f);
        hi[a] = (int)((m[12 + a] + m[5 * a] * 0.1f * (float)last[a]) * 10.0f);
    }
}

static int order(vxl_ctx* ctx, vxl_grid* grid, const std::string& list, int n) {
    static const uint8_t voxels[64] = {};
    const vxl_model model{voxels, 4, 4, 4};
    std::mt19937 rng(n);
    std::uniform_real_distribution<float> at(0.2f, 2.6f);
    std::vector<vxl_instance> inst((size_t)n);
    for (int i = 0; i < n; i++) {
        vxl_instance& I = inst[(size_t)i];
        std::memset(&I, 0, sizeof I);
        I.matrix[0] = I.matrix[5] = I.matrix[10] = I.matrix[15] = 1.0f;
        for (int a = 0; a < 3; a++) I.matrix[12 + a] = at(rng);
        I.op = list == "one" ? (i != n / 2) : list == "halves" ? (i >= n / 2) : list == "pairs" ? i % 2 : rng() % 3 != 0;
    }
    double best = 1e9;
    for (int rep = 0; rep < 3; rep++) {
        vxl::levels_.clear();
        const auto t = std::chrono::steady_clock::now();
        if (vxl_voxelize(ctx, grid, &model, 1, inst.data(), n, nullptr, nullptr)) return 2;
        best = std::min(best, std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t).count());
    }
    // every instance once, and after the earlier ones of the other op that share cells with it
    std::vector<int> level((size_t)n, -1);
    for (size_t l = 0; l < vxl::levels_.size(); l++)
        for (int k = vxl::levels_[l]; k < (l + 1 < vxl::levels_.size() ? vxl::levels_[l + 1] : n); k++) {
            const vxl::VoxJob& J = vxl::jobs_[k];
            if (J.index < 0 || J.index >= n || level[(size_t)J.index] >= 0) return 3;
            if (J.op != inst[(size_t)J.index].op || std::memcmp(J.m, inst[(size_t)J.index].matrix, sizeof J.m)) return 4;
            level[(size_t)J.index] = (int)l;
        }
    for (int i = 0; i < n; i++)
        for (int j = i > 3000 ? i - 3000 : 0; j < i; j++) {
            if (inst[(size_t)i].op == inst[(size_t)j].op || level[(size_t)j] < level[(size_t)i]) continue;
            int a[6], b[6];
            cells(inst[(size_t)i].matrix, model, a, a + 3);
            cells(inst[(size_t)j].matrix, model, b, b + 3);
            bool meet = true;
            for (int k = 0; k < 3; k++) meet = meet && std::max(a[k], b[k]) <= std::min(a[3 + k], b[3 + k]);
            if (meet) return 5;
        }
    std::printf("%zu %.3f\n", vxl::levels_.size(), best);
    return 0;
}

int main(int argc, char** argv) {
    vxl_ctx* ctx = nullptr;
    vxl_grid* grid = nullptr;
    if (vxl_ctx_create(0, &ctx) || vxl_grid_create(ctx, 32, 32, 32, &grid)) return 1;
    if (argc > 2) return order(ctx, grid, argv[1], std::atoi(argv[2]));
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
