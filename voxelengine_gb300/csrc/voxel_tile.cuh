// voxel_tile.cuh — one tile of a placed model written into the grid: the inner
// loops of ShadowVoxSystem::OnUpdate (Sources/World/Systems/
// ShadowVoxSystem.cpp:137-177) with SetVolumeAt (:82-94), shared by the
// voxelizer's two kernels.
//
// A block of kVoxThreads threads takes a tile of 1024 source voxels and collects its
// bits in shared memory, one 64-bit word per brick of the tile's image, then
// applies each non-empty word with one 64-bit atomic. A tile's voxels are
// neighbours, so about 400 of them (the usual 40% fill) land in 50 to 150
// bricks. One atomic per voxel bound the earlier form: two thousand models
// (95 M source voxels, 38 M of them set) took 1780 us, now 575 us (640 with
// one tile shape, bounds tests on every voxel and divisions for every tile's
// and brick's place).
#pragma once
#include <climits>

#include "vxl_device.cuh"

namespace vxl {

constexpr int kVoxThreads = 128;
constexpr int kVoxPer = 8;           // source voxels per thread
constexpr uint32_t kVoxBricks = 512;  // bricks of a tile's image held in shared memory

struct VoxTileShared {
    unsigned long long bits[kVoxBricks];  // all zero between tiles
    int lo[3], hi[3];                     // the tile's mapped voxels; INT_MAX / INT_MIN between tiles
};

// by all threads, before the first tile
__device__ __forceinline__ void voxel_tile_init(VoxTileShared& sh) {
    for (uint32_t i = threadIdx.x; i < kVoxBricks; i += kVoxThreads) sh.bits[i] = 0ull;
    if (threadIdx.x < 3) {
        sh.lo[threadIdx.x] = INT_MAX;
        sh.hi[threadIdx.x] = INT_MIN;
    }
    __syncthreads();
}

// A model's tiles run along x, then y, then z.
struct VoxTileAt {
    uint32_t x, y, z, nx, ny;  // tile coordinates, tiles along x and y
    VoxTileShape S;
    __device__ __forceinline__ VoxTileAt(const DevModel& M, uint32_t k) {
        S = vox_tile_shape(M.sx, M.sy, M.sz);
        nx = vox_tiles(M.sx, S.lx);
        ny = vox_tiles(M.sy, S.ly);
        z = k / (nx * ny);
        const uint32_t r = k - z * (nx * ny);
        y = r / nx;
        x = r - y * nx;
    }
    __device__ __forceinline__ void next() {
        if (++x == nx) {
            x = 0;
            if (++y == ny) {
                y = 0;
                z++;
            }
        }
    }
};

// One tile of a model, by all threads of a block. m: the placement's 16
// floats; aabb: the instance's six values or NULL.
__device__ __forceinline__ void voxel_tile(const GridView& g, unsigned long long* __restrict__ words,
                                           const float* __restrict__ m, const DevModel& M, const VoxTileAt& at, bool set,
                                           int32_t* aabb, VoxTileShared& sh) {
    const VoxTileShape S = at.S;
    const uint32_t kx = at.x, ky = at.y, kz = at.z;
    const int x0 = (int)(kx << S.lx), y0 = (int)(ky << S.ly), z0 = (int)(kz << S.lz);
    const int x1 = min(x0 + (1 << S.lx), M.sx) - 1, y1 = min(y0 + (1 << S.ly), M.sy) - 1,
              z1 = min(z0 + (1 << S.lz), M.sz) - 1;

    // The source voxels of this thread: its x and y are fixed, z advances
    const int t = (int)threadIdx.x, x = x0 + (t & ((1 << S.lx) - 1)), y = y0 + ((t >> S.lx) & ((1 << S.ly) - 1));
    const int zf = z0 + (t >> (S.lx + S.ly)), zs = kVoxThreads >> (S.lx + S.ly);
    const bool mine = x <= x1 && y <= y1;
    uint8_t pal[kVoxPer];
#pragma unroll
    for (int j = 0; j < kVoxPer; j++) {
        const int z = zf + j * zs;
        pal[j] = mine && z <= z1 ? __ldg(M.data + ((size_t)x + (size_t)M.sx * ((size_t)y + (size_t)M.sy * (size_t)z))) : 0;
    }

    // The cells the tile's image can touch, clipped to the grid. Every
    // operation of the mapping is monotone in x, y and z (rounding is), so per
    // axis the least and greatest cell are those of two corners. Lane 0-2:
    // least cell of axis 0-2, lane 3-5: greatest.
    int edge;
    bool clipped;
    {
        const int lane = t & 31, a = lane % 3;
        const bool high = lane >= 3;
        const float dx = m[a] * 0.1f, dy = m[4 + a] * 0.1f, dz = m[8 + a] * 0.1f;
        const float cx = (float)(((dx >= 0.0f) == high) ? x1 : x0), cy = (float)(((dy >= 0.0f) == high) ? y1 : y0),
                    cz = (float)(((dz >= 0.0f) == high) ? z1 : z0);
        const float w = ((m[12 + a] + dx * cx) + dy * cy) + dz * cz;
        const int c = (int)(w * 10.0f), n = a == 0 ? g.nx : (a == 1 ? g.ny : g.nz);
        edge = high ? min(c, n - 1) : max(c, 0);
        clipped = !(fabsf(w) < 1e6f) || c < 0 || c >= n;
    }
    const int lx = __shfl_sync(0xffffffffu, edge, 0), ly = __shfl_sync(0xffffffffu, edge, 1),
              lz = __shfl_sync(0xffffffffu, edge, 2);
    const int hx = __shfl_sync(0xffffffffu, edge, 3), hy = __shfl_sync(0xffffffffu, edge, 4),
              hz = __shfl_sync(0xffffffffu, edge, 5);
    const bool some = lx <= hx && ly <= hy && lz <= hz;
    const uint32_t wx = (uint32_t)((hx >> 2) - (lx >> 2) + 1), wy = (uint32_t)((hy >> 2) - (ly >> 2) + 1),
                   wz = (uint32_t)((hz >> 2) - (lz >> 2) + 1);
    // a scaled placement can spread the tile over more bricks than fit: its
    // voxels go to the grid one by one
    const bool gather = some && (uint64_t)wx * wy * wz <= kVoxBricks;
    const uint32_t wxy = wx * wy;
    // the whole image lies inside the grid (the usual tile): its voxels need no
    // bounds, and z is counted up as a float, which holds whole numbers to 2^24
    const bool inside = gather && M.sz <= 1 << 24 && !(__ballot_sync(0xffffffffu, clipped) & 63u);

    // o = M[3], dx,dy,dz = M[0..2] * 0.1f; wp = o + x*dx + y*dy + z*dz; fwp = ivec3(wp * 10) (:137-147)
    const f3 dz = mk(m[8] * 0.1f, m[9] * 0.1f, m[10] * 0.1f);
    const f3 oxy = add(add(mk(m[12], m[13], m[14]), mul(mk(m[0] * 0.1f, m[1] * 0.1f, m[2] * 0.1f), (float)x)),
                       mul(mk(m[4] * 0.1f, m[5] * 0.1f, m[6] * 0.1f), (float)y));
    int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {INT_MIN, INT_MIN, INT_MIN};
    if (inside) {
        const uint32_t i0 = (uint32_t)(lx >> 2) + (uint32_t)(ly >> 2) * wx + (uint32_t)(lz >> 2) * wxy;
        uint32_t* bits = reinterpret_cast<uint32_t*>(sh.bits) - 2u * i0;
        float zc = (float)zf;
#pragma unroll
        for (int j = 0; j < kVoxPer; j++, zc += (float)zs) {
            if (pal[j] < 16) continue;
            const f3 wp = add(oxy, mul(dz, zc));
            const int fx = (int)(wp.x * 10.0f), fy = (int)(wp.y * 10.0f), fz = (int)(wp.z * 10.0f);
            if (aabb) {
                lo[0] = min(lo[0], fx);
                lo[1] = min(lo[1], fy);
                lo[2] = min(lo[2], fz);
                hi[0] = max(hi[0], fx);
                hi[1] = max(hi[1], fy);
                hi[2] = max(hi[2], fz);
            }
            const uint32_t i = (uint32_t)(fx >> 2) + (uint32_t)(fy >> 2) * wx + (uint32_t)(fz >> 2) * wxy;
            // bits 0-4 of bit_index, bit 5 in the half's address; the shift takes its count modulo 32
            atomicOr(bits + 2u * i + (((uint32_t)fz >> 1) & 1u), 1u << (((fx & 3) | ((fy & 3) << 2) | (fz << 4)) & 31));
        }
    } else {
#pragma unroll
        for (int j = 0; j < kVoxPer; j++) {
            if (pal[j] < 16) continue;
            const f3 wp = add(oxy, mul(dz, (float)(zf + j * zs)));
            const int fx = (int)(wp.x * 10.0f), fy = (int)(wp.y * 10.0f), fz = (int)(wp.z * 10.0f);
            if (aabb) {
                lo[0] = min(lo[0], fx);
                lo[1] = min(lo[1], fy);
                lo[2] = min(lo[2], fz);
                hi[0] = max(hi[0], fx);
                hi[1] = max(hi[1], fy);
                hi[2] = max(hi[2], fz);
            }
            const uint32_t b = bit_index(fx, fy, fz);
            if (gather && fx >= lx && fx <= hx && fy >= ly && fy <= hy && fz >= lz && fz <= hz) {
                const uint32_t i = (uint32_t)((fx >> 2) - (lx >> 2)) + (uint32_t)((fy >> 2) - (ly >> 2)) * wx +
                                   (uint32_t)((fz >> 2) - (lz >> 2)) * wxy;
                atomicOr(reinterpret_cast<uint32_t*>(sh.bits) + 2u * i + (b >> 5), 1u << (b & 31u));
            } else if ((unsigned)fx < (unsigned)g.nx && (unsigned)fy < (unsigned)g.ny && (unsigned)fz < (unsigned)g.nz) {
                // SetVolumeAt bounds: 0 <= x < 2*SizeX (:83). Without a gathered
                // image, or outside it (a placement that is not finite)
                unsigned long long* w = words + word_index(g, fx, fy, fz);
                if (set)
                    atomicOr(w, 1ull << b);
                else
                    atomicAnd(w, ~(1ull << b));
            }
        }
    }
    if (aabb) {
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const int l = __reduce_min_sync(0xffffffffu, lo[a]), h = __reduce_max_sync(0xffffffffu, hi[a]);
            // l > h: no voxel. (Not l == INT_MAX, which a far cell is, too: conversions saturate.)
            if ((t & 31) == 0 && l <= h) {
                atomicMin(&sh.lo[a], l);
                atomicMax(&sh.hi[a], h);
            }
        }
    }
    __syncthreads();
    if (gather) {
        const float inv_wxy = 1.0f / (float)wxy, inv_wx = 1.0f / (float)wx;
        for (uint32_t i = threadIdx.x; i < wxy * wz; i += kVoxThreads) {
            const unsigned long long b = sh.bits[i];
            if (b == 0ull) continue;
            sh.bits[i] = 0ull;
            // i < 512, and (i + 0.5) / w lies 0.5 / w or more from every whole number: exact
            const uint32_t iz = (uint32_t)(((float)i + 0.5f) * inv_wxy), r = i - iz * wxy,
                           iy = (uint32_t)(((float)r + 0.5f) * inv_wx), ix = r - iy * wx;
            unsigned long long* w = words + ((uint32_t)(lx >> 2) + ix) + ((uint32_t)(ly >> 2) + iy) * (uint32_t)g.bx +
                                    ((uint32_t)(lz >> 2) + iz) * g.bxy;
            if (set)
                atomicOr(w, b);
            else
                atomicAnd(w, ~b);
        }
    }
    if (aabb && threadIdx.x < 3 && sh.lo[threadIdx.x] <= sh.hi[threadIdx.x]) {
        atomicMin(aabb + threadIdx.x, sh.lo[threadIdx.x]);
        atomicMax(aabb + 3 + threadIdx.x, sh.hi[threadIdx.x]);
        sh.lo[threadIdx.x] = INT_MAX;
        sh.hi[threadIdx.x] = INT_MIN;
    }
    __syncthreads();
}

}  // namespace vxl
