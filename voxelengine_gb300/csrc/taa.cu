// taa.cu — temporal accumulation of the lighting buffer (the pass after the
// occlusion path): Sources/Shaders/LightTAA.frag:37-141, one thread per
// pixel, operation for operation. texture() is this library's sampler for the
// pass (bilinear, clamp to edge, texel centres at (i + 0.5) / size; the
// engine's light images use its default linear filter) and sin/cos are the
// library's own (sincos_own), as in the oracle.
//
// Every spiral tap samples six images at the same coordinates, 16 floats of
// four texels each. The L1 data pipe bounds the pass (a warp's taps land on
// unrelated texels, so a 16-byte load costs about seven wavefronts), and what
// helps is loading less, with the same floats combined in the same order:
//  - a streaming pre-pass (k_taa_pack) packs (light rgb, depth), (colour,
//    flags) and the normal as float4 planes, and notes per texel whether the
//    four texels of a tap there have one colour, one normal and material: such
//    a tap loads one texel's and interpolates that value with itself;
//  - a tap whose colour differs from the pixel's has factor 0 (:119), so its
//    normal and material are not loaded, unless a value near it is not finite
//    (flagged too: 0 times that is not 0);
//  - the motion test (> 0.1 apart, :120) needs no loads where the pre-pass's
//    per-tile maxima show that no tap in reach can fail it.
// 1080p: 1171 + 37 us (every tap 16 16-byte loads) -> 456 + 126 + 41 us, 68%
// issue-bound, the rest load latency.
// Planes rather than records: the 16-byte loads of scattered taps then spread
// over eight L1 bank groups (texel mod 8).
#include <climits>

#include "vxl_device.cuh"
#include "vxl_internal.h"

namespace vxl {
namespace {

struct TaaIn {
    const float* light;     // 4 channels
    const float* last;      // 4
    const float* color;     // 3
    const float* normal;    // 3
    const float* material;  // 4
    const float* depth;     // 1
    const float* motion;    // 2
    const float* noise;     // 4
    int W, H;
};

// The pass's launches follow one another with their starts overlapped (taa_launch):
// this waits for the one before to end and its writes to be seen. The pointers
// to what the pass itself has written are given anew after the wait: loads
// through the read-only path, which the compiler may take for constants of the
// launch, cannot be moved before it then.
template <class... P>
__device__ __forceinline__ void after_previous(P&... p) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    auto anew = [](auto& q) { asm volatile("" : "+l"(q)::"memory"); };
    (anew(p), ...);
}

__device__ __forceinline__ float gmax(float x, float y) { return (x < y) ? y : x; }
__device__ __forceinline__ float gmin(float x, float y) { return (y < x) ? y : x; }
__device__ __forceinline__ float clampg(float x, float lo, float hi) { return gmin(gmax(x, lo), hi); }

// texture() of a 4-channel image with the pass's sampler (16-byte texels: one
// vector load each)
__device__ __forceinline__ void tex4(const float* __restrict__ p, int W, int H, float u, float v, float* out) {
    const float x = u * (float)W - 0.5f, y = v * (float)H - 0.5f;
    const float fx = floorf(x), fy = floorf(y);
    const float ax = x - fx, ay = y - fy;
    int x0 = (int)fx, y0 = (int)fy, x1 = x0 + 1, y1 = y0 + 1;
    x0 = x0 < 0 ? 0 : (x0 > W - 1 ? W - 1 : x0);
    x1 = x1 < 0 ? 0 : (x1 > W - 1 ? W - 1 : x1);
    y0 = y0 < 0 ? 0 : (y0 > H - 1 ? H - 1 : y0);
    y1 = y1 < 0 ? 0 : (y1 > H - 1 ? H - 1 : y1);
    const float bx = 1.0f - ax, by = 1.0f - ay;
    const float4* q = reinterpret_cast<const float4*>(p);
    const float4 a = __ldg(q + ((size_t)y0 * W + x0)), b = __ldg(q + ((size_t)y0 * W + x1));
    const float4 c = __ldg(q + ((size_t)y1 * W + x0)), d = __ldg(q + ((size_t)y1 * W + x1));
    const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
    const float cv[4] = {c.x, c.y, c.z, c.w}, dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float top = av[k] * bx + bv[k] * ax;
        const float bot = cv[k] * bx + dv[k] * ax;
        out[k] = top * by + bot * ay;
    }
}
__device__ __forceinline__ float len2(float x, float y) { return sqrtf(x * x + y * y); }
__device__ __forceinline__ float len3(const float* a, const float* b) {
    const float dx = a[0] - b[0], dy = a[1] - b[1], dz = a[2] - b[2];
    float d = dx * dx + dy * dy;
    d = d + dz * dz;
    return sqrtf(d);
}
__device__ __forceinline__ float len4(const float* a, const float* b) {
    const float d0 = a[0] - b[0], d1 = a[1] - b[1], d2 = a[2] - b[2], d3 = a[3] - b[3];
    float d = d0 * d0 + d1 * d1;
    d = d + d2 * d2;
    d = d + d3 * d3;
    return sqrtf(d);
}
__device__ __forceinline__ float dot3(const float* a, const float* b) {
    float d = a[0] * b[0] + a[1] * b[1];
    return d + a[2] * b[2];
}

// Texel planes (n texels each): (light rgb, depth), (colour, flags), (normal, -).
// The flags of texel (x, y) tell of the texels (x..x+1, y..y+1) inside the image.
constexpr int kTaaPlanes = 3;
constexpr int kTaaColor = 1;    // one colour, bit for bit
constexpr int kTaaSurface = 2;  // one normal and one material
constexpr int kTaaWild = 4;     // a value that is not below 1e15 in magnitude
// bits 3-5, with kTaaSurface: the normal where it is a coordinate axis (2 * axis, + 1 for the negative one; 7: another)
constexpr int kTaaNormal = 3, kTaaOther = 7;
// bits 6-29, with kTaaSurface: the material in 1/63 steps, 6 bits a channel 
constexpr int kTaaMaterial = 6, kTaaOdd = 1 << 30;  // kTaaOdd: no such material (not uniform, or outside [0, 1])
constexpr int kPackW = 32, kPackH = 8;  // texels per block of the pre-pass

__device__ __forceinline__ bool tame(float x) { return fabsf(x) < 1e15f; }

// One texel a thread, with the row and column beyond the block's for the
// flags. rec, per block the greatest |motion| component (a NaN counts as
// infinite), and an empty list of disoccluded pixels. HBM-bound: 68 bytes read and 48 written per texel.
__global__ void __launch_bounds__(kPackW* kPackH) k_taa_pack(const TaaIn I, float4* __restrict__ rec,
                                                            float* __restrict__ motion_max, int* __restrict__ list) {
    constexpr int SW = kPackW + 1, SH = kPackH + 1;
    __shared__ float s_val[10][SW * SH];  // colour, normal, material
    __shared__ bool s_wild[SW * SH];
    __shared__ float s_max[kPackW * kPackH / 32];
    const int t0 = threadIdx.x, x0 = blockIdx.x * kPackW, y0 = blockIdx.y * kPackH;
    const size_t n = (size_t)I.W * I.H;
    float top = 0.0f;
#pragma unroll
    for (int t = t0; t < SW * SH; t += kPackW * kPackH) {
        // texels of the block first, so that thread t0 holds texel t0 of the block
        const bool own = t < kPackW * kPackH;
        const int e = t - kPackW * kPackH;
        const int lx = own ? t % kPackW : (e < SH ? kPackW : e - SH), ly = own ? t / kPackW : (e < SH ? e : kPackH);
        const int x = min(x0 + lx, I.W - 1), y = min(y0 + ly, I.H - 1);
        const size_t i = (size_t)y * I.W + x;
        const float4 m = __ldg(reinterpret_cast<const float4*>(I.material) + i);
        const float4 l = __ldg(reinterpret_cast<const float4*>(I.light) + i);
        const float v[10] = {__ldg(I.color + 3 * i),      __ldg(I.color + 3 * i + 1),  __ldg(I.color + 3 * i + 2),
                             __ldg(I.normal + 3 * i),     __ldg(I.normal + 3 * i + 1), __ldg(I.normal + 3 * i + 2),
                             m.x, m.y, m.z, m.w};
        const float de = __ldg(I.depth + i);
        bool ok = tame(l.x) && tame(l.y) && tame(l.z) && tame(de);
#pragma unroll
        for (int k = 0; k < 10; k++) {
            ok = ok && tame(v[k]);
            s_val[k][ly * SW + lx] = v[k];
        }
        s_wild[ly * SW + lx] = !ok;
        if (own && x0 + lx < I.W && y0 + ly < I.H) {
            rec[i] = make_float4(l.x, l.y, l.z, de);
            rec[2 * n + i] = make_float4(v[3], v[4], v[5], 0.0f);
            const float2 mo = __ldg(reinterpret_cast<const float2*>(I.motion) + i);
            const float a = fabsf(mo.x), b = fabsf(mo.y);
            top = a == a && b == b ? fmaxf(a, b) : INFINITY;
        }
    }
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    if ((t0 & 31) == 0) s_max[t0 >> 5] = top;
    __syncthreads();
    const int lx = t0 % kPackW, ly = t0 / kPackW, c = ly * SW + lx;
    if (x0 + lx < I.W && y0 + ly < I.H) {
        const int q[3] = {c + 1, c + SW, c + SW + 1};
        bool color = true, surface = true, wild = s_wild[c];
#pragma unroll
        for (int j = 0; j < 3; j++) {
#pragma unroll
            for (int k = 0; k < 10; k++) {
                const bool same = __float_as_uint(s_val[k][c]) == __float_as_uint(s_val[k][q[j]]);
                if (k < 3) color = color && same;
                else surface = surface && same;
            }
            wild = wild || s_wild[q[j]];
        }
        int axis = kTaaOther, bins = 0;
        bool small = true;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float m = s_val[6 + k][c];
            small = small && m >= 0.0f && m <= 1.0f;
            bins |= (int)(m * 63.0f) << (6 * k);
        }
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const uint32_t v = __float_as_uint(s_val[3 + k][c]) & 0x7fffffffu;
            const uint32_t rest = __float_as_uint(s_val[3 + (k + 1) % 3][c]) | __float_as_uint(s_val[3 + (k + 2) % 3][c]);
            if (v == 0x3f800000u && rest == 0u) axis = 2 * k + (s_val[3 + k][c] < 0.0f ? 1 : 0);
        }
        const int f = (wild ? kTaaWild : 0) | (color ? kTaaColor : 0) |
                      (surface ? kTaaSurface | (axis << kTaaNormal) | (small ? bins << kTaaMaterial : kTaaOdd) : kTaaOdd);
        rec[n + (size_t)(y0 + ly) * I.W + x0 + lx] = make_float4(s_val[0][c], s_val[1][c], s_val[2][c], __int_as_float(f));
    }
    if (t0 == 0) {
        if (blockIdx.x == 0 && blockIdx.y == 0) list[0] = list[1] = 0;
        for (int w = 1; w < kPackW * kPackH / 32; w++) top = fmaxf(top, s_max[w]);
        motion_max[blockIdx.y * gridDim.x + blockIdx.x] = top;
    }
}

__device__ __forceinline__ void lerp4(const float4& a, const float4& b, const float4& c, const float4& d, float ax,
                                      float bx, float ay, float by, float* o) {
    const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
    const float cv[4] = {c.x, c.y, c.z, c.w}, dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float top = av[k] * bx + bv[k] * ax;
        const float bot = cv[k] * bx + dv[k] * ax;
        o[k] = top * by + bot * ay;
    }
}

// A tap's place: the coordinates, clamping and weights of tex4.
struct TapAt {
    int i00, dx, dy;  // texel (x0, y0), offsets to x1 and y1
    float ax, ay, bx, by;
    __device__ __forceinline__ TapAt(int W, int H, float u, float v) {
        const float x = u * (float)W - 0.5f, y = v * (float)H - 0.5f;
        const float fx = floorf(x), fy = floorf(y);
        ax = x - fx;
        ay = y - fy;
        int x0 = (int)fx, y0 = (int)fy, x1 = x0 + 1, y1 = y0 + 1;
        x0 = x0 < 0 ? 0 : (x0 > W - 1 ? W - 1 : x0);
        x1 = x1 < 0 ? 0 : (x1 > W - 1 ? W - 1 : x1);
        y0 = y0 < 0 ? 0 : (y0 > H - 1 ? H - 1 : y0);
        y1 = y1 < 0 ? 0 : (y1 > H - 1 ? H - 1 : y1);
        bx = 1.0f - ax;
        by = 1.0f - ay;
        i00 = y0 * W + x0;
        dx = x1 - x0;
        dy = (y1 - y0) * W;
    }
    // a float4 image here; a: its texel (x0, y0), which all four equal where `one`
    __device__ __forceinline__ void get(const float4* __restrict__ img, float4 a, bool one, float* o) const {
        float4 b = a, c = a, d = a;
        if (!one) {
            const float4* q = img + i00;
            b = __ldg(q + dx);
            c = __ldg(q + dy);
            d = __ldg(q + dx + dy);
        }
        lerp4(a, b, c, d, ax, bx, ay, by, o);
    }
    __device__ __forceinline__ void motion(const float* __restrict__ img, float* o) const {
        const float2* q = reinterpret_cast<const float2*>(img) + i00;
        const float2 a = __ldg(q), b = __ldg(q + dx), c = __ldg(q + dy), d = __ldg(q + dx + dy);
        const float tx = a.x * bx + b.x * ax, ux = c.x * bx + d.x * ax;
        const float ty = a.y * bx + b.y * ax, uy = c.y * bx + d.y * ax;
        o[0] = tx * by + ux * ay;
        o[1] = ty * by + uy * ay;
    }
};

// Centre values a disocclusion tap compares against.
struct Centre {
    float uvx, uvy, no[3], ma[4], de, co[3], mo[2];
};

// dot3 of the centre's normal with a tap's, and whether the materials are
// alike (LightTAA.frag's step(0.8, 1 - distance)), with no loads where the
// flags decide. f: the tap's flags, here: the centre's.
__device__ __forceinline__ float taa_like(const float4* __restrict__ mat, const TapAt& t, const Centre& c, int f, int here) {
    // materials of one bin per channel lie within 0.04 of one another
    if (((f | here) & kTaaWild) == 0 && ((f ^ here) >> kTaaMaterial) == 0 && !(f & kTaaOdd)) return 1.0f;
    float ma[4];
    t.get(mat, __ldg(mat + t.i00), f & kTaaSurface, ma);
    return glsl_step(0.8f, 1.0f - len4(c.ma, ma));
}
__device__ __forceinline__ float taa_facing(const float4* __restrict__ normals, const TapAt& t, const Centre& c, int f,
                                            int here) {
    const int axis = (f >> kTaaNormal) & 7;
    if (((f | here) & kTaaWild) || !(f & kTaaSurface) || axis == kTaaOther) {
        float no[4];
        t.get(normals, __ldg(normals + t.i00), f & kTaaSurface, no);
        return dot3(c.no, no);
    }
    // an axis interpolated with itself: its one component, and zeros
    const float w = t.bx + t.ax;
    const float c1 = axis < 2 ? c.no[0] : (axis < 4 ? c.no[1] : c.no[2]);
    return c1 * ((axis & 1) ? -(w * t.by + w * t.ay) : w * t.by + w * t.ay);
}

// One tap (x, y) of the 19x19 disocclusion neighbourhood (LightTAA.frag:61-80):
// (factor * light.rgb, factor), the terms its sums add in order.
__device__ __forceinline__ float4 disocc_tap(const TaaIn& I, const float4* __restrict__ rec, float iResx, float iResy,
                                             const Centre& c, int here, bool still, int x, int y) {
    const float FAR = 4096.0f;
    const float ox = (float)x * iResx, oy = (float)y * iResy;
    const float u = clampg(c.uvx + ox, 0.001f, 0.999f), v = clampg(c.uvy + oy, 0.001f, 0.999f);
    const TapAt t(I.W, I.H, u, v);
    const size_t n = (size_t)I.W * I.H;
    const float4 c00 = __ldg(rec + n + t.i00);
    const int f = __float_as_int(c00.w);
    const float like = taa_like(reinterpret_cast<const float4*>(I.material), t, c, f, here);
    if (like == 0.0f && !((f | here) & kTaaWild)) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);  // adds nothing
    float ld[4], co[4];
    t.get(rec, __ldg(rec + t.i00), false, ld);
    t.get(rec + n, c00, f & kTaaColor, co);
    float factor = gmax(taa_facing(rec + 2 * n, t, c, f, here), 0.0f);
    factor *= like;
    factor *= 1.0f - clampg(fabsf(c.de - ld[3]) * FAR, 0.0f, 1.0f);
    factor *= 1.0f - clampg(len3(c.co, co), 0.0f, 1.0f);
    if (!still) {
        float mo[2];
        t.motion(I.motion, mo);
        if (len2(c.mo[0] - mo[0], c.mo[1] - mo[1]) > 0.1f) factor = 0.0f;
    }
    return make_float4(factor * ld[0], factor * ld[1], factor * ld[2], factor);
}

// The same with every texel loaded at once: a warp of neighbouring pixels,
// which together need most of them, waits for memory once a tap.
__device__ __forceinline__ float4 disocc_tap_all(const TaaIn& I, const float4* __restrict__ rec, float iResx, float iResy,
                                                 const Centre& c, bool still, int x, int y) {
    const float FAR = 4096.0f;
    const float ox = (float)x * iResx, oy = (float)y * iResy;
    const float u = clampg(c.uvx + ox, 0.001f, 0.999f), v = clampg(c.uvy + oy, 0.001f, 0.999f);
    const TapAt t(I.W, I.H, u, v);
    const size_t n = (size_t)I.W * I.H;
    const float4* mat = reinterpret_cast<const float4*>(I.material);
    float ld[4], co[4], no[4], ma[4];
    t.get(mat, __ldg(mat + t.i00), false, ma);
    t.get(rec + 2 * n, __ldg(rec + 2 * n + t.i00), false, no);
    t.get(rec + n, __ldg(rec + n + t.i00), false, co);
    t.get(rec, __ldg(rec + t.i00), false, ld);
    float factor = gmax(dot3(c.no, no), 0.0f);
    factor *= glsl_step(0.8f, 1.0f - len4(c.ma, ma));
    factor *= 1.0f - clampg(fabsf(c.de - ld[3]) * FAR, 0.0f, 1.0f);
    factor *= 1.0f - clampg(len3(c.co, co), 0.0f, 1.0f);
    if (!still) {
        float mo[2];
        t.motion(I.motion, mo);
        if (len2(c.mo[0] - mo[0], c.mo[1] - mo[1]) > 0.1f) factor = 0.0f;
    }
    return make_float4(factor * ld[0], factor * ld[1], factor * ld[2], factor);
}

// 1.212 - radius / 12 of the spiral's taps (LightTAA.frag:115)
__constant__ float c_ring[12] = {1.212f - 2.0f / 12.0f, 1.212f - 3.0f / 12.0f,  1.212f - 4.0f / 12.0f,  1.212f - 5.0f / 12.0f,
                                 1.212f - 6.0f / 12.0f, 1.212f - 7.0f / 12.0f,  1.212f - 8.0f / 12.0f,  1.212f - 9.0f / 12.0f,
                                 1.212f - 10.0f / 12.0f, 1.212f - 11.0f / 12.0f, 1.212f - 12.0f / 12.0f, 1.212f - 13.0f / 12.0f};

constexpr int kDisTaps = 19 * 19;

// The list of disoccluded pixels: how many lie in warps of few and in warps of
// more than kTaaFew, then the former from the front, the latter from the back.
// A pixel costs k_taa_edge 6.3 ns and a lane of k_taa_many's warp 4: 20 of 32
// (16: 1080p with scattered ones 4593 us, now 4458, a quarter of the columns
// 3000, now 2628).
constexpr int kTaaFew = 20;
__device__ __forceinline__ unsigned taa_entry(unsigned n, bool many, int at) {
    return many ? n + 1u - (unsigned)at : 2u + (unsigned)at;
}

// The centre of a pixel: everything its taps are compared with; returns its
// flags. A warp's centres are neighbours, so all four texels are loaded at
// once rather than the flags first.
__device__ __forceinline__ int taa_centre(const TaaIn& I, const float4* __restrict__ rec, int px, int py, Centre& c) {
    const size_t n = (size_t)I.W * I.H;
    const float4* mat = reinterpret_cast<const float4*>(I.material);
    c.uvx = ((float)px + 0.5f) / (float)I.W;
    c.uvy = ((float)py + 0.5f) / (float)I.H;
    const TapAt t(I.W, I.H, c.uvx, c.uvy);
    float q[4];
    const float4 c00 = __ldg(rec + n + t.i00);
    const int f = __float_as_int(c00.w);
    t.get(rec + n, c00, false, q);
    c.co[0] = q[0];
    c.co[1] = q[1];
    c.co[2] = q[2];
    t.get(rec + 2 * n, __ldg(rec + 2 * n + t.i00), false, q);
    c.no[0] = q[0];
    c.no[1] = q[1];
    c.no[2] = q[2];
    t.get(mat, __ldg(mat + t.i00), false, c.ma);
    t.get(rec, __ldg(rec + t.i00), false, q);
    c.de = q[3];
    t.motion(I.motion, c.mo);
    return f;
}

// Reach of a pixel's taps, in texels, within which the motion test is decided
// by the pre-pass's maxima: they lie at most 14.5 away, their texels at most
// 16, so the block's own and its neighbouring tiles of 32 x 8 hold them, two
// rows of tiles up and down. Motions below 0.035 differ by less than 0.1.
constexpr float kTaaReach = 14.5f, kTaaStill = 0.035f;

// By a whole warp: no tap in reach of a pixel of tile (tx, ty) can fail the motion test.
__device__ __forceinline__ bool taa_still(int W, int H, int tx, int ty, const float* __restrict__ motion_max) {
    const int lane = threadIdx.x & 31, nx = (W + kPackW - 1) / kPackW, ny = (H + kPackH - 1) / kPackH;
    const int x = tx - 1 + lane % 3, y = ty - 2 + lane / 3;
    bool still = W <= 14000 && H <= 14000;
    if (lane < 15 && x >= 0 && y >= 0 && x < nx && y < ny) still = still && __ldg(motion_max + y * nx + x) < kTaaStill;
    return __all_sync(0xffffffffu, still);
}

// The pixels whose reprojection leaves the screen (listed by k_taa), up to
// kEdgeGroup at a time per block: the current frame's 19x19 neighbourhood only.
// The threads compute a pixel's taps row by row (their texels are then
// adjacent) into shared memory, and four lanes per pixel add its four sums up
// column by column, the shader's loop order, so the result is the same float.
// 361 taps instead of 12: inside the spiral's kernel the few warps with such
// pixels, at the screen's edge, ran on after all others (1080p, 1% of the
// pixels: 958 us, now 456 for the spiral and 126 here).
// A block of 384 threads makes a pixel's taps in one go, for few pixels; many
// run better in blocks of 128. `apart` or more pixels in warps of many are left
// to k_taa_many.
constexpr int kEdgeGroup = 4;
template <int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == 128 ? 8 : 2) k_taa_edge(const TaaIn I, const float4* __restrict__ rec,
                                                  const float* __restrict__ motion_max, const int* __restrict__ list,
                                                  int apart, float* __restrict__ out) {
    __shared__ float4 s_dis[kEdgeGroup][kDisTaps];
    __shared__ Centre s_centre[kEdgeGroup];
    __shared__ int s_flags[kEdgeGroup], s_pixel[kEdgeGroup];
    __shared__ bool s_still[kEdgeGroup];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const float iResx = 1.0f / (float)I.W, iResy = 1.0f / (float)I.H;
    const unsigned n = (unsigned)I.W * (unsigned)I.H;
    after_previous(rec, motion_max, list);
    const int few = list[0], many = list[1], count = many >= apart ? few : few + many;
    const int group = min(kEdgeGroup, (count + (int)gridDim.x - 1) / (int)gridDim.x);
    for (int k = blockIdx.x * group; k < count; k += gridDim.x * group) {
        const int m = min(group, count - k);
        if (wib < m) {
            const int e = k + wib, i = list[taa_entry(n, e >= few, e < few ? e : e - few)];
            Centre c;
            const int f = taa_centre(I, rec, i % I.W, i / I.W, c);
            const bool still = taa_still(I.W, I.H, i % I.W / kPackW, i / I.W / kPackH, motion_max);
            if (lane == 0) {
                s_still[wib] = still;
                s_centre[wib] = c;
                s_flags[wib] = f;
                s_pixel[wib] = i;
            }
        }
        __syncthreads();
        for (int e = 0; e < m; e++)
            for (int t = threadIdx.x; t < kDisTaps; t += THREADS) {
                const int x = t % 19, y = t / 19;
                s_dis[e][x * 19 + y] = disocc_tap(I, rec, iResx, iResy, s_centre[e], s_flags[e], s_still[e], x - 9, y - 9);
            }
        __syncthreads();
        if (wib == 0) {
            float acc = 0.0f;
            if (lane < 4 * m) {
                const float* f = reinterpret_cast<const float*>(s_dis[lane >> 2]) + (lane & 3);
                for (int x = 0; x < 19; x++) {
#pragma unroll
                    for (int y = 0; y < 19; y++) acc += f[4 * (x * 19 + y)];
                }
            }
            const float total = __shfl_sync(0xffffffffu, acc, lane | 3);
            if (lane < 4 * m)
                out[4 * (size_t)s_pixel[lane >> 2] + (lane & 3)] = (lane & 3) < 3 ? acc / total : 1.0f;
        }
        __syncthreads();
    }
}

// The pixels in warps of many, one a lane, where there are enough of them to
// fill the GPU that way (a fast pan, a camera that jumps): a warp's pixels
// share texels, and all 16 loads of a tap are in flight. That takes 128
// registers, which is why this is a kernel of its own: with k_taa_edge's 64 it
// took a third longer, and k_taa_edge 8% longer with 128. us a frame at 1080p
// for 2, 4, 8, 25 and 100% of the frame's rows, by k_taa_edge / here: 732 /
// 786, 993 / 1045, 1486 / 1275, 3640 / 2562, 13061 / 8172; at 640x360 for 25,
// 50 and 100%: 437 / 433, 773 / 665, 1473 / 931. L1 wavefronts bound it (71%).
constexpr int kTaaMany = 560;  // pixels per SM from which on it runs
constexpr int kManyThreads = 128;
__global__ void __launch_bounds__(kManyThreads, 4) k_taa_many(const TaaIn I, const float4* __restrict__ rec,
                                                              const int* __restrict__ list, int apart,
                                                              float* __restrict__ out) {
    after_previous(rec, list);
    const int many = list[1], lane = threadIdx.x & 31;
    if (many >= apart) {
        const unsigned n = (unsigned)I.W * (unsigned)I.H;
        const float iResx = 1.0f / (float)I.W, iResy = 1.0f / (float)I.H;
        for (int k = blockIdx.x * kManyThreads + threadIdx.x - lane; k < many; k += gridDim.x * kManyThreads) {
            const bool on = k + lane < many;
            const int i = list[taa_entry(n, true, on ? k + lane : k)], px = i % I.W, py = i / I.W;
            // The motion test loads nothing where the motions of all texels in
            // reach (9 pixels and the clamp at 0.001, and one for the second
            // texel) differ by less than 0.1, rounding included.
            const int x0 = max(__reduce_min_sync(0xffffffffu, px) - 10, 0);
            const int x1 = min(__reduce_max_sync(0xffffffffu, px) + 10, I.W - 1);
            const int y0 = max(__reduce_min_sync(0xffffffffu, py) - 10, 0);
            const int y1 = min(__reduce_max_sync(0xffffffffu, py) + 10, I.H - 1);
            const int w = x1 - x0 + 1, texels = w * (y1 - y0 + 1);
            bool still = I.W <= 9000 && I.H <= 9000 && texels <= 4096;
            if (still) {
                float lo0 = INFINITY, hi0 = -INFINITY, lo1 = INFINITY, hi1 = -INFINITY;
                bool ok = true;
                for (int t = lane; t < texels; t += 32) {
                    const size_t at = (size_t)(y0 + t / w) * I.W + x0 + t % w;
                    const float2 m = __ldg(reinterpret_cast<const float2*>(I.motion) + at);
                    ok = ok && fabsf(m.x) < 256.0f && fabsf(m.y) < 256.0f;
                    lo0 = fminf(lo0, m.x);
                    hi0 = fmaxf(hi0, m.x);
                    lo1 = fminf(lo1, m.y);
                    hi1 = fmaxf(hi1, m.y);
                }
                for (int o = 16; o > 0; o >>= 1) {
                    lo0 = fminf(lo0, __shfl_xor_sync(0xffffffffu, lo0, o));
                    hi0 = fmaxf(hi0, __shfl_xor_sync(0xffffffffu, hi0, o));
                    lo1 = fminf(lo1, __shfl_xor_sync(0xffffffffu, lo1, o));
                    hi1 = fmaxf(hi1, __shfl_xor_sync(0xffffffffu, hi1, o));
                }
                still = __all_sync(0xffffffffu, ok) && hi0 - lo0 < 2.0f * kTaaStill && hi1 - lo1 < 2.0f * kTaaStill;
            }
            if (!on) continue;
            Centre c;
            taa_centre(I, rec, px, py, c);
            float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            for (int x = -9; x <= 9; x++)
#pragma unroll 1
                for (int y = -9; y <= 9; y++) {
                    const float4 t = disocc_tap_all(I, rec, iResx, iResy, c, still, x, y);
                    sum.x += t.x;
                    sum.y += t.y;
                    sum.z += t.z;
                    sum.w += t.w;
                }
            float* o = out + 4 * (size_t)i;
            o[0] = sum.x / sum.w;
            o[1] = sum.y / sum.w;
            o[2] = sum.z / sum.w;
            o[3] = 1.0f;
        }
    }
}

// 32x4-pixel blocks: the spiral taps of neighbouring pixels overlap in L1.
// Four rows and 7 blocks per SM (72 registers, 48 bytes of spills) measured
// 456 us at 1080p; 6 blocks 504, 8 blocks 484, two rows 484, eight rows 510.
constexpr int kTaaRows = 4;
// SPLIT lanes share a pixel: lane s of them makes the taps s, s + SPLIT, ..,
// and all add them up in the shader's order.
template <int SPLIT, int BLOCKS>
__global__ void __launch_bounds__(32 * kTaaRows, BLOCKS) k_taa(const TaaIn I, const float4* __restrict__ rec,
                                                               const float* __restrict__ motion_max,
                                                               int* __restrict__ list, float* __restrict__ out) {
    constexpr int WIDE = 32 / SPLIT;  // pixels per warp
    const int W = I.W, H = I.H;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, share = lane % SPLIT;
    const int px = blockIdx.x * WIDE + lane / SPLIT, py = blockIdx.y * kTaaRows + wib;
    const bool valid = px < W && py < H;
    const int i = valid ? py * W + px : 0;
    const size_t n = (size_t)W * H;
    const float4* mat = reinterpret_cast<const float4*>(I.material);
    after_previous(rec, motion_max, list);
    const bool still = taa_still(W, H, (int)(blockIdx.x * WIDE / kPackW), (int)(blockIdx.y * kTaaRows / kPackH), motion_max);
    const float GR = 2.118033988749895f;
    const float iResx = 1.0f / (float)W, iResy = 1.0f / (float)H;
    float* o = out + 4 * (size_t)i;
    Centre c;
    float cl[4], ll[4];
    int mode = 0;  // 0 done, 1 disoccluded, 2 spiral
    int here = 0;  // the centre's flags
    if (valid) {
        here = taa_centre(I, rec, px, py, c);
        tex4(I.light, W, H, c.uvx, c.uvy, cl);
        if (c.de == 1.0f) {
            o[0] = cl[0];
            o[1] = cl[1];
            o[2] = cl[2];
            o[3] = cl[3];
        } else {
            const float oux = c.uvx + c.mo[0], ouy = c.uvy + c.mo[1];
            tex4(I.last, W, H, oux, ouy, ll);
            mode = (clampg(oux, 0.0f, 1.0f) != oux || clampg(ouy, 0.0f, 1.0f) != ouy) ? 1 : 2;
        }
    }
    const unsigned dis = __ballot_sync(0xffffffffu, mode == 1 && share == 0);
    if (dis != 0u) {
        const bool many = __popc(dis) > kTaaFew;
        int at = 0;
        if (lane == 0) at = atomicAdd(list + many, __popc(dis));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(dis & ((1u << lane) - 1u));
        if (mode == 1 && share == 0) list[taa_entry((unsigned)n, many, at)] = i;
    }
    if (mode != 2) return;  // with its pixel's other lanes
    const float* motion = c.mo;
    const float* cc = c.co;
    const float depth = c.de;
    const float uvx = c.uvx, uvy = c.uvy;
    const float FAR = 4096.0f;
    float lastVariance = ll[3];
    // 12-tap golden-angle spiral, neighbourhood clip, variance-driven blend
    float nmin[3] = {10000.0f, 10000.0f, 10000.0f}, nmax[3] = {0.0f, 0.0f, 0.0f};
    float ncol[3] = {0.0f, 0.0f, 0.0f};
    float diffSum = 1.0f, count = 0.0f;
    const float size = 12.0f;
    float radius = 1.0f;
    const float dscale = gmin(gmax(0.1f, 0.5f), 1.0f / depth);
    const bool near = still && fabsf((size + 1.0f) * (lastVariance + 1.0f) * dscale) < kTaaReach;
    const float n0 = __ldg(I.noise + 4 * (size_t)i);
    float angle = n0 * 3.1415f * GR;
    // the pixel's lanes, which are all here
    const unsigned group = SPLIT == 1 ? 1u << lane : ((1u << SPLIT) - 1u) << (lane - share);
#pragma unroll 1
    for (int k0 = 0; k0 < 12; k0 += SPLIT) {
        float own = angle;  // of this lane's tap: the shader's sum, term by term
        float rad = radius + 1.0f;
        for (int j = 0; j < SPLIT; j++) {
            if (j < share) {
                own += 2.39f;
                rad += 1.0f;
            }
            angle += 2.39f;
            radius += 1.0f;
        }
        float sn, cs;
        sincos_own(own, &sn, &cs);
        const float rv = rad * (lastVariance + 1.0f);
        const float ox = cs * iResx * rv * dscale, oy = sn * iResy * rv * dscale;
        const float u = clampg(uvx + ox, 0.001f, 0.999f), v = clampg(uvy + oy, 0.001f, 0.999f);
        const TapAt t(W, H, u, v);
        float ld[4], co[4];
        t.get(rec, __ldg(rec + t.i00), false, ld);
        const float4 c00 = __ldg(rec + n + t.i00);
        const int f = __float_as_int(c00.w);
        t.get(rec + n, c00, f & kTaaColor, co);
        const float apart = len3(cc, co) * 10000.0f;
        float factor = 0.0f;
        if (!(apart >= 1.0f) || ((f | here) & kTaaWild)) {
            factor = c_ring[k0 + share];
            factor *= taa_like(mat, t, c, f, here);
            factor *= gmax(taa_facing(rec + 2 * n, t, c, f, here), 0.0f);
            factor *= 1.0f - clampg(fabsf(depth - ld[3]) * FAR, 0.0f, 1.0f);
            factor *= 1.0f - clampg(apart, 0.0f, 1.0f);
            if (!near) {
                float mo[2];
                t.motion(I.motion, mo);
                if (len2(motion[0] - mo[0], motion[1] - mo[1]) > 0.1f) factor = 0.0f;
            }
        }
        const float differ = len3(ld, cl) * factor;
#pragma unroll
        for (int j = 0; j < SPLIT; j++) {
            float nli[3] = {ld[0], ld[1], ld[2]}, fj = factor, dj = differ;
            if (SPLIT > 1) {
                const int from = lane - share + j;
#pragma unroll
                for (int k = 0; k < 3; k++) nli[k] = __shfl_sync(group, ld[k], from);
                fj = __shfl_sync(group, factor, from);
                dj = __shfl_sync(group, differ, from);
            }
#pragma unroll
            for (int k = 0; k < 3; k++) {
                nmin[k] = gmin(nmin[k], nli[k]);
                nmax[k] = gmax(nmax[k], nli[k]);
                ncol[k] += fj * nli[k];
            }
            count += fj;
            diffSum += dj;
        }
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        cl[k] += ncol[k];
        cl[k] /= count + 1.0f;
    }
    diffSum /= radius;
#pragma unroll
    for (int k = 0; k < 3; k++) ll[k] = gmin(gmax(ll[k], nmin[k]), nmax[k]);
    const float a0 = fabsf(cl[0] - ll[0]), a1 = fabsf(cl[1] - ll[1]), a2 = fabsf(cl[2] - ll[2]);
    float lum = a0 * 0.2125f + a1 * 0.7154f;
    lum = lum + a2 * 0.0721f;
    const float variance = clampg(lum * 5.5f, 0.0f, 1.0f);
    lastVariance += variance;
    lastVariance -= diffSum * 0.08f;
    lastVariance += len2(motion[0], motion[1]) * 20.0f;
    const float t = clampg(1.0f - lastVariance, 0.3f, 0.9f);
    const float omt = 1.0f - t;
    if (share != 0) return;
    o[0] = cl[0] * omt + ll[0] * t;
    o[1] = cl[1] * omt + ll[1] * t;
    o[2] = cl[2] * omt + ll[2] * t;
    o[3] = clampg(lastVariance * 0.7f, 0.0f, 1.0f);
}

// A launch whose start overlaps the end of the one before it in the stream
// (after_previous waits in the kernel): 1 to 2 us less between two of them.
template <class... P, class... A>
cudaError_t taa_launch(void (*kernel)(P...), dim3 grid, unsigned threads, cudaStream_t s, A... args) {
    cudaLaunchAttribute overlap[1];
    overlap[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.stream = s;
    cfg.attrs = overlap;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, (P)args...);
}

}  // namespace

vxl_status launch_light_taa(vxl_ctx* ctx, const vxl_taa_frame* f, float* out, cudaStream_t s) {
    TaaIn I{f->light, f->last_light, f->color, f->normal, f->material, f->depth, f->motion, f->noise, f->width,
            f->height};
    const size_t n = (size_t)f->width * f->height;
    const dim3 pack((unsigned)((f->width + kPackW - 1) / kPackW), (unsigned)((f->height + kPackH - 1) / kPackH));
    // planes, the pre-pass's maxima, and the list of disoccluded pixels (its lengths first)
    const size_t planes = n * kTaaPlanes * sizeof(float4), maxima = (size_t)pack.x * pack.y * sizeof(float);
    VXL_TRY(ctx_grow(&ctx->d_taa, &ctx->taa_bytes, planes + maxima + (n + 2) * sizeof(int)));
    float4* rec = (float4*)ctx->d_taa;
    float* motion_max = (float*)((char*)ctx->d_taa + planes);
    int* list = (int*)((char*)ctx->d_taa + planes + maxima);
    k_taa_pack<<<pack, kPackW * kPackH, 0, s>>>(I, rec, motion_max, list);
    ctx->launches++;
    const dim3 grid((unsigned)((f->width + 31) / 32), (unsigned)((f->height + kTaaRows - 1) / kTaaRows));
    // A frame whose warps the GPU holds all at once takes as long as one pixel's
    // 12 taps one after another: there four lanes share a pixel, and the edge
    // runs in larger blocks (us, four lanes a pixel / one: 5,000 pixels 25 / 42,
    // 40,000 38 / 47, 58,000 44 / 49, 80,000 54 / 54, 120,000 66 / 60).
    const bool small = n <= (size_t)ctx->sm_count * 448;
    const int apart = small ? INT_MAX : ctx->sm_count * kTaaMany;
    const unsigned edge = (unsigned)std::min<size_t>(n, (size_t)ctx->sm_count * (small ? 2 : 8));
    if (small) {
        const dim3 quarter((unsigned)((f->width + 7) / 8), grid.y);
        VXL_TRY_CUDA(taa_launch(k_taa<4, 7>, quarter, 32 * kTaaRows, s, I, rec, motion_max, list, out));
        VXL_TRY_CUDA(taa_launch(k_taa_edge<384>, edge, 384, s, I, rec, motion_max, list, apart, out));
        ctx->launches += 2;
    } else {
        VXL_TRY_CUDA(taa_launch(k_taa<1, 7>, grid, 32 * kTaaRows, s, I, rec, motion_max, list, out));
        VXL_TRY_CUDA(taa_launch(k_taa_edge<128>, edge, 128, s, I, rec, motion_max, list, apart, out));
        VXL_TRY_CUDA(taa_launch(k_taa_many, (unsigned)ctx->sm_count * 4, kManyThreads, s, I, rec, list, apart, out));
        ctx->launches += 3;
    }
    VXL_TRY_CUDA(cudaGetLastError());
    return VXL_OK;
}

}  // namespace vxl
