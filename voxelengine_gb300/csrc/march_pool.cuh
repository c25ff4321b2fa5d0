// march_pool.cuh — the marchers raycastShadowVolumeSparse / SuperSparse
// (Sources/Shaders/lib/Light.frag:131-217) for many rays per warp: the same
// positions, fetches and results as march() of vxl_device.cuh, bit for bit.
//
// What bounds march() one ray a thread is instructions: six conversions and
// rounding operations a step at a quarter of the FMA rate, steps taken after
// the ray has left the grid, where nothing can be hit (half of all steps of a
// view from outside the grid), and lanes idle behind their warp's longest ray
// (four of five for incoherent rays). Here
//  - a warp keeps a pool of up to kMarchRays rays in shared memory and its
//    lanes take the next ones as theirs end; rays that survive the fine part
//    (steps of step0 up to 16) go back to the pool for the coarse part, so
//    each part runs its own loop;
//  - floor() is one addition of a large constant that rounds down, whose low
//    bits are the cell, and the mod(pos, 0.5) > 0.25 test of the fine part
//    (Light.frag:142-148) is the difference of two such additions; the word's
//    address and the bit in it are sums of multiples of those, which run on
//    the FMA pipe (in shifts and masks, on the ALU pipe: 2 to 6% slower);
//  - positions are monotone, so one bounds test covers the four steps of a
//    batch, and a ray outside the grid on the side it moves to is a miss at
//    once; with records its positions still advance to the last one, after the
//    other rays' tests, 32 such rays side by side (march_away).
// Before -> after, at 1080p on a 512^3 grid: sun shadow + ambient 391 -> 226
// us, reflection 364 -> 186 us, the pairs of 64 lights 287 -> 181 us; 1 M
// incoherent sparse rays with records 271 -> 157 us. Still bound by the
// instructions it issues (a fine test is about 37, a coarse one 22).
#pragma once
#include <cstdint>
#include <type_traits>

#include "vxl_device.cuh"

namespace vxl {

constexpr int kMarchRays = 128;   // rays of a warp's pool
constexpr int kMarchWarps = 2;    // warps per block: fewer wait for their block's slowest pool (4: 3% slower)
constexpr int kMarchBlocks = 16;  // blocks per SM (64 registers)
constexpr int kMarchFirst = 4;    // tests made before a ray enters the pool
constexpr int kMarchBatch = 4;    // tests between looks at the warp's state (2 or 8: 10 to 20% slower)
constexpr int kMarchRefill = 24;  // a pool refills when no more lanes than this run (8 to 28: within 3%)

struct MarchPool {
    float4 a[kMarchRays];  // position, dist
    float4 b[kMarchRays];  // step, id
};
// with records: slots of the rays for the coarse part, and of those that left the grid
struct MarchPoolRec : MarchPool {
    uint8_t keep[kMarchRays], away[kMarchRays];
};
// id: the ray's index in the tile; kMarchSuper set for the SuperSparse marcher.
// Of a ray that left the grid also twice its next test's distance from bit 8
// on, and kMarchFine where that test is one of the fine part.
constexpr uint32_t kMarchSuper = 0x80000000u, kMarchRay = 0xffu, kMarchFine = 1u << 20;

// x + 1.5 * 2^(23 - k), rounded down, holds floor(2^k x) in its low bits
// (|x| < 2^20): floor(x / 4), floor(x / 2) and floor(2 x) of a position.
constexpr float kBrick = 50331648.0f, kBlock = 25165824.0f, kHalf = 6291456.0f;
constexpr uint32_t kBrickBits = 0x4C400000u, kBlockBits = 0x4BC00000u;

// The 32 bits (half a brick) with the 2^3 block of position p (0 <= p < n) and
// the block's first bit in them, modulo 32. Everything after the additions is
// a sum of multiples of their bits, so it runs on the FMA pipe; the pipe of
// shifts, masks and compares bounds this kernel.
__device__ __forceinline__ uint32_t march_word(const GridView& g, f3 p, bool on, uint32_t* shift) {
    const uint32_t bx = __float_as_uint(__fadd_rd(p.x, kBlock)), by = __float_as_uint(__fadd_rd(p.y, kBlock)),
                   bz = __float_as_uint(__fadd_rd(p.z, kBlock));
    const uint32_t wx = __float_as_uint(__fadd_rd(p.x, kBrick)), wy = __float_as_uint(__fadd_rd(p.y, kBrick)),
                   wz = __float_as_uint(__fadd_rd(p.z, kBrick));
    const uint32_t brick = wx + wy * (uint32_t)g.bx + wz * g.bxy - kBrickBits * (1u + (uint32_t)g.bx + g.bxy);
    const uint32_t half = bz - 2u * wz - (kBlockBits - 2u * kBrickBits);
    *shift = 2u * bx - 4u * wx + 8u * by - 16u * wy;  // the constants are multiples of 32
    return on ? __ldg(reinterpret_cast<const uint32_t*>(g.words + brick) + half) : 0u;
}
// bit of the fine part's cell: its block's voxel by mod(pos, 0.5) > 0.25 per axis (Light.frag:142-148).
// For x >= 0 that is ceil(2x - 0.5) - floor(2x): x - 0.25 is exact from 0.125 up, and below
// both are 0 whatever its rounding.
__device__ __forceinline__ bool march_fine_bit(const GridView& g, f3 p) {
    const uint32_t fx = __float_as_uint(__fadd_rd(p.x, kHalf)), fy = __float_as_uint(__fadd_rd(p.y, kHalf)),
                   fz = __float_as_uint(__fadd_rd(p.z, kHalf));
    const uint32_t cx = __float_as_uint(__fadd_ru(p.x - 0.25f, kHalf)), cy = __float_as_uint(__fadd_ru(p.y - 0.25f, kHalf)),
                   cz = __float_as_uint(__fadd_ru(p.z - 0.25f, kHalf));
    uint32_t sh;
    const uint32_t w = march_word(g, p, true, &sh);
    sh += (cx - fx) + 4u * (cy - fy) + 16u * (cz - fz);
    return __funnelshift_r(w, w, sh) & 1u;
}
// any voxel of the coarse part's block
__device__ __forceinline__ bool march_coarse_bit(const GridView& g, f3 p) {
    uint32_t sh;
    const uint32_t w = march_word(g, p, true, &sh);
    return (__funnelshift_r(w, w, sh) & 0x00330033u) != 0u;
}
// Either test where p may lie below 0 (above -2: the shader's conversions
// truncate, so such a coordinate reads block 0) or, with `on` false, anywhere.
// Below 0 the shader's mod() rounds; this is its arithmetic.
template <bool FINE>
__device__ __forceinline__ bool march_bit(const GridView& g, f3 p, bool on) {
    uint32_t sh;
    const uint32_t w = march_word(g, mk(fmaxf(p.x, 0.0f), fmaxf(p.y, 0.0f), fmaxf(p.z, 0.0f)), on, &sh);
    if (!FINE) return (__funnelshift_r(w, w, sh) & 0x00330033u) != 0u;
    const bool qx = p.x - (__fadd_rd(p.x, kHalf) - kHalf) > 0.25f, qy = p.y - (__fadd_rd(p.y, kHalf) - kHalf) > 0.25f,
               qz = p.z - (__fadd_rd(p.z, kHalf) - kHalf) > 0.25f;
    sh += (qx ? 1u : 0u) + (qy ? 4u : 0u) + (qz ? 16u : 0u);
    return __funnelshift_r(w, w, sh) & 1u;
}
// The tested voxel as the shader computes it.
template <bool FINE>
__device__ __forceinline__ void march_voxel(f3 p, int* v) {
    const float q[3] = {p.x, p.y, p.z};
    for (int k = 0; k < 3; k++)
        v[k] = FINE ? (int)(q[k] * 0.5f) * 2 + (mod_half(q[k]) > 0.25f) : (int)q[k] / 2 * 2;
}
__device__ __forceinline__ unsigned march_lanes_below() {
    unsigned m;
    asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// inside the cells that the shader reads (see march_bit); outside them it reads 0
__device__ __forceinline__ bool march_inside(const GridView& g, f3 p) {
    return p.x > -2.0f && p.y > -2.0f && p.z > -2.0f && p.x < (float)g.nx && p.y < (float)g.ny && p.z < (float)g.nz;
}
// Nothing can be hit from here on: outside and not moving back.
__device__ __forceinline__ bool march_gone(const GridView& g, f3 p, f3 s) {
    return (p.x <= -2.0f && s.x <= 0.0f) || (p.y <= -2.0f && s.y <= 0.0f) || (p.z <= -2.0f && s.z <= 0.0f) ||
           (p.x >= (float)g.nx && s.x >= 0.0f) || (p.y >= (float)g.ny && s.y >= 0.0f) ||
           (p.z >= (float)g.nz && s.z >= 0.0f);
}

// All positions from p to about e lie outside, on the same side. The half cell
// covers the rounding of the positions and of e for steps below kMarchSlack: a
// position near the grid is then at most 2^21 away from p and from the origin,
// where the at most four roundings make 1/4 (at 2^24 a step, two cells).
constexpr float kMarchSlack = 524288.0f;
__device__ __forceinline__ bool march_small(f3 s) {
    return fmaxf(fmaxf(fabsf(s.x), fabsf(s.y)), fabsf(s.z)) < kMarchSlack;
}
__device__ __forceinline__ bool march_outside(const GridView& g, f3 p, f3 e) {
    return fmaxf(p.x, e.x + 0.5f) <= -2.0f || fmaxf(p.y, e.y + 0.5f) <= -2.0f || fmaxf(p.z, e.z + 0.5f) <= -2.0f ||
           fminf(p.x, e.x - 0.5f) >= (float)g.nx || fminf(p.y, e.y - 0.5f) >= (float)g.ny ||
           fminf(p.z, e.z - 0.5f) >= (float)g.nz;
}

// The rounding of a batch's positions inside the grid, which is below 32768
// cells: four times 2^-9 at most. A ray within this of a face, and for good if
// it runs along it, sends its warp through the tests that look at every
// position (at half a cell, one ray in 85 on 256^3: 30,000 such rays 43 us).
constexpr float kMarchEdge = 1.0f / 32.0f;
// The N tests from p on, s apart: bit j of the result set where test j finds a
// voxel. q becomes the position after them. `in`: p is known to lie in [0, n)
// (it becomes so for q's batch); small: march_small(s); left: nothing can be hit from q on. lanes: those that call it
// together, from a vote of the whole warp. EDGE: tests at once on the grid's
// edge (2 for sparse rays, 30,000 along an axis 41 -> 33 us; the light passes
// have no room for it, 1080p with records 418 -> 464 us).
template <bool FINE, int N, int EDGE>
__device__ __forceinline__ unsigned march_tests(unsigned lanes, const GridView& g, f3 p, f3 s, f3& q, bool& in, bool small,
                                                bool& left) {
    // where the last test lies, to less than what the bounds leave
    const f3 e = mk(__fmaf_rn(s.x, (float)(N - 1), p.x), __fmaf_rn(s.y, (float)(N - 1), p.y),
                    __fmaf_rn(s.z, (float)(N - 1), p.z));
    const bool in_e = e.x >= kMarchEdge && e.y >= kMarchEdge && e.z >= kMarchEdge && e.x <= (float)g.nx - kMarchEdge &&
                      e.y <= (float)g.ny - kMarchEdge && e.z <= (float)g.nz - kMarchEdge;
    unsigned hits = 0u;
    q = p;
    const bool inner = in && in_e;  // every position from p to e is inside
    const bool none = !inner && small && march_outside(g, p, e);
    // One lane on the grid's edge sends its whole warp through the tests that
    // look at every position: a branch per lane would run both loops.
    if (__all_sync(lanes, inner || none)) {
        if (inner) {
#pragma unroll
            for (int j = 0; j < N; j++) {
                hits |= (FINE ? march_fine_bit(g, q) : march_coarse_bit(g, q)) ? 1u << j : 0u;
                q = add(q, s);
            }
        } else {
            for (int j = 0; j < N; j++) q = add(q, s);
            left = march_gone(g, q, s);
        }
    } else {
#pragma unroll EDGE
        for (int j = 0; j < N; j++) {
            hits |= march_bit<FINE>(g, q, !none && march_inside(g, q)) ? 1u << j : 0u;
            q = add(q, s);
        }
        left = !inner && march_gone(g, q, s);
    }
    in = in_e;
    return hits;
}

__device__ __forceinline__ float march_step0(uint32_t id) { return (id & kMarchSuper) ? 2.5f : 0.5f; }
// the coarse part's first distance: the first multiple of step0 from 16 up
__device__ __forceinline__ float march_dcoarse(uint32_t id) { return (id & kMarchSuper) ? 17.5f : 16.0f; }

// One part of the march for the pool's `count` rays. done(id, hit, t, fine,
// last, steps) is called once per ray that ends in this part: t the hit
// distance or dist, `last` the last position tested, steps the tests made (the
// last two for REC only). Returns the number of rays that go on to the coarse
// part: the pool's first ones then, or with REC those of P.keep. With REC rays
// that left the grid are put by in P.away, `away` of them. Rays that ended wait
// until no more than kMarchRefill lanes run: their ends and the refill cost
// about as much as a batch of tests.
template <bool FINE, bool REC, int EDGE, class Pool, class Done>
__device__ __forceinline__ int march_part(const GridView& g, Pool& P, int count, int& away, Done done) {
    constexpr int N = kMarchBatch;
    int base = 0, kept = 0, slot = 0;
    bool busy = false, in = false, small = true;
    f3 p = mk(0.0f, 0.0f, 0.0f), s = p;
    float d = 0.0f, ds = 0.0f, lim = 0.0f, dist = 0.0f;
    uint32_t id = 0;
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !busy);
        bool off = false;  // left the grid, tests to go
        if (base < count) {
            const int at = base + __popc(idle & march_lanes_below());
            if (!busy && at < count) {
                if constexpr (REC) slot = FINE ? at : P.keep[at];
                const float4 a = P.a[REC ? slot : at], b = P.b[REC ? slot : at];
                p = mk(a.x, a.y, a.z);
                s = mk(b.x, b.y, b.z);
                dist = a.w;
                id = __float_as_uint(b.w);
                ds = march_step0(id) * (FINE ? 1.0f : 2.0f);
                d = FINE ? ds * (float)(kMarchFirst + 1) : march_dcoarse(id);
                lim = FINE ? 16.0f : (dist < 164.0f ? dist : 164.0f);
                in = p.x >= 0.0f && p.y >= 0.0f && p.z >= 0.0f && march_inside(g, p);
                small = march_small(s);
                off = REC && FINE && march_gone(g, p, s);
                busy = !off;
            }
            base = min(base + __popc(idle), count);
            __syncwarp();
        } else if (idle == 0xffffffffu) {
            break;
        }
        float next = d;  // of the tests to go, and whether they are fine ones
        bool fine = FINE;
        const int waiting = base < count ? kMarchRefill : 0;
        bool run = busy, left = false;
        unsigned hits = 0u, lanes = __ballot_sync(0xffffffffu, run);
        do {
            if (run) {
                f3 q;
                hits = march_tests<FINE, N, EDGE>(lanes, g, p, s, q, in, small, left);
                const float dn = d + (float)N * ds;  // small multiples of 0.5: exact
                if (hits != 0u || !(dn < lim) || left) {
                    run = false;
                } else {
                    p = q;
                    d = dn;
                }
            }
            lanes = __ballot_sync(0xffffffffu, run);
        } while (__popc(lanes) > waiting);
        bool keep = false;
        if (busy && !run) {
            int nv = 1;  // the batch's tests that the shader makes: those at a distance below lim
#pragma unroll
            for (int j = 1; j < N; j++) nv += d + (float)j * ds < lim ? 1 : 0;
            const int first = __ffs(hits) - 1;
            const bool hit = hits != 0u && first < nv;
            const float dcoarse = march_dcoarse(id), dn = d + (float)N * ds;
            if (FINE && !hit && !(dn < lim) && dcoarse < (dist < 164.0f ? dist : 164.0f)) {
                for (int j = 0; j < nv; j++) p = add(p, s);
                keep = !march_gone(g, p, s);
                s = mul(s, 2.0f);
                off = REC && !keep;
                next = dcoarse;
                fine = false;
            } else if (REC && !hit && dn < lim) {
                for (int j = 0; j < N; j++) p = add(p, s);
                off = true;
                next = dn;
            }
            if (!keep && !off) {
                const int k = hit ? first : nv - 1;
                const float t = d + (float)k * ds;
                if (REC)
                    for (int j = 0; j < k; j++) p = add(p, s);
                const int steps =
                    REC ? (int)((t - (FINE ? ds : dcoarse)) / ds) + 1 + (FINE ? 0 : ((id & kMarchSuper) ? 6 : 31)) : 0;
                done(id & kMarchRay, hit, hit ? t : dist, FINE, p, steps);
            }
            busy = false;
        }
        if constexpr (REC) {
            const unsigned km = __ballot_sync(0xffffffffu, keep), om = __ballot_sync(0xffffffffu, off);
            if (keep || off) {
                const uint32_t rest = off ? (uint32_t)(2.0f * next) << 8 | (fine ? kMarchFine : 0u) : 0u;
                P.a[slot] = make_float4(p.x, p.y, p.z, dist);
                P.b[slot] = make_float4(s.x, s.y, s.z, __uint_as_float(id | rest));
                if (keep)
                    P.keep[kept + __popc(km & march_lanes_below())] = (uint8_t)slot;
                else
                    P.away[away + __popc(om & march_lanes_below())] = (uint8_t)slot;
            }
            kept += __popc(km);
            away += __popc(om);
        } else if constexpr (FINE) {
            const unsigned km = __ballot_sync(0xffffffffu, keep);
            if (keep) {
                const int at = kept + __popc(km & march_lanes_below());
                P.a[at] = make_float4(p.x, p.y, p.z, dist);
                P.b[at] = make_float4(s.x, s.y, s.z, __uint_as_float(id));
            }
            kept += __popc(km);
        }
    }
    __syncwarp();
    return kept;
}

// The records of rays that left the grid: their last position and test count.
template <class Done>
__device__ __forceinline__ void march_away(const MarchPoolRec& P, int count, Done done) {
    for (int i = threadIdx.x & 31; i < count; i += 32) {
        const float4 a = P.a[P.away[i]], b = P.b[P.away[i]];
        f3 p = mk(a.x, a.y, a.z), s = mk(b.x, b.y, b.z), last = p;
        const uint32_t id = __float_as_uint(b.w);
        float d = 0.5f * (float)(id >> 8 & 0x1ffu), ds = march_step0(id);
        if (id & kMarchFine) {
            for (; d < 16.0f; d += ds) {
                last = p;
                p = add(p, s);
            }
            s = mul(s, 2.0f);
        }
        ds *= 2.0f;
        const float lim = a.w < 164.0f ? a.w : 164.0f, dcoarse = march_dcoarse(id);
        for (; d < lim; d += ds) {
            last = p;
            p = add(p, s);
        }
        const int coarse = (int)((d - dcoarse) / ds);
        done(id & kMarchRay, false, a.w, coarse == 0, last, ((id & kMarchSuper) ? 6 : 31) + coarse);
    }
}

// Both parts. The warp has written the pool's rays; those whose origin or
// direction is outside ray_domain_ok are left out by the caller (misses).
template <bool REC, int EDGE = 1, class Pool, class Done>
__device__ __forceinline__ void march_pool(const GridView& g, Pool& P, int count, Done done) {
    __syncwarp();
    int away = 0;
    const int kept = march_part<true, REC, EDGE>(g, P, count, away, done);
    march_part<false, REC, EDGE>(g, P, kept, away, done);
    if constexpr (REC) march_away(P, away, done);
}

// The first kMarchFirst tests of one ray per lane with `on` set (a quarter of
// the rays or more end there, and neighbours' first tests run alike), then
// the ray into the pool unless it has ended.
template <bool REC, int EDGE = 1, class Done>
__device__ __forceinline__ void march_push(const GridView& g, MarchPool& P, int& count, bool on, f3 o, f3 d,
                                           float dist, uint32_t id, Done done) {
    static_assert(kMarchFirst < 6, "the SuperSparse marcher's fine part is 6 tests");
    on = on && ray_domain_ok(o, d) && (REC || !march_gone(g, o, d));
    const float step0 = march_step0(id);
    const f3 s = mul(d, step0);
    f3 q = o;
    const unsigned lanes = __ballot_sync(0xffffffffu, on);
    if (on) {
        bool in = o.x >= 0.0f && o.y >= 0.0f && o.z >= 0.0f && march_inside(g, o), left = false;
        const unsigned hits = march_tests<true, kMarchFirst, EDGE>(lanes, g, o, s, q, in, march_small(s), left);
        if (hits) {
            const int k = __ffs(hits) - 1;
            f3 p = o;
            if (REC)
                for (int j = 0; j < k; j++) p = add(p, s);
            done(id & kMarchRay, true, step0 * (float)(k + 1), true, p, k + 1);
            on = false;
        } else if (!REC && left) {
            done(id & kMarchRay, false, dist, true, o, 0);
            on = false;
        }
    }
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (on) {
        const int at = count + __popc(m & march_lanes_below());
        P.a[at] = make_float4(q.x, q.y, q.z, dist);
        P.b[at] = make_float4(s.x, s.y, s.z, __uint_as_float(id));
    }
    count += __popc(m);
}

__device__ __forceinline__ Hit march_hit(bool hit, float t, bool fine, f3 last, int steps) {
    Hit h{0, 0, 0, t, steps, hit ? VXL_RF_HIT | (fine ? 0 : VXL_RF_COARSE) : 0};
    int v[3];
    if (fine)
        march_voxel<true>(last, v);
    else
        march_voxel<false>(last, v);
    h.vx = v[0];
    h.vy = v[1];
    h.vz = v[2];
    return h;
}

}  // namespace vxl
