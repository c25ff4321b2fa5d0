// trace.cu — occlusion tracing kernels: raw ray batches (DDA / Sparse /
// SuperSparse), the DDA-mode occlusion pass over a G-buffer, and the
// reference light passes (ambient, reflection, point/spot).
#include "march_pool.cuh"
#include "vxl_device.cuh"

namespace vxl {

// ------------------------------------------------------------ ray batches
// DDA rays with records. Independent rays end after very different step counts
// (one ray a thread kept 19% of the lanes busy on rays from random points), so
// a warp sets up 32 rays at a time in shared memory and its lanes take the next
// one as theirs end; when the 32 are gone it sets up the next 32 beside the
// rays still running. 1 M rays on a 384^3 grid: 415 -> 171 us (208 with pools
// of 128 that each drain before the next). Issue-bound, 30 iterations a ray.
constexpr int kRayBatch = 8;  // iterations between refills
struct RayPool {
    float4 a[32];  // cell (x, y as 16 bits each), t_max
    float4 b[32];  // cell z and signs, t_delta
    float maxt[32];
    int lane[32];  // of the ray in its 32
};

template <bool CACHE>
__global__ void __launch_bounds__(32 * kMarchWarps, kMarchBlocks)
    k_trace_rays(const __grid_constant__ GridView g, const float* __restrict__ rays, int64_t n,
                 vxl_ray_record* __restrict__ rec) {
    __shared__ RayPool pools[kMarchWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    RayPool& P = pools[warp];
    int64_t next = ((int64_t)blockIdx.x * kMarchWarps + warp) * 32;  // first ray of the next 32
    int64_t first = 0, id = 0;                                       // of the pool's 32; this lane's ray
    int count = 0, base = 0;
    DState s;
    s.leap = false;
    bool busy = false;
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !busy);
        if (base == count && next < n) {
            const int64_t i = next + lane;
            bool on = i < n;
            DState t;
            if (on) {
                const float* q = rays + 7 * i;
                const f3 o = mk(q[0], q[1], q[2]), d = mk(q[3], q[4], q[5]);
                if (ray_domain_ok(o, d) && dir_fast_ok(d)) {
                    dda_init(t, o, d, q[6]);
                    if ((unsigned)t.cx > g.ux || (unsigned)t.cy > g.uy || (unsigned)t.cz > g.uz) {
                        // the first bounds test ends it
                        store_record(rec + i, Hit{t.cx, t.cy, t.cz, 0.0f, 0, VXL_RF_EXIT_BOUNDS});
                        on = false;
                    }
                } else {
                    store_record(rec + i, dda(g, o, d, q[6]));  // a miss, or the literal form
                    on = false;
                }
            }
            const unsigned m = __ballot_sync(0xffffffffu, on);
            if (on) {
                const int at = __popc(m & march_lanes_below());
                const int sg = (t.sx < 0 ? 1 : 0) | (t.sy < 0 ? 2 : 0) | (t.sz < 0 ? 4 : 0);
                P.a[at] = make_float4(__int_as_float(t.cx | (t.cy << 16)), t.tx, t.ty, t.tz);
                P.b[at] = make_float4(__int_as_float(t.cz | (sg << 16)), t.tdx, t.tdy, t.tdz);
                P.maxt[at] = t.maxt;
                P.lane[at] = lane;
            }
            first = next;
            next += (int64_t)gridDim.x * kMarchWarps * 32;
            base = 0;
            count = __popc(m);
            __syncwarp();
        }
        if (base < count) {
            const int at = base + __popc(idle & march_lanes_below());
            if (!busy && at < count) {
                const float4 a = P.a[at], b = P.b[at];
                const int xy = __float_as_int(a.x), zs = __float_as_int(b.x);
                s.cx = xy & 0xffff;
                s.cy = (int)((unsigned)xy >> 16);
                s.cz = zs & 0xffff;
                s.sx = (zs & 0x10000) ? -1 : 1;
                s.sy = (zs & 0x20000) ? -1 : 1;
                s.sz = (zs & 0x40000) ? -1 : 1;
                s.tx = a.y;
                s.ty = a.z;
                s.tz = a.w;
                s.tdx = b.y;
                s.tdy = b.z;
                s.tdz = b.w;
                s.maxt = P.maxt[at];
                s.tot = 0.0f;
                s.n = 0;
                s.wcur = 0xffffffffu;
                id = first + P.lane[at];
                busy = true;
            }
            base = min(base + __popc(idle), count);
            __syncwarp();  // the slots are read before the next 32 rays are written
        } else if (idle == 0xffffffffu && next >= n) {
            break;
        }
        const unsigned running = __ballot_sync(0xffffffffu, busy);
        if (busy) {
            Hit h;
            if (dda_run<false, CACHE, !CACHE, true>(g, s, h, kRayBatch, running)) {
                store_record(rec + id, h);
                busy = false;
            }
        }
    }
}

// SuperSparse rays with records, one a thread: at most 29 tests a ray leave a
// pool nothing to gain (400,000 rays from random points: 29 us, pooled 36).
__global__ void __launch_bounds__(128) k_super_rays(GridView g, const float* __restrict__ rays, int64_t n,
                                                    vxl_ray_record* __restrict__ rec) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float* q = rays + 7 * i;
        store_record(rec + i, march(g, mk(q[0], q[1], q[2]), mk(q[3], q[4], q[5]), q[6], 2.5f));
    }
}

// Sparse rays with records: `tile` rays (a multiple of 32) per warp. 1 M rays
// from random points 133 us (246 one ray a thread). An image's rays, which run
// alike, gain nothing from a pool: 1 M of one view 185 us, 161 one a thread.
__global__ void __launch_bounds__(32 * kMarchWarps, kMarchBlocks) k_march_rays(const __grid_constant__ GridView g,
                                                                    const float* __restrict__ rays, int64_t n, int tile,
                                                                    vxl_ray_record* __restrict__ rec) {
    __shared__ MarchPoolRec pools[kMarchWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t at = ((int64_t)blockIdx.x * kMarchWarps + warp) * tile;
    MarchPoolRec& P = pools[warp];
    auto done = [&](uint32_t id, bool hit, float t, bool fine, f3 last, int steps) {
        store_record(rec + at + id, march_hit(hit, t, fine, last, steps));
    };
    int count = 0;
    for (int k = lane; k < tile; k += 32) {
        const int64_t i = at + k;
        f3 o = mk(0.0f, 0.0f, 0.0f), d = o;
        float dist = 0.0f;
        if (i < n) {
            const float* q = rays + 7 * i;
            o = mk(q[0], q[1], q[2]);
            d = mk(q[3], q[4], q[5]);
            dist = q[6];
            if (!ray_domain_ok(o, d)) store_record(rec + i, Hit{0, 0, 0, dist, 0, 0});
        }
        march_push<true, 2>(g, P, count, i < n, o, d, dist, (uint32_t)k, done);
    }
    march_pool<true, 2>(g, P, count, done);
}

// ------------------------------------------------------ DDA-mode occlusion
struct TraceConsts {
    f3 light;
    f3 cam;
    float bias, shadow_len, ao_len, spec_len, default_rough;
    int n_shadow, n_ao, n_spec;
    uint32_t seed_h;
};

// One thread per pixel; rays of a pixel in the order shadow, AO 0..n-1,
// spec 0..n-1. Same ray generation as the oracle's occlusion_pixel.
template <bool RECORDS>
__global__ void __launch_bounds__(128) k_occlusion(GridView g, const float* __restrict__ pos,
                                                   const float* __restrict__ nrm, const float* __restrict__ rough,
                                                   int64_t npix, TraceConsts c, float* __restrict__ o_shadow,
                                                   float* __restrict__ o_ao, float* __restrict__ o_vis,
                                                   float* __restrict__ o_spec, float* __restrict__ o_spec_t,
                                                   vxl_ray_record* __restrict__ rec) {
    const int R = c.n_shadow + c.n_ao + c.n_spec;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < npix;
         i += (int64_t)gridDim.x * blockDim.x) {
        f3 P = ld3(pos + 3 * i), N = ld3(nrm + 3 * i);
        float sh = 1.0f, ao = 1.0f, vis = 1.0f, sp = 1.0f, st = c.spec_len;
        if (!(N.x == 0.0f && N.y == 0.0f && N.z == 0.0f)) {
            f3 O = add(P, mul(N, c.bias));
            int slot = 0;
            if (c.n_shadow > 0) {
                Hit h = dda(g, O, c.light, c.shadow_len);
                sh = (h.flags & VXL_RF_HIT) ? 0.0f : 1.0f;
                if (RECORDS) store_record(rec + i * R + slot, h);
                slot++;
            }
            f3 T, B;
            tangent_frame(N, &T, &B);
            float acc = 0.0f, v = 0.0f;
            for (int k = 0; k < c.n_ao; k++) {
                float u1 = rand01(c.seed_h, (uint32_t)i, 64u + 2u * k);
                float u2 = rand01(c.seed_h, (uint32_t)i, 65u + 2u * k);
                f3 d = frame_dir(T, B, N, cosine_sample(u1, u2));
                Hit h = dda(g, O, d, c.ao_len);
                bool hit = h.flags & VXL_RF_HIT;
                float tt = hit ? (h.t < c.ao_len ? h.t : c.ao_len) : c.ao_len;
                float q = tt / c.ao_len;
                acc += q * q;
                v += hit ? 0.0f : 1.0f;
                if (RECORDS) store_record(rec + i * R + slot, h);
                slot++;
            }
            if (c.n_ao > 0) {
                ao = acc / (float)c.n_ao;
                vis = v / (float)c.n_ao;
            }
            if (c.n_spec > 0) {
                float ro = rough ? rough[i] : c.default_rough;
                float a = ro * ro;
                float a2 = a * a;
                f3 V = normalize(sub(c.cam, P));
                float spa = 0.0f, sta = 0.0f;
                for (int j = 0; j < c.n_spec; j++) {
                    float u1 = rand01(c.seed_h, (uint32_t)i, 2u * j);
                    float u2 = rand01(c.seed_h, (uint32_t)i, 2u * j + 1u);
                    float ct = sqrtf((1.0f - u1) / (1.0f + (a2 - 1.0f) * u1));
                    float st2 = 1.0f - ct * ct;
                    float sn = sqrtf(st2 > 0.0f ? st2 : 0.0f);
                    float s, cs;
                    sincos_own(6.2831855f * u2, &s, &cs);
                    f3 H = frame_dir(T, B, N, mk(sn * cs, sn * s, ct));
                    float vh = dot(V, H);
                    f3 d = normalize(sub(mul(H, 2.0f * vh), V));
                    Hit h = dda(g, O, d, c.spec_len);
                    bool hit = h.flags & VXL_RF_HIT;
                    spa += hit ? 0.0f : 1.0f;
                    sta += hit ? h.t : c.spec_len;
                    if (RECORDS) store_record(rec + i * R + slot, h);
                    slot++;
                }
                sp = spa / (float)c.n_spec;
                st = sta / (float)c.n_spec;
            }
        } else if (RECORDS) {
            Hit z{0, 0, 0, 0.0f, 0, 0};
            for (int k = 0; k < R; k++) store_record(rec + i * R + k, z);
        }
        if (o_shadow) o_shadow[i] = sh;
        if (o_ao) o_ao[i] = ao;
        if (o_vis) o_vis[i] = vis;
        if (o_spec) o_spec[i] = sp;
        if (o_spec_t) o_spec_t[i] = st;
    }
}

// -------------------------------------------------- reference light passes
// LightAmbient.frag:148-173: two rays a pixel, `tile` pixels (a multiple of
// 32, two rays each in the pool) per warp.
template <bool REC>
__global__ void __launch_bounds__(32 * kMarchWarps, kMarchBlocks)
    k_light_ambient(const __grid_constant__ GridView g, const float* __restrict__ wcp_in, const float* __restrict__ nrm,
                    const float* __restrict__ depth, const float4* __restrict__ noise, int64_t npix, f3 sun, int tile,
                    float* __restrict__ shadow, float* __restrict__ irr, vxl_ray_record* __restrict__ rec) {
    using Pool = std::conditional_t<REC, MarchPoolRec, MarchPool>;
    __shared__ Pool pools[kMarchWarps];
    __shared__ float res[kMarchWarps][kMarchRays];  // t of ray 2 * pixel + {0: sun, 1: hemisphere}
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t at = ((int64_t)blockIdx.x * kMarchWarps + warp) * tile;
    Pool& P = pools[warp];
    float* rt = res[warp];
    auto done = [&](uint32_t id, bool hit, float t, bool fine, f3 last, int steps) {
        if (hit) rt[id] = t;
        if (REC) store_record(rec + 2 * at + id, march_hit(hit, t, fine, last, steps));
    };
    int count = 0;
    for (int k = lane; k < tile; k += 32) {
        const int64_t i = at + k;
        f3 o = mk(0.0f, 0.0f, 0.0f), wd = o, dir = o;
        if (i < npix) {
            float4 nz = noise[i];
            f3 normal = ld3(nrm + 3 * i);
            f3 wcp = ld3(wcp_in + 3 * i);
            const f3 cosv = cosine_sample(nz.x, nz.y);
            f3 randomVec = mul(cosv, 0.1f);
            randomVec.z *= glsl_sign(nz.z - 0.5f);
            wd = normalize(mix(sun, randomVec, 0.5f));
            wcp = add(wcp, mul(wd, nz.w * 1.0f));
            wcp = add(wcp, mul(randomVec, 2.5f));
            float bias = smoothstep(0.0f, 0.2f, depth[i]) * 50.0f + 1.5f;
            o = add(wcp, mul(normal, bias));
            f3 T, B;
            tangent_frame(normal, &T, &B);
            dir = frame_dir(T, B, normal, cosv);
            rt[2 * k] = rt[2 * k + 1] = 128.0f;
            if (REC) {
                if (!ray_domain_ok(o, wd)) store_record(rec + 2 * i, Hit{0, 0, 0, 128.0f, 0, 0});
                if (!ray_domain_ok(o, dir)) store_record(rec + 2 * i + 1, Hit{0, 0, 0, 128.0f, 0, 0});
            }
        }
        march_push<REC>(g, P, count, i < npix, o, wd, 128.0f, 2u * k, done);
        march_push<REC>(g, P, count, i < npix, o, dir, 128.0f, (2u * k + 1u) | kMarchSuper, done);
    }
    march_pool<REC>(g, P, count, done);
    __syncwarp();
    for (int k = lane; k < tile; k += 32) {
        const int64_t i = at + k;
        if (i >= npix) break;
        shadow[i] = (rt[2 * k] != 128.0f) ? 0.0f : 1.0f;
        float dd = rt[2 * k + 1] / 128.0f;
        irr[i] = dd * dd * 0.05f;
    }
}

// LightReflection.frag:92-113, `tile` pixels (a multiple of 32) per warp
template <bool REC>
__global__ void __launch_bounds__(32 * kMarchWarps, kMarchBlocks)
    k_light_reflection(const __grid_constant__ GridView g, const float* __restrict__ wcp_in,
                       const float* __restrict__ nrm, const float* __restrict__ view_r,
                       const float* __restrict__ rough, const float4* __restrict__ noise, int64_t npix, int tile,
                       float* __restrict__ t_out, vxl_ray_record* __restrict__ rec) {
    using Pool = std::conditional_t<REC, MarchPoolRec, MarchPool>;
    __shared__ Pool pools[kMarchWarps];
    __shared__ float res[kMarchWarps][kMarchRays];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t at = ((int64_t)blockIdx.x * kMarchWarps + warp) * tile;
    Pool& P = pools[warp];
    float* rt = res[warp];
    auto done = [&](uint32_t id, bool hit, float t, bool fine, f3 last, int steps) {
        if (hit) rt[id] = t;
        if (REC) store_record(rec + at + id, march_hit(hit, t, fine, last, steps));
    };
    int count = 0;
    for (int k = lane; k < tile; k += 32) {
        const int64_t i = at + k;
        f3 o = mk(0.0f, 0.0f, 0.0f), wd = o;
        if (i < npix) {
            float4 nz = noise[i];
            f3 normal = ld3(nrm + 3 * i);
            wd = normalize(ld3(view_r + 3 * i));
            f3 wcp = ld3(wcp_in + 3 * i);
            f3 randomVec = cosine_sample(nz.x, nz.y);
            randomVec.z *= glsl_sign(nz.z - 0.5f);
            wd = mix(wd, randomVec, rough[i] * 0.1f);
            wcp = add(wcp, mul(normal, nz.w));
            wd = mul(wd, 1.0f + nz.w * 0.5f);
            o = add(wcp, normal);
            rt[k] = 256.0f;
            if (REC && !ray_domain_ok(o, wd)) store_record(rec + i, Hit{0, 0, 0, 256.0f, 0, 0});
        }
        march_push<REC>(g, P, count, i < npix, o, wd, 256.0f, (uint32_t)k, done);
    }
    march_pool<REC>(g, P, count, done);
    __syncwarp();
    for (int k = lane; k < tile; k += 32)
        if (at + k < npix) t_out[at + k] = rt[k];
}

// LightPoint.frag:234-267 (spot = 0), LightSpot.frag:83-117 (spot = 1)
__global__ void k_light_point(GridView g, const float* __restrict__ wpos, const float* __restrict__ nrm,
                              const float4* __restrict__ noise, int64_t npix, f3 L, float range, int spot,
                              float* __restrict__ shadow, vxl_ray_record* __restrict__ rec) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < npix;
         i += (int64_t)gridDim.x * blockDim.x) {
        float4 nz = noise[i];
        f3 worldPos = ld3(wpos + 3 * i);
        f3 normal = ld3(nrm + 3 * i);
        f3 lightDir = sub(L, worldPos);
        float lightDistance = sqrtf(dot(lightDir, lightDir));
        if (lightDistance > range) {  // discard: output untouched
            if (rec) {
                Hit z{0, 0, 0, -1.0f, 0, 0};
                store_record(rec + i, z);
            }
            continue;
        }
        f3 wd;
        float hitDist;
        if (spot) {
            wd = mul(normalize(lightDir), 10.0f);
            hitDist = lightDistance * 10.0f;
        } else {
            wd = lightDir;
            hitDist = lightDistance * 10.5f;
        }
        f3 wcp = mul(worldPos, 10.0f);
        f3 randomVec = mul(cosine_sample(nz.x, nz.y), 0.1f);
        randomVec.z *= glsl_sign(nz.z - 0.5f);
        wd = normalize(mix(wd, randomVec, 0.5f));
        wcp = add(wcp, mul(wd, nz.w * 1.0f));
        wcp = add(wcp, mul(randomVec, 2.5f));
        Hit h = march(g, add(wcp, mul(normal, 0.5f)), wd, hitDist, spot ? 2.5f : 0.5f);
        shadow[i] = (h.t < hitDist) ? 0.0f : 1.0f;
        if (rec) store_record(rec + i, h);
    }
}

// Fused point / spot shadows for up to 64 lights (vxl_light_points): a light
// grid narrows each pixel's candidate lights, pass 1 runs the exact range
// tests and lists the pairs in range, pass 2 traces each listed pair's ray --
// the one k_light_point traces for that light alone -- and sets its bit in the
// pixel's 64-bit mask.
struct LightDev {
    f3 pos;
    float range;
    int spot;
};
struct LightTable {
    LightDev l[64];
    int n;
};

// The shadow ray of one (pixel, light) pair in range, as vxl_light_point traces
// it (LightPoint.frag:105-129, LightSpot.frag:93-117): origin, direction and
// length; step 2.5 for a spot light, 0.5 for a point light.
__device__ __forceinline__ void light_pair_ray(f3 worldPos, f3 normal, float4 nz, const LightDev& Lt, f3 lightDir,
                                               float lightDistance, f3* o, f3* dir, float* hitDist) {
    f3 wd;
    if (Lt.spot) {
        wd = mul(normalize(lightDir), 10.0f);
        *hitDist = lightDistance * 10.0f;
    } else {
        wd = lightDir;
        *hitDist = lightDistance * 10.5f;
    }
    f3 wcp = mul(worldPos, 10.0f);
    f3 randomVec = mul(cosine_sample(nz.x, nz.y), 0.1f);
    randomVec.z *= glsl_sign(nz.z - 0.5f);
    wd = normalize(mix(wd, randomVec, 0.5f));
    wcp = add(wcp, mul(wd, nz.w * 1.0f));
    wcp = add(wcp, mul(randomVec, 2.5f));
    *o = add(wcp, mul(normal, 0.5f));
    *dir = wd;
}
// true when the pair is unshadowed
__device__ __forceinline__ bool light_pair_lit(const GridView& g, f3 worldPos, f3 normal, float4 nz, const LightDev& Lt,
                                               f3 lightDir, float lightDistance) {
    f3 o, wd;
    float hitDist;
    light_pair_ray(worldPos, normal, nz, Lt, lightDir, lightDistance, &o, &wd, &hitDist);
    const Hit h = march(g, o, wd, hitDist, Lt.spot ? 2.5f : 0.5f);
    return !(h.t < hitDist);
}

// Light grid of the fused lights: kLightCells^3 cells over the box that holds
// every light's sphere; each cell keeps the mask of lights whose sphere, grown
// by a margin, touches the cell grown by a margin, so a pixel needs the exact
// range test for its cell's lights only (a pixel outside the box is in range
// of none). The margins cover the fp32 rounding of the cell index and of the
// box distance.
constexpr int kLightCells = 32;
struct LightGrid {
    f3 lo;         // box corner
    float cell;    // cell edge
    float inv;     // 1 / cell
    float slack;   // absolute margin: a few ulps of the largest light coordinate
    int on;        // 0: every pixel tests every light
};

__global__ void k_light_grid(const __grid_constant__ LightTable T, LightGrid LG, unsigned long long* __restrict__ masks) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= kLightCells * kLightCells * kLightCells) return;
    const int cx = c % kLightCells, cy = (c / kLightCells) % kLightCells, cz = c / (kLightCells * kLightCells);
    const float m = LG.cell * 0.01f + LG.slack;
    const f3 a = mk(LG.lo.x + (float)cx * LG.cell - m, LG.lo.y + (float)cy * LG.cell - m,
                    LG.lo.z + (float)cz * LG.cell - m);
    const f3 b = mk(a.x + LG.cell + 2.0f * m, a.y + LG.cell + 2.0f * m, a.z + LG.cell + 2.0f * m);
    unsigned long long mask = 0ull;
    for (int l = 0; l < T.n; l++) {
        const LightDev& Lt = T.l[l];
        const float dx = fmaxf(fmaxf(a.x - Lt.pos.x, Lt.pos.x - b.x), 0.0f);
        const float dy = fmaxf(fmaxf(a.y - Lt.pos.y, Lt.pos.y - b.y), 0.0f);
        const float dz = fmaxf(fmaxf(a.z - Lt.pos.z, Lt.pos.z - b.z), 0.0f);
        const float r = fabsf(Lt.range) * 1.0001f + 1e-4f;
        if (!(dx * dx + dy * dy + dz * dz > r * r)) mask |= 1ull << l;
    }
    masks[c] = mask;
}

// Pass 1 of the fused lights: one thread per pixel. The pixel's candidate
// lights come from the light grid (all lights for a NaN position or without a
// grid); the exact per-pixel range test of each candidate sets the in-range
// mask. Pairs in range are appended to a list (one atomic per warp) for pass 2,
// which traces them with full warps; pairs past the list's capacity are traced
// here.
__global__ void __launch_bounds__(256) k_light_points(GridView g, const float* __restrict__ wpos,
                                                      const float* __restrict__ nrm, const float4* __restrict__ noise,
                                                      int64_t npix, const __grid_constant__ LightTable T, LightGrid LG,
                                                      const unsigned long long* __restrict__ masks,
                                                      unsigned long long* __restrict__ lit,
                                                      unsigned long long* __restrict__ in_range,
                                                      unsigned long long* __restrict__ pairs,
                                                      unsigned long long* __restrict__ npairs, uint64_t cap) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned long long all = T.n >= 64 ? ~0ull : ((1ull << T.n) - 1ull);
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < npix; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = base + threadIdx.x;
        const bool valid = i < npix;
        const f3 worldPos = valid ? ld3(wpos + 3 * i) : mk(0.0f, 0.0f, 0.0f);
        unsigned long long cand = 0ull;
        if (valid) {
            cand = all;
            const bool nan_pos = worldPos.x != worldPos.x || worldPos.y != worldPos.y || worldPos.z != worldPos.z;
            if (LG.on && !nan_pos) {
                const float fx = floorf((worldPos.x - LG.lo.x) * LG.inv), fy = floorf((worldPos.y - LG.lo.y) * LG.inv),
                            fz = floorf((worldPos.z - LG.lo.z) * LG.inv);
                const float top = (float)kLightCells;
                if (fx >= 0.0f && fy >= 0.0f && fz >= 0.0f && fx < top && fy < top && fz < top)
                    cand = masks[((int)fz * kLightCells + (int)fy) * kLightCells + (int)fx];
                else
                    cand = 0ull;  // outside every light's sphere
            }
        }
        unsigned long long inr = 0ull;
        for (unsigned long long c = cand; c; c &= c - 1ull) {
            const int l = __ffsll((long long)c) - 1;
            const LightDev& Lt = T.l[l];
            const f3 lightDir = sub(Lt.pos, worldPos);
            const float lightDistance = sqrtf(dot(lightDir, lightDir));
            if (!(lightDistance > Lt.range)) inr |= 1ull << l;  // else the light's pass discards this pixel
        }
        // one list slot per pair in range: warp prefix sum, one atomic per warp
        const int cnt = __popcll(inr);
        int pre = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(full, pre, o);
            if (lane >= o) pre += y;
        }
        const int total = __shfl_sync(full, pre, 31);
        unsigned long long at0 = 0ull;
        if (lane == 0 && total > 0) at0 = atomicAdd(npairs, (unsigned long long)total);
        at0 = __shfl_sync(full, at0, 0) + (unsigned long long)(pre - cnt);
        unsigned long long litm = 0ull;
        for (unsigned long long c = inr; c; c &= c - 1ull, at0++) {
            const int l = __ffsll((long long)c) - 1;
            if (at0 < cap) {
                pairs[at0] = ((unsigned long long)i << 6) | (unsigned long long)l;
            } else {
                const LightDev& Lt = T.l[l];
                const f3 lightDir = sub(Lt.pos, worldPos);
                const float lightDistance = sqrtf(dot(lightDir, lightDir));
                if (light_pair_lit(g, worldPos, ld3(nrm + 3 * i), noise[i], Lt, lightDir, lightDistance))
                    litm |= 1ull << l;
            }
        }
        if (valid) {
            lit[i] = litm;
            if (in_range) in_range[i] = inr;
        }
    }
}

// Pass 2: the listed (pixel, light) pairs, up to kMarchRays per pool. The
// list's length is known on the device only: few pairs are spread over all
// warps of the launch in pools of 32 or 64.
__global__ void __launch_bounds__(32 * kMarchWarps, kMarchBlocks)
    k_light_pairs(const __grid_constant__ GridView g, const float* __restrict__ wpos, const float* __restrict__ nrm,
                  const float4* __restrict__ noise, const __grid_constant__ LightTable T,
                  const unsigned long long* __restrict__ pairs, const unsigned long long* __restrict__ npairs,
                  uint64_t cap, unsigned long long* __restrict__ lit) {
    __shared__ MarchPool pools[kMarchWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    MarchPool& P = pools[warp];
    const unsigned long long n = *npairs < cap ? *npairs : cap;
    const unsigned long long warps = (unsigned long long)gridDim.x * kMarchWarps;
    int tile = kMarchRays;
    while (tile > 32 && n < warps * tile) tile >>= 1;
    for (unsigned long long at = ((unsigned long long)blockIdx.x * kMarchWarps + warp) * tile; at < n;
         at += warps * tile) {
        auto done = [&](uint32_t id, bool hit, float t, bool, f3, int) {
            // a hit can lie at or beyond a short hitDist: the fine part always runs to 16
            const unsigned long long pr = pairs[at + id];
            const int64_t i = (int64_t)(pr >> 6);
            const LightDev& Lt = T.l[(int)(pr & 63ull)];
            if (hit) {
                const f3 lightDir = sub(Lt.pos, ld3(wpos + 3 * i));
                const float lightDistance = sqrtf(dot(lightDir, lightDir));
                if (t < lightDistance * (Lt.spot ? 10.0f : 10.5f)) return;
            }
            atomicOr(lit + i, 1ull << (pr & 63ull));
        };
        int count = 0;
        for (int k = lane; k < tile; k += 32) {
            const bool on = at + k < n;
            f3 o = mk(0.0f, 0.0f, 0.0f), wd = o;
            float hitDist = 0.0f;
            uint32_t id = (uint32_t)k;
            if (on) {
                const unsigned long long pr = pairs[at + k];
                const int64_t i = (int64_t)(pr >> 6);
                const LightDev& Lt = T.l[(int)(pr & 63ull)];
                const f3 worldPos = ld3(wpos + 3 * i);
                const f3 lightDir = sub(Lt.pos, worldPos);
                light_pair_ray(worldPos, ld3(nrm + 3 * i), noise[i], Lt, lightDir, sqrtf(dot(lightDir, lightDir)), &o,
                               &wd, &hitDist);
                if (Lt.spot) id |= kMarchSuper;
                // not marched (march_push): t = hitDist, unshadowed
                if (!ray_domain_ok(o, wd) || march_gone(g, o, wd)) atomicOr(lit + i, 1ull << (pr & 63ull));
            }
            march_push<false>(g, P, count, on, o, wd, hitDist, id, done);
        }
        march_pool<false>(g, P, count, done);
    }
}

// ---------------------------------------------------------------- launchers
static unsigned grid_blocks(vxl_ctx* ctx, int64_t n, int threads, int per_sm) {
    int64_t need = (n + threads - 1) / threads;
    int64_t cap = (int64_t)ctx->sm_count * per_sm;
    if (need > cap) need = cap;
    if (need < 1) need = 1;
    return (unsigned)need;
}

// Pixels (or rays) of a march kernel's warp: as many as its pool holds, fewer
// (down to 32) while that would leave the GPU's warps without work: a pool's
// lanes are busier the more rays it holds, but a call of few rays waits for
// its slowest warp.
static int march_tile(const vxl_ctx* ctx, int64_t n, int rays_each) {
    int tile = kMarchRays / rays_each;
    while (tile > 32 && n < (int64_t)ctx->sm_count * kMarchBlocks * kMarchWarps * tile) tile >>= 1;
    return tile;
}
static unsigned march_blocks(int64_t n, int tile) {
    return (unsigned)((n + (int64_t)tile * kMarchWarps - 1) / ((int64_t)tile * kMarchWarps));
}

vxl_status launch_trace_rays(vxl_ctx* ctx, const vxl_grid* g, const float* rays, int64_t n, int mode,
                             vxl_ray_record* rec, cudaStream_t s) {
    if (n <= 0) return VXL_OK;
    GridView v = view_of(g);
    if (mode == VXL_MODE_DDA) {
        // grids beyond 64 MiB of words keep the brick in registers, as the occlusion pool does
        const unsigned b = (unsigned)std::min<int64_t>(march_blocks(n, 32), (int64_t)ctx->sm_count * kMarchBlocks);
        (g->nwords > (8ull << 20) ? k_trace_rays<true> : k_trace_rays<false>)<<<b, 32 * kMarchWarps, 0, s>>>(v, rays, n, rec);
    } else if (mode == VXL_MODE_SPARSE) {
        const int tile = march_tile(ctx, n, 1);
        k_march_rays<<<march_blocks(n, tile), 32 * kMarchWarps, 0, s>>>(v, rays, n, tile, rec);
    } else {
        k_super_rays<<<grid_blocks(ctx, n, 128, 16), 128, 0, s>>>(v, rays, n, rec);
    }
    ctx->launches++;
    VXL_TRY_CUDA(cudaGetLastError());
    return VXL_OK;
}

vxl_status launch_trace_occlusion(vxl_ctx* ctx, const vxl_grid* g, const vxl_gbuffer* gb, const vxl_trace_params* p,
                                  const vxl_outputs* out, cudaStream_t s) {
    if (gb->npix <= 0) return VXL_OK;
    if (occl_pool_supported(g, p)) {
        unsigned long long* counter = nullptr;
        VXL_TRY(ctx_take_counter(ctx, s, &counter));
        return launch_trace_occlusion_pool(ctx, g, gb, p, out, counter, ctx->tune, s);
    }
    GridView v = view_of(g);
    TraceConsts c;
    c.light = mk(p->light_dir[0], p->light_dir[1], p->light_dir[2]);
    c.cam = mk(p->cam_pos[0], p->cam_pos[1], p->cam_pos[2]);
    c.bias = p->bias;
    c.shadow_len = p->shadow_len;
    c.ao_len = p->ao_len;
    c.spec_len = p->spec_len;
    c.default_rough = p->default_rough;
    c.n_shadow = p->n_shadow;
    c.n_ao = p->n_ao;
    c.n_spec = p->n_spec;
    c.seed_h = pcg(p->seed);
    unsigned b = grid_blocks(ctx, gb->npix, 128, 16);
    if (out->records)
        k_occlusion<true><<<b, 128, 0, s>>>(v, gb->pos, gb->nrm, gb->rough, gb->npix, c, out->shadow, out->ao,
                                            out->ao_vis, out->spec, out->spec_t, out->records);
    else
        k_occlusion<false><<<b, 128, 0, s>>>(v, gb->pos, gb->nrm, gb->rough, gb->npix, c, out->shadow, out->ao,
                                             out->ao_vis, out->spec, out->spec_t, nullptr);
    ctx->launches++;
    VXL_TRY_CUDA(cudaGetLastError());
    return VXL_OK;
}

// SUN_DIR = normalize(vec3(0.3,0.4,0.5)) (LightAmbient.frag:15), glm's form
static f3 sun_dir() {
    float x = 0.3f, y = 0.4f, z = 0.5f;
    float d = x * x + y * y;
    d = d + z * z;
    float r = 1.0f / sqrtf(d);
    return mk(x * r, y * r, z * r);
}

vxl_status launch_light_ambient(vxl_ctx* ctx, const vxl_grid* g, const float* wcp, const float* nrm,
                                const float* depth, const float* noise, int64_t npix, float* shadow, float* irr,
                                vxl_ray_record* rec, cudaStream_t s) {
    if (npix <= 0) return VXL_OK;
    GridView v = view_of(g);
    const int tile = march_tile(ctx, npix, 2);
    (rec ? k_light_ambient<true> : k_light_ambient<false>)<<<march_blocks(npix, tile), 32 * kMarchWarps, 0, s>>>(
        v, wcp, nrm, depth, (const float4*)noise, npix, sun_dir(), tile, shadow, irr, rec);
    ctx->launches++;
    VXL_TRY_CUDA(cudaGetLastError());
    return VXL_OK;
}

vxl_status launch_light_reflection(vxl_ctx* ctx, const vxl_grid* g, const float* wcp, const float* nrm,
                                   const float* view_r, const float* rough, const float* noise, int64_t npix,
                                   float* t, vxl_ray_record* rec, cudaStream_t s) {
    if (npix <= 0) return VXL_OK;
    GridView v = view_of(g);
    const int tile = march_tile(ctx, npix, 1);
    (rec ? k_light_reflection<true> : k_light_reflection<false>)<<<march_blocks(npix, tile), 32 * kMarchWarps, 0, s>>>(
        v, wcp, nrm, view_r, rough, (const float4*)noise, npix, tile, t, rec);
    ctx->launches++;
    VXL_TRY_CUDA(cudaGetLastError());
    return VXL_OK;
}

vxl_status launch_light_point(vxl_ctx* ctx, const vxl_grid* g, const float* wpos, const float* nrm,
                              const float* noise, int64_t npix, const float lp[3], float range, int spot,
                              float* shadow, vxl_ray_record* rec, cudaStream_t s) {
    if (npix <= 0) return VXL_OK;
    GridView v = view_of(g);
    k_light_point<<<grid_blocks(ctx, npix, 128, 16), 128, 0, s>>>(v, wpos, nrm, (const float4*)noise, npix,
                                                                  mk(lp[0], lp[1], lp[2]), range, spot, shadow, rec);
    ctx->launches++;
    VXL_TRY_CUDA(cudaGetLastError());
    return VXL_OK;
}

vxl_status launch_light_points(vxl_ctx* ctx, const vxl_grid* g, const float* wpos, const float* nrm,
                               const float* noise, int64_t npix, const vxl_light* lights, int nlights,
                               unsigned long long* lit, unsigned long long* in_range, cudaStream_t s) {
    if (npix <= 0) return VXL_OK;
    LightTable T;
    T.n = nlights > 0 ? nlights : 0;
    for (int l = 0; l < T.n; l++) {
        T.l[l].pos = mk(lights[l].pos[0], lights[l].pos[1], lights[l].pos[2]);
        T.l[l].range = lights[l].range;
        T.l[l].spot = lights[l].spot ? 1 : 0;
    }
    // light grid over the box of every light's sphere (off when a light's
    // position or range is not finite)
    constexpr int kCells = kLightCells * kLightCells * kLightCells;
    LightGrid LG{mk(0.0f, 0.0f, 0.0f), 1.0f, 1.0f, 0.0f, T.n > 0 ? 1 : 0};
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY}, maxabs = 0.0f;
    for (int l = 0; l < T.n; l++) {
        const float r = std::fabs(lights[l].range);
        for (int a = 0; a < 3; a++) {
            if (!std::isfinite(lights[l].pos[a]) || !std::isfinite(r)) LG.on = 0;
            lo[a] = std::min(lo[a], lights[l].pos[a] - r);
            hi[a] = std::max(hi[a], lights[l].pos[a] + r);
            maxabs = std::max(maxabs, std::fabs(lights[l].pos[a]) + r);
        }
    }
    if (LG.on) {
        LG.slack = 1e-4f + maxabs * 4e-7f;
        float ext = 0.0f;
        for (int a = 0; a < 3; a++) ext = std::max(ext, hi[a] - lo[a]);
        ext = std::max(ext + 2.0f * LG.slack, 1e-3f) * 1.002f;
        LG.cell = ext / (float)kLightCells;
        LG.inv = 1.0f / LG.cell;
        LG.lo = mk(lo[0] - LG.slack - 0.001f * ext, lo[1] - LG.slack - 0.001f * ext, lo[2] - LG.slack - 0.001f * ext);
        if (!std::isfinite(LG.cell) || !std::isfinite(LG.inv) || !std::isfinite(maxabs)) LG.on = 0;
    }
    // pair list: two pairs per pixel (frames with more trace the rest in pass 1)
    const uint64_t cap = (uint64_t)std::max<int64_t>(2 * npix, 1 << 16);
    VXL_TRY(ctx_grow(&ctx->d_lpairs, &ctx->lpairs_bytes, (size_t)(cap + 1 + kCells) * sizeof(unsigned long long)));
    unsigned long long* npairs = (unsigned long long*)ctx->d_lpairs;
    unsigned long long* masks = npairs + 1;
    unsigned long long* pairs = masks + kCells;
    VXL_TRY_CUDA(cudaMemsetAsync(npairs, 0, sizeof(unsigned long long), s));
    GridView v = view_of(g);
    if (LG.on) {
        k_light_grid<<<(kCells + 255) / 256, 256, 0, s>>>(T, LG, masks);
        ctx->launches++;
    }
    const int64_t bx = std::min<int64_t>((npix + 255) / 256, (int64_t)ctx->sm_count * 8);
    k_light_points<<<(unsigned)bx, 256, 0, s>>>(v, wpos, nrm, (const float4*)noise, npix, T, LG, masks, lit, in_range,
                                                pairs, npairs, cap);
    ctx->launches++;
    VXL_TRY_CUDA(cudaGetLastError());
    if (T.n > 0) {
        k_light_pairs<<<(unsigned)ctx->sm_count * kMarchBlocks, 32 * kMarchWarps, 0, s>>>(v, wpos, nrm, (const float4*)noise, T, pairs, npairs,
                                                                  cap, lit);
        ctx->launches++;
        VXL_TRY_CUDA(cudaGetLastError());
    }
    return VXL_OK;
}

}  // namespace vxl
