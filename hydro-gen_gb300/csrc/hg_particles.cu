// Particle (droplet) erosion, src/erosion.cpp:132-156: movement
// (glsl/particle.glsl:64-136), erosion (glsl/particle_erosion.glsl:22-128),
// the thermal passes and smoothing with its particle branch
// (glsl/smoothing.glsl:22-103).
//
// The shader serialises the droplets' updates of a texel with a spinlock per
// texel, in whatever order the droplets win it.  Here the order is fixed and
// no thread waits on another:
//   k_pmove                        moves the droplets, counts their four corner
//                                  records per texel (a record's place in its
//                                  texel's bucket is what the count was) and
//                                  packs what a record reads of its droplet
//   k_palloc / k_pscatter          give each texel a bucket, and the texels to
//                                  lists by record count; keys into the buckets
//   k_papply                       each texel applies its records in
//                                  droplet-id order (a texel update needs only
//                                  the droplet's state from before the pass)
//                                  and stores what each corner left for the
//                                  droplet's sediment; a texel with up to 8
//                                  records sorts them in its thread's
//                                  registers, one with more across a warp's
//                                  lanes
//   k_pfinal                       each droplet replays its corners 0..3
// which is a sequential pass over droplets in id order, corners in order.
// Spawn positions come from Philox4x32-10 (counter: droplet id, step,
// 'part', 0; key: the rain seed), 24-bit uniforms; the shader's
// fract(1e4 sin(...)) hash of the frame time has no portable bits.
#include "hg_internal.h"

#include <algorithm>

namespace hg {

namespace {

constexpr int PB = 256;

__device__ __forceinline__ float fract_(float x) { return x - floorf(x); }
__device__ __forceinline__ bool inb(int n, int x, int y) { return x >= 0 && x < n && y >= 0 && y < n; }

// img_bilinear (glsl/img_interpolation.glsl:3-22) of a field, 0 outside
__device__ __forceinline__ float bilin(const float* f, int n, float sx, float sy) {
    const int ix = (int)sx, iy = (int)sy;
    const float fx = fract_(sx), fy = fract_(sy);
    auto t = [&](int xx, int yy) { return inb(n, xx, yy) ? f[(size_t)yy * n + xx] : 0.0f; };
    const float v1 = gmix(t(ix, iy), t(ix + 1, iy), fx);
    const float v2 = gmix(t(ix, iy + 1), t(ix + 1, iy + 1), fx);
    return gmix(v1, v2, fy);
}

// corner k of a droplet: texel (cx, cy) and the droplet's offset in its texel.
// A live droplet sits in (1, n - 2) on both axes (movement reverts steps that
// leave it), so the clamp only keeps a non-finite position's texels inside the map.
__device__ __forceinline__ void corner(float px, float py, int k, int n, int& cx, int& cy, float& ofx, float& ofy) {
    const int bx = min(max((int)(px * 1.0f), 0), n - 2), by = min(max((int)(py * 1.0f), 0), n - 2);
    ofx = fract_(px * 1.0f);
    ofy = fract_(py * 1.0f);
    cx = (k == 1 || k == 2) ? bx + 1 : bx;
    cy = (k >= 2) ? by + 1 : by;
}
__device__ __forceinline__ float corner_weight(float ofx, float ofy, int k) {
    const float wx = (k == 1 || k == 2) ? ofx : 1.0f - ofx;
    const float wy = (k >= 2) ? ofy : 1.0f - ofy;
    return wx * wy;
}

struct MoveArgs {
    StepConsts c;
    hg_erosion_settings es;
    Drops d;
    const float* rock;
    const float* dirt;
    const float* water;
    const float* mx;
    const float* my;
    uint32_t step1;
    uint32_t seed_lo, seed_hi;
    int should_rain;
    uint32_t* cnt;  // records per texel, zero before
    uint4* rank;    // per droplet: its records' places in their buckets
    float4* pack;   // per droplet, two: offset x (sign bit: kill), offset y, capacity, volume; sediments, velocity
};

// Terrain normal's height differences and the samples at (px, py), see k_pmove
struct Around {
    float rr, rg, lr, lg, br, bg, tr, tg, mx, my, water;
};
__device__ __forceinline__ Around look_around(const MoveArgs& a, int n, float px, float py) {
    Around o;
    o.rr = bilin(a.rock, n, px + 1.0f, py); o.rg = bilin(a.dirt, n, px + 1.0f, py);
    o.lr = bilin(a.rock, n, px - 1.0f, py); o.lg = bilin(a.dirt, n, px - 1.0f, py);
    o.br = bilin(a.rock, n, px, py - 1.0f); o.bg = bilin(a.dirt, n, px, py - 1.0f);
    o.tr = bilin(a.rock, n, px, py + 1.0f); o.tg = bilin(a.dirt, n, px, py + 1.0f);
    o.mx = bilin(a.mx, n, px, py);
    o.my = bilin(a.my, n, px, py);
    o.water = bilin(a.water, n, px, py);
    return o;
}
// The same from 16-byte loads.  A warp's droplets lie anywhere, so a load costs
// a cache line per lane whatever its width, and the kernel is bound by those:
// 44 loads of a texel each against about 20 of an aligned quad, of which a row's
// four neighbouring texels need one or two (n is a multiple of 8: rows are whole
// quads).  Needs the whole cross of texels inside the map.
// With the count (9 us by itself before) and the packing the launch takes 41 us
// (262144 droplets on 1024²), without them it took as long from single texels.
__device__ __forceinline__ Around look_around_quads(const MoveArgs& a, int n, float px, float py, int ix, int iy) {
    // texels first .. first + M - 1 of a row
    const int s1 = (ix - 1) & 3, q1 = (ix - 1) & ~3, s0 = ix & 3, q0 = ix & ~3;
    auto row4 = [&](const float* f, int y, float t[4]) {
        const float4* p = reinterpret_cast<const float4*>(f + (size_t)y * n + q1);
        const float4 u = __ldg(p);
        float4 v = u;
        if (s1) v = __ldg(p + 1);
        t[0] = s1 == 0 ? u.x : s1 == 1 ? u.y : s1 == 2 ? u.z : u.w;
        t[1] = s1 == 0 ? u.y : s1 == 1 ? u.z : s1 == 2 ? u.w : v.x;
        t[2] = s1 == 0 ? u.z : s1 == 1 ? u.w : s1 == 2 ? v.x : v.y;
        t[3] = s1 == 0 ? u.w : s1 == 1 ? v.x : s1 == 2 ? v.y : v.z;
    };
    auto row2 = [&](const float* f, int y, float t[2]) {
        const float4* p = reinterpret_cast<const float4*>(f + (size_t)y * n + q0);
        const float4 u = __ldg(p);
        float v = 0.0f;
        if (s0 == 3) v = __ldg(reinterpret_cast<const float*>(p + 1));
        t[0] = s0 == 0 ? u.x : s0 == 1 ? u.y : s0 == 2 ? u.z : u.w;
        t[1] = s0 == 0 ? u.y : s0 == 1 ? u.z : s0 == 2 ? u.w : v;
    };
    const float fx = fract_(px), fy = fract_(py), fr = fract_(px + 1.0f), fl = fract_(px - 1.0f),
                ft = fract_(py + 1.0f), fb = fract_(py - 1.0f);
    Around o;
    auto cross = [&](const float* f, float& r, float& l, float& b, float& t) {
        float c0[4], c1[4], dn[2], up[2];
        row4(f, iy, c0);
        row4(f, iy + 1, c1);
        row2(f, iy - 1, dn);
        row2(f, iy + 2, up);
        r = gmix(gmix(c0[2], c0[3], fr), gmix(c1[2], c1[3], fr), fy);
        l = gmix(gmix(c0[0], c0[1], fl), gmix(c1[0], c1[1], fl), fy);
        b = gmix(gmix(dn[0], dn[1], fx), gmix(c0[1], c0[2], fx), fb);
        t = gmix(gmix(c1[1], c1[2], fx), gmix(up[0], up[1], fx), ft);
    };
    cross(a.rock, o.rr, o.lr, o.br, o.tr);
    cross(a.dirt, o.rg, o.lg, o.bg, o.tg);
    auto here = [&](const float* f) {
        float c0[2], c1[2];
        row2(f, iy, c0);
        row2(f, iy + 1, c1);
        return gmix(gmix(c0[0], c0[1], fx), gmix(c1[0], c1[1], fx), fy);
    };
    o.mx = here(a.mx);
    o.my = here(a.my);
    o.water = here(a.water);
    return o;
}

__global__ void __launch_bounds__(PB, 4) k_pmove(const MoveArgs a) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= a.d.count) return;
    const int n = a.c.n;
    const float dt = a.es.d_t;
    uint32_t iters = a.d.iters[id];
    int kill = a.d.kill[id];
    if (iters == 0 && !a.should_rain) return;
    float px = a.d.px[id], py = a.d.py[id], vx = a.d.vx[id], vy = a.d.vy[id], vol = a.d.vol[id];
    float s0 = a.d.s0[id], s1 = a.d.s1[id], sc = a.d.sc[id];
    if (s0 < 0.0f || iters == 0) s0 = 0.0f;
    if (s1 < 0.0f || iters == 0) s1 = 0.0f;
    bool done = false;
    if (iters == 0 || kill) {
        uint32_t w[4] = {(uint32_t)id, a.step1, 0x70617274u, 0u};
        philox4x32_10(w, a.seed_lo, a.seed_hi);
        const float span = (float)n - 4.0f;
        kill = 0;
        px = (float)(w[0] >> 8) * 0x1p-24f * span / 1.0f + 2.0f;
        py = (float)(w[1] >> 8) * 0x1p-24f * span / 1.0f + 2.0f;
        vx = 0.0f;
        vy = 0.0f;
        vol = a.es.init_volume;
        iters = a.should_rain ? 1u : 0u;
        done = !a.should_rain;
    }
    if (!done) {
        // get_terr_normal (:48-60)
        const int ix = (int)px, iy = (int)py;
        const bool quads = ix >= 1 && ix <= n - 3 && iy >= 1 && iy <= n - 3 &&
                           (int)(px + 1.0f) == ix + 1 && (int)(px - 1.0f) == ix - 1 && (int)(py + 1.0f) == iy + 1 &&
                           (int)(py - 1.0f) == iy - 1;
        const Around o = quads ? look_around_quads(a, n, px, py, ix, iy) : look_around(a, n, px, py);
        const float dx = o.rr + o.rg - o.lr - o.lg;
        const float dz = o.tr + o.tg - o.br - o.bg;
        const float cx = dx * 2.0f - 0.0f * dz, cy = 0.0f * 0.0f - 2.0f * 2.0f, cz = 2.0f * dz - dx * 0.0f;
        const float len = sqrtf(cx * cx + cy * cy + cz * cz);
        const float nx = cx / len, ny = cy / len, nz = cz / len;
        const float mxv = o.mx, myv = o.my, water = o.water;
        vx -= (dt * nx) / vol * a.es.G;
        vy -= (dt * nz) / vol * a.es.G;
        const float lm = sqrtf(mxv * mxv + myv * myv);
        float lv = sqrtf(vx * vx + vy * vy);
        if (lm > 0.0f && lv > 0.0f) {
            const float d = (mxv / lm) * (vx / lv) + (myv / lm) * (vy / lv);
            const float k = a.es.inertia * d / (vol + 1e5f * water);
            vx += k * mxv;
            vy += k * myv;
        }
        lv = sqrtf(vx * vx + vy * vy);
        if (lv > 1.0f) {  // capped speed: no tunnelling through the terrain
            vx = vx / lv;
            vy = vy / lv;
        }
        const float ox = px, oy = py;
        px += dt * vx;
        py += dt * vy;
        if (px <= 1.0f || py <= 1.0f || px * 1.0f >= (float)(n - 2) || py * 1.0f >= (float)(n - 2)) {
            px = ox; py = oy; vx = 0.0f; vy = 0.0f; kill = 1;
        }
        const float fr = 1.0f - dt * a.es.friction * ny;
        vx *= fr;
        vy *= fr;
        vol -= dt * a.es.Ke;
        const float sin_a = fabsf(sqrtf(1.0f - ny * ny));
        lv = sqrtf(vx * vx + vy * vy);
        sc = gmax(0.0f, a.es.Kc * vol * lv * gmax(0.02f, sin_a));
        iters++;
        if (vol <= a.es.min_volume || lv < a.es.min_velocity || iters >= a.es.ttl) kill = 1;
    }
    a.d.px[id] = px; a.d.py[id] = py; a.d.vx[id] = vx; a.d.vy[id] = vy; a.d.vol[id] = vol;
    a.d.s0[id] = s0; a.d.s1[id] = s1; a.d.sc[id] = sc; a.d.iters[id] = iters; a.d.kill[id] = kill;
    if (iters == 0) return;
    uint32_t rank[4];
    float ofx, ofy;
    for (int k = 0; k < 4; ++k) {
        int cx, cy;
        corner(px, py, k, n, cx, cy, ofx, ofy);
        rank[k] = atomicAdd(a.cnt + (size_t)cy * n + cx, 1u);
    }
    a.pack[2 * id] = make_float4(copysignf(ofx, kill ? -1.0f : 1.0f), ofy, sc, vol);
    a.pack[2 * id + 1] = make_float4(s0, s1, vx, vy);
    a.rank[id] = make_uint4(rank[0], rank[1], rank[2], rank[3]);
}

constexpr int SMALL = 8;       // records a texel's own thread sorts and applies
constexpr int HALF = 4;        // of those, the ones with a network of half the size
constexpr int MID = 32;        // records a warp sorts in registers, one per lane
constexpr int HOT_KEYS = 512;  // records a warp sorts at a time in a busier texel
enum { L_BIG = 0, L_MID, L_SMALL, L_HALF, LISTS };
enum { C_TOTAL = LISTS, C_NEXT, COUNTERS };  // records in all; next work item of k_papply

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sums, uint32_t& total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint32_t s = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        warp_sums[lane] = s;  // inclusive
    }
    __syncthreads();
    total = warp_sums[(blockDim.x >> 5) - 1];
    const uint32_t before = wid > 0 ? warp_sums[wid - 1] : 0u;
    return before + x - v;
}

struct TexelLists {
    uint32_t* counters;      // COUNTERS of them: texels per list, then C_*; zero before
    uint32_t* list[LISTS];
    uint32_t cap[LISTS];
};

// Buckets for the texels' records, in whatever order the blocks come (a texel
// sorts its own), and the texels by record count: 4096 texels per block, one
// counter update per block and list.  One pass over the counts in place of a
// scan's three (17 us at 1024², now 9).
constexpr int AL_T = 1024, AL_E = 4;
__global__ void __launch_bounds__(AL_T) k_palloc(const uint32_t* __restrict__ cnt, uint32_t* __restrict__ offs,
                                                 size_t count, TexelLists tl) {
    __shared__ uint32_t ws[32], num[LISTS], first[LISTS], base_sh;
    const size_t base = ((size_t)blockIdx.x * AL_T + threadIdx.x) * AL_E;
    if (threadIdx.x < LISTS) num[threadIdx.x] = 0;
    __syncthreads();
    uint32_t v[AL_E] = {0, 0, 0, 0}, sum = 0, place[AL_E];
    if (base < count) {  // (n is a multiple of 8: whole quads)
        const uint4 q = *reinterpret_cast<const uint4*>(cnt + base);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    }
    auto which = [](uint32_t k) { return k > MID ? L_BIG : k > SMALL ? L_MID : k > HALF ? L_SMALL : L_HALF; };
#pragma unroll
    for (int e = 0; e < AL_E; ++e) {
        sum += v[e];
        if (v[e]) place[e] = atomicAdd(&num[which(v[e])], 1u);
    }
    uint32_t total;
    uint32_t run = block_exclusive_scan(sum, ws, total);  // (its barriers order num)
    if (threadIdx.x < LISTS) first[threadIdx.x] = num[threadIdx.x] ? atomicAdd(tl.counters + threadIdx.x, num[threadIdx.x]) : 0u;
    if (threadIdx.x == LISTS) base_sh = total ? atomicAdd(tl.counters + C_TOTAL, total) : 0u;
    __syncthreads();
    run += base_sh;
#pragma unroll
    for (int e = 0; e < AL_E; ++e) {
        if (v[e]) {
            offs[base + e] = run;
            const int w = which(v[e]);
            const uint32_t slot = first[w] + place[e];
            if (slot < tl.cap[w]) tl.list[w][slot] = (uint32_t)(base + e);
        }
        run += v[e];
    }
}

__global__ void k_pscatter(Drops d, int n, const uint32_t* __restrict__ offs, const uint4* __restrict__ rank,
                           uint32_t* __restrict__ keys) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= d.count || d.iters[id] == 0) return;
    const float px = d.px[id], py = d.py[id];
    const uint4 r = rank[id];
    const uint32_t rk[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        int cx, cy;
        float ofx, ofy;
        corner(px, py, k, n, cx, cy, ofx, ofy);
        keys[offs[(size_t)cy * n + cx] + rk[k]] = (uint32_t)id * 4u + (uint32_t)k;
    }
}

struct ApplyArgs {
    hg_erosion_settings es;
    const float4* pack;
    const uint32_t* cnt;
    const uint32_t* offs;
    uint32_t* keys;        // records bucketed by texel, any order within a bucket
    uint32_t* sorted;      // big texels: their bucket in droplet-id order
    TexelLists tl;
    float* rock;
    float* dirt;
    float* water;
    float* mz;
    float* mw;
    float2* rec;           // per record (droplet * 4 + corner): the sediment it left of dirt and of
                           // rock, UNSET for a layer it did not reach
};

// A record's inputs: all from before the pass
struct Rec {
    uint32_t key;
    float multipl, sc, vol, s0, s1, vx, vy;
    int kill;
};

__device__ __forceinline__ Rec load_rec(const ApplyArgs& a, uint32_t key) {
    Rec r;
    r.key = key;
    const float4 p = __ldg(a.pack + 2 * (size_t)(key >> 2)), q = __ldg(a.pack + 2 * (size_t)(key >> 2) + 1);
    r.multipl = corner_weight(fabsf(p.x), p.y, (int)(key & 3u));
    r.kill = __float_as_int(p.x) < 0;
    r.sc = p.z;
    r.vol = p.w;
    r.s0 = q.x;
    r.s1 = q.y;
    r.vx = q.z;
    r.vy = q.w;
    return r;
}

struct Texel {
    float terr[2], wat, mz, mw;
};

// A NaN that no arithmetic gives (that is 0x7fffffff), and every sediment stored comes from an add.
constexpr uint32_t UNSET = 0x7fc0dead;
// what a record leaves for its droplet's sediment replay (mask bit 1: dirt, bit 0: rock)
struct RecOut {
    float s_dirt, s_rock;
    uint32_t mask;
};

// one droplet corner on its texel (glsl/particle_erosion.glsl:66-122): the
// layer loop from dirt down to rock, then water and momentum
__device__ __forceinline__ RecOut apply_record(const ApplyArgs& a, const Rec& r, Texel& T) {
    const float old_sed[2] = {r.s0, r.s1};
    float s_out[2] = {0.0f, 0.0f};
    uint32_t mask = 0;
    float cap = 0.0f;
    for (int l = 1; l >= 0; --l) {
        if (r.kill) {
            T.terr[l] += old_sed[l] * r.multipl;
            continue;
        }
        const float Kls = a.es.d_t * a.es.Ks[l], Kld = a.es.d_t * a.es.Kd[l];
        const float c = gmax(0.0f, r.sc - cap);
        float s1 = old_sed[l];
        const float old_terr = T.terr[l];
        mask |= 1u << l;
        if (c > s1) {
            const float eroded = r.multipl * Kls * (c - s1);
            s1 += eroded;
            T.terr[l] -= eroded;
            if (T.terr[l] < 0.0f) {
                s1 += T.terr[l];
                T.terr[l] = 0.0f;
                cap += old_terr;
            } else {
                s_out[l] = s1;
                break;
            }
        } else {
            const float deposit = r.multipl * Kld * (s1 - c);
            s1 -= deposit;
            T.terr[l] += deposit;
        }
        s_out[l] = s1;
    }
    T.wat += 1e-5f * r.vol * r.multipl;
    T.mz += r.vol * r.vx * r.multipl;
    T.mw += r.vol * r.vy * r.multipl;
    return RecOut{s_out[1], s_out[0], mask};
}

// A record's amounts with no layer exhausted, which do not depend on the texel
// (computed in parallel across a warp's lanes): the dirt step, then the rock step.
// mode 0: kill (both layers take their share back); 1: dirt dissolves and the
// loop breaks; 2: dirt deposits, rock dissolves; 3: both deposit.
struct Pre {
    uint32_t key;
    int mode;
    float d1, d0;    // kill: the returned sediment; else the dissolved / deposited amounts
    float s1n, s0n;  // the dirt / rock sediment after their step
    float wi, mzi, mwi;
};

__device__ __forceinline__ Pre prep_record(const ApplyArgs& a, const Rec& r) {
    Pre p;
    p.key = r.key;
    p.wi = 1e-5f * r.vol * r.multipl;
    p.mzi = r.vol * r.vx * r.multipl;
    p.mwi = r.vol * r.vy * r.multipl;
    p.s1n = 0.0f;
    p.s0n = 0.0f;
    if (r.kill) {
        p.mode = 0;
        p.d1 = r.s1 * r.multipl;
        p.d0 = r.s0 * r.multipl;
        return p;
    }
    const float c = gmax(0.0f, r.sc - 0.0f);  // cap is 0 until a layer is exhausted
    if (c > r.s1) {
        p.mode = 1;
        p.d1 = r.multipl * (a.es.d_t * a.es.Ks[1]) * (c - r.s1);
        p.s1n = r.s1 + p.d1;
        p.d0 = 0.0f;
        return p;
    }
    p.d1 = r.multipl * (a.es.d_t * a.es.Kd[1]) * (r.s1 - c);
    p.s1n = r.s1 - p.d1;
    if (c > r.s0) {
        p.mode = 2;
        p.d0 = r.multipl * (a.es.d_t * a.es.Ks[0]) * (c - r.s0);
        p.s0n = r.s0 + p.d0;
    } else {
        p.mode = 3;
        p.d0 = r.multipl * (a.es.d_t * a.es.Kd[0]) * (r.s0 - c);
        p.s0n = r.s0 - p.d0;
    }
    return p;
}

__device__ __forceinline__ void store_rec(const ApplyArgs& a, uint32_t key, const RecOut& o) {
    a.rec[key] = make_float2(o.mask & 2u ? o.s_dirt : __uint_as_float(UNSET), o.mask & 1u ? o.s_rock : __uint_as_float(UNSET));
}

__device__ __forceinline__ Texel load_texel(const ApplyArgs& a, size_t t) {
    return Texel{{a.rock[t], a.dirt[t]}, a.water[t], a.mz[t], a.mw[t]};
}
__device__ __forceinline__ void store_texel(const ApplyArgs& a, size_t t, const Texel& T) {
    a.rock[t] = T.terr[0];
    a.dirt[t] = T.terr[1];
    a.water[t] = T.wat;
    a.mz[t] = T.mz;
    a.mw[t] = T.mw;
}

// A texel with k <= S records, by one thread: sorting network on registers
// (odd-even transposition, S rounds), then the records in droplet-id order
// (each loaded when its turn comes: two or four loaded ahead cost registers, so
// warps: 1193 and 1248 us for 8 steps against 1161).
template <int S>
__device__ __forceinline__ void apply_small(const ApplyArgs& a, size_t t) {
    const uint32_t lo = a.offs[t], k = a.cnt[t];
    uint32_t kk[S];
#pragma unroll
    for (int i = 0; i < S; ++i) kk[i] = (uint32_t)i < k ? a.keys[lo + i] : 0xffffffffu;
    Texel T = load_texel(a, t);
#pragma unroll
    for (int r = 0; r < S; ++r)
#pragma unroll
        for (int i = r & 1; i + 1 < S; i += 2) {
            const uint32_t u = min(kk[i], kk[i + 1]), v = max(kk[i], kk[i + 1]);
            kk[i] = u;
            kk[i + 1] = v;
        }
#pragma unroll
    for (int i = 0; i < S; ++i)
        if ((uint32_t)i < k) store_rec(a, kk[i], apply_record(a, load_rec(a, kk[i]), T));
    store_texel(a, t, T);
}

constexpr int AP_WARPS = 4, AP_BLOCKS = 7;  // warps per block of k_papply, blocks per SM

// Bitonic network over a warp's 32 * E keys, element lane * E + e in k[e]: the
// smaller strides between a lane's registers, the others between lanes.
template <int E>
__device__ __forceinline__ void warp_sort(uint32_t (&k)[E], int lane) {
#pragma unroll
    for (int size = 2; size <= 32 * E; size <<= 1)
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            const bool lane_up = (lane & (size / E)) == 0;  // (size >= E: a lane's keys go one way)
            if (stride >= E) {
                const bool low = ((lane & (stride / E)) == 0) == lane_up;
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const uint32_t other = __shfl_xor_sync(0xffffffffu, k[e], stride / E);
                    k[e] = low ? min(k[e], other) : max(k[e], other);
                }
            } else {
#pragma unroll
                for (int e = 0; e < E; ++e)
                    if ((e & stride) == 0) {
                        const bool up = size < E ? (e & size) == 0 : lane_up;
                        const uint32_t u = min(k[e], k[e + stride]), v = max(k[e], k[e + stride]);
                        k[e] = up ? u : v;
                        k[e + stride] = up ? v : u;
                    }
            }
        }
}
// len <= 32 * E keys of src, sorted into sk
template <int E>
__device__ __forceinline__ void sort_chunk(const uint32_t* src, uint32_t len, uint32_t* sk, int lane) {
    uint32_t k[E];
#pragma unroll
    for (int e = 0; e < E; ++e) k[e] = 32u * e + lane < len ? src[32 * e + lane] : 0xffffffffu;
    warp_sort<E>(k, lane);
#pragma unroll
    for (int e = 0; e < E; ++e) sk[lane * E + e] = k[e];
}

// A warp applies up to 32 records of one texel in order.  With no layer
// exhausted each of the texel's five values is a plain running sum of amounts
// that do not depend on the texel, and so is what a record leaves for its
// droplet: lane c keeps sum c (dirt, rock, water, mz, mw) and adds the records'
// amounts, transposed through shared memory, one add per record for all five.
// A dirt or rock sum that gets below zero may mean an exhausted layer: then every
// lane runs these two again from the values they started with, a record at a
// time without a branch, and keeps those its own record met; from them it works
// out what the record leaves.
// Bound by the latency of the chains: about 25 cycles a record, and 105 more where
// a layer is exhausted (790 when the whole record went from lane to lane).
constexpr int SUMS = 5, SUM_PITCH = 36;  // (16-byte rows, lanes 0 to 4 on different banks)
struct WarpSums {
    float v[SUMS][SUM_PITCH];
    float4 w[2][32];  // exhausted layers: dirt and rock amounts, capacity, rock sediment; rock's
                      // rates, whether the record dissolves dirt, rock
};
__device__ __forceinline__ float* texel_sum(const ApplyArgs& a, int c) {
    return c == 0 ? a.dirt : c == 1 ? a.rock : c == 2 ? a.water : c == 3 ? a.mz : a.mw;
}
// mine: lane's record (of m); acc: lane c's sum (lanes above 4 follow lane 4)
__device__ __forceinline__ void warp_apply(const ApplyArgs& a, WarpSums& ws, int lane, uint32_t m, const Rec& mine,
                                           float& acc) {
    const unsigned FULL = 0xffffffffu;
    const bool have = (uint32_t)lane < m;
    Pre p{};
    if (have) p = prep_record(a, mine);
    // (x + -0 is x: what a record leaves alone, and the lanes without one)
    ws.v[0][lane] = !have ? -0.0f : p.mode == 1 ? -p.d1 : p.d1;
    ws.v[1][lane] = !have || p.mode == 1 ? -0.0f : p.mode == 2 ? -p.d0 : p.d0;
    ws.v[2][lane] = have ? p.wi : -0.0f;
    ws.v[3][lane] = have ? p.mzi : -0.0f;
    ws.v[4][lane] = have ? p.mwi : -0.0f;
    __syncwarp();
    const float* row = ws.v[min(lane, SUMS - 1)];
    float sum = acc, least = 0.0f;
    for (uint32_t i = 0; i < m; i += 8) {
        const float4 lo = *reinterpret_cast<const float4*>(row + i), hi = *reinterpret_cast<const float4*>(row + i + 4);
        const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            sum += v[e];
            least = fminf(least, sum);
        }
    }
    __syncwarp();  // the rows are read: the next batch may write them
    if (!__any_sync(FULL, lane < 2 && least < 0.0f)) {
        acc = sum;
        if (have) {
            store_rec(a, p.key, p.mode == 1   ? RecOut{p.s1n, 0.0f, 2u}
                                : p.mode == 0 ? RecOut{0.0f, 0.0f, 0u}
                                              : RecOut{p.s1n, p.s0n, 3u});
        }
        return;
    }
    ws.w[0][lane] = make_float4(p.mode == 1 ? -p.d1 : p.d1, p.mode == 1 ? -0.0f : p.mode == 2 ? -p.d0 : p.d0, mine.sc, mine.s0);
    ws.w[1][lane] = make_float4(mine.multipl * (a.es.d_t * a.es.Ks[0]), mine.multipl * (a.es.d_t * a.es.Kd[0]),
                                p.mode == 1 ? 1.0f : 0.0f, p.mode == 2 ? 1.0f : 0.0f);
    __syncwarp();
    float dirt = __shfl_sync(FULL, acc, 0), rock = __shfl_sync(FULL, acc, 1), met_dirt = 0.0f, met_rock = 0.0f;
#pragma unroll 4
    for (uint32_t i = 0; i < m; ++i) {
        const float4 u = ws.w[0][i], v = ws.w[1][i];
        const bool here = (uint32_t)lane == i;
        met_dirt = here ? dirt : met_dirt;
        met_rock = here ? rock : met_rock;
        const float d = dirt + u.x;
        const bool gone = (v.z != 0.0f) & (d < 0.0f);
        // the rock below an exhausted dirt layer: what the dirt held counts
        // against the capacity
        const float c = gmax(0.0f, u.z - dirt);
        const bool more = c > u.w;
        const float e = (more ? v.x : v.y) * (more ? c - u.w : u.w - c);
        const float r = rock + (gone ? (more ? -e : e) : u.y);
        dirt = gone ? 0.0f : d;
        rock = ((gone ? more : v.w != 0.0f) & (r < 0.0f)) ? 0.0f : r;
    }
    __syncwarp();  // the rows are read
    if (have) {
        Texel T{{met_rock, met_dirt}, 0.0f, 0.0f, 0.0f};
        const RecOut o = apply_record(a, mine, T);
        store_rec(a, p.key, o);
    }
    acc = lane == 0 ? dirt : lane == 1 ? rock : sum;  // (no layer enters the water's and the momentum's sums)
}

// a texel of SMALL + 1 to MID records, by a warp: lane i holds record i; a
// bitonic network over the lanes sorts the keys by droplet id
__device__ __forceinline__ void apply_mid(const ApplyArgs& a, WarpSums& ws, int lane, size_t t) {
    const uint32_t lo = a.offs[t], k = a.cnt[t];
    uint32_t key[1] = {(uint32_t)lane < k ? a.keys[lo + lane] : 0xffffffffu};
    float* f = texel_sum(a, min(lane, SUMS - 1)) + t;
    float acc = *f;
    warp_sort<1>(key, lane);
    Rec mine{};
    if ((uint32_t)lane < k) mine = load_rec(a, key[0]);
    warp_apply(a, ws, lane, k, mine, acc);
    if (lane < SUMS) *f = acc;
}

// a texel of more than MID records, by a warp: sort the bucket by droplet id,
// chunks of HOT_KEYS merged by rank, then apply it 32 records at a time
__device__ __noinline__ void apply_big(const ApplyArgs& a, WarpSums& ws, uint32_t* sk, int lane, size_t t) {
    const uint32_t lo = a.offs[t], k = a.cnt[t], hi = lo + k;
    float* f = texel_sum(a, min(lane, SUMS - 1)) + t;
    float acc = *f;
    for (uint32_t c0 = 0; c0 < k; c0 += HOT_KEYS) {
        const uint32_t len = min((uint32_t)HOT_KEYS, k - c0);
        const uint32_t* src = a.keys + lo + c0;
        if (len <= 64) sort_chunk<2>(src, len, sk, lane);
        else if (len <= 128) sort_chunk<4>(src, len, sk, lane);
        else if (len <= 256) sort_chunk<8>(src, len, sk, lane);
        else sort_chunk<16>(src, len, sk, lane);
        __syncwarp();
        if (k > HOT_KEYS) {
            for (uint32_t i = lane; i < len; i += 32) a.sorted[lo + c0 + i] = sk[i];
            __syncwarp();
        }
    }
    // merge the sorted chunks, two neighbouring runs at a time: a record's place is
    // its place in its run plus the records of the other run below it
    // (every chunk searched by every record took 16.3 ms a step at 64² with 262144
    // droplets after 80 steps, so 9.0)
    uint32_t *src = a.sorted + lo, *dst = a.keys + lo;
    for (uint32_t run = HOT_KEYS; run < k; run *= 2) {
        for (uint32_t i = lane; i < k; i += 32) {
            const uint32_t key = src[i], own = i & ~(run - 1), pair = i & ~(2 * run - 1);
            const uint32_t other = pair + (own == pair ? run : 0u), len = other < k ? min(run, k - other) : 0u;
            uint32_t l = 0, h = len;  // records of the other run below key
            while (l < h) {
                const uint32_t m = (l + h) >> 1;
                if (src[other + m] < key) l = m + 1; else h = m;
            }
            dst[pair + (i - own) + l] = key;
        }
        __syncwarp();
        uint32_t* t2 = src;
        src = dst;
        dst = t2;
    }
    const uint32_t* order = k > HOT_KEYS ? src : sk;
    for (uint32_t base = lo; base < hi; base += 32) {
        const uint32_t m = min(32u, hi - base);
        Rec mine{};
        if ((uint32_t)lane < m) mine = load_rec(a, order[base - lo + lane]);
        warp_apply(a, ws, lane, m, mine, acc);
    }
    __syncwarp();  // sk is read: the warp's next texel may sort
    if (lane < SUMS) *f = acc;
}

// Every texel with records: warps take the next item until none is left, the
// busiest texels first (they are the longest), then those of a warp each, then
// 32 at a time those of a thread each.  Bound by latency: the records' droplets
// lie anywhere, two loads of 16 bytes each (nine of 4 bytes before).  262144
// droplets on 1024² after 100 steps (buckets up to 317 records): one launch over
// all texels and one each over the busier two kinds took 33, 40 and 130 us, this
// 46.  8 steps, three worlds in turn / alone: 7 blocks per SM 1143 / 1289 us, 6
// 1161 / 1292, 8 1135 / 1328.
__global__ void __launch_bounds__(32 * AP_WARPS, AP_BLOCKS) k_papply(const ApplyArgs a) {
    __shared__ __align__(16) WarpSums sums[AP_WARPS];
    __shared__ uint32_t sk[AP_WARPS][HOT_KEYS];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    uint32_t num[LISTS];
#pragma unroll
    for (int l = 0; l < LISTS; ++l) num[l] = min(a.tl.counters[l], a.tl.cap[l]);
    const uint32_t small = (num[L_SMALL] + 31) / 32, half = (num[L_HALF] + 31) / 32;
    for (;;) {
        uint32_t i = lane == 0 ? atomicAdd(a.tl.counters + C_NEXT, 1u) : 0u;
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i < num[L_BIG]) {
            apply_big(a, sums[wl], sk[wl], lane, a.tl.list[L_BIG][i]);
        } else if ((i -= num[L_BIG]) < num[L_MID]) {
            apply_mid(a, sums[wl], lane, a.tl.list[L_MID][i]);
        } else if ((i -= num[L_MID]) < small) {
            if (32 * i + lane < num[L_SMALL]) apply_small<SMALL>(a, a.tl.list[L_SMALL][32 * i + lane]);
        } else if ((i -= small) < half) {
            if (32 * i + lane < num[L_HALF]) apply_small<HALF>(a, a.tl.list[L_HALF][32 * i + lane]);
        } else {
            return;
        }
        __syncwarp();
    }
}

// each droplet replays its corners 0..3 for its sediment
__global__ void k_pfinal(const hg_erosion_settings es, Drops d, const float2* __restrict__ rec) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= d.count || d.iters[id] == 0) return;
    const float old_sed[2] = {d.s0[id], d.s1[id]};
    float sed[2] = {old_sed[0], old_sed[1]};
    const bool kill = d.kill[id] != 0;
    const float ofx = fract_(d.px[id] * 1.0f), ofy = fract_(d.py[id] * 1.0f);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (kill) {
            const float multipl = corner_weight(ofx, ofy, k);
            sed[1] -= old_sed[1] * multipl;
            sed[0] -= old_sed[0] * multipl;
        } else {
            const float2 r = rec[(size_t)id * 4 + k];
            if (__float_as_uint(r.x) != UNSET) sed[1] = r.x;
            if (__float_as_uint(r.y) != UNSET) sed[0] = r.y;
        }
        const float conv = sed[0] * es.Kconv * es.d_t;
        sed[1] += conv;
        sed[0] -= conv;
    }
    d.s0[id] = sed[0];
    d.s1[id] = sed[1];
}

}  // namespace

size_t particle_counters() { return COUNTERS; }
int particle_lists() { return LISTS; }
size_t particle_list_capacity(int list, size_t cells, int count) {
    static_assert(LISTS == 4, "one capacity per list");
    const size_t least[LISTS] = {MID + 1, SMALL + 1, HALF + 1, 1};  // records of its texels
    return std::min(cells, (size_t)4 * (size_t)count / least[list] + 1);
}

void launch_particle_step(const StepConsts& c, const hg_erosion_settings& es, const ParticleBufs& pb,
                          const PWorld& pw, uint32_t step1, uint64_t seed, bool should_rain, cudaStream_t st) {
    const int n = c.n;
    const size_t cells = (size_t)n * n;
    const int pgrid = (pb.d.count + PB - 1) / PB;
    MoveArgs ma{c, es, pb.d, pw.rock, pw.dirt, pw.water, pw.mom[0], pw.mom[1], step1, (uint32_t)seed,
                (uint32_t)(seed >> 32), should_rain ? 1 : 0, pb.cnt, pb.rank, pb.pack};
    TexelLists tl;
    tl.counters = pb.cnt + cells;
    for (int l = 0; l < LISTS; ++l) {
        tl.list[l] = pb.list[l];
        tl.cap[l] = (uint32_t)particle_list_capacity(l, cells, pb.d.count);
    }
    cudaMemsetAsync(pb.cnt, 0, (cells + COUNTERS) * sizeof(uint32_t), st);
    k_pmove<<<pgrid, PB, 0, st>>>(ma);
    k_palloc<<<(unsigned)((cells + AL_T * AL_E - 1) / (AL_T * AL_E)), AL_T, 0, st>>>(pb.cnt, pb.offs, cells, tl);
    k_pscatter<<<pgrid, PB, 0, st>>>(pb.d, n, pb.offs, pb.rank, pb.keys);
    ApplyArgs aa{es, pb.pack, pb.cnt, pb.offs, pb.keys, pb.sorted, tl, pw.rock, pw.dirt, pw.water,
                 pw.mom[2], pw.mom[3], pb.rec};
    k_papply<<<152 * AP_BLOCKS, 32 * AP_WARPS, 0, st>>>(aa);
    k_pfinal<<<pgrid, PB, 0, st>>>(es, pb.d, pb.rec);
    count_launch(5);
}

}  // namespace hg
