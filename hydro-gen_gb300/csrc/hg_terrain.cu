// hydro-gen's own terrain generator and rain, on the GPU.
//
//   hg_init_reference_heightmap   glsl/heightmap.glsl:52-158 (masks :25-43),
//                                 via World::gen_heightmap (src/state.cpp:116-147)
//   HG_RAIN_REFERENCE             glsl/rain.glsl:32-56 (cadence src/main.cpp:315-319)
//
// Noise (the shaders take these from glNoise, glsl/simplex_noise.glsl):
//   simplex2   2-D simplex noise as published by McEwan, Sheets, Gustavson and
//              Richardson ("Efficient computational noise in GLSL", JGT 2012):
//              skewed lattice, permutation polynomial (34 x^2 + x) mod 289,
//              gradients from 41 points on a line folded onto a diamond
//   gnoise_d   gradient noise with quintic fade and analytic derivatives
//              (Inigo Quilez's formulation), corner gradients from Hugo
//              Elias's integer hash (wrap-around int32 arithmetic)
//   fbm_*      octave sums; the "erosion" variant divides each octave by
//              1 + |running sum of derivatives|^2
// Float arithmetic in the shaders' operation order (the library is built
// without contraction), so the CPU restatement reproduces every bit except
// where exp() enters (the exponential mask).  pow(x, 2) and pow(x, 3) of
// possibly negative bases are x*x and x*x*x (GLSL leaves pow undefined for
// x < 0) and pow(r, 1) is r.
#include <cmath>

#include "hg_internal.h"

namespace hg {

namespace {

constexpr int BX = 32, BY = 8;

struct Fbm {  // gln_tFBMOpts with redistribution 1 (what every call site passes)
    float seed, persistance, lacunarity, scale;
    int octaves;
    bool turbulence, ridge;
};

__device__ __forceinline__ float fract_(float x) { return x - floorf(x); }
__device__ __forceinline__ float mod289(float x) { return x - 289.0f * floorf(x / 289.0f); }
__device__ __forceinline__ float perm(float x) { return mod289((x * 34.0f + 1.0f) * x); }

__device__ float simplex2(float vx, float vy) {
    const float F = 0.366025403784439f;   // (sqrt(3) - 1) / 2
    const float G = 0.211324865405187f;   // (3 - sqrt(3)) / 6
    const float G2 = -0.577350269189626f; // 2 G - 1
    const float R = 0.024390243902439f;   // 1 / 41
    const float s = vx * F + vy * F;
    float ix = floorf(vx + s), iy = floorf(vy + s);
    const float t = ix * G + iy * G;
    const float x0 = vx - ix + t, y0 = vy - iy + t;
    const float ox = x0 > y0 ? 1.0f : 0.0f, oy = x0 > y0 ? 0.0f : 1.0f;
    const float cx[3] = {x0, x0 + G - ox, x0 + G2};
    const float cy[3] = {y0, y0 + G - oy, y0 + G2};
    ix = mod289(ix);
    iy = mod289(iy);
    const float row[3] = {perm(iy + 0.0f), perm(iy + oy), perm(iy + 1.0f)};
    const float col[3] = {0.0f, ox, 1.0f};
    float sum = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float h = perm(row[k] + ix + col[k]);
        float w = gmax(0.5f - (cx[k] * cx[k] + cy[k] * cy[k]), 0.0f);
        w = w * w;
        w = w * w;
        const float gx = 2.0f * fract_(h * R) - 1.0f;
        const float gy = fabsf(gx) - 0.5f;
        const float a = gx - floorf(gx + 0.5f);
        w *= 1.79284291400159f - 0.85373472095314f * (a * a + gy * gy);
        const float d = a * cx[k] + gy * cy[k];
        sum = k == 0 ? w * d : sum + w * d;
    }
    return 130.0f * sum;
}

__device__ float fbm_simplex(float vx, float vy, const Fbm& o) {
    vx += o.seed * 100.0f;
    vy += o.seed * 100.0f;
    float acc = 0.0f, amp = 1.0f, freq = 1.0f, norm = amp;
    for (int i = 0; i < o.octaves && i < 30; ++i) {  // MAX_FBM_ITERATIONS
        float v = simplex2(vx * freq * o.scale, vy * freq * o.scale);
        if (o.turbulence) v = fabsf(v);
        if (o.turbulence && o.ridge) v = 1.0f - v;
        acc += v * amp;
        freq *= o.lacunarity;
        amp *= o.persistance;
        norm += amp;
    }
    return acc / norm;
}

// ---- gradient noise of two points ------------------------------------------------------
// 32 noise evaluations per cell with 8 octaves, first bounded by issue slots
// (97 % busy), half of them for the corner gradients' integer hash.
//   - A thread makes two adjacent cells, one per f32x2 lane: every float
//     operation of the noise is one instruction for both, with the shader's
//     operations and order per lane.
//   - A block's 64 x 8 cells lie in few lattice cells (10 to 1333 cells wide
//     at the default scale), so per fBm the block hashes the corners of its
//     lattice box once, into shared memory.  A box of more than LUT_CAP
//     corners (scales near a cell's size) or coordinates past 2^21 are hashed
//     per cell instead.
//   - The octaves' frequencies and amplitudes come from the host.
// 2048² with the default map: 662 us (one cell per thread), 535 (pairs), 379
// with the corner table.
constexpr int LUT_CAP = 768;
struct Lut {
    float gx[LUT_CAP], gy[LUT_CAP];  // corner gradients, octave by octave, row-major
    int x0[30], y0[30], w[30], off[31];
    int lo[2], hi[2];                // the block's coordinates (warped fBm), order-preserving integers
    float lof[2], hif[2];
};
struct Octaves {  // of one fBm: frequency and amplitude per octave, their sum plus the next
    float freq[30], amp[30];  // (amp: half the amplitude, for (value + 1) / 2)
    float norm;
};
struct MapArgs {
    hg_map_settings cfg;
    int n, octaves;
    float offset;           // seed * 100
    Octaves plain, eroded;  // starting frequency 1 and 1.5
    float* rock;
    float* dirt;            // nullptr: one layer
    float* zero[20];        // fields to clear
    int nzero;
};

// corner gradient component of both lanes, from Hugo Elias's integer hash:
// -1 + 2 h / 268435455 (the divisor is 2^28 as a float), h the low 28 bits of
// v * (v * v * 15731 + 789221) + 1376312589.  All constants times 16: the
// word then holds 16 h without masking, and every step scales exactly.
__device__ __forceinline__ float2 elias2(uint32_t n0, uint32_t n1) {
    auto h16 = [](uint32_t n) {
        const uint32_t v = (n << 13) ^ n;
        return (float)(v * (v * v * (15731u * 16u) + 789221u * 16u) + 1376312589u * 16u);
    };
    return fma2(make_float2(h16(n0), h16(n1)), pf(0x1p-31f), pf(-1.0f));
}
__device__ __forceinline__ float2 add_rm2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "add.rm.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ void corner_words(int32_t ix, int32_t iy, uint32_t& n0, uint32_t& n1) {
    n0 = (uint32_t)ix * 3u + (uint32_t)iy * 311u;
    n1 = (uint32_t)ix * 37u + (uint32_t)iy * 113u;
}
// floor and fraction of both lanes; |p| < 2^22 takes the integer part from an
// add of 1.5 * 2^23 that rounds down
__device__ __forceinline__ float2 split2(float2 p, int32_t i[2]) {
    if (fabsf(p.x) + fabsf(p.y) < 0x1p22f) {  // (not with a NaN)
        const float2 t = add_rm2(p, pf(0x1.8p23f));
        i[0] = __float_as_int(t.x) - 0x4b400000;
        i[1] = __float_as_int(t.y) - 0x4b400000;
        return sub2(p, add2(t, pf(-0x1.8p23f)));
    }
    const float2 f = make_float2(floorf(p.x), floorf(p.y));
    i[0] = (int32_t)f.x;
    i[1] = (int32_t)f.y;
    return sub2(p, f);
}

// value (and with D the gradient dx, dy) of the gradient noise at (px, py) in
// octave `oct`; TAB: corner gradients from the block's table
template <bool D, bool TAB>
__device__ __forceinline__ float2 gnoise2(float2 px, float2 py, const Lut& t, int oct, float2* ddx, float2* ddy) {
    int32_t ix[2], iy[2];
    const float2 fx = split2(px, ix), fy = split2(py, iy);
    auto fade = [](float2 f) {
        return mul2(mul2(mul2(f, f), f), add2(mul2(f, add2(mul2(f, pf(6.0f)), pf(-15.0f))), pf(10.0f)));
    };
    const float2 ux = fade(fx), uy = fade(fy);
    const float2 gx1 = add2(fx, pf(-1.0f)), gy1 = add2(fy, pf(-1.0f));
    // corners (0,0), (1,0), (0,1), (1,1)
    float2 ax, ay, bx, by, cx, cy, ex, ey;
    if (TAB) {
        const int w = t.w[oct], base = t.off[oct] - t.y0[oct] * w - t.x0[oct];
        const int p0 = base + iy[0] * w + ix[0], p1 = base + iy[1] * w + ix[1];
        ax = make_float2(t.gx[p0], t.gx[p1]);
        ay = make_float2(t.gy[p0], t.gy[p1]);
        bx = make_float2(t.gx[p0 + 1], t.gx[p1 + 1]);
        by = make_float2(t.gy[p0 + 1], t.gy[p1 + 1]);
        cx = make_float2(t.gx[p0 + w], t.gx[p1 + w]);
        cy = make_float2(t.gy[p0 + w], t.gy[p1 + w]);
        ex = make_float2(t.gx[p0 + w + 1], t.gx[p1 + w + 1]);
        ey = make_float2(t.gy[p0 + w + 1], t.gy[p1 + w + 1]);
    } else {
        uint32_t n0[2], n1[2];
#pragma unroll
        for (int l = 0; l < 2; ++l) corner_words(ix[l], iy[l], n0[l], n1[l]);
        ax = elias2(n0[0], n0[1]), ay = elias2(n1[0], n1[1]);
        bx = elias2(n0[0] + 3u, n0[1] + 3u), by = elias2(n1[0] + 37u, n1[1] + 37u);
        cx = elias2(n0[0] + 311u, n0[1] + 311u), cy = elias2(n1[0] + 113u, n1[1] + 113u);
        ex = elias2(n0[0] + 314u, n0[1] + 314u), ey = elias2(n1[0] + 150u, n1[1] + 150u);
    }
    const float2 va = add2(mul2(ax, fx), mul2(ay, fy));
    const float2 vb = add2(mul2(bx, gx1), mul2(by, fy));
    const float2 vc = add2(mul2(cx, fx), mul2(cy, gy1));
    const float2 vd = add2(mul2(ex, gx1), mul2(ey, gy1));
    const float2 k = add2(sub2(sub2(va, vb), vc), vd);
    const float2 uu = mul2(ux, uy);
    if (D) {
        auto dfade = [](float2 f) {
            return mul2(mul2(mul2(pf(30.0f), f), f), add2(mul2(f, add2(f, pf(-2.0f))), pf(1.0f)));
        };
        auto grad = [&](float2 a, float2 b, float2 c, float2 e, float2 du, float2 u, float2 v1) {
            const float2 lin = add2(add2(a, mul2(ux, sub2(b, a))), mul2(uy, sub2(c, a)));
            const float2 quad = mul2(uu, add2(sub2(sub2(a, b), c), e));
            return add2(add2(lin, quad), mul2(du, sub2(add2(mul2(u, k), v1), va)));
        };
        *ddx = grad(ax, bx, cx, ex, dfade(fx), uy, vb);
        *ddy = grad(ay, by, cy, ey, dfade(fy), ux, vc);
    }
    return add2(add2(add2(va, mul2(ux, sub2(vb, va))), mul2(uy, sub2(vc, va))), mul2(uu, k));
}

// Integers in the order of the floats (a NaN at an end).
__device__ __forceinline__ int ordered(float f) {
    const int b = __float_as_int(f);
    return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float unordered(int b) { return __int_as_float(b ^ ((b >> 31) & 0x7fffffff)); }

// Fills the block's corner table for an fBm at the threads' (vx, vy); false
// (for the whole block) when the box does not fit.  WARPED: the coordinates
// do not grow with the cell's, so their range is reduced over the block.
template <bool WARPED>
__device__ bool build_lut(Lut& t, float2 vx, float2 vy, const Octaves& o, const MapArgs& m) {
    const int tid = threadIdx.y * BX + threadIdx.x;
    __syncthreads();  // the last fBm's readers are done
    if (WARPED) {
        if (tid < 2) {
            t.lo[tid] = 0x7fffffff;
            t.hi[tid] = (int)0x80000000;
        }
        __syncthreads();
        const int xl = __reduce_min_sync(0xffffffffu, min(ordered(vx.x), ordered(vx.y)));
        const int xh = __reduce_max_sync(0xffffffffu, max(ordered(vx.x), ordered(vx.y)));
        const int yl = __reduce_min_sync(0xffffffffu, min(ordered(vy.x), ordered(vy.y)));
        const int yh = __reduce_max_sync(0xffffffffu, max(ordered(vy.x), ordered(vy.y)));
        if (threadIdx.x == 0) {
            atomicMin(&t.lo[0], xl);
            atomicMax(&t.hi[0], xh);
            atomicMin(&t.lo[1], yl);
            atomicMax(&t.hi[1], yh);
        }
        __syncthreads();
        if (tid < 2) {
            t.lof[tid] = unordered(t.lo[tid]);
            t.hif[tid] = unordered(t.hi[tid]);
        }
    } else {
        if (tid == 0) {
            t.lof[0] = vx.x;
            t.lof[1] = vy.x;
        }
        if (tid == BX * BY - 1) {
            t.hif[0] = vx.y;
            t.hif[1] = vy.x;
        }
    }
    __syncthreads();
    if (tid < m.octaves) {
        int org[2], ext[2];
        bool ok = true;
        for (int d = 0; d < 2; ++d) {
            const float a = t.lof[d] * o.freq[tid] * m.cfg.scale, b = t.hif[d] * o.freq[tid] * m.cfg.scale;
            const float lo = fminf(a, b), hi = fmaxf(a, b);
            ok = ok && fabsf(a) + fabsf(b) < 0x1p21f;  // (not with a NaN)
            org[d] = ok ? (int)floorf(lo) : 0;
            ext[d] = ok ? (int)floorf(hi) - org[d] + 2 : 2;
            ok = ok && ext[d] <= LUT_CAP;
        }
        t.x0[tid] = org[0];
        t.y0[tid] = org[1];
        t.w[tid] = ext[0];
        t.off[tid + 1] = ok ? min(ext[0] * ext[1], LUT_CAP + 1) : LUT_CAP + 1;
    }
    __syncthreads();
    if (tid == 0) {
        int sum = 0;
        t.off[0] = 0;
        for (int k = 1; k <= m.octaves; ++k) {
            sum = min(sum + t.off[k], LUT_CAP + 1);
            t.off[k] = sum;
        }
    }
    __syncthreads();
    const int total = t.off[m.octaves];
    if (total > LUT_CAP) return false;
    for (int e = tid, k = 0; e < total; e += BX * BY) {
        while (e >= t.off[k + 1]) ++k;
        const int q = e - t.off[k], w = t.w[k];
        uint32_t n0, n1;
        corner_words(t.x0[k] + q % w, t.y0[k] + q / w, n0, n1);
        const float2 g = elias2(n0, n1);
        t.gx[e] = g.x;
        t.gy[e] = g.y;
    }
    __syncthreads();
    return true;
}

__device__ __forceinline__ float2 fbm_gradient2(float2 vx, float2 vy, bool warped, Lut& t, const MapArgs& m) {
    vx = add2(vx, pf(m.offset));
    vy = add2(vy, pf(m.offset));
    const bool tab = warped ? build_lut<true>(t, vx, vy, m.plain, m) : build_lut<false>(t, vx, vy, m.plain, m);
    const float2 scale = pf(m.cfg.scale);
    float2 acc = pf(0.0f);
#pragma unroll 1
    for (int i = 0; i < m.octaves; ++i) {
        const float2 fr = pf(m.plain.freq[i]);
        const float2 px = mul2(mul2(vx, fr), scale), py = mul2(mul2(vy, fr), scale);
        const float2 nv = tab ? gnoise2<false, true>(px, py, t, i, nullptr, nullptr)
                              : gnoise2<false, false>(px, py, t, i, nullptr, nullptr);
        acc = add2(acc, mul2(add2(nv, pf(1.0f)), pf(m.plain.amp[i])));
    }
    return make_float2(acc.x / m.plain.norm, acc.y / m.plain.norm);
}

// erosion-like fBm: octaves damped by the running sum of derivatives
__device__ __forceinline__ float2 fbm_eroded2(float2 vx, float2 vy, Lut& t, const MapArgs& m) {
    vx = add2(vx, pf(m.offset));
    vy = add2(vy, pf(m.offset));
    const bool tab = build_lut<true>(t, vx, vy, m.eroded, m);
    const float2 scale = pf(m.cfg.scale);
    float2 acc = pf(0.0f), sx = pf(0.0f), sy = pf(0.0f);
#pragma unroll 1
    for (int i = 0; i < m.octaves; ++i) {
        const float2 fr = pf(m.eroded.freq[i]);
        const float2 px = mul2(mul2(vx, fr), scale), py = mul2(mul2(vy, fr), scale);
        float2 dx, dy;
        const float2 nv = tab ? gnoise2<true, true>(px, py, t, i, &dx, &dy)
                              : gnoise2<true, false>(px, py, t, i, &dx, &dy);
        sx = add2(sx, dx);
        sy = add2(sy, dy);
        const float2 num = mul2(add2(nv, pf(1.0f)), pf(m.eroded.amp[i]));
        const float2 den = add2(pf(1.0f), add2(mul2(sx, sx), mul2(sy, sy)));
        float2 q;
        if (num_range(num.x) & num_range(num.y) & den_range(den.x) & den_range(den.y) &
            (fmaxf(fabsf(num.x), fabsf(num.y)) <= 0x1p80f))
            q = div_recip2(num, make_float2(-den.x, -den.y), rcp_newton2(den));
        else
            q = make_float2(num.x / den.x, num.y / den.y);
        acc = add2(acc, q);
    }
    return make_float2(acc.x / m.eroded.norm, acc.y / m.eroded.norm);
}

// masks, terraces and height of one cell from its eroded fBm value
__device__ __forceinline__ float map_height(const hg_map_settings& cfg, int n, float fx, float fy, float val) {
    const float uvx = fx / (float)n, uvy = fy / (float)n;
    float hm = cfg.height_mult;
    if (cfg.uplift != 0) {  // :85-101
        const Fbm up_opts{cfg.seed, cfg.persistance, cfg.lacunarity, cfg.scale / cfg.uplift_scale, cfg.octaves,
                          true, true};
        const float up = fbm_simplex(fx - 7.3f, fy + 19.9f, up_opts);
        if (cfg.mask_exp != 0) hm += 2.5f;
        hm += 1.0f;
        val *= up;
    }
    if (cfg.mask_round != 0) {  // :102-107, round_mask :25-29
        if (cfg.mask_exp != 0) hm += 16.0f;
        const float ax = uvx - 0.5f, ay = uvy - 0.5f;
        const float v = 1.0f - (ax * ax + ay * ay + 0.75f);
        val = val * gmax(0.0f, v * 1.0f);
    }
    if (cfg.mask_exp != 0) {  // :108-111, exp_mask :42-44
        hm += 2.0f;
        val = val * (expf(val) - 1.0f) / 1.718f;
    }
    if (cfg.mask_power != 0) {  // :112-118, power_mask :38-40
        hm += 1.25f;
        if (cfg.mask_exp != 0) hm += 2.0f;
        const float b = val + 0.5f;
        val = val * (((b * b * b - 0.125f) / 3.25f) * 0.55f + 0.45f);
    }
    if (cfg.mask_slope != 0) val = 0.25f * val + 0.75f * (val * uvx * uvy);  // slope_mask :34-36
    val = val + (float)(4u * cfg.mask_round) * val;
    if (cfg.terrace > 0) {  // :124-129
        const float q = 1.0f / ((float)cfg.terrace * hm);
        const float lvl = floorf(val / q);
        const float t = cfg.terrace_scale;
        val = (t * lvl * q) + val * (1.0f - t);
    }
    return gmin(cfg.max_height, val * cfg.max_height * hm);  // :131
}

__global__ void __launch_bounds__(BX* BY) k_ref_heightmap(const __grid_constant__ MapArgs m) {
    __shared__ Lut t;
    const int n = m.n;
    const int x = min(2 * (int)(blockIdx.x * BX + threadIdx.x), n - 2), y = min((int)(blockIdx.y * BY + threadIdx.y), n - 1);
    // (n is even; threads past the map repeat its last cells, for the block's barriers)
    const bool own = 2 * (blockIdx.x * BX + threadIdx.x) < n && blockIdx.y * BY + threadIdx.y < n;
    const hg_map_settings& cfg = m.cfg;
    const size_t i = (size_t)y * n + x;
    // the world's other fields start at zero: stores under the arithmetic
    if (own)
        for (int k = 0; k < m.nzero; ++k) *reinterpret_cast<float2*>(m.zero[k] + i) = pf(0.0f);
    const float2 fx = make_float2((float)x, (float)(x + 1)), fy = pf((float)y);
    const float2 ws = pf(cfg.domain_warp_scale);
    // domain warp (:65-77)
    float2 wx = pf(1.0f), wy = pf(1.0f);
    if (cfg.domain_warp != 0) {
        wx = fbm_gradient2(add2(fx, pf(2.3f)), add2(fy, pf(2.9f)), false, t, m);
        wy = fbm_gradient2(add2(fx, pf(-3.1f)), add2(fy, pf(-4.3f)), false, t, m);
        if (cfg.domain_warp == 2) {
            const float2 qx = add2(fx, mul2(ws, wx)), qy = add2(fy, mul2(ws, wy));
            wx = fbm_gradient2(add2(qx, pf(-5.7f)), add2(qy, pf(27.9f)), true, t, m);
            wy = fbm_gradient2(add2(qx, pf(11.5f)), add2(qy, pf(-23.7f)), true, t, m);
        }
    }
    const float2 val = fbm_eroded2(add2(fx, mul2(ws, wx)), add2(fy, mul2(ws, wy)), t, m);  // :78-83
    const float2 h = make_float2(map_height(cfg, n, fx.x, fy.x, val.x), map_height(cfg, n, fx.y, fy.y, val.y));
    if (own) *reinterpret_cast<float2*>(m.rock + i) = h;
    if (m.dirt) {  // :133-135
        const float2 d = fbm_gradient2(add2(fx, pf(13.7f)), add2(fy, pf(27.1f)), false, t, m);
        if (own) *reinterpret_cast<float2*>(m.dirt + i) = mul2(add2(d, pf(1.5f)), pf(cfg.max_dirt));
    }
}

struct RefRain {
    float seed, amount, mountain_thresh, mountain_multip, drops, max_height;
};

// water += amount r + mountain bonus, r = max(0, simplex fBm); total height
// (rock + dirt) + water
__global__ void k_ref_rain(const RefRain rr, int n, const float* __restrict__ rock, const float* __restrict__ dirt,
                           float* __restrict__ water) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= n || y >= n) return;
    const size_t i = (size_t)y * n + x;
    const Fbm opts{rr.seed, 0.5f, 2.0f, rr.drops, 8, false, false};
    const float r = gmax(0.0f, fbm_simplex((float)x, (float)y, opts));
    float incr = rr.amount * r;
    const float total = (dirt ? rock[i] + dirt[i] : rock[i] + 0.0f) + water[i];
    const float mountain = total - rr.max_height * rr.mountain_thresh;
    if (mountain > 0.0f)
        incr += mountain * rr.mountain_multip * r / ((1.0f - rr.mountain_thresh) * rr.max_height);
    water[i] = water[i] + incr;
}

dim3 grid_for(int n) { return dim3((n + BX - 1) / BX, (n + BY - 1) / BY); }
dim3 grid_for2(int n) { return dim3((n / 2 + BX - 1) / BX, (n + BY - 1) / BY); }

}  // namespace

namespace {
// one rounding per operation, as the shader's loop does
void fill_octaves(Octaves& o, const hg_map_settings& cfg, float freq) {
    volatile float f = freq, a = 1.0f, norm = 1.0f;
    for (int i = 0; i < 30; ++i) {
        o.freq[i] = f;
        o.amp[i] = 0.5f * a;
        if (i >= cfg.octaves) continue;
        f = f * cfg.lacunarity;
        a = a * cfg.persistance;
        norm = norm + a;
    }
    o.norm = norm;
}
}  // namespace

void launch_ref_heightmap(const hg_map_settings& cfg, int n, float* rock, float* dirt, float* const* zero, int nzero,
                          cudaStream_t st) {
    MapArgs m{};
    m.cfg = cfg;
    m.n = n;
    m.octaves = cfg.octaves < 30 ? cfg.octaves : 30;  // MAX_FBM_ITERATIONS
    volatile float off = cfg.seed * 100.0f;
    m.offset = off;
    fill_octaves(m.plain, cfg, 1.0f);
    fill_octaves(m.eroded, cfg, 1.5f);
    m.rock = rock;
    m.dirt = dirt;
    m.nzero = nzero;
    for (int k = 0; k < nzero; ++k) m.zero[k] = zero[k];
    k_ref_heightmap<<<grid_for2(n), dim3(BX, BY), 0, st>>>(m);
    count_launch();
}

void launch_ref_rain(const hg_rain_settings& rs, const hg_map_settings& map, float time, int n, const float* rock,
                     const float* dirt, float* water, cudaStream_t st) {
    RefRain rr;
    volatile float tf = time * 1.372914227e3f;  // glsl/rain.glsl:36: fract(time * 1.372914227e3) * 1000
    rr.seed = ((float)tf - std::floor((float)tf)) * 1000.0f;
    rr.amount = rs.amount;
    rr.mountain_thresh = rs.mountain_thresh;
    rr.mountain_multip = rs.mountain_multip;
    rr.drops = rs.drops;
    rr.max_height = map.max_height;
    k_ref_rain<<<grid_for(n), dim3(BX, BY), 0, st>>>(rr, n, rock, dirt, water);
    count_launch();
}

}  // namespace hg
