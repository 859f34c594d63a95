// Per-pass kernels: one kernel per GLSL pass of the grid step, FP32
// structure-of-arrays fields, two adjacent cells per thread (rows of 64 cells
// per warp, 8-byte accesses, both cells in f32x2 instructions; the maps' side
// is even), Jacobi ping-pong between passes as in the reference
// (src/erosion.cpp:158-200).  A step of whole maps joins passes that need
// nothing of their neighbours' results: uniform rain, flux, erosion and
// evaporation in one kernel, both talus passes in another.  Bound by issue slots
// and, at sides around 1000, by launches.  A step with Bernoulli rain and talus
// at 1000²: 52 us with one cell per thread and built-in divisions (flux and
// talus outflows 83 and 86 % busy), 35 with two, 30 with the passes joined.
#include "hg_internal.h"
#include "hg_tile.cuh"

namespace hg {

namespace {

constexpr int BX = 32, BY = 8;

__device__ __forceinline__ size_t at(int n, int x, int y) { return (size_t)y * n + x; }

// glsl/rain.glsl:32-56 — four cells per thread share one Philox call.
__global__ void k_rain(StepConsts c, RainStep r, float* __restrict__ water) {
    int x0 = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x0 >= c.n || y < c.row_lo || y >= c.row_hi) return;
    float4* p = reinterpret_cast<float4*>(water + at(c.n, x0, y));
    float4 d = *p;
    uint32_t w[4] = {0, 0, 0, 0};
    if (r.bernoulli) rain_words4(r, x0, y, w);
    d.x += rain_incr(r, w[0]);
    d.y += rain_incr(r, w[1]);
    d.z += rain_incr(r, w[2]);
    d.w += rain_incr(r, w[3]);
    *p = d;
}

// the thread's pair of cells (x, y), (x + 1, y); false past the map or the rows
__device__ __forceinline__ bool pair_at(const StepConsts& c, int& x, int& y, size_t& i) {
    x = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    y = blockIdx.y * blockDim.y + threadIdx.y;
    i = at(c.n, x, y);
    return x < c.n && y >= c.row_lo && y < c.row_hi;
}

// glsl/hydro_flux.glsl:77-166; ERODE: and glsl/hydro_erosion.glsl:37-92, which
// needs nothing of the neighbours' flux, and the step's evaporation
struct FluxArgs {
    const float *rock, *water, *fl, *fr, *ft, *fb;
    float *water_o, *fl_o, *fr_o, *ft_o, *fb_o, *u, *v, *vz;
    float *rock_o, *sed;  // ERODE: eroded rock; sediment, in place
    float rain;           // falls on every cell before the step (-0: none, which leaves a depth's bits)
};
template <bool ERODE>
__global__ void k_flux(StepConsts c, const FluxArgs a) {
    int x, y;
    size_t i;
    if (!pair_at(c, x, y, i)) return;
    const int n = c.n;
    const bool hl = x > 0, hr = x + 2 < n, hb = y > 0, ht = y < n - 1;
    const float2 rain = pf(a.rain), d1 = add2(ldg2(a.water + i), rain), f_l = ldg2(a.fl + i), f_r = ldg2(a.fr + i);
    // heights of the neighbours: 0 outside, as the erosion's normal has it
    float2 b = ldg2(a.rock + i);
    const float2 bl = make_float2(hl ? __ldg(a.rock + i - 1) : 0.0f, b.x);
    const float2 br = make_float2(b.y, hr ? __ldg(a.rock + i + 2) : 0.0f);
    const float2 bt = ht ? ldg2(a.rock + i + n) : pf(0.0f), bb = hb ? ldg2(a.rock + i - n) : pf(0.0f);
    const float2 w = add2(b, d1);
    const float2 wl = make_float2(hl ? bl.x + (__ldg(a.water + i - 1) + a.rain) : FAR_HEIGHT, w.x);
    const float2 wr = make_float2(w.y, hr ? br.y + (__ldg(a.water + i + 2) + a.rain) : FAR_HEIGHT);
    const float2 wt = ht ? add2(bt, add2(ldg2(a.water + i + n), rain)) : pf(FAR_HEIGHT);
    const float2 wb = hb ? add2(bb, add2(ldg2(a.water + i - n), rain)) : pf(FAR_HEIGHT);
    const float2 inl = make_float2(hl ? __ldg(a.fr + i - 1) : 0.0f, f_r.x);
    const float2 inr = make_float2(f_l.y, hr ? __ldg(a.fl + i + 2) : 0.0f);
    const Flux2 o = cell_flux2(c, x, y, true, w, d1, f_l, f_r, ldg2(a.ft + i), ldg2(a.fb + i), wl, wr, wt, wb, inl, inr,
                               ht ? ldg2(a.fb + i + n) : pf(0.0f), hb ? ldg2(a.ft + i - n) : pf(0.0f));
    st2(a.fl_o + i, o.fl);
    st2(a.fr_o + i, o.fr);
    st2(a.ft_o + i, o.ft);
    st2(a.fb_o + i, o.fb);
    st2(a.water_o + i, ERODE ? mul2(o.d2, pf(c.evap)) : o.d2);
    st2(a.u + i, o.u);
    st2(a.v + i, o.v);
    st2(a.vz + i, o.vz);
    if (ERODE) {
        float2 s = ld2(a.sed + i);
        const float2 Kls0 = c.ks_field ? mul2(pf(c.dt), ldg2(c.ks_field + i)) : pf(c.Kls0);
        cell_erosion_pair(c, Kls0, o.vz, o.len, b, s, br, bl, bb, bt);
        st2(a.rock_o + i, b);
        st2(a.sed + i, s);
    }
}

// glsl/hydro_erosion.glsl:37-92
__global__ void k_erosion(StepConsts c, const float* __restrict__ u, const float* __restrict__ v,
                          const float* __restrict__ vz, const float* __restrict__ rock,
                          float* __restrict__ rock_o, float* __restrict__ sed) {
    int x, y;
    size_t i;
    if (!pair_at(c, x, y, i)) return;
    const int n = c.n;
    float2 b = ld2(rock + i), s = ld2(sed + i);
    const float2 bl = make_float2(x > 0 ? rock[i - 1] : 0.0f, b.x), br = make_float2(b.y, x + 2 < n ? rock[i + 2] : 0.0f);
    const float2 bb = y > 0 ? ld2(rock + i - n) : pf(0.0f), bt = y < n - 1 ? ld2(rock + i + n) : pf(0.0f);
    const float2 Kls0 = c.ks_field ? mul2(pf(c.dt), ld2(c.ks_field + i)) : pf(c.Kls0);
    cell_erosion_pair(c, Kls0, ld2(vz + i), speed2(ld2(u + i), ld2(v + i)), b, s, br, bl, bb, bt);
    st2(rock_o + i, b);
    st2(sed + i, s);
}

// glsl/sediment_transport.glsl:66-93
template <bool EVAPORATE>
__global__ void k_sediment(StepConsts c, const float* __restrict__ u, const float* __restrict__ v,
                           const float* __restrict__ sed, float* __restrict__ sed_o,
                           float* __restrict__ water) {
    int x, y;
    size_t i;
    if (!pair_at(c, x, y, i)) return;
    st2(sed_o + i, gather_sediment(c, sed, x, y, ld2(u + i), ld2(v + i)));
    if (EVAPORATE) st2(water + i, mul2(ld2(water + i), pf(c.evap)));
}

// glsl/thermal_erosion.glsl:28-115, layer 0
__global__ void k_thermal_out(StepConsts c, const float* __restrict__ rock, float4* __restrict__ tc,
                              float4* __restrict__ td) {
    int x, y;
    size_t i;
    if (!pair_at(c, x, y, i)) return;
    const int n = c.n;
    const bool hl = x > 0, hr = x + 2 < n;
    auto row = [&](bool ok, size_t j, float2& m, float2& l, float2& r) {
        m = ok ? ld2(rock + j) : pf(FAR_HEIGHT);
        l = make_float2(ok && hl ? rock[j - 1] : FAR_HEIGHT, m.x);
        r = make_float2(m.y, ok && hr ? rock[j + 2] : FAR_HEIGHT);
    };
    float2 b, bl, br, t, tl, tr, d, dl, dr;
    row(true, i, b, bl, br);
    row(y < n - 1, i + n, t, tl, tr);
    row(y > 0, i - n, d, dl, dr);
    float2 dm[8] = {sub2(b, bl), sub2(b, br), sub2(b, t), sub2(b, d), sub2(b, tl), sub2(b, tr), sub2(b, dl), sub2(b, dr)};
    float2 o[8];
    cell_thermal_outflows_dh2(c.dt, c.Kalpha0, c.Kspeed0, c.talus_x_cross, c.talus_b_diag, c.fast_div, b, dm, o);
    tc[i] = make_float4(o[0].x, o[1].x, o[2].x, o[3].x);
    tc[i + 1] = make_float4(o[0].y, o[1].y, o[2].y, o[3].y);
    td[i] = make_float4(o[4].x, o[5].x, o[6].x, o[7].x);
    td[i + 1] = make_float4(o[4].y, o[5].y, o[6].y, o[7].y);
}

// glsl/thermal_transport.glsl:31-65, layer 0
__global__ void k_thermal_in(StepConsts c, const float* __restrict__ rock, const float4* __restrict__ tc,
                             const float4* __restrict__ td, float* __restrict__ rock_o) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y * blockDim.y + threadIdx.y;
    const int n = c.n;
    if (x >= n || y < c.row_lo || y >= c.row_hi) return;
    size_t i = at(n, x, y);
    auto ok = [&](int xx, int yy) { return xx >= 0 && xx < n && yy >= 0 && yy < n; };
    float in[8];
    in[0] = ok(x - 1, y) ? tc[i - 1].y : 0.0f;
    in[1] = ok(x + 1, y) ? tc[i + 1].x : 0.0f;
    in[2] = ok(x, y + 1) ? tc[i + n].w : 0.0f;
    in[3] = ok(x, y - 1) ? tc[i - n].z : 0.0f;
    in[4] = ok(x - 1, y + 1) ? td[i + n - 1].w : 0.0f;
    in[5] = ok(x + 1, y + 1) ? td[i + n + 1].z : 0.0f;
    in[6] = ok(x - 1, y - 1) ? td[i - n - 1].y : 0.0f;
    in[7] = ok(x + 1, y - 1) ? td[i - n + 1].x : 0.0f;
    float4 a = tc[i], b4 = td[i];
    float own[8] = {a.x, a.y, a.z, a.w, b4.x, b4.y, b4.z, b4.w};
    rock_o[i] = cell_thermal_apply(rock[i], own, in);
}

// Both talus passes of layer 0 in one launch (see talus_rows; two launches with
// the outflows in memory between them took 15 us at 1000²), SED: with the
// sediment gather.  Steps with talus, gather in the same launch / in its own, in
// three worlds in turn: 136² 9.9 / 11.6 us, 520² 10.6 / 12.6, 1000² 32.6 / 29.6,
// 1496² 71 / 60; ROWS_MAX_N is the line here too.
template <bool SED>
__global__ void __launch_bounds__(32 * R_WARPS, SED ? 2 : 3) k_talus(StepConsts c, const float* __restrict__ rock,
                                                                   float* __restrict__ rock_o, const float* __restrict__ u,
                                                                   const float* __restrict__ v, const float* __restrict__ sed,
                                                                   float* __restrict__ sed_o) {
    Taps<1> taps;
    talus_rows(
        c, rock, rock_o, blockIdx.x, blockIdx.y * R_ROWS,
        [&](int x, int y, size_t i) {
            const float* const se[1] = {sed};
            if (SED) load_taps<1>(c, se, x, y, ldg2(u + i), ldg2(v + i), taps);
        },
        [&](int, int, size_t i) {
            if (SED) st2(sed_o + i, mix_taps(taps, 0));
        });
}

// glsl/smoothing.glsl:22-103, rock channel (see cell_smooth)
__global__ void k_smooth(StepConsts c, const float* __restrict__ rock, float* __restrict__ rock_o) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y * blockDim.y + threadIdx.y;
    const int n = c.n;
    if (x >= n || y < c.row_lo || y >= c.row_hi) return;
    size_t i = at(n, x, y);
    if (x == 0 || y == 0 || x == n - 1 || y == n - 1) {  // border texels are copied (:27-33)
        rock_o[i] = rock[i];
        return;
    }
    rock_o[i] = cell_smooth(c.smooth_m, rock[i], rock[i - 1], rock[i + 1], rock[i + n], rock[i - n]);
}

dim3 grid_for(int n) { return dim3((n + BX - 1) / BX, (n + BY - 1) / BY); }
dim3 pairs_for(int n) { return dim3((n / 2 + BX - 1) / BX, (n + BY - 1) / BY); }

}  // namespace

void launch_rain(const StepConsts& c, const RainStep& r, float* water, cudaStream_t st) {
    dim3 blk(BX, BY), grd((c.n / 4 + BX - 1) / BX, (c.n + BY - 1) / BY);
    k_rain<<<grd, blk, 0, st>>>(c, r, water);
    count_launch();
}

void launch_flux(const StepConsts& c, const float* rock, const float* water, const float* fl, const float* fr,
                 const float* ft, const float* fb, float* water_o, float* fl_o, float* fr_o, float* ft_o,
                 float* fb_o, float* u, float* v, float* vz, cudaStream_t st) {
    const FluxArgs a{rock, water, fl, fr, ft, fb, water_o, fl_o, fr_o, ft_o, fb_o, u, v, vz, nullptr, nullptr,
                     -0.0f};
    k_flux<false><<<pairs_for(c.n), dim3(BX, BY), 0, st>>>(c, a);
    count_launch();
}

void launch_flux_erosion(const StepConsts& c, float rain, const float* const in[S_COUNT], float* const out[S_COUNT],
                         float* sed, float* u, float* v, float* vz, cudaStream_t st) {
    const FluxArgs a{in[S_ROCK],  in[S_WATER], in[S_FL],  in[S_FR],  in[S_FT],  in[S_FB], out[S_WATER], out[S_FL],
                     out[S_FR],   out[S_FT],   out[S_FB], u,         v,         vz,       out[S_ROCK],  sed,
                     rain};
    k_flux<true><<<pairs_for(c.n), dim3(BX, BY), 0, st>>>(c, a);
    count_launch();
}

void launch_gather(const StepConsts& c, const float* u, const float* v, const float* sed, float* sed_o,
                   cudaStream_t st) {
    k_sediment<false><<<pairs_for(c.n), dim3(BX, BY), 0, st>>>(c, u, v, sed, sed_o, nullptr);
    count_launch();
}

// From this side up warps march (hg_fused.cu): steps with talus, a row per warp /
// marching, in three worlds in turn and (alone): 1496² 60 / 58 us (81 / 86), 1752²
// 72 / 67 (93 / 94), 2296² 123 / 111 (149 / 148), 3000² 234 / 210 (274 / 270);
// 1000² 29.3 / 30.1 (45 / 50).
constexpr int MARCH_MIN_N = 2048;

void launch_talus(const StepConsts& c, const float* rock, float* rock_o, cudaStream_t st) {
    if (c.n >= MARCH_MIN_N) return launch_talus_march(c, rock, rock_o, st);
    k_talus<false><<<dim3(strips(c.n), c.n / R_ROWS), 32 * R_WARPS, 0, st>>>(c, rock, rock_o, nullptr, nullptr, nullptr,
                                                                            nullptr);
    count_launch();
}

void launch_gather_talus(const StepConsts& c, const float* rock, float* rock_o, const float* u, const float* v,
                         const float* sed, float* sed_o, cudaStream_t st) {
    if (c.n > ROWS_MAX_N) {
        launch_gather(c, u, v, sed, sed_o, st);
        launch_talus(c, rock, rock_o, st);
        return;
    }
    k_talus<true><<<dim3(strips(c.n), c.n / R_ROWS), 32 * R_WARPS, 0, st>>>(c, rock, rock_o, u, v, sed, sed_o);
    count_launch();
}

void launch_erosion(const StepConsts& c, const float* u, const float* v, const float* vz, const float* rock,
                    float* rock_o, float* sed_inout, cudaStream_t st) {
    k_erosion<<<pairs_for(c.n), dim3(BX, BY), 0, st>>>(c, u, v, vz, rock, rock_o, sed_inout);
    count_launch();
}

void launch_sediment(const StepConsts& c, const float* u, const float* v, const float* sed, float* sed_o,
                     float* water_inout, cudaStream_t st) {
    k_sediment<true><<<pairs_for(c.n), dim3(BX, BY), 0, st>>>(c, u, v, sed, sed_o, water_inout);
    count_launch();
}

void launch_thermal_out(const StepConsts& c, const float* rock, float4* tc, float4* td, cudaStream_t st) {
    k_thermal_out<<<pairs_for(c.n), dim3(BX, BY), 0, st>>>(c, rock, tc, td);
    count_launch();
}

void launch_thermal_in(const StepConsts& c, const float* rock, const float4* tc, const float4* td,
                       float* rock_o, cudaStream_t st) {
    k_thermal_in<<<grid_for(c.n), dim3(BX, BY), 0, st>>>(c, rock, tc, td, rock_o);
    count_launch();
}

void launch_smooth(const StepConsts& c, const float* rock, float* rock_o, cudaStream_t st) {
    k_smooth<<<grid_for(c.n), dim3(BX, BY), 0, st>>>(c, rock, rock_o);
    count_launch();
}

}  // namespace hg
