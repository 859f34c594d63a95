// Per-pass kernels of the two-layer world (rock + dirt): the reference's
// full material model.  Rock sits in heightmap.r, dirt in heightmap.g, rock
// sediment in sedimap.r and dirt sediment in sedimap.g
// (glsl/heightmap.glsl:138-146, src/rendering.cpp:214); the total height the
// flux pass compares is (rock + dirt) + water, the order in which every pass
// before it leaves the total channel.  Rain reuses k_rain.  As in the one-layer
// step (hg_plain.cu) a thread has a pair of cells and passes that need nothing
// of their neighbours' results are joined: flux, erosion and evaporation in one
// kernel, each layer's two talus passes in another.  Bound by issue slots and
// launches: 8 steps with the reference's defaults at 1000² took 697 us in eight
// launches a step of one cell per thread with built-in divisions, 381 so.
#include "hg_internal.h"
#include "hg_tile.cuh"

namespace hg {

namespace {

constexpr int BX = 32, BY = 8;

// the thread's pair of cells (x, y), (x + 1, y); false past the map
__device__ __forceinline__ bool pair_at(int n, int& x, int& y, size_t& i) {
    x = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    y = blockIdx.y * blockDim.y + threadIdx.y;
    i = (size_t)y * n + x;
    return x < n && y < n;
}

// glsl/hydro_flux.glsl:77-166 with the two-layer total, glsl/hydro_erosion.glsl:23-92
// on both layers and the step's evaporation
struct Flux2Args {
    const float *rock, *dirt, *water, *fl, *fr, *ft, *fb;
    float *water_o, *fl_o, *fr_o, *ft_o, *fb_o, *u, *v, *vz, *rock_o, *dirt_o;
    float *s0, *s1;  // in place
};
__global__ void k2_flux_erosion(StepConsts c, const Flux2Args a) {
    int x, y;
    size_t i;
    const int n = c.n;
    if (!pair_at(n, x, y, i)) return;
    const bool hl = x > 0, hr = x + 2 < n, hb = y > 0, ht = y < n - 1;
    const float2 z = pf(0.0f);
    const float2 d1 = ldg2(a.water + i), f_l = ldg2(a.fl + i), f_r = ldg2(a.fr + i);
    // heights of the neighbours: 0 outside, as the erosion's normal has them
    auto row = [&](const float* f, float2& m, float2& l, float2& r, float2& t, float2& b) {
        m = ldg2(f + i);
        l = make_float2(hl ? __ldg(f + i - 1) : 0.0f, m.x);
        r = make_float2(m.y, hr ? __ldg(f + i + 2) : 0.0f);
        t = ht ? ldg2(f + i + n) : z;
        b = hb ? ldg2(f + i - n) : z;
    };
    float2 r, rl, rr, rt, rb, g, gl, gr, gt, gb;
    row(a.rock, r, rl, rr, rt, rb);
    row(a.dirt, g, gl, gr, gt, gb);
    const float2 w = add2(add2(r, g), d1);
    const float2 wl = make_float2(hl ? (rl.x + gl.x) + __ldg(a.water + i - 1) : FAR_HEIGHT, w.x);
    const float2 wr = make_float2(w.y, hr ? (rr.y + gr.y) + __ldg(a.water + i + 2) : FAR_HEIGHT);
    const float2 wt = ht ? add2(add2(rt, gt), ldg2(a.water + i + n)) : pf(FAR_HEIGHT);
    const float2 wb = hb ? add2(add2(rb, gb), ldg2(a.water + i - n)) : pf(FAR_HEIGHT);
    const float2 inl = make_float2(hl ? __ldg(a.fr + i - 1) : 0.0f, f_r.x);
    const float2 inr = make_float2(f_l.y, hr ? __ldg(a.fl + i + 2) : 0.0f);
    const Flux2 o = cell_flux2(c, x, y, true, w, d1, f_l, f_r, ldg2(a.ft + i), ldg2(a.fb + i), wl, wr, wt, wb, inl, inr,
                               ht ? ldg2(a.fb + i + n) : z, hb ? ldg2(a.ft + i - n) : z);
    st2(a.fl_o + i, o.fl);
    st2(a.fr_o + i, o.fr);
    st2(a.ft_o + i, o.ft);
    st2(a.fb_o + i, o.fb);
    st2(a.water_o + i, mul2(o.d2, pf(c.evap)));
    st2(a.u + i, o.u);
    st2(a.v + i, o.v);
    st2(a.vz + i, o.vz);
    float2 s0 = ld2(a.s0 + i), s1 = ld2(a.s1 + i);
    const float2 Kls0 = c.ks_field ? mul2(pf(c.dt), ldg2(c.ks_field + i)) : pf(c.Kls0);
    cell_erosion2_pair(c, Kls0, o.vz, o.len, r, g, s0, s1, rr, gr, rl, gl, rt, gt, rb, gb);
    st2(a.rock_o + i, r);
    st2(a.dirt_o + i, g);
    st2(a.s0 + i, s0);
    st2(a.s1 + i, s1);
}

// glsl/sediment_transport.glsl:66-93, both sediment channels
__global__ void k2_gather(StepConsts c, const float* __restrict__ u, const float* __restrict__ v,
                          const float* __restrict__ s0, const float* __restrict__ s1, float* __restrict__ s0_o,
                          float* __restrict__ s1_o) {
    int x, y;
    size_t i;
    if (!pair_at(c.n, x, y, i)) return;
    float2 q0, q1;
    gather_sediment2(c, s0, s1, x, y, ldg2(u + i), ldg2(v + i), q0, q1);
    st2(s0_o + i, q0);
    st2(s1_o + i, q1);
}

// Both talus passes of layer 1 in one launch (glsl/thermal_erosion.glsl:28-109,
// glsl/thermal_transport.glsl:31-65): drops summed over rock and dirt, H capped
// by the dirt height, dirt moves
__global__ void __launch_bounds__(32 * R_WARPS, 2) k2_talus1(StepConsts c, Talus1 t1, const float* __restrict__ rock,
                                                             const float* __restrict__ dirt, float* __restrict__ dirt_o) {
    talus_rows<true>(
        c, TalusRates{c.Kalpha1, c.Kspeed1, t1.x_cross, t1.b_diag, t1.fast_div}, rock, dirt, dirt_o, blockIdx.x,
        blockIdx.y * R_ROWS, [](int, int, size_t) {}, [](int, int, size_t) {});
}

// glsl/smoothing.glsl:22-103, both channels; PARTICLE: with the particle branch
// (:76-95); border texels are copied (:27-33)
template <bool PARTICLE>
__global__ void k2_smooth(StepConsts c, const float* __restrict__ rock, const float* __restrict__ dirt,
                          float* __restrict__ rock_o, float* __restrict__ dirt_o, const ParticleCells pc) {
    int x, y;
    size_t i;
    const int n = c.n;
    if (!pair_at(n, x, y, i)) return;
    const float2 r0 = ldg2(rock + i), g0 = ldg2(dirt + i);
    float2 r = r0, g = g0;
    if (y > 0 && y < n - 1) {
        const bool hl = x > 0, hr = x + 2 < n;
        cell_smooth2_pair(c.smooth_m, r, g, make_float2(hl ? __ldg(rock + i - 1) : 0.0f, r0.x),
                          make_float2(hl ? __ldg(dirt + i - 1) : 0.0f, g0.x),
                          make_float2(r0.y, hr ? __ldg(rock + i + 2) : 0.0f),
                          make_float2(g0.y, hr ? __ldg(dirt + i + 2) : 0.0f), ldg2(rock + i + n), ldg2(dirt + i + n),
                          ldg2(rock + i - n), ldg2(dirt + i - n));
        if (!hl) {
            r.x = r0.x;
            g.x = g0.x;
        }
        if (!hr) {
            r.y = r0.y;
            g.y = g0.y;
        }
    }
    st2(rock_o + i, r);
    st2(dirt_o + i, g);
    if (PARTICLE) particle_cells(pc, n, i, x, y);
}

dim3 pairs_for(int n) { return dim3((n / 2 + BX - 1) / BX, (n + BY - 1) / BY); }

}  // namespace

void launch_flux_erosion2(const StepConsts& c, const float* const in[S_COUNT], const float* dirt,
                          float* const out[S_COUNT], float* dirt_o, float* s0, float* s1, float* u, float* v, float* vz,
                          cudaStream_t st) {
    const Flux2Args a{in[S_ROCK], dirt,      in[S_WATER], in[S_FL],  in[S_FR], in[S_FT], in[S_FB],    out[S_WATER], out[S_FL],
                      out[S_FR],  out[S_FT], out[S_FB],   u,         v,        vz,       out[S_ROCK], dirt_o,       s0,
                      s1};
    k2_flux_erosion<<<pairs_for(c.n), dim3(BX, BY), 0, st>>>(c, a);
    count_launch();
}

void launch_gather2(const StepConsts& c, const float* u, const float* v, const float* s0, const float* s1, float* s0_o,
                    float* s1_o, cudaStream_t st) {
    k2_gather<<<pairs_for(c.n), dim3(BX, BY), 0, st>>>(c, u, v, s0, s1, s0_o, s1_o);
    count_launch();
}

void launch_talus1(const StepConsts& c, const Talus1& t1, const float* rock, const float* dirt, float* dirt_o,
                   cudaStream_t st) {
    k2_talus1<<<dim3(strips(c.n), c.n / R_ROWS), 32 * R_WARPS, 0, st>>>(c, t1, rock, dirt, dirt_o);
    count_launch();
}

void launch_smooth2(const StepConsts& c, const float* rock, const float* dirt, float* rock_o, float* dirt_o,
                    cudaStream_t st) {
    k2_smooth<false><<<pairs_for(c.n), dim3(BX, BY), 0, st>>>(c, rock, dirt, rock_o, dirt_o, ParticleCells{});
    count_launch();
}

void launch_particle_smooth(const StepConsts& c, float count, const PWorld& in, const PWorld& out, cudaStream_t st) {
    const ParticleCells pc = particle_cells_of(count, in, out);
    k2_smooth<true><<<pairs_for(c.n), dim3(BX, BY), 0, st>>>(c, in.rock, in.dirt, out.rock, out.dirt, pc);
    count_launch();
}

}  // namespace hg
