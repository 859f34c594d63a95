// Fused step of a two-layer (rock + dirt) world, the reference's own model,
// in three kernels per step (up to four in a chain's last) instead of the nine
// per-pass launches:
//   k2f_hydro   [the previous step's sediment gather, both channels ->] rain ->
//               hydro_flux -> hydro_erosion (both layers, Kconv) ->
//               evaporation; 64 x 16 tiles, the fields TMA-staged with a
//               4-column, 1-row halo, pairs of cells in f32x2
//   k2f_rock    the rock talus pass (thermal_erosion/thermal_transport, layer
//               0), a row per warp
//   k2f_gather  a chain's last step (or a single step): the sediment gather of
//               both channels on its own (up to 768² within k2f_rock)
//   k2f_layer1  the dirt talus pass (layer 1: cumulative rock + dirt drops,
//               capped by the dirt height) and smoothing of both channels, on
//               64 x 16 tiles staged with a 3-cell halo
// (src/erosion.cpp:158-200; glsl/hydro_flux.glsl, hydro_erosion.glsl,
// sediment_transport.glsl, thermal_erosion.glsl, thermal_transport.glsl,
// smoothing.glsl).  Steps launched together form a chain, as in the one-layer
// step (hg_fused.cu).  Per-cell arithmetic is the per-pass kernels'
// operations, so the fused step equals them bit for bit.  The particle step
// (src/erosion.cpp:132-156) reuses the last two: the rock talus pass alone,
// then the dirt talus pass with smoothing's particle branch (momentum fold,
// water decay; glsl/smoothing.glsl:76-95).
//
// 2048² with the reference's defaults, per launch: k2f_hydro 62 us and 383
// instructions per cell with one cell at a time, 51 and 198 with pairs (60 and
// 251 in a chain, the gather included); rock talus pass and gather 45 us, now
// 40 without the gather; k2f_layer1 64 us and 467, now 55 and 280.
#include "hg_internal.h"
#include "hg_tile.cuh"
#include "hg_tma.cuh"

namespace hg {

namespace {

constexpr int TH = 16, NT = 256;  // k2f_hydro: tile height, threads per block
enum { F_B = 0, F_G, F_D, F_FL, F_FR, F_FT, F_FB, F_S0, F_S1, F_N };
constexpr int H_RH = TH + 2, H_BOX = RW * H_RH, H_RC = ((H_BOX + 31) / 32) * 32;

struct HydroArgs {
    CUtensorMap maps[F_N];  // rock, dirt, water, fL, fR, fT, fB, sediment rock / dirt (72 x 18 boxes)
    StepConsts c;
    RainStep r;
    const float *s0_prev, *s1_prev;  // chained: the previous step's eroded sediment
    float *water, *fl, *fr, *ft, *fb, *u, *v;
    float *s0, *s1;      // eroded sediment (rock, dirt)
    float *rock, *dirt;  // eroded rock and dirt
};

// ---- k2f_hydro ----------------------------------------------------------------
__device__ __forceinline__ void store_flux(const HydroArgs& a, size_t gi, const Flux2& o, float evap) {
    st2(a.fl + gi, o.fl);
    st2(a.fr + gi, o.fr);
    st2(a.ft + gi, o.ft);
    st2(a.fb + gi, o.fb);
    st2(a.water + gi, mul2(o.d2, pf(evap)));  // sediment_transport's evaporation
    st2(a.u + gi, o.u);
    st2(a.v + gi, o.v);
}

template <bool EDGE, bool CHAIN>
__device__ __forceinline__ void hydro_tile(const HydroArgs& a, float* sm, uint64_t* bar, int tx0, int ty0,
                                           int* err) {
    const StepConsts& c = a.c;
    const RainStep& r = a.r;
    const int n = c.n;
    const int tid = threadIdx.x;
    const int gx0 = tx0 - HX, gy0 = ty0 - 1;
    constexpr int PLANES = CHAIN ? F_S0 : F_N, PAIRS = TW * TH / NT / 2, STEP = NT / (TW / 2);
    if (tid == 0) {
        mbar_arrive_expect_tx(bar, PLANES * H_BOX * sizeof(float));
#pragma unroll
        for (int f = 0; f < PLANES; ++f) tma_load_2d(sm + f * H_RC, &a.maps[f], gx0, gy0, bar);
    }
    // the thread's pairs: column ix, rows iy, iy + STEP, ...
    const int ix = (tid % (TW / 2)) * 2, iy0 = tid / (TW / 2), x = tx0 + ix;
    const size_t g0 = (size_t)(ty0 + iy0) * n + x;
    float2 sed0[PAIRS], sed1[PAIRS], pu[PAIRS], pv[PAIRS];
    if (CHAIN) {  // (plain loads: this thread overwrites u and v below)
#pragma unroll
        for (int k = 0; k < PAIRS; ++k) {
            pu[k] = ld2(a.u + g0 + (size_t)(k * STEP) * n);
            pv[k] = ld2(a.v + g0 + (size_t)(k * STEP) * n);
        }
    }
    // rain: uniform amounts are added as water is read, Bernoulli drops (and
    // amounts that could round the out-of-range height) in the staged box
    const bool stage = r.active && (r.bernoulli || !(fabsf(r.amount) <= 16384.0f));
    const float2 shower = pf(r.active && !stage ? r.amount : 0.0f);
    constexpr int RG = (RW / 4) * H_RH;
    constexpr int RGK = (RG + NT - 1) / NT;
    uint32_t hits[RGK];
#pragma unroll
    for (int k = 0; k < RGK; ++k) {
        hits[k] = 0;
        const int q = tid + k * NT;
        if (q < RG && stage) {
            const int gx = gx0 + (q % (RW / 4)) * 4, gy = gy0 + q / (RW / 4);
            if (!EDGE || (gx >= 0 && gx < n && gy >= 0 && gy < n)) {
                if (r.bernoulli) {
                    uint32_t w[4];
                    rain_words4(r, gx, gy, w);
#pragma unroll
                    for (int j = 0; j < 4; ++j) hits[k] |= (w[j] < r.threshold ? 1u : 0u) << j;
                } else {
                    hits[k] = 15u;
                }
            }
        }
    }
    if (CHAIN) {
#pragma unroll
        for (int k = 0; k < PAIRS; ++k)
            gather_sediment2(c, a.s0_prev, a.s1_prev, x, ty0 + iy0 + k * STEP, pu[k], pv[k], sed0[k], sed1[k]);
    }
    bool ok = mbar_wait(bar, 0);
    if (stage || EDGE) ok = __syncthreads_and(ok);
    if (!ok) {
        atomicExch(err, 1);
        mbar_wait(bar, 0);
        return;
    }
    if (stage) {
        float* D = sm + F_D * H_RC;
#pragma unroll
        for (int k = 0; k < RGK; ++k) {
            if (hits[k] == 0) continue;
            const int q = tid + k * NT;
            float* p = D + (q / (RW / 4)) * RW + (q % (RW / 4)) * 4;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (hits[k] >> j & 1u) p[j] += r.amount;
        }
    }
    // out-of-grid water becomes the shader's out-of-range height: with rock,
    // dirt and flux 0 there, neighbour reads need no test
    if (EDGE) fill_outside<H_RH, 1, NT>(sm + F_D * H_RC, gx0, gy0, n, FAR_HEIGHT, tid);
    if (stage || EDGE) __syncthreads();
    const float* B = sm + F_B * H_RC;
    const float* G = sm + F_G * H_RC;
    const float* D = sm + F_D * H_RC;
    const float* FL = sm + F_FL * H_RC;
    const float* FR = sm + F_FR * H_RC;
    const float* FT = sm + F_FT * H_RC;
    const float* FB = sm + F_FB * H_RC;
    // pair of field f at `o`, and the pairs one column to the left and right
    auto row = [](const float* f, int o, float2& m, float2& l, float2& rr) {
        m = ld2(f + o);
        l = make_float2(f[o - 1], m.x);
        rr = make_float2(m.y, f[o + 2]);
    };
#pragma unroll 1
    for (int k = 0; k < PAIRS; ++k) {
        const int y = ty0 + iy0 + k * STEP;
        const int si = (1 + iy0 + k * STEP) * RW + HX + ix;
        const size_t gi = g0 + (size_t)(k * STEP) * n;
        float2 b, bl, br, g, gl, gr, d1, dl, dr;
        row(B, si, b, bl, br);
        row(G, si, g, gl, gr);
        row(D, si, d1, dl, dr);
        const float2 bb = ld2(B + si - RW), bt = ld2(B + si + RW), gb = ld2(G + si - RW), gt = ld2(G + si + RW);
        d1 = add2(d1, shower);
        // the two-layer total (rock + dirt) + water
        const float2 w = add2(add2(b, g), d1);
        const float2 wl = add2(add2(bl, gl), add2(dl, shower)), wr = add2(add2(br, gr), add2(dr, shower));
        const float2 wt = add2(add2(bt, gt), add2(ld2(D + si + RW), shower));
        const float2 wb = add2(add2(bb, gb), add2(ld2(D + si - RW), shower));
        const float2 fl = ld2(FL + si), fr = ld2(FR + si);
        const Flux2 o = cell_flux2(c, x, y, EDGE, w, d1, fl, fr, ld2(FT + si), ld2(FB + si), wl, wr, wt, wb,
                                   make_float2(FR[si - 1], fr.x), make_float2(fl.y, FL[si + 2]), ld2(FB + si + RW),
                                   ld2(FT + si - RW));
        store_flux(a, gi, o, c.evap);
        float2 s0 = !CHAIN ? ld2(sm + F_S0 * H_RC + si) : k == 0 ? sed0[0] : sed0[PAIRS - 1];
        float2 s1 = !CHAIN ? ld2(sm + F_S1 * H_RC + si) : k == 0 ? sed1[0] : sed1[PAIRS - 1];
        float2 Kls0 = pf(c.Kls0);
        if (c.ks_field) Kls0 = mul2(pf(c.dt), ldg2(c.ks_field + gi));
        cell_erosion2_pair(c, Kls0, o.vz, o.len, b, g, s0, s1, br, gr, bl, gl, bt, gt, bb, gb);
        st2(a.s0 + gi, s0);
        st2(a.s1 + gi, s1);
        st2(a.rock + gi, b);
        st2(a.dirt + gi, g);
    }
}

template <bool CHAIN>
__global__ void __launch_bounds__(NT, 4) k2f_hydro(const __grid_constant__ HydroArgs a, int* err) {
    __shared__ __align__(128) float sm[(CHAIN ? F_S0 : F_N) * H_RC];
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    const int n = a.c.n;
    const int tx0 = blockIdx.x * TW, ty0 = blockIdx.y * TH;
    const bool inner = tx0 - HX >= 0 && tx0 + TW + HX <= n && ty0 - 1 >= 0 && ty0 + TH + 1 <= n;
    if (inner) hydro_tile<false, CHAIN>(a, sm, &bar, tx0, ty0, err);
    else hydro_tile<true, CHAIN>(a, sm, &bar, tx0, ty0, err);
}

// ---- k2f_rock --------------------------------------------------------------------
struct RockArgs {
    StepConsts c;
    const float *u, *v, *s0, *s1;  // velocity, eroded sediment (rock, dirt)
    float *s0_o, *s1_o;            // transported sediment
    const float* rock;             // eroded rock
    float* rock_o;                 // rock after the layer-0 talus pass
};

// One row per warp (see talus_rows), whatever the size: short blocks, which
// share the SMs with the other kernels of worlds stepped together.  (Warps
// marching up strips take 32 us against 40 at 2048², but 8 steps of three
// worlds in turn 1.28 ms against 1.18; of one world 1.34 against 1.38.)
// SED: with the sediment gather of both channels (a chain's last step of a small
// world, see ROWS_MAX_N: one launch less; at 2048² the pair takes 45 us together,
// 40 and 12 apart, but a single step 215 us together, 200 apart)
template <bool SED>
__global__ void __launch_bounds__(32 * R_WARPS, SED ? 2 : 3) k2f_rock(const __grid_constant__ RockArgs a) {
    Taps<2> taps;
    talus_rows(
        a.c, a.rock, a.rock_o, blockIdx.x, blockIdx.y * R_ROWS,
        [&](int x, int y, size_t gi) {
            const float* const se[2] = {a.s0, a.s1};
            if (SED) load_taps<2>(a.c, se, x, y, ldg2(a.u + gi), ldg2(a.v + gi), taps);
        },
        [&](int, int, size_t gi) {
            if (SED) {
                st2(a.s0_o + gi, mix_taps(taps, 0));
                st2(a.s1_o + gi, mix_taps(taps, 1));
            }
        });
}

// sediment_transport of both channels, for a chain's last step.
__global__ void __launch_bounds__(NT) k2f_gather(const __grid_constant__ RockArgs a) {
    const int x = 2 * (blockIdx.x * 32 + (threadIdx.x & 31)), y = blockIdx.y * (NT / 32) + (threadIdx.x >> 5);
    const size_t gi = (size_t)y * a.c.n + x;
    float2 q0, q1;
    gather_sediment2(a.c, a.s0, a.s1, x, y, ldg2(a.u + gi), ldg2(a.v + gi), q0, q1);
    st2(a.s0_o + gi, q0);
    st2(a.s1_o + gi, q1);
}

// ---- k2f_layer1 -----------------------------------------------------------------
struct Layer1Args {
    CUtensorMap map_r, map_g;  // rock after layer 0, dirt after erosion: 72 x 22 boxes
    StepConsts c;
    Talus1 t1;
    int thermal1;              // layer-1 talus pass on (Kspeed[1] != 0)
    float *rock_o, *dirt_o;
    ParticleCells pc;          // particle mode
};
constexpr int L_RH = TH + 6, L_BOX = RW * L_RH, L_RC = ((L_BOX + 31) / 32) * 32;  // 3-row halo
constexpr int P_W = TW + 4, P_H = TH + 4, P_C = P_W * P_H;                        // outflows of the tile plus 2
constexpr size_t LAYER1_SMEM = (2 * L_RC + 8 * P_C) * sizeof(float) + 16;

// A 64 x 16 tile of rock and dirt staged with a 3-row, 4-column halo; pairs of
// cells throughout: outflows of the tile plus two rings into shared memory,
// dirt transport on the tile plus one ring in place in the dirt box, smoothing
// on the tile.  Bound by the shared-memory pipe and issue slots alike.  (Warps
// marching up strips with the passes in registers took 71 us against 64 for
// the one-cell tile form at 2048², and twice its time below 768²: 118
// registers, and chunks that recompute four rows.)
// Region (rx, ry) of the boxes <-> global (tx0 - HX + rx, ty0 - 3 + ry);
// outflow planes cover rx in [2, 70), ry in [1, 21): index (ry - 1) * P_W + rx - 2
template <bool PARTICLE>
__global__ void __launch_bounds__(NT, 4) k2f_layer1(const __grid_constant__ Layer1Args a, int* err) {
    extern __shared__ __align__(128) float dyn[];
    float* R = dyn;
    float* Gd = dyn + L_RC;
    float* P = dyn + 2 * L_RC;
    uint64_t* bar = reinterpret_cast<uint64_t*>(dyn + 2 * L_RC + 8 * P_C);
    const StepConsts& c = a.c;
    const int n = c.n, tid = threadIdx.x;
    const int tx0 = blockIdx.x * TW, ty0 = blockIdx.y * TH;
    const int gx0 = tx0 - HX, gy0 = ty0 - 3;
    const bool edge = gx0 < 0 || tx0 + TW + HX > n || gy0 < 0 || ty0 + TH + 3 > n;
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_arrive_expect_tx(bar, 2 * L_BOX * sizeof(float));
        tma_load_2d(R, &a.map_r, gx0, gy0, bar);
        tma_load_2d(Gd, &a.map_g, gx0, gy0, bar);
    }
    __syncthreads();
    const bool ok = __syncthreads_and(mbar_wait(bar, 0));
    if (!ok) {
        if (tid == 0) atomicExch(err, 1);
        mbar_wait(bar, 0);
        return;
    }
    if (edge) {  // the talus pass reads FAR_HEIGHT outside the grid (nothing else reads there)
        fill_outside<L_RH, 3, NT>(R, gx0, gy0, n, FAR_HEIGHT, tid);
        fill_outside<L_RH, 3, NT>(Gd, gx0, gy0, n, FAR_HEIGHT, tid);
        __syncthreads();
    }
    if (a.thermal1) {
#pragma unroll 1
        for (int q = tid; q < P_C / 2; q += NT) {
            const int px = (q % (P_W / 2)) * 2, py = q / (P_W / 2);
            const int si = (py + 1) * RW + px + 2;
            const float2 r = ld2(R + si), g = ld2(Gd + si);
            auto drop = [&](float2 nr, float2 ng) { return add2(sub2(r, nr), sub2(g, ng)); };
            const float2 rt = ld2(R + si + RW), gt = ld2(Gd + si + RW), rb = ld2(R + si - RW), gb = ld2(Gd + si - RW);
            auto left = [&](const float* f, int o, float2 m) { return make_float2(f[o - 1], m.x); };
            auto right = [&](const float* f, int o, float2 m) { return make_float2(m.y, f[o + 2]); };
            float2 dm[8], o[8];
            dm[0] = drop(left(R, si, r), left(Gd, si, g));
            dm[1] = drop(right(R, si, r), right(Gd, si, g));
            dm[2] = drop(rt, gt);
            dm[3] = drop(rb, gb);
            dm[4] = drop(left(R, si + RW, rt), left(Gd, si + RW, gt));
            dm[5] = drop(right(R, si + RW, rt), right(Gd, si + RW, gt));
            dm[6] = drop(left(R, si - RW, rb), left(Gd, si - RW, gb));
            dm[7] = drop(right(R, si - RW, rb), right(Gd, si - RW, gb));
            cell_thermal_outflows_dh2(c.dt, c.Kalpha1, c.Kspeed1, a.t1.x_cross, a.t1.b_diag, a.t1.fast_div, g, dm, o);
            if (edge) {  // a pair lies inside the grid or outside it (even columns)
                const int gx = gx0 + px + 2, gy = gy0 + py + 1;
                if (gx < 0 || gx >= n || gy < 0 || gy >= n) {
#pragma unroll
                    for (int d = 0; d < 8; ++d) o[d] = pf(0.0f);
                }
            }
#pragma unroll
            for (int d = 0; d < 8; ++d) st2(P + d * P_C + py * P_W + px, o[d]);
        }
        __syncthreads();
        // every pair of the planes' columns and the tile's rows plus one ring
        // (the outermost columns' results are read by nobody)
        constexpr int TQ = (P_W / 2) * (TH + 2), TK = (TQ + NT - 1) / NT;
        float2 res[TK];
#pragma unroll
        for (int k = 0; k < TK; ++k) {
            const int q = tid + k * NT;
            res[k] = pf(0.0f);
            if (q >= TQ) continue;
            const int px = (q % (P_W / 2)) * 2, py = 1 + q / (P_W / 2), pi = py * P_W + px;
            auto own = [&](int d) { return ld2(P + d * P_C + pi); };
            float2 o[8];
            float2 sum = pf(0.0f);
#pragma unroll
            for (int d = 0; d < 8; ++d) {
                o[d] = own(d);
                sum = sub2(sum, o[d]);
            }
            // inflows in the shader's order: L.R, R.L, T.B, B.T, LT.RB, RT.LB, LB.RT, RB.LT
            auto from_l = [&](int d, int row, float2 m) { return make_float2(P[d * P_C + pi + row - 1], m.x); };
            auto from_r = [&](int d, int row, float2 m) { return make_float2(m.y, P[d * P_C + pi + row + 2]); };
            auto at = [&](int d, int row) { return ld2(P + d * P_C + pi + row); };
            float2 inf = add2(from_l(1, 0, o[1]), from_r(0, 0, o[0]));
            inf = add2(inf, at(3, P_W));
            inf = add2(inf, at(2, -P_W));
            inf = add2(inf, from_l(7, P_W, at(7, P_W)));
            inf = add2(inf, from_r(6, P_W, at(6, P_W)));
            inf = add2(inf, from_l(5, -P_W, at(5, -P_W)));
            inf = add2(inf, from_r(4, -P_W, at(4, -P_W)));
            res[k] = add2(ld2(Gd + (py + 1) * RW + px + 2), add2(sum, inf));
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < TK; ++k) {
            const int q = tid + k * NT;
            if (q < TQ) st2(Gd + (2 + q / (P_W / 2)) * RW + (q % (P_W / 2)) * 2 + 2, res[k]);
        }
        __syncthreads();
    }
    // smoothing of the tile (border texels of the grid are copied)
#pragma unroll 1
    for (int k = 0; k < TW * TH / NT / 2; ++k) {
        const int q = tid + k * NT;
        const int ix = (q % (TW / 2)) * 2, iy = q / (TW / 2);
        const int x = tx0 + ix, y = ty0 + iy, si = (3 + iy) * RW + HX + ix;
        const size_t gi = (size_t)y * n + x;
        const float2 r = ld2(R + si), g = ld2(Gd + si);
        float2 nr = r, ng = g;
        if ((PARTICLE || c.smooth_m != 0.0f) && y > 0 && y < n - 1) {
            cell_smooth2_pair(c.smooth_m, nr, ng, make_float2(R[si - 1], r.x), make_float2(Gd[si - 1], g.x),
                              make_float2(r.y, R[si + 2]), make_float2(g.y, Gd[si + 2]), ld2(R + si + RW),
                              ld2(Gd + si + RW), ld2(R + si - RW), ld2(Gd + si - RW));
            if (x == 0) {
                nr.x = r.x;
                ng.x = g.x;
            }
            if (x + 2 == n) {
                nr.y = r.y;
                ng.y = g.y;
            }
        }
        st2(a.rock_o + gi, nr);
        st2(a.dirt_o + gi, ng);
        if (PARTICLE) particle_cells(a.pc, n, gi, x, y);
    }
}

void launch_rock(const RockArgs& a, bool gather, cudaStream_t st) {
    const dim3 grid(strips(a.c.n), a.c.n / R_ROWS);
    if (gather) k2f_rock<true><<<grid, 32 * R_WARPS, 0, st>>>(a);
    else k2f_rock<false><<<grid, 32 * R_WARPS, 0, st>>>(a);
    count_launch();
}

int launch_layer1(Layer1Args& a, const float* rock, const float* dirt, bool particle, TmaCache& tma, int* err,
                  cudaStream_t st) {
    const int n = a.c.n;
    if (!tma.get(rock, n, L_RH, &a.map_r) || !tma.get(dirt, n, L_RH, &a.map_g)) return HG_ERR_CUDA;
    auto* k = particle ? k2f_layer1<true> : k2f_layer1<false>;
    // per device and cheap: set on every launch rather than cached
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LAYER1_SMEM);
    k<<<dim3(n / TW, n / TH), NT, LAYER1_SMEM, st>>>(a, err);
    count_launch();
    return HG_OK;
}

}  // namespace

bool fused2_ok(int n) { return n % TW == 0 && n % TH == 0; }

int launch_fused2_step(const StepConsts& c, const Talus1& t1, const RainStep& r, const Fused2Bufs& b, ChainPos pos,
                       TmaCache& tma, int* err, cudaStream_t st) {
    const int n = c.n;
    const bool l0 = c.thermal != 0, chained = pos.index > 0;
    const bool l1 = c.Kspeed1 != 0.0f || c.smooth_m != 0.0f;  // k2f_layer1 runs
    // where each stage leaves rock and dirt
    float* rock_eroded = l0 ? b.b_ero : (l1 ? b.rock_mid : b.rock_o);
    float* rock_l0 = l1 ? b.rock_mid : b.rock_o;
    float* dirt_eroded = l1 ? b.g_ero : b.dirt_o;

    HydroArgs ha{};
    const float* ins[F_N] = {b.rock, b.dirt, b.water, b.fl, b.fr, b.ft, b.fb, b.s0, b.s1};
    for (int f = 0; f < (chained ? F_S0 : F_N); ++f)
        if (!tma.get(ins[f], n, H_RH, &ha.maps[f])) return HG_ERR_CUDA;
    ha.c = c;
    ha.r = r;
    ha.s0_prev = b.s0_prev;
    ha.s1_prev = b.s1_prev;
    ha.water = b.water_o; ha.fl = b.fl_o; ha.fr = b.fr_o; ha.ft = b.ft_o; ha.fb = b.fb_o;
    ha.u = b.u; ha.v = b.v;
    ha.s0 = b.s0_ero; ha.s1 = b.s1_ero;
    ha.rock = rock_eroded;
    ha.dirt = dirt_eroded;
    const dim3 tiles(n / TW, n / TH);
    if (chained) k2f_hydro<true><<<tiles, NT, 0, st>>>(ha, err);
    else k2f_hydro<false><<<tiles, NT, 0, st>>>(ha, err);
    count_launch();

    if (l0 || pos.last) {
        RockArgs ra{};
        ra.c = c;
        ra.u = b.u; ra.v = b.v;
        ra.s0 = b.s0_ero; ra.s1 = b.s1_ero;
        ra.s0_o = b.s0_o; ra.s1_o = b.s1_o;
        ra.rock = b.b_ero;
        ra.rock_o = rock_l0;
        const bool together = l0 && pos.last && n <= ROWS_MAX_N;
        if (l0) launch_rock(ra, together, st);
        if (pos.last && !together) {
            k2f_gather<<<dim3(n / 64, n / (NT / 32)), NT, 0, st>>>(ra);
            count_launch();
        }
    }
    if (l1) {
        Layer1Args la{};
        la.c = c;
        la.t1 = t1;
        la.thermal1 = c.Kspeed1 != 0.0f ? 1 : 0;
        la.rock_o = b.rock_o;
        la.dirt_o = b.dirt_o;
        return launch_layer1(la, rock_l0, dirt_eroded, false, tma, err, st);
    }
    return HG_OK;
}

int launch_particle_thermal_smooth(const StepConsts& c, const Talus1& t1, float count, const PWorld& in,
                                   const PWorld& out, float* rock_mid, TmaCache& tma, int* err, cudaStream_t st) {
    const float* rock_l0 = in.rock;
    if (c.thermal) {  // the rock talus pass alone
        RockArgs ra{};
        ra.c = c;
        ra.rock = in.rock;
        ra.rock_o = rock_mid;
        launch_rock(ra, false, st);
        rock_l0 = rock_mid;
    }
    Layer1Args la{};
    la.c = c;
    la.t1 = t1;
    la.thermal1 = c.Kspeed1 != 0.0f ? 1 : 0;
    la.rock_o = out.rock;
    la.dirt_o = out.dirt;
    la.pc = particle_cells_of(count, in, out);
    return launch_layer1(la, rock_l0, in.dirt, true, tma, err, st);
}

}  // namespace hg
