// Fused grid step in two kernels:
//   k_hydro:      [previous step's sediment_transport ->] rain -> hydro_flux
//                 -> hydro_erosion (+ evaporation)
//   k_transport:  thermal_erosion -> thermal_transport [, sediment_transport]
// replacing the reference's six dispatches per step (src/erosion.cpp:158-200).
//
// Why two and not one: every pass of k_hydro needs only its neighbours'
// INPUTS (rock, water, flux), so it runs with no redundant work; the talus
// and sediment passes need neighbours' RESULTS of k_hydro.  The sediment
// back-trace reach |u|*dt is unbounded (velocity divides by the water depth,
// and thin films give reaches of thousands of cells), so no halo can hold
// it; after k_hydro has written the eroded sediment of every cell, the
// gather takes any tap straight from L2/HBM.
//
// Chains: steps launched together form a chain.  hydro_erosion reads the
// sediment of its own cell only, so inside a chain a step's gather runs at
// the start of the next step's k_hydro: the gathered sediment is never
// written and read back (8 B per cell-step less), its two dependent loads
// (velocity, taps) overlap the tile's copies instead of stalling a kernel of
// their own, and a world without talus passes needs one launch per step.
// Only a chain's last step gathers in k_transport.  Two buffers of eroded
// sediment alternate.  Per step, three worlds in turn: 1024² without talus
// 15.3 -> 12.2 us, 4096² with it 279 -> 256 us, 8192² 1050 -> 925 us.
//
// Edge tiles (whose box leaves the grid) run either their own copy of the
// tile code or the inner tiles' code with block-uniform edge branches: the
// latter for batches and worlds below 4096² (see hydro_block).
//
// Both kernels are table driven: one launch covers any number of worlds
// ("terrains") of different sizes and settings.  A block (a marching warp)
// finds its terrain by binary search and reads the terrain's record (step constants, rain settings, buffers, step counter;
// TMA tensor maps in global memory).  A single world takes its whole descriptor, tensor
// maps included, as a kernel parameter.  The rain step number is the
// terrain's device step counter (advanced at a chain's end) plus the step's
// place in the chain, so a captured CUDA graph of a few steps can be replayed
// any number of times.
//
//   k_hydro stages rock, water, the four fluxes (and a chain's first step the
//   sediment) of a 64 x TH tile plus a halo (4 columns, 1 row) with TMA 2-D
//   tile loads; while they fly, threads draw this step's Philox rain words
//   and gather the sediment.  Each thread computes pairs of adjacent cells,
//   one per iteration, a warp covering a row of the tile.
//   k_transport marches warps up strips of columns, the talus pass in
//   registers; smaller launches run it by tiles in shared memory, the
//   smallest worlds by a row per warp (see below).
//
// Per-cell arithmetic is the code of the per-pass kernels (hg_device.cuh),
// evaluated two cells per f32x2 instruction where cells pair up, so the
// fused step reproduces the per-pass kernels bit for bit.
#include <cudaTypedefs.h>

#include <mutex>
#include <vector>

#include "hg_internal.h"
#include "hg_tile.cuh"
#include "hg_tma.cuh"

namespace hg {

namespace {

enum { H_B = 0, H_D, H_FL, H_FR, H_FT, H_FB, H_S, H_N };

// Geometry of a 64 x TH tile, TH = 16 or 8, of NT threads: two pairs of cells per
// thread, or one in small launches' 8-row tiles (256 threads), where the time is
// latency.  4096² by 8 rows, one step without talus / eight with it: 282 / 2800 us
// with one pair per thread, 243 / 2611 with two (16 rows: 246 / 2673).
template <int TH, int NT>
struct Geo {
    static constexpr int NTH = NT, BLOCKS = 1024 / NT;  // (64 registers)
    static constexpr int H_RH = TH + 2, H_BOX = RW * H_RH;
    static constexpr int H_RC = ((H_BOX + 31) / 32) * 32;  // 128-byte aligned array stride
    static constexpr int CPT = TW * TH / NTH;             // cells per thread in k_hydro (4)
};

__device__ __forceinline__ int find_terrain(const int* tile0, int nterr, int tile) {
    int lo = 0, hi = nterr - 1;
    while (lo < hi) {  // last terrain whose first tile <= tile
        int mid = (lo + hi + 1) >> 1;
        if (tile0[mid] <= tile) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ RainStep rain_for(const RainBase& rb, unsigned long long step1) {
    RainStep r;
    // uniform and Bernoulli rain only: the reference rain runs as its own
    // kernel before the step (the host inserts it)
    // (a 64-bit remainder costs over a hundred instructions per thread: only
    // for a step count that needs it)
    bool due = rb.period == 1;
    if (rb.period > 1)
        due = (step1 >> 32) == 0 ? (uint32_t)step1 % (uint32_t)rb.period == 0u
                                 : step1 % (unsigned long long)rb.period == 0ull;
    r.active = ((rb.mode == 1 || rb.mode == 2) && due) ? 1 : 0;
    r.bernoulli = rb.mode == 2 ? 1 : 0;
    r.amount = rb.amount;
    r.threshold = rb.threshold;
    r.seed_lo = rb.seed_lo;
    r.seed_hi = rb.seed_hi;
    r.terrain_id = rb.terrain_id;
    r.step = (uint32_t)step1;
    return r;
}

// ---------------------------------------------------------------------------
// k_hydro
// ---------------------------------------------------------------------------
// EM: 0 inner tile, 1 edge tile (each its own code), 2 either, told at run
// time by edge_rt (one code path for both)
template <int TH, int NT, int EM, bool CHAIN>
__device__ __forceinline__ void hydro_tile(const TerrainHot& td, const CUtensorMap* maps, float* sm, uint64_t* bar,
                                           int tx0, int ty0, int index, bool edge_rt, int* err) {
    const bool EDGE = EM == 2 ? edge_rt : EM == 1;
    using G = Geo<TH, NT>;
    constexpr int NTH = G::NTH, H_RC = G::H_RC, H_RH = G::H_RH;
    const StepConsts1& c = td.c;
    const int n = c.n;
    const int tid = threadIdx.x;
    const int gx0 = tx0 - HX, gy0 = ty0 - 1;
    constexpr int PLANES = CHAIN ? H_S : H_N;  // a chained step gathers its sediment
    if (tid == 0) {
        mbar_arrive_expect_tx(bar, PLANES * G::H_BOX * sizeof(float));
#pragma unroll
        for (int f = 0; f < PLANES; ++f) tma_load_2d(sm + f * H_RC, &maps[f], gx0, gy0, bar);
    }
    constexpr int PAIRS = G::CPT / 2;  // pairs per thread
    // a chained step starts with the previous step's sediment_transport: the
    // velocities of all its pairs first, then (after the rain words) all
    // their taps, so that the two dependent loads overlap the tiles' copies.
    // (u and v may be overwritten below, by this thread: plain loads)
    const size_t g0 = (size_t)(ty0 + tid / (TW / 2)) * n + tx0 + (tid % (TW / 2)) * 2;
    float2 sed[PAIRS], pu[PAIRS], pv[PAIRS];
    if (CHAIN) {
#pragma unroll
        for (int k = 0; k < PAIRS; ++k) {
            const size_t gi = g0 + (size_t)(k * (NTH / (TW / 2))) * n + td.uv_prev;
            pu[k] = ld2(td.u + gi);
            pv[k] = ld2(td.v + gi);
        }
    }
    // the step counter's load overlaps the tiles' copies
    const RainStep r = rain_for(td.rain, *td.step + 1ull + (unsigned long long)index);
    // Uniform rain is added to the water as it is read; Bernoulli rain (and an
    // amount that could round the out-of-range height) in the staged box
    // first.  Words of the region's row groups are drawn while the tiles load.
    const bool stage = r.active && (r.bernoulli || !(fabsf(r.amount) <= 16384.0f));
    const float2 shower = pf(r.active && !stage ? r.amount : 0.0f);
    constexpr int RG = (RW / 4) * H_RH;
    constexpr int RGK = (RG + NTH - 1) / NTH;
    uint32_t hits[RGK];  // bit j: it rains on cell j of the group
#pragma unroll
    for (int k = 0; k < RGK; ++k) {
        hits[k] = 0;
        const int q = tid + k * NTH;
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
            sed[k] = gather_sediment(c, td.s_prev, tx0 + (tid % (TW / 2)) * 2,
                                     ty0 + tid / (TW / 2) + k * (NTH / (TW / 2)), pu[k], pv[k]);
        if (td.s_keep) {
#pragma unroll
            for (int k = 0; k < PAIRS; ++k) st2(td.s_keep + g0 + (size_t)(k * (NTH / (TW / 2))) * n, sed[k]);
        }
    }
    bool ok = mbar_wait(bar, 0);
    if (stage || EDGE) ok = __syncthreads_and(ok);
    if (!ok) {  // the tile never arrived: record, give the copies one more bounded wait, skip the tile
        atomicExch(err, 1);
        mbar_wait(bar, 0);
        return;
    }
    if (stage) {
        float* D = sm + H_D * H_RC;
#pragma unroll
        for (int k = 0; k < RGK; ++k) {
            if (hits[k] == 0) continue;
            const int q = tid + k * NTH;
            float* p = D + (q / (RW / 4)) * RW + (q % (RW / 4)) * 4;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (hits[k] >> j & 1u) p[j] += r.amount;
        }
    }
    if (EDGE) {  // water outside the grid (zero-filled by the copy) becomes the shader's
                 // out-of-range height: with rock 0 there, the neighbour's total height
                 // rock + water is exactly FAR_HEIGHT; rock 0 and flux 0 outside are
                 // what the shader reads there too, so neighbour reads need no test
        fill_outside<H_RH, 1, NTH>(sm + H_D * H_RC, gx0, gy0, n, FAR_HEIGHT, tid);
    }
    if (stage || EDGE) __syncthreads();

    const float* B = sm + H_B * H_RC;
    const float* D = sm + H_D * H_RC;
    const float* S = sm + H_S * H_RC;
    const float* FL = sm + H_FL * H_RC;
    const float* FR = sm + H_FR * H_RC;
    const float* FT = sm + H_FT * H_RC;
    const float* FB = sm + H_FB * H_RC;
    // Pairs of horizontally adjacent cells, a row of the tile per warp: 8-byte
    // shared loads and global stores, both cells in one f32x2 instruction
    // (cell_flux2, cell_erosion_pair).  Neighbours outside the grid read rock 0, flux 0 and
    // total height FAR_HEIGHT from the tile (see the fill above); the
    // closed-boundary outflow zeroing runs in edge tiles.
    float* const rock_o = c.thermal ? td.b_ero : td.out[S_ROCK];  // no thermal pass: eroded rock is final
#pragma unroll 1
    for (int k = 0; k < PAIRS; ++k) {
        const int q = tid + k * NTH;
        const int ix = (q % (TW / 2)) * 2, iy = q / (TW / 2);
        const int x = tx0 + ix, y = ty0 + iy;
        const int si = (1 + iy) * RW + HX + ix;
        const size_t gi = (size_t)y * n + x;
        const float2 b = ld2(B + si), d1 = add2(ld2(D + si), shower);
        const float2 bl = make_float2(B[si - 1], b.x), br = make_float2(b.y, B[si + 2]);
        const float2 bb = ld2(B + si - RW), bt = ld2(B + si + RW);
        const float2 wl = add2(bl, make_float2(D[si - 1] + shower.x, d1.x));
        const float2 wr = add2(br, make_float2(d1.y, D[si + 2] + shower.x));
        const float2 wt = add2(bt, add2(ld2(D + si + RW), shower)), wb = add2(bb, add2(ld2(D + si - RW), shower));
        const float2 fl = ld2(FL + si), fr = ld2(FR + si);
        const float2 inl = make_float2(FR[si - 1], fr.x), inr = make_float2(fl.y, FL[si + 2]);
        const float2 s = !CHAIN ? ld2(S + si) : k == 0 ? sed[0] : sed[PAIRS - 1];
        float2 Kls0 = pf(c.Kls0);
        if (c.ks_field) Kls0 = mul2(pf(c.dt), __ldg(reinterpret_cast<const float2*>(c.ks_field + gi)));
        const Flux2 o = cell_flux2(c, x, y, EDGE, add2(b, d1), d1, fl, fr, ld2(FT + si), ld2(FB + si), wl, wr, wt, wb,
                                   inl, inr, ld2(FB + si + RW), ld2(FT + si - RW));
        float2 be = b, se = s;
        cell_erosion_pair(c, Kls0, o.vz, o.len, be, se, br, bl, bb, bt);
        st2(td.out[S_FL] + gi, o.fl);
        st2(td.out[S_FR] + gi, o.fr);
        st2(td.out[S_FT] + gi, o.ft);
        st2(td.out[S_FB] + gi, o.fb);
        // sediment_transport's evaporation (glsl/sediment_transport.glsl:75)
        st2(td.out[S_WATER] + gi, mul2(o.d2, pf(c.evap)));
        st2(td.u + gi, o.u);
        st2(td.v + gi, o.v);
        st2(td.s_ero + gi, se);
        st2(rock_o + gi, be);
    }
}

template <int TH, int NT, bool SPLIT, bool CHAIN>
__device__ __forceinline__ void hydro_block(const TerrainHot& td, const CUtensorMap* maps, int tx0, int ty0, int index,
                                            int* err) {
    using G = Geo<TH, NT>;
    __shared__ __align__(128) float sm[(CHAIN ? H_S : H_N) * G::H_RC];
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    const int n = td.c.n;
    bool inner = tx0 - HX >= 0 && tx0 + TW + HX <= n && ty0 - 1 >= 0 && ty0 + TH + 1 <= n;
    // Small terrains are mostly edge tiles, interleaved with inner ones on
    // every SM: !SPLIT runs one code path for both (two unrolled copies
    // missed in the instruction cache: 4.6 stalls per issue on an empty
    // instruction buffer, 11 % more time at 256²).  A large world is almost
    // all inner tiles and keeps a copy specialised for them (SPLIT).
    if (!SPLIT) hydro_tile<TH, NT, 2, CHAIN>(td, maps, sm, &bar, tx0, ty0, index, !inner, err);
    else if (inner) hydro_tile<TH, NT, 0, CHAIN>(td, maps, sm, &bar, tx0, ty0, index, false, err);
    else hydro_tile<TH, NT, 1, CHAIN>(td, maps, sm, &bar, tx0, ty0, index, true, err);
}

// Batch form: the terrain records are a kernel parameter (constant bank),
// the block finds its terrain by binary search.
template <int TH, int NT, bool CHAIN>
__global__ void __launch_bounds__(NT, Geo<TH, NT>::BLOCKS) k_hydro(const __grid_constant__ BatchParams bp,
                                                        const CUtensorMap* __restrict__ maps, int index, int* err) {
    const int t = find_terrain(bp.tile0, bp.nterr, blockIdx.x);
    const unsigned tile = blockIdx.x - bp.tile0[t], tiles_x = bp.t[t].tiles_x;
    hydro_block<TH, NT, false, CHAIN>(bp.t[t], maps + MAPS_PER_TERRAIN * t, (tile % tiles_x) * TW, (tile / tiles_x) * TH,
                                  index, err);
}

// Single-world form: the whole descriptor, tensor maps included, is a kernel
// parameter.  SPLIT as for hydro_block: the host picks it by world size.
template <int TH, int NT, bool SPLIT, bool CHAIN>
__global__ void __launch_bounds__(NT, Geo<TH, NT>::BLOCKS) k_hydro1(const __grid_constant__ TerrainDesc td, int index, int* err) {
    hydro_block<TH, NT, SPLIT, CHAIN>(td.h, td.maps, blockIdx.x * TW, td.row_lo + blockIdx.y * TH, index, err);
}

// ---------------------------------------------------------------------------
// k_transport of large launches: sediment_transport, then
// thermal_erosion/thermal_transport (layer 0).  A warp marches up a strip of
// columns, two adjacent cells per lane (one f32x2 pair), and keeps the talus pass in registers: the eroded
// rock of three rows, the current row's eight outflows, and of the row below
// what its neighbours need.  Neighbours across lanes come by shuffle, so
// there is no shared memory and no block barrier.
//
// The 64-column strip gives 60 columns (a cell's inflow needs the outflows
// one column around it, and those the rock one further), a chunk of R rows
// recomputes the outflows of two rows.
// ---------------------------------------------------------------------------
constexpr int T_WARPS = 4;       // warps per block, each with its own strip
// Blocks per SM: with the gather 5 (96 registers), without 6 (80).  More warps
// at fewer registers spill, and leave no room for another world's k_hydro
// beside them (4096², three worlds in turn: 262 us a step at 6 blocks, 299 at
// 7, 324 at 8).
constexpr int T_BLOCKS_SED = 5, T_BLOCKS = 6;
// Most warps a launch should have (two rounds of 152 SMs x 24 warps): fewer
// leave SMs idle at the end of the launch, more recompute more rows, and just
// over a round leaves the last one nearly empty.  One step at
// 4096², alone / among other worlds' steps: one round 331 / 265 us, two 310 /
// 262, three 302 / 266.
constexpr int T_FILL = 2 * 152 * T_WARPS * T_BLOCKS;

// rows [y0, y1) of strip `strip`; SED: with the sediment gather
template <bool SED>
__device__ __forceinline__ void transport_strip(const TerrainHot& td, int strip, int y0, int y1) {
    const StepConsts1& c = td.c;
    const int n = c.n;
    const int lane = threadIdx.x & 31;
    const int x = strip * SW - 2 + 2 * lane;
    const bool in = x >= 0 && x < n;                      // n is even: the grid's edge lies between lanes
    const bool own = in && lane >= 1 && lane <= SW / 2;   // columns this warp writes
    const bool edge = strip == 0 || strip * SW + SW + 2 > n;
    const float2 zero = pf(0.0f);
    if (!c.thermal) {
        if (!SED || !own) return;
        size_t gi = (size_t)y0 * n + x;
#pragma unroll 2
        for (int y = y0; y < y1; ++y, gi += n)
            st2(td.out[S_SED] + gi, gather_sediment(c, td.s_ero, x, y, ldg2(td.u + gi), ldg2(td.v + gi)));
        return;
    }
    auto rock = [&](int y) {
        return in && y >= 0 && y < n ? ldg2(td.b_ero + (size_t)y * n + x) : pf(FAR_HEIGHT);
    };
    RockRow dn = rock_row(rock(y0 - 2)), md = rock_row(rock(y0 - 1));
    float2 next = rock(y0), un = zero, vn = zero;
    // of the row below the current one: its inflow from left and right, minus
    // its outflows, its rock; of that row and the one below it: the outflows
    // upward (T, and RT and LT already at the receiving column)
    float2 lr = zero, osum = zero, rk = zero, t1 = zero, rt1 = zero, lt1 = zero, t0 = zero, rt0 = zero, lt0 = zero;
#pragma unroll 1
    for (int r = y0 - 1; r <= y1; ++r) {
        const RockRow up = rock_row(next);
        next = rock(r + 2);
        const size_t gi = (size_t)r * n + x;
        const bool sed_row = SED && own && r >= y0 && r < y1;
        const float2 u = un, v = vn;
        if (SED && own && r + 1 < y1) {
            un = ldg2(td.u + gi + n);
            vn = ldg2(td.v + gi + n);
        }
        float2 o[8];
        if (r >= 0 && r < n) {
            float2 dm[8] = {sub2(md.c, md.l), sub2(md.c, md.r), sub2(md.c, up.c), sub2(md.c, dn.c),
                            sub2(md.c, up.l), sub2(md.c, up.r), sub2(md.c, dn.l), sub2(md.c, dn.r)};
            cell_thermal_outflows_dh2(c.dt, c.Kalpha0, c.Kspeed0, c.talus_x_cross, c.talus_b_diag, c.fast_div, md.c,
                                      dm, o);
            if (edge && !in) {
#pragma unroll
                for (int d = 0; d < 8; ++d) o[d] = zero;
            }
        } else {
#pragma unroll
            for (int d = 0; d < 8; ++d) o[d] = zero;
        }
        // the row below: its inflows in the shader's order (L, R, T, B, LT,
        // RT, LB, RB), then rock + (its outflows' sum + inflow)
        const float2 rb = from_left(o[7]), lb = from_right(o[6]);
        if (own && r > y0) {
            const float2 inf = add2(add2(add2(add2(add2(add2(lr, o[3]), t0), rb), lb), rt0), lt0);
            st2(td.out[S_ROCK] + gi - n, add2(rk, add2(osum, inf)));
        }
        lr = add2(from_left(o[1]), from_right(o[0]));
        osum = sub2(zero, o[0]);
#pragma unroll
        for (int d = 1; d < 8; ++d) osum = sub2(osum, o[d]);
        rk = md.c;
        t0 = t1; rt0 = rt1; lt0 = lt1;
        t1 = o[2];
        rt1 = from_left(o[5]);
        lt1 = from_right(o[4]);
        if (sed_row) st2(td.out[S_SED] + gi, gather_sediment(c, td.s_ero, x, r, u, v));
        dn = md;
        md = up;
    }
}

// Task `task` of a terrain whose rows [lo, hi) are done: chunks of td.t_rows
// rows of each strip, strips fastest.  steps: what the device step counter
// advances by (0 within a chain, else the chain's length).
template <bool SED>
__device__ __forceinline__ void transport_task(const TerrainHot& td, int task, int lo, int hi, int steps) {
    const int ns = strips(td.c.n);
    const int y0 = lo + (task / ns) * td.t_rows;
    transport_strip<SED>(td, task % ns, y0, min(y0 + td.t_rows, hi));
    // the chain's k_hydro launches have finished (stream order) and the next
    // chain's start after this launch
    if (SED && task == 0 && (threadIdx.x & 31) == 0) *td.step += (unsigned long long)steps;
}

template <bool SED>
__global__ void __launch_bounds__(32 * T_WARPS, SED ? T_BLOCKS_SED : T_BLOCKS)
    k_transport(const __grid_constant__ BatchParams bp, int steps) {
    const int w = blockIdx.x * T_WARPS + (threadIdx.x >> 5);
    if (w >= bp.tasks) return;
    const int t = find_terrain(bp.task0, bp.nterr, w);
    transport_task<SED>(bp.t[t], w - bp.task0[t], 0, bp.t[t].c.n, steps);
}

template <bool SED>
__global__ void __launch_bounds__(32 * T_WARPS, SED ? T_BLOCKS_SED : T_BLOCKS)
    k_transport1(const __grid_constant__ TerrainDesc td, int tasks, int steps) {
    const int w = blockIdx.x * T_WARPS + (threadIdx.x >> 5);
    if (w < tasks) transport_task<SED>(td.h, w, td.row_lo, td.row_hi, steps);
}

// ---------------------------------------------------------------------------
// k_transport_tile: the same by 64 x 16 tiles, 256 threads with a row group of
// four cells (two pairs) each: the eroded rock of the tile and a two-row halo
// and the outflows of the tile and a ring of one go through shared memory.  A
// block is short and the SM holds 32 warps of it, where a marching warp works
// through its rows one after the other at 20 to 24 warps per SM: the form for
// launches whose time is latency.  The marching form recomputes less once it can
// march far, and leaves the SMs room for other worlds' kernels.
// Bound by issue slots and the barriers.
// ---------------------------------------------------------------------------
constexpr int TT_H = 16, TT_NTH = 256, TT_BH = TT_H + 4, TT_OC = RW * (TT_H + 2);
struct TileShared {
    float rock[RW * TT_BH];  // region (rx, ry): global (tx0 - HX + rx, ty0 - 2 + ry)
    float out[8 * TT_OC];    // outflows at (rx, ry), ry in [1, TT_H + 2]: index (ry - 1) * RW + rx
};

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// outflows of the pair at index si of the staged rock
__device__ __forceinline__ void tile_outflows(const StepConsts1& c, const float* rock, int si, float2 o[8]) {
    const float2 m = ld2(rock + si), up = ld2(rock + si + RW), dn = ld2(rock + si - RW);
    auto left = [&](int i, float2 v) { return make_float2(rock[i - 1], v.x); };
    auto right = [&](int i, float2 v) { return make_float2(v.y, rock[i + 2]); };
    float2 dm[8] = {sub2(m, left(si, m)),       sub2(m, right(si, m)),       sub2(m, up),
                    sub2(m, dn),                sub2(m, left(si + RW, up)),  sub2(m, right(si + RW, up)),
                    sub2(m, left(si - RW, dn)), sub2(m, right(si - RW, dn))};
    cell_thermal_outflows_dh2(c.dt, c.Kalpha0, c.Kspeed0, c.talus_x_cross, c.talus_b_diag, c.fast_div, m, dm, o);
}

template <bool SED>
__device__ __forceinline__ void transport_tile(const TerrainHot& td, TileShared& sm, int tx0, int ty0) {
    const StepConsts1& c = td.c;
    const int n = c.n, tid = threadIdx.x;
    const int gx0 = tx0 - HX, gy0 = ty0 - 2;
    const int ix = 4 * (tid % (TW / 4)), iy = tid / (TW / 4);
    const size_t gi = (size_t)(ty0 + iy) * n + tx0 + ix;
    // the rock (the shader's out-of-range height outside the grid) and the
    // sediment taps are in flight together
    constexpr int BP = RW / 2 * TT_BH, BK = (BP + TT_NTH - 1) / TT_NTH;
    float2 box[BK];
    if (c.thermal) {
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            const int q = tid + k * TT_NTH, gx = gx0 + 2 * (q % (RW / 2)), gy = gy0 + q / (RW / 2);
            const bool in = q < BP && gx >= 0 && gx < n && gy >= 0 && gy < n;
            box[k] = in ? ldg2(td.b_ero + (size_t)gy * n + gx) : pf(FAR_HEIGHT);
        }
    }
    Taps<1> taps[2];
    if (SED) {
        const float4 u = __ldg(reinterpret_cast<const float4*>(td.u + gi));
        const float4 v = __ldg(reinterpret_cast<const float4*>(td.v + gi));
        const float* const se[1] = {td.s_ero};
        load_taps<1>(c, se, tx0 + ix, ty0 + iy, make_float2(u.x, u.y), make_float2(v.x, v.y), taps[0]);
        load_taps<1>(c, se, tx0 + ix + 2, ty0 + iy, make_float2(u.z, u.w), make_float2(v.z, v.w), taps[1]);
    }
    if (c.thermal) {
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            const int q = tid + k * TT_NTH;
            if (q < BP) st2(sm.rock + 2 * q, box[k]);
        }
        __syncthreads();
    }
    if (SED) {
        const float2 a = mix_taps(taps[0], 0), b = mix_taps(taps[1], 0);
        *reinterpret_cast<float4*>(td.out[S_SED] + gi) = make_float4(a.x, a.y, b.x, b.y);
    }
    if (!c.thermal) return;
    // outflows of the ring: 34 pairs in the row below and above the tile (from
    // two columns before it), a pair at either end of its rows
    constexpr int CAP = TW / 2 + 2, RING = 2 * CAP + 2 * TT_H;
    if (tid < RING) {
        const bool cap = tid < 2 * CAP;
        const int rx = cap ? HX - 2 + 2 * (tid % CAP) : tid & 1 ? HX + TW : HX - 2;
        const int ry = cap ? (tid < CAP ? 1 : TT_H + 2) : 2 + (tid - 2 * CAP) / 2;
        float2 o[8];
        tile_outflows(c, sm.rock, ry * RW + rx, o);
        const int gx = gx0 + rx, gy = gy0 + ry;
        const bool in = gx >= 0 && gx < n && gy >= 0 && gy < n;  // (a pair lies inside the grid or outside it)
#pragma unroll
        for (int d = 0; d < 8; ++d) st2(sm.out + d * TT_OC + (ry - 1) * RW + rx, in ? o[d] : pf(0.0f));
    }
    const int si = (iy + 2) * RW + HX + ix, oi = si - RW;
    float2 osum[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        float2 o[8];
        tile_outflows(c, sm.rock, si + 2 * p, o);
        osum[p] = pf(0.0f);
#pragma unroll
        for (int d = 0; d < 8; ++d) {
            osum[p] = sub2(osum[p], o[d]);
            st2(sm.out + d * TT_OC + oi + 2 * p, o[d]);
        }
    }
    __syncthreads();
    // inflows in the shader's order: L, R, T, B, LT, RT, LB, RB
    float2 inf[2] = {pf(0.0f), pf(0.0f)};
    auto add = [&](float2 a, float2 b) {
        inf[0] = add2(inf[0], a);
        inf[1] = add2(inf[1], b);
    };
    auto sides = [&](int dl, int dr, int off) {  // left neighbour's dl, right neighbour's dr
        const float *a = sm.out + dl * TT_OC + oi + off, *b = sm.out + dr * TT_OC + oi + off;
        const float4 l = ld4(a), r = ld4(b);
        add(make_float2(a[-1], l.x), make_float2(l.y, l.z));
        add(make_float2(r.y, r.z), make_float2(r.w, b[4]));
    };
    auto above = [&](int d, int off) {
        const float4 v = ld4(sm.out + d * TT_OC + oi + off);
        add(make_float2(v.x, v.y), make_float2(v.z, v.w));
    };
    sides(1, 0, 0);
    above(3, RW);
    above(2, -RW);
    sides(7, 6, RW);
    sides(5, 4, -RW);
    const float4 b = ld4(sm.rock + si);
    const float2 r0 = add2(make_float2(b.x, b.y), add2(osum[0], inf[0]));
    const float2 r1 = add2(make_float2(b.z, b.w), add2(osum[1], inf[1]));
    *reinterpret_cast<float4*>(td.out[S_ROCK] + gi) = make_float4(r0.x, r0.y, r1.x, r1.y);
}

template <bool SED>
__global__ void __launch_bounds__(TT_NTH, 4) k_transport_tile1(const __grid_constant__ TerrainDesc td, int steps) {
    __shared__ __align__(16) TileShared sm;
    transport_tile<SED>(td.h, sm, blockIdx.x * TW, td.row_lo + blockIdx.y * TT_H);
    if (SED && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *td.h.step += (unsigned long long)steps;
}

// shift: 0 when k_hydro's tiles have 16 rows as these, 1 when they have 8
template <bool SED>
__global__ void __launch_bounds__(TT_NTH, 4) k_transport_tile(const __grid_constant__ BatchParams bp, int shift, int steps) {
    __shared__ __align__(16) TileShared sm;
    const int t = find_terrain(bp.tile0, bp.nterr, blockIdx.x << shift);
    const unsigned tile = blockIdx.x - (bp.tile0[t] >> shift), tiles_x = bp.t[t].tiles_x;
    transport_tile<SED>(bp.t[t], sm, (tile % tiles_x) * TW, (tile / tiles_x) * TT_H);
    if (SED && tile == 0 && threadIdx.x == 0) *bp.t[t].step += (unsigned long long)steps;
}

template <bool SED>
__global__ void __launch_bounds__(32 * R_WARPS, SED ? 2 : 3) k_transport_rows(const __grid_constant__ TerrainDesc td, int steps) {
    const TerrainHot& h = td.h;
    Taps<1> taps;
    talus_rows(
        h.c, h.b_ero, h.out[S_ROCK], blockIdx.x, td.row_lo + blockIdx.y * R_ROWS,
        [&](int x, int y, size_t gi) {
            const float* const se[1] = {h.s_ero};
            if (SED) load_taps<1>(h.c, se, x, y, ldg2(h.u + gi), ldg2(h.v + gi), taps);
        },
        [&](int, int, size_t gi) {
            if (SED) st2(h.out[S_SED] + gi, mix_taps(taps, 0));
        });
    if (SED && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *td.h.step += (unsigned long long)steps;
}

// ---------------------------------------------------------------------------
// tensor maps
// ---------------------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::once_flag g_encode_once;

bool encode_box(CUtensorMap* map, const float* base, int n, int box_h) {
    std::call_once(g_encode_once, [] {
        cudaDriverEntryPointQueryResult q;
        void* fn = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    });
    if (!g_encode) return false;
    cuuint64_t dims[2] = {(cuuint64_t)n, (cuuint64_t)n};
    cuuint64_t strides[1] = {(cuuint64_t)n * sizeof(float)};
    cuuint32_t box[2] = {(cuuint32_t)RW, (cuuint32_t)box_h};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box,
                          estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

}  // namespace

bool TmaCache::get(const float* base, int n, int box_h, CUtensorMap* out) {
    for (auto& e : entries)
        if (e.base == base && e.n == n && e.box_h == box_h) {
            *out = e.map;
            return true;
        }
    Entry e{base, n, box_h, {}};
    if (!encode_box(&e.map, base, n, box_h)) return false;
    entries.push_back(e);
    *out = e.map;
    return true;
}

bool fused_tile_ok(int n, int th) { return (th == 16 || th == 8) && n % TW == 0 && n % th == 0; }

int fused_tiles(int n, int th) { return (n / TW) * (n / th); }

int chunk_rows(const int* sides, const int* rows, int count) {
    int most = 0;
    size_t cells = 0;
    for (int i = 0; i < count; ++i) {
        most = rows[i] > most ? rows[i] : most;
        cells += (size_t)sides[i] * rows[i];
    }
    size_t r = cells / SW / T_FILL;
    for (r = r < 4 ? 4 : r; r < (size_t)most; ++r) {
        size_t tasks = 0;
        for (int i = 0; i < count; ++i) tasks += transport_tasks(sides[i], rows[i], (int)r);
        if (tasks <= (size_t)T_FILL) break;
    }
    return (int)r;
}

int transport_tasks(int n, int rows, int t_rows) { return strips(n) * ((rows + t_rows - 1) / t_rows); }

namespace {
int task_blocks(int tasks) { return (tasks + T_WARPS - 1) / T_WARPS; }
}  // namespace

bool fill_desc(TerrainDesc& d, const TerrainSrc& s, int th, TmaCache& cache) {
    TerrainHot& h = d.h;
    h.c = s.c;
    h.rain = s.rain;
    for (int f = 0; f < S_COUNT; ++f) h.out[f] = s.out[f];
    h.u = s.u;
    h.v = s.v;
    h.s_ero = s.s_ero;
    h.b_ero = s.b_ero;
    h.s_prev = s.s_prev;
    h.s_keep = s.s_keep;
    h.uv_prev = s.uv_prev;
    h.step = s.step;
    h.tiles_x = s.c.n / TW;
    h.t_rows = chunk_rows(&s.c.n, &s.c.n, 1);
    d.row_lo = 0;
    d.row_hi = s.c.n;
    const int in_fields[H_N] = {S_ROCK, S_WATER, S_FL, S_FR, S_FT, S_FB, S_SED};
    for (int f = 0; f < H_N; ++f)
        if (!cache.get(s.in[in_fields[f]], s.c.n, th + 2, &d.maps[f])) return false;
    return true;
}

namespace {
// Worlds from this side up keep separate inner and edge code in k_hydro (edge
// tiles are under 4 % of a 4096² launch at tile height 16); smaller ones,
// where edge tiles are 8 % (2048²) to 56 % (256²) of the launch, run one code
// path.
constexpr int SPLIT_MIN_N = 4096;

// Forms of the talus launch: a single world up to this side runs talus_rows, a
// larger one and batches tiles up to the cells below, above them warps march.
// One step of one world, alone / three worlds in turn, us, by tiles, marching:
// 1024² 37 / 20, 44 / 24; 2048² 98 / 76, 106 / 77; 3072² 188 / 166, 198 / 158
// (smoothing, 16 such steps: 3596 / 3424, 3887 / 3383); 4096² 347 / 315, 377 / 312.
// 16 chained steps, of which two gather: 1024² 372 / 297, 462 / 325; 1536² 825 / 646,
// 892 / 645; 1792² 1071 / 876, 1158 / 847; 2048² 1322 / 1131, 1409 / 1078.  Eight by
// rows, tiles: 256² 68 / 25, 76 / 28; 384² 80 / 31, 82 / 36; 448² 87 / 39, 92 / 40,
// four worlds of 448² on their own streams 164 / 166, 152 / 140.
constexpr int ROWS1_MAX_N = 384;
bool tiled(size_t cells, bool thermal, bool last) {
    if (!thermal) return true;  // the gather alone, nothing to march for
    return last ? cells < (size_t)4096 * 4096 : cells <= (size_t)1536 * 1536;
}

template <int TH, int NT>
void launch_hydro1(const TerrainDesc& td, int index, int* err, cudaStream_t st) {
    const dim3 tiles(td.h.tiles_x, (td.row_hi - td.row_lo) / TH);
    const bool split = td.h.c.n >= SPLIT_MIN_N;
    if (index > 0) {
        if (split) k_hydro1<TH, NT, true, true><<<tiles, NT, 0, st>>>(td, index, err);
        else k_hydro1<TH, NT, false, true><<<tiles, NT, 0, st>>>(td, index, err);
    } else {
        if (split) k_hydro1<TH, NT, true, false><<<tiles, NT, 0, st>>>(td, 0, err);
        else k_hydro1<TH, NT, false, false><<<tiles, NT, 0, st>>>(td, 0, err);
    }
    count_launch();
}
// 8-row tiles have 256 threads up to these cells, 128 above: 16 steps without talus,
// alone / three worlds in turn, us, by 256 and 128 threads: 256² 75 / 28 and 87 / 31,
// 448² 93 / 39 and 99 / 41, 640² 134 / 78 and 125 / 62, 1024² 235 / 244 and 212 / 193.
bool small_launch(size_t cells) { return cells <= (size_t)512 * 512; }
void launch_hydro1(const TerrainDesc& td, int th, int index, int* err, cudaStream_t st) {
    if (th == 16) launch_hydro1<16, 256>(td, index, err, st);
    else if (small_launch((size_t)td.h.c.n * (td.row_hi - td.row_lo))) launch_hydro1<8, 256>(td, index, err, st);
    else launch_hydro1<8, 128>(td, index, err, st);
}

template <int TH, int NT>
void launch_hydro_table(const BatchParams& bp, const CUtensorMap* maps, int tiles, int index, int* err,
                        cudaStream_t st) {
    if (index > 0) k_hydro<TH, NT, true><<<tiles, NT, 0, st>>>(bp, maps, index, err);
    else k_hydro<TH, NT, false><<<tiles, NT, 0, st>>>(bp, maps, 0, err);
    count_launch();
}

void launch_transport1(const TerrainDesc& td, bool last, int steps, cudaStream_t st) {
    const int rows = td.row_hi - td.row_lo;
    if (td.h.c.thermal && td.h.c.n <= ROWS1_MAX_N) {
        const dim3 grid(strips(td.h.c.n), rows / R_ROWS);
        if (last) k_transport_rows<true><<<grid, 32 * R_WARPS, 0, st>>>(td, steps);
        else k_transport_rows<false><<<grid, 32 * R_WARPS, 0, st>>>(td, 0);
        count_launch();
        return;
    }
    if (tiled((size_t)td.h.c.n * rows, td.h.c.thermal, last)) {
        const dim3 grid(td.h.tiles_x, rows / TT_H);
        if (last) k_transport_tile1<true><<<grid, TT_NTH, 0, st>>>(td, steps);
        else k_transport_tile1<false><<<grid, TT_NTH, 0, st>>>(td, 0);
        count_launch();
        return;
    }
    const int tasks = transport_tasks(td.h.c.n, rows, td.h.t_rows);
    if (last) k_transport1<true><<<task_blocks(tasks), 32 * T_WARPS, 0, st>>>(td, tasks, steps);
    else k_transport1<false><<<task_blocks(tasks), 32 * T_WARPS, 0, st>>>(td, tasks, 0);
    count_launch();
}
}  // namespace

void launch_talus_march(const StepConsts& c, const float* rock, float* rock_o, cudaStream_t st) {
    TerrainDesc td{};
    td.h.c = c;
    td.h.b_ero = const_cast<float*>(rock);  // (read only)
    td.h.out[S_ROCK] = rock_o;
    td.h.t_rows = chunk_rows(&c.n, &c.n, 1);
    td.row_hi = c.n;
    const int tasks = transport_tasks(c.n, c.n, td.h.t_rows);
    k_transport1<false><<<task_blocks(tasks), 32 * T_WARPS, 0, st>>>(td, tasks, 0);
    count_launch();
}

void launch_fused_table(const BatchParams& bp, const CUtensorMap* maps, int total_tiles, int th, bool thermal,
                        ChainPos pos, int* err, cudaStream_t st) {
    const size_t cells = (size_t)total_tiles * TW * th;
    if (th == 16) launch_hydro_table<16, 256>(bp, maps, total_tiles, pos.index, err, st);
    else if (small_launch(cells)) launch_hydro_table<8, 256>(bp, maps, total_tiles, pos.index, err, st);
    else launch_hydro_table<8, 128>(bp, maps, total_tiles, pos.index, err, st);
    if (!pos.last && !thermal) return;
    if (tiled(cells, thermal, pos.last)) {
        const int shift = th == TT_H ? 0 : 1, tiles = total_tiles >> shift;
        if (pos.last) k_transport_tile<true><<<tiles, TT_NTH, 0, st>>>(bp, shift, pos.index + 1);
        else k_transport_tile<false><<<tiles, TT_NTH, 0, st>>>(bp, shift, 0);
        count_launch();
        return;
    }
    if (pos.last) k_transport<true><<<task_blocks(bp.tasks), 32 * T_WARPS, 0, st>>>(bp, pos.index + 1);
    else k_transport<false><<<task_blocks(bp.tasks), 32 * T_WARPS, 0, st>>>(bp, 0);
    count_launch();
}

void launch_fused_half(const TerrainDesc& td, int th, int which, int* err, cudaStream_t st) {
    if (td.row_hi <= td.row_lo) return;
    if (which == 1) launch_transport1(td, true, 1, st);
    else launch_hydro1(td, th, 0, err, st);
}

void launch_fused_one(const TerrainDesc& td, int th, ChainPos pos, int* err, cudaStream_t st) {
    launch_hydro1(td, th, pos.index, err, st);
    if (pos.last || td.h.c.thermal) launch_transport1(td, pos.last, pos.index + 1, st);
}

}  // namespace hg
