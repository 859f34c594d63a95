// Shared pieces of the fused steps' kernels: the staged box, 8-byte accesses,
// and the talus pass with a row of a strip per warp.
#pragma once
#include "hg_device.cuh"
#include "hg_internal.h"

namespace hg {

constexpr int TW = 64;           // tile width
constexpr int HX = 4;            // halo columns: 16-byte aligned TMA boxes
constexpr int RW = TW + 2 * HX;  // 72

__device__ __forceinline__ float2 ld2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 ldg2(const float* p) { return __ldg(reinterpret_cast<const float2*>(p)); }
__device__ __forceinline__ void st2(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }

// Sets the cells of a staged box that lie outside the grid to v.  The box
// (ROWS x RW cells, row 0 at global row gy0, column 0 at global column
// gx0 = tx0 - HX) reaches past the grid only through its HX outer columns
// on either side and its HALO outer rows on either side, so only those
// are visited (a corner cell twice, with the same value).
template <int ROWS, int HALO, int NTH>
__device__ __forceinline__ void fill_outside(float* box, int gx0, int gy0, int n, float v, int tid) {
    constexpr int SIDE = ROWS * 2 * HX;  // the outer columns of every row
    constexpr int CAP = 2 * HALO * RW;   // the outer rows
    for (int i = tid; i < SIDE + CAP; i += NTH) {
        int r, col;
        if (i < SIDE) {
            r = i / (2 * HX);
            const int k = i % (2 * HX);
            col = k < HX ? k : RW - 2 * HX + k;
        } else {
            const int j = i - SIDE, rr = j / RW;
            col = j % RW;
            r = rr < HALO ? rr : ROWS - 2 * HALO + rr;
        }
        const int gx = gx0 + col, gy = gy0 + r;
        if (gx < 0 || gx >= n || gy < 0 || gy >= n) box[r * RW + col] = v;
    }
}

// A pair of a row's heights and the pairs one column to the left and right
// (the neighbouring lanes' cells; the warp's outermost two are the lane's own).
struct RockRow {
    float2 c, l, r;
};
__device__ __forceinline__ float2 from_left(float2 a) { return make_float2(__shfl_up_sync(0xffffffffu, a.y, 1), a.x); }
__device__ __forceinline__ float2 from_right(float2 a) {
    return make_float2(a.y, __shfl_down_sync(0xffffffffu, a.x, 1));
}
__device__ __forceinline__ RockRow rock_row(float2 c) { return RockRow{c, from_left(c), from_right(c)}; }

constexpr int SW = 60;  // columns a warp's strip delivers
__host__ __device__ constexpr int strips(int n) { return (n + SW - 1) / SW; }

// A small world's rock talus pass: a block takes 8 rows of a strip, one warp
// per row (and one for the row above and below), so a launch is one pass over
// short straight code instead of a march of several rows per warp: there the
// time is latency, and chunks of few rows recompute half of their outflows.
// Rows exchange the outflows they send each other through shared memory.
// begin(x, y, gi) runs after the rock's loads are issued and end(x, y, gi) after
// the outflows, in lanes whose pair this block delivers: a sediment gather
// leaves its taps in flight between them.
constexpr int R_ROWS = 8, R_WARPS = R_ROWS + 2;
struct TalusRates {
    float Kalpha, Kspeed, x_cross, b_diag;
    int fast_div;
};
// DIRT: layer 1, whose drops are rock's plus dirt's and whose dirt moves;
// else in_dirt is not read and rock moves
template <bool DIRT, class Begin, class End>
__device__ __forceinline__ void talus_rows(const StepConsts1& c, const TalusRates& t, const float* __restrict__ in_rock,
                                           const float* __restrict__ in_dirt, float* __restrict__ out, int strip, int y0,
                                           Begin begin, End end) {
    __shared__ float2 to_up[R_WARPS][3][32], to_down[R_WARPS][3][32];  // T, RT, LT / B, RB, LB at the receiving column
    const int n = c.n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x = strip * SW - 2 + 2 * lane, y = y0 - 1 + warp;
    const bool in = x >= 0 && x < n;
    const bool own = in && lane >= 1 && lane <= SW / 2 && warp >= 1 && warp <= R_ROWS;
    const size_t gi = (size_t)y * n + x;
    auto height = [&](const float* f, int r) {
        return in && r >= 0 && r < n ? ldg2(f + (size_t)r * n + x) : pf(FAR_HEIGHT);
    };
    const float2 c0 = height(in_rock, y - 1), c1 = height(in_rock, y), c2 = height(in_rock, y + 1);
    float2 g0, g1, g2;
    if (DIRT) {
        g0 = height(in_dirt, y - 1);
        g1 = height(in_dirt, y);
        g2 = height(in_dirt, y + 1);
    }
    if (own) begin(x, y, gi);
    float2 o[8];
    if (y >= 0 && y < n) {
        const RockRow dn = rock_row(c0), md = rock_row(c1), up = rock_row(c2);
        float2 dm[8] = {sub2(md.c, md.l), sub2(md.c, md.r), sub2(md.c, up.c), sub2(md.c, dn.c),
                        sub2(md.c, up.l), sub2(md.c, up.r), sub2(md.c, dn.l), sub2(md.c, dn.r)};
        if (DIRT) {
            const RockRow dg = rock_row(g0), mg = rock_row(g1), ug = rock_row(g2);
            const float2 ng[8] = {mg.l, mg.r, ug.c, dg.c, ug.l, ug.r, dg.l, dg.r};
#pragma unroll
            for (int k = 0; k < 8; ++k) dm[k] = add2(dm[k], sub2(mg.c, ng[k]));
        }
        cell_thermal_outflows_dh2(c.dt, t.Kalpha, t.Kspeed, t.x_cross, t.b_diag, t.fast_div, DIRT ? g1 : md.c, dm, o);
    }
    if (!in || y < 0 || y >= n) {
#pragma unroll
        for (int d = 0; d < 8; ++d) o[d] = pf(0.0f);
    }
    to_up[warp][0][lane] = o[2];
    to_up[warp][1][lane] = from_left(o[5]);
    to_up[warp][2][lane] = from_right(o[4]);
    to_down[warp][0][lane] = o[3];
    to_down[warp][1][lane] = from_left(o[7]);
    to_down[warp][2][lane] = from_right(o[6]);
    const float2 lr = add2(from_left(o[1]), from_right(o[0]));
    float2 osum = sub2(pf(0.0f), o[0]);
#pragma unroll
    for (int d = 1; d < 8; ++d) osum = sub2(osum, o[d]);
    if (own) end(x, y, gi);
    __syncthreads();
    if (!own) return;
    // the shader's order: L, R, T, B, LT, RT, LB, RB
    float2 inf = add2(add2(lr, to_down[warp + 1][0][lane]), to_up[warp - 1][0][lane]);
    inf = add2(add2(inf, to_down[warp + 1][1][lane]), to_down[warp + 1][2][lane]);
    inf = add2(add2(inf, to_up[warp - 1][1][lane]), to_up[warp - 1][2][lane]);
    st2(out + gi, add2(DIRT ? g1 : c1, add2(osum, inf)));
}
template <class Begin, class End>
__device__ __forceinline__ void talus_rows(const StepConsts1& c, const float* __restrict__ in_rock,
                                           float* __restrict__ out_rock, int strip, int y0, Begin begin, End end) {
    const TalusRates t{c.Kalpha0, c.Kspeed0, c.talus_x_cross, c.talus_b_diag, c.fast_div};
    talus_rows<false>(c, t, in_rock, nullptr, out_rock, strip, y0, begin, end);
}
// Maps up to this side gather the sediment within the rock's talus launch: one
// launch less (two layers, one step: 384² 109 us apart, 103 together; 2048² 200
// apart, 215 together).
constexpr int ROWS_MAX_N = 768;

// smoothing's particle branch (glsl/smoothing.glsl:76-95), per cell: momentum
// fold and water decay
struct ParticleCells {
    float count;  // droplets
    const float* water;
    float* water_o;
    const float* mom[4];
    float* mom_o[4];
};
inline ParticleCells particle_cells_of(float count, const PWorld& in, const PWorld& out) {
    ParticleCells p{count, in.water, out.water, {}, {}};
    for (int k = 0; k < 4; ++k) {
        p.mom[k] = in.mom[k];
        p.mom_o[k] = out.mom[k];
    }
    return p;
}
// smoothing's particle branch at the cells (x, y), (x + 1, y): border texels
// copy their water and leave the momentum map's write buffer as it was
__device__ __forceinline__ void particle_cells(const ParticleCells& a, int n, size_t gi, int x, int y) {
    const bool row = y == 0 || y == n - 1;
    const bool b0 = row || x == 0, b1 = row || x + 2 == n;
    const float2 wat = ldg2(a.water + gi);
    float2 w = mul2(wat, pf(gclamp(1.0f - 8e-8f * a.count, 0.0f, 1.0f)));
    w = make_float2(w.x < 1e-6f ? 0.0f : w.x, w.y < 1e-6f ? 0.0f : w.y);
    st2(a.water_o + gi, make_float2(b0 ? wat.x : w.x, b1 ? wat.y : w.y));
    const float2 keep = pf(gclamp(1.0f - 1e-12f * a.count, 0.0f, 1.0f)), take = pf(1e-12f * a.count);
    float2 mx = add2(mul2(ldg2(a.mom[0] + gi), keep), mul2(take, ldg2(a.mom[2] + gi)));
    float2 my = add2(mul2(ldg2(a.mom[1] + gi), keep), mul2(take, ldg2(a.mom[3] + gi)));
    const float2 len = sqrt_newton2(add2(mul2(mx, mx), mul2(my, my)));  // (below 2^-100 it stays far below 1e-12)
    const bool zx = len.x < 1e-12f, zy = len.y < 1e-12f;
    mx = make_float2(zx ? 0.0f : mx.x, zy ? 0.0f : mx.y);
    my = make_float2(zx ? 0.0f : my.x, zy ? 0.0f : my.y);
    const float2 z = pf(0.0f), v[4] = {mx, my, z, z};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (!b0 && !b1) {
            st2(a.mom_o[k] + gi, v[k]);
        } else {
            if (!b0) a.mom_o[k][gi] = v[k].x;
            if (!b1) a.mom_o[k][gi + 1] = v[k].y;
        }
    }
}

}  // namespace hg
