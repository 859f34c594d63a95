// Reverse-mode adjoint of the one-layer grid step (talus passes included).
//
// One reversed step j works on the step's input state X_j, the step's
// forward intermediates kept by the segment recompute (velocity u, v and the
// eroded sediment se of every cell: the fused forward step writes them
// anyway) and the adjoint A of the step's outputs.  The adjoint of a state is
// kept as twelve fields (AdjState) from which a reader takes each cell's own
// terms and adds what its neighbours pass, in a fixed order (deterministic),
// so no separate gather pass runs.  One kernel per step:
//   k_adj_cell      64 x 8 tiles of X_j and of A's fields that neighbours
//                   read, staged by TMA with a one-row halo, this step's rain
//                   added in shared memory; one thread per pair of cells
//                   (f32x2) recomputes the forward flux and erosion (the
//                   operations of hg_device.cuh, so every branch is the
//                   forward's) and reverses them; it writes the adjoint of
//                   X_j, accumulates the Ks gradient and clears its
//                   sediment-adjoint cells (double buffer); then, with the
//                   sediment adjoint of step j - 1 now final, it reverses
//                   that step's semi-Lagrangian gather: a scatter to the
//                   back-trace's four taps (atomicAdd: the taps are data
//                   dependent) and the back-trace velocity adjoint
//   k_adj_sediment  the same scatter on its own, for a segment's last step
//                   (its intermediates exist only after the recompute)
//   k_adj_final     the gathered rock adjoint of the first state
//   k_adj_thermal   the talus passes reversed: gathers the output rock's
//                   adjoint over its box while the eroded rock's box flies,
//                   and yields the adjoint of the eroded rock, which
//                   k_adj_cell then takes
//
// Subgradients: max(0, x) and min(1, q) pass the derivative of the taken
// argument (ties take the constant side), clamps pass 0 when clamped,
// dissolve/deposit/exhaustion use the taken branch, floor() is locally
// constant, and in water films below FILM_DEPTH the velocity and the flux
// scale are locally constant.  The formulas follow the shaders cited in hg_device.cuh.  The
// reversed arithmetic divides through correctly rounded reciprocals
// (x * (1/y), within two ulps of x / y); the recomputed forward's quotients
// and roots are the forward's own, so its values and branches are too.
#include "hg_internal.h"
#include "hg_tile.cuh"
#include "hg_tma.cuh"

namespace hg {

namespace {

constexpr int BX = 32, BY = 8;
__device__ __forceinline__ size_t at(int n, int x, int y) { return (size_t)y * n + x; }

// Water films thinner than this (the depth below which the erosion ignores
// the velocity, glsl/hydro_erosion.glsl:45-52) pass no adjoint through the
// velocity (u = flux difference / depth) or the flux scale (K = depth /
// outflow): both derivatives grow like 1/depth and overflow float in the
// films that intermittent rain leaves (depths reach 1e-35), where they carry
// no usable gradient anyway.
constexpr float FILM_DEPTH = 5e-4f;

// ---- sediment_transport reversed ------------------------------------------------
// Cells (x, y) and (x + 1, y) of a step whose output sediment adjoint is `a`,
// with the back-trace's taps of the eroded sediment in q: scatter to the taps
// of dse, back-trace velocity adjoint into du, dv.  Neighbouring cells mostly
// trace to neighbouring taps: the column they share is added once.
__device__ __forceinline__ void sediment_adjoint(const StepConsts& c, const Taps<1>& q, size_t i, float2 a, float* dse,
                                                 float* du, float* dv) {
    const int n = c.n;
    const float2 fx = q.tr.fx, fy = q.tr.fy, ox = sub2(pf(1.0f), fx), oy = sub2(pf(1.0f), fy);
    const float2 a0 = mul2(a, ox), a1 = mul2(a, fx);
    float2 w00 = mul2(a0, oy), w01 = mul2(a0, fy);
    float2 w10 = mul2(a1, oy), w11 = mul2(a1, fy);
    const int x0 = (int)q.tr.ix[0], y0 = (int)q.tr.iy[0], x1 = (int)q.tr.ix[1], y1 = (int)q.tr.iy[1];
    const bool shared = x0 + 1 < n && x1 == x0 + 1 && y1 == y0;
    if (shared) {
        w10.x += w00.y;
        w11.x += w01.y;
        w00.y = w01.y = 0.0f;
    }
    auto add = [&](int xx, int yy, float v) {
        if (xx < n && yy < n && v != 0.0f) atomicAdd(dse + at(n, xx, yy), v);
    };
    add(x0, y0, w00.x);
    add(x0 + 1, y0, w10.x);
    add(x0, y0 + 1, w01.x);
    add(x0 + 1, y0 + 1, w11.x);
    add(x1, y1, w00.y);
    add(x1 + 1, y1, w10.y);
    add(x1, y1 + 1, w01.y);
    add(x1 + 1, y1 + 1, w11.y);
    auto s = [&](int k) { return make_float2(q.t[0][k][0], q.t[0][k][1]); };  // 00, 10, 01, 11
    const float2 dfx = add2(mul2(sub2(s(1), s(0)), oy), mul2(sub2(s(3), s(2)), fy));
    const float2 dfy = sub2(add2(mul2(s(2), ox), mul2(s(3), fx)), add2(mul2(s(0), ox), mul2(s(1), fx)));
    const float2 gx = mul2(mul2(a, dfx), pf(-c.dt)), gy = mul2(mul2(a, dfy), pf(-c.dt));
    // a point clamped to the grid passes nothing on (the last texel holds only
    // points at its very edge or beyond)
    auto inside = [&](int t, float f) { return (t > 0 || f > 0.0f) && t < n - 1; };
    st2(du + i, make_float2(inside(x0, fx.x) ? gx.x : 0.0f, inside(x1, fx.y) ? gx.y : 0.0f));
    st2(dv + i, make_float2(inside(y0, fy.x) ? gy.x : 0.0f, inside(y1, fy.y) ? gy.y : 0.0f));
}

__global__ void k_adj_sediment(StepConsts c, AdjSlot sl, const float* __restrict__ as_, float* __restrict__ dse,
                               float* __restrict__ du, float* __restrict__ dv) {
    const int x = 2 * (blockIdx.x * BX + threadIdx.x), y = blockIdx.y * BY + threadIdx.y;
    const size_t i = at(c.n, x, y);
    Taps<1> q;
    const float* const se[1] = {sl.se};
    load_taps<1>(c, se, x, y, ldg2(sl.u + i), ldg2(sl.v + i), q);
    sediment_adjoint(c, q, i, ldg2(as_ + i), dse, du, dv);
}

// A state's adjoint at the cells (x, y), (x + 1, y): own terms plus what the
// neighbours pass (L, R, T, B neighbours, fixed order).
// nbw: what the neighbours' height differences toward the cell pass to its total
// (w = rock + water enters those with a minus sign)
template <bool EDGE>
__device__ __forceinline__ float2 adj_nbw(const StepConsts1& c, const AdjState& A, int x, int y, size_t i, float2 h0,
                                          float2 h1) {
    const int n = c.n;
    const float2 z = pf(0.0f), w = pf(c.dt * c.G);
    const float l = !EDGE || x > 0 ? __ldg(A.h[1] + i - 1) : 0.0f;      // left neighbour's R
    const float r = !EDGE || x + 2 < n ? __ldg(A.h[0] + i + 2) : 0.0f;  // right neighbour's L
    const float2 t = !EDGE || y < n - 1 ? ldg2(A.h[3] + i + n) : z;     // top neighbour's B
    const float2 b = !EDGE || y > 0 ? ldg2(A.h[2] + i - n) : z;         // bottom neighbour's T
    const float2 s = add2(mul2(w, make_float2(l, h1.x)), mul2(w, make_float2(h0.y, r)));
    return add2(add2(s, mul2(w, t)), mul2(w, b));
}
// the neighbours' terrain-normal terms
template <bool EDGE>
__device__ __forceinline__ float2 adj_normal(const AdjState& A, int n, int x, int y, size_t i) {
    const float2 z = pf(0.0f), nx = ldg2(A.nx + i);
    const float l = !EDGE || x > 0 ? __ldg(A.nx + i - 1) : 0.0f;
    const float r = !EDGE || x + 2 < n ? __ldg(A.nx + i + 2) : 0.0f;
    const float2 b = !EDGE || y > 0 ? ldg2(A.nz + i - n) : z, t = !EDGE || y < n - 1 ? ldg2(A.nz + i + n) : z;
    return sub2(add2(sub2(make_float2(l, nx.x), make_float2(nx.y, r)), b), t);
}

// ---- k_adj_cell ------------------------------------------------------------------
// A warp per row of 32 pairs of cells, in f32x2; the tile is staged with a
// one-row halo.  Bound by the latency of its loads under too few warps (80
// registers, 24 warps per SM) before DRAM (131 MB at 1024²): what a thread
// alone reads goes into shared memory by cp.async and to registers only where
// it is used, and so do the neighbours' terms.  1024² with talus, per launch:
// one cell at a time with every neighbour's share stored by itself 45 us (827
// instructions per cell, 172 MB); pairs with the inputs in registers 44
// (16 warps per SM); as here 33 (460).  64 x 4 tiles take 1 % longer, 4 blocks
// per SM 8 % (spills), 2 blocks 10 %.
constexpr int TH = 8, NTH = TW / 2 * TH;
constexpr int H_RH = TH + 2, H_BOX = RW * H_RH, H_RC = ((H_BOX + 31) / 32) * 32;
// the pair's own inputs: rock, water, sediment adjoint, back-trace velocity
// adjoint, Ks, velocity of step j - 1
enum { O_B = 0, O_D, O_S, O_DU, O_DV, O_KS, O_PU, O_PV, O_N };
enum { X_B = 0, X_D, X_S, X_FL, X_FR, X_FT, X_FB, X_H, X_P = X_H + 4, X_GU, X_GV, X_N };  // state, adjoint

__device__ __forceinline__ float2 sel(bool x, bool y, float2 a, float2 b) {
    return make_float2(x ? a.x : b.x, y ? a.y : b.y);
}
__device__ __forceinline__ float2 frcp2(float2 a) { return make_float2(__frcp_rn(a.x), __frcp_rn(a.y)); }

// Forward flux of two cells with the intermediates its adjoint needs: the
// operations of cell_flux2 (hg_device.cuh), so every branch is the forward's.
// Directions L, R, T, B; wn[] neighbour totals, in[] neighbours' facing flux.
// A direction is live where g > 0.
struct FluxFwd2 {
    float2 g[4];  // outflows before scaling
    float2 sum_out, K, arg, vz, u, v, len;
    float2 rden, rvz, rlen;      // reciprocals, of 1 where no use is made of them
    bool scaled_x, scaled_y;
};
__device__ __forceinline__ FluxFwd2 flux_fwd2(const StepConsts& c, int x, int y, float2 w, float2 d1,
                                              const float2 f[4], const float2 wn[4], const float2 in[4], bool border) {
    FluxFwd2 o;
    const float2 EK = pf(c.EK), dt = pf(c.dt), G = pf(c.G);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 t = add2(mul2(EK, f[k]), mul2(dt, mul2(G, sub2(w, wn[k]))));
        o.g[k] = make_float2(fmaxf(0.0f, t.x), fmaxf(0.0f, t.y));
    }
    if (border) {
        if (x <= 0) o.g[0].x = 0.0f;
        if (x + 1 >= c.n - 1) o.g[1].y = 0.0f;
        if (y <= 0) o.g[3] = pf(0.0f);
        else if (y >= c.n - 1) o.g[2] = pf(0.0f);
    }
    const float2 sum_in = add2(add2(add2(in[0], in[1]), in[2]), in[3]);
    o.sum_out = add2(add2(add2(o.g[0], o.g[1]), o.g[2]), o.g[3]);
    const float2 den = mul2(o.sum_out, dt);
    const bool fullx = d1.x >= den.x, fully = d1.y >= den.y;
    o.K = o.rden = pf(1.0f);
    o.scaled_x = o.scaled_y = false;
    if (!(fullx & fully)) {
        const float2 dn = make_float2(fullx ? 1.0f : den.x, fully ? 1.0f : den.y);
        float2 q;
        if (depth_range(d1) & den_range(dn.x) & den_range(dn.y)) {
            o.rden = rcp_newton2(dn);
            q = div_recip2(d1, make_float2(-dn.x, -dn.y), o.rden);
        } else {
            o.rden = frcp2(dn);
            q = make_float2(d1.x / dn.x, d1.y / dn.y);
        }
        o.scaled_x = !fullx && q.x < 1.0f;
        o.scaled_y = !fully && q.y < 1.0f;
        o.K = sel(o.scaled_x, o.scaled_y, q, o.K);
    }
    o.arg = add2(d1, mul2(dt, sub2(sum_in, mul2(o.sum_out, o.K))));
    o.vz = add2(d1, make_float2(fmaxf(0.0f, o.arg.x), fmaxf(0.0f, o.arg.y)));
    const float2 nu = sub2(add2(sub2(in[0], f[0]), f[1]), in[1]), nv = sub2(add2(sub2(in[3], f[3]), f[2]), in[2]);
    const bool wetx = o.vz.x > 0.0f, wety = o.vz.y > 0.0f;
    const float2 vs = sel(wetx, wety, o.vz, pf(1.0f)), nd = make_float2(-vs.x, -vs.y);
    o.rvz = rcp_newton2(vs);
    o.u = sel(wetx, wety, div_recip2(nu, nd, o.rvz), pf(0.0f));
    o.v = sel(wetx, wety, div_recip2(nv, nd, o.rvz), pf(0.0f));
    float2 ss = add2(mul2(o.u, o.u), mul2(o.v, o.v));
    const bool ok = num_range(nu.x) & num_range(nu.y) & num_range(nv.x) & num_range(nv.y) & den_range(vs.x) &
                    den_range(vs.y) & root_range(ss.x) & root_range(ss.y);
    if (ok) {
        o.len = sqrt_newton2(ss);
        o.rlen = rcp_newton2(sel(o.len.x > 0.0f, o.len.y > 0.0f, o.len, pf(1.0f)));
    } else {
        o.rvz = frcp2(vs);
        o.u = make_float2(wetx ? nu.x / vs.x : 0.0f, wety ? nu.y / vs.y : 0.0f);
        o.v = make_float2(wetx ? nv.x / vs.x : 0.0f, wety ? nv.y / vs.y : 0.0f);
        ss = add2(mul2(o.u, o.u), mul2(o.v, o.v));
        o.len = make_float2(sqrtf(ss.x), sqrtf(ss.y));
        o.rlen = frcp2(o.len);
    }
    return o;
}

// 8 bytes of global memory into shared memory, in flight until copy_async_wait
// (of the same thread)
__device__ __forceinline__ void copy_async8(void* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const float* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <bool EDGE>
__device__ __forceinline__ void adj_tile(const AdjCellArgs& a, float* sm, uint64_t* bar, int tx0, int ty0,
                                         int* err) {
    const StepConsts& c = a.c;
    const RainStep& r = a.rain;
    const int n = c.n;
    const int tid = threadIdx.x;
    const int gx0 = tx0 - HX, gy0 = ty0 - 1;
    if (tid == 0) {
        mbar_arrive_expect_tx(bar, X_N * H_BOX * sizeof(float));
#pragma unroll
        for (int f = 0; f < X_N; ++f) tma_load_2d(sm + f * H_RC, &a.maps[f], gx0, gy0, bar);
    }
    // the pair's adjoint inputs, loaded while the tile flies, and the taps of
    // step j - 1's sediment gather, which the end reverses
    const int ix = (tid % (TW / 2)) * 2, iy = tid / (TW / 2);
    const int x = tx0 + ix, y = ty0 + iy;
    const size_t i = (size_t)y * n + x;
    const float2 z = pf(0.0f), one = pf(1.0f);
    float2* own = reinterpret_cast<float2*>(sm + X_N * H_RC) + tid;
    auto fetch = [&](int k, const float* p) { copy_async8(own + k * NTH, p + i); };
    if (a.scatter_prev) {
        fetch(O_PU, a.prev.u);
        fetch(O_PV, a.prev.v);
        prefetch_l2(a.prev.se + i);  // near the taps read at the end
    }
    fetch(O_B, a.gbe ? a.gbe : a.A.b);  // thermal on: the eroded rock's adjoint (k_adj_thermal)
    fetch(O_D, a.A.d);
    fetch(O_S, a.dse);
    fetch(O_DU, a.du);
    fetch(O_DV, a.dv);
    if (c.ks_field) fetch(O_KS, c.ks_field);
    const float2 Anrm = a.gbe ? z : adj_normal<EDGE>(a.A, n, x, y, i);
    constexpr int RG = (RW / 4) * H_RH;  // groups of four cells, at most one per thread
    static_assert(RG <= NTH, "one rain group per thread");
    uint32_t words[4] = {0, 0, 0, 0};
    const int rrx = (tid % (RW / 4)) * 4, rry = tid / (RW / 4), rgx = gx0 + rrx, rgy = gy0 + rry;
    const bool rains = r.active && tid < RG && (!EDGE || (rgx >= 0 && rgx < n && rgy >= 0 && rgy < n));
    if (rains && r.bernoulli) rain_words4(r, rgx, rgy, words);
    copy_async_wait();
    bool ok = __syncthreads_and(mbar_wait(bar, 0));
    if (!ok) {
        if (tid == 0) atomicExch(err, 1);
        mbar_wait(bar, 0);
        return;
    }
    if (r.active) {
        if (rains) {
            float* p = sm + X_D * H_RC + rry * RW + rrx;
            p[0] += rain_incr(r, words[0]);
            p[1] += rain_incr(r, words[1]);
            p[2] += rain_incr(r, words[2]);
            p[3] += rain_incr(r, words[3]);
        }
        __syncthreads();
    }
    const float* B = sm + X_B * H_RC;
    const float* D = sm + X_D * H_RC;
    const float* F[4] = {sm + X_FL * H_RC, sm + X_FR * H_RC, sm + X_FT * H_RC, sm + X_FB * H_RC};
    const int si = (1 + iy) * RW + HX + ix;
    const bool has_l = !EDGE || x > 0, has_r = !EDGE || x + 2 < n;
    const bool has_b = !EDGE || y > 0, has_t = !EDGE || y < n - 1;
    auto left = [&](const float* p, float2 m) { return make_float2(p[si - 1], m.x); };
    auto right = [&](const float* p, float2 m) { return make_float2(m.y, p[si + 2]); };
    // ---- adjoint of the step's output (0 outside the grid) ---------------
    float2 Ab, Ad;
    const float *h = sm + X_H * H_RC, *P = sm + X_P * H_RC, *GU = sm + X_GU * H_RC, *GV = sm + X_GV * H_RC;
    {
        const float2 w = pf(c.dt * c.G), h0 = ld2(h + si), h1 = ld2(h + H_RC + si);
        float2 nbw = add2(mul2(w, left(h + H_RC, h1)), mul2(w, right(h, h0)));
        nbw = add2(nbw, mul2(w, ld2(h + 3 * H_RC + si + RW)));
        nbw = add2(nbw, mul2(w, ld2(h + 2 * H_RC + si - RW)));
        Ab = own[O_B * NTH];
        if (!a.gbe) Ab = add2(sub2(Ab, nbw), Anrm);
        Ad = sub2(own[O_D * NTH], nbw);
    }
    // ---- forward recompute: flux --------------------------------------
    const float2 b = ld2(B + si), d1 = ld2(D + si);
    float2 bl = left(B, b), br = right(B, b), bb = ld2(B + si - RW), bt = ld2(B + si + RW);
    const float2 f[4] = {ld2(F[0] + si), ld2(F[1] + si), ld2(F[2] + si), ld2(F[3] + si)};
    float2 wn[4] = {add2(bl, left(D, d1)), add2(br, right(D, d1)), add2(bt, ld2(D + si + RW)),
                    add2(bb, ld2(D + si - RW))};
    // (outside the grid the staged tile is 0, what the normal and the inflows read there)
    const float2 in[4] = {left(F[1], f[1]), right(F[0], f[0]), ld2(F[3] + si + RW), ld2(F[2] + si - RW)};
    if (EDGE) {
        if (!has_l) wn[0].x = FAR_HEIGHT;
        if (!has_r) wn[1].y = FAR_HEIGHT;
        if (!has_t) wn[2] = pf(FAR_HEIGHT);
        if (!has_b) wn[3] = pf(FAR_HEIGHT);
    }
    const FluxFwd2 fw = flux_fwd2(c, x, y, add2(b, d1), d1, f, wn, in, EDGE);
    // ---- forward recompute: erosion speed and tilt ---------------------
    const float2 u = fw.u, v = fw.v, vz = fw.vz, len = fw.len;
    float2 ero = len, dero_dlen = one, dero_dvz = z;
    if ((vz.x < 1e-3f) | (vz.y < 1e-3f)) {  // (see capacity2; a depth from 1e-3 up has t = 0)
        constexpr float DD = 5e-4f - 1e-3f, RD = 1.0f / DD;
        const float2 dd = make_float2(fminf(fmaxf(5e-4f, vz.x), 1e-3f), fminf(fmaxf(5e-4f, vz.y), 1e-3f));
        const float2 t = div_recip2(add2(dd, pf(-1e-3f)), pf(-DD), pf(RD));
        const float2 fade = sub2(one, mul2(mul2(t, t), sub2(pf(3.0f), mul2(pf(2.0f), t))));
        const bool sx = vz.x < 1e-3f, sy = vz.y < 1e-3f;
        dero_dlen = sel(sx, sy, fade, one);
        ero = sel(sx, sy, mul2(len, fade), len);
        // d(smoothstep)/d(vz): 6 t (1 - t) / (5e-4 - 1e-3)
        const float2 dv = mul2(mul2(mul2(mul2(len, pf(6.0f)), t), sub2(one, t)), pf(2000.0f));
        dero_dvz = sel(sx && vz.x > 5e-4f && t.x > 0.0f && t.x < 1.0f, sy && vz.y > 5e-4f && t.y > 0.0f && t.y < 1.0f,
                       dv, z);
    }
    const float2 dx = sub2(br, bl), dz = sub2(bt, bb);
    const float2 cx = add2(dx, dx), cz = add2(dz, dz);
    const float2 L2 = add2(add2(mul2(cx, cx), pf(16.0f)), mul2(cz, cz));
    float2 L3 = sqrt_newton2(L2), r3 = rcp_newton2(L3);
    float2 ny = div_recip2(pf(-4.0f), make_float2(-L3.x, -L3.y), r3);
    float2 sin_a = sqrt_newton2(sub2(one, mul2(ny, ny)));
    if (!((L2.x <= 0x1p80f) & (L2.y <= 0x1p80f))) {
        auto tilt = [](float ddx, float ddz, float& nyl, float& r3l) {
            const float x1 = ddx * 2.0f - 0.0f * ddz, z1 = 2.0f * ddz - ddx * 0.0f;
            const float l = sqrtf(x1 * x1 + 16.0f + z1 * z1);
            nyl = -4.0f / l;
            r3l = __frcp_rn(l);
            return fabsf(sqrtf(1.0f - nyl * nyl));
        };
        sin_a.x = tilt(dx.x, dz.x, ny.x, r3.x);
        sin_a.y = tilt(dx.y, dz.y, ny.y, r3.y);
    }
    const float2 sa = make_float2(gmax(0.02f, sin_a.x), gmax(0.02f, sin_a.y));
    const float2 craw = mul2(mul2(pf(c.Kc), sa), ero);
    const float2 cc = make_float2(fmaxf(0.0f, craw.x), fmaxf(0.0f, craw.y));
    const float2 s = ld2(sm + X_S * H_RC + si);
    // ---- erosion reversed ----------------------------------------------
    st2(a.dse + i, z);  // free for the step after next
    // dissolve (K = dt Ks) and deposit (K = dt Kd) are one form; identity where
    // the empty dirt layer ends the layer loop, and where the rock is exhausted
    // (b' = 0, s' = s + b) both inputs take the sediment's adjoint
    const float2 e = sub2(cc, s), k1 = mul2(pf(c.Kls1), cc);
    const bool morex = cc.x > s.x, morey = cc.y > s.y;
    const bool endx = (cc.x > 0.0f) & !(k1.x > 0.0f), endy = (cc.y > 0.0f) & !(k1.y > 0.0f);
    const float2 Kls = mul2(pf(c.dt), c.ks_field ? own[O_KS * NTH] : pf(c.Ks0)), K = sel(morex, morey, Kls, pf(c.Kld0));
    const float2 left_b = sub2(b, mul2(Kls, e));
    const bool gonex = !endx & morex & (left_b.x < 0.0f), goney = !endy & morey & (left_b.y < 0.0f);
    const bool keepx = endx | gonex, keepy = endy | goney;
    const float2 as = own[O_S * NTH], diff = sub2(as, Ab);
    const float2 gs = sel(keepx, keepy, as, add2(mul2(Ab, K), mul2(as, sub2(one, K))));
    const float2 gb = sel(gonex, goney, as, Ab);
    const float2 gc = sel(keepx, keepy, z, mul2(diff, K));
    const float2 gKs = sel(!keepx & morex, !keepy & morey, mul2(diff, e), z);
    const bool ks_any = (gKs.x != 0.0f) | (gKs.y != 0.0f);
    float2 dks = z;
    if (ks_any) dks = ld2(a.dks + i);  // (added at the end)
    // capacity reversed
    const bool cx0 = craw.x > 0.0f, cy0 = craw.y > 0.0f;
    const float2 gk = mul2(gc, pf(c.Kc));
    const float2 gsa = mul2(gk, ero), gero = sel(cx0, cy0, mul2(gk, sa), z);
    const bool tx = cx0 & (sin_a.x > 0.02f), ty = cy0 & (sin_a.y > 0.02f);
    const float2 rsin = rcp_newton2(sel(tx, ty, sin_a, one));
    const float2 gny = mul2(gsa, mul2(make_float2(-ny.x, -ny.y), rsin));
    const float2 gL = mul2(mul2(gny, mul2(mul2(pf(4.0f), r3), r3)), pf(4.0f));
    st2(a.R.nx + i, sel(tx, ty, mul2(mul2(gL, dx), r3), z));
    st2(a.R.nz + i, sel(tx, ty, mul2(mul2(gL, dz), r3), z));
    const float2 glen = mul2(gero, dero_dlen);
    const bool mx = len.x > 0.0f, my = len.y > 0.0f;
    const float2 DU = add2(own[O_DU * NTH], sel(mx, my, mul2(mul2(glen, u), fw.rlen), z));
    const float2 DV = add2(own[O_DV * NTH], sel(mx, my, mul2(mul2(glen, v), fw.rlen), z));
    float2 gvz = mul2(gero, dero_dvz);
    // ---- flux reversed -------------------------------------------------
    const bool wx = vz.x >= FILM_DEPTH, wy = vz.y >= FILM_DEPTH;  // thinner films: velocity locally constant
    const float2 gu = sel(wx, wy, mul2(DU, fw.rvz), z), gv = sel(wx, wy, mul2(DV, fw.rvz), z);
    gvz = sel(wx, wy, sub2(gvz, mul2(add2(mul2(DU, u), mul2(DV, v)), fw.rvz)), gvz);
    st2(a.R.gu + i, gu);
    st2(a.R.gv + i, gv);
    const float2 gd2 = add2(gvz, mul2(Ad, pf(c.evap)));
    const float2 garg = make_float2(fw.arg.x > 0.0f ? gd2.x : 0.0f, fw.arg.y > 0.0f ? gd2.y : 0.0f);
    float2 gd1 = add2(gvz, garg);
    st2(a.R.p + i, mul2(pf(c.dt), garg));
    float2 Af[4];
    {
        const float2 EK = pf(c.EK), p = ld2(P + si), nu = ld2(GU + si), nv = ld2(GV + si);
        // a cell's own flux term: its outflow's energy part and its place in its
        // own velocity; the neighbour it flows to has it as an inflow
        Af[0] = add2(sub2(mul2(EK, ld2(h + si)), nu), sub2(left(P, p), left(GU, nu)));
        Af[1] = add2(add2(mul2(EK, ld2(h + H_RC + si)), nu), add2(right(P, p), right(GU, nu)));
        Af[2] = add2(add2(mul2(EK, ld2(h + 2 * H_RC + si)), nv), add2(ld2(P + si + RW), ld2(GV + si + RW)));
        Af[3] = add2(sub2(mul2(EK, ld2(h + 3 * H_RC + si)), nv), sub2(ld2(P + si - RW), ld2(GV + si - RW)));
    }
    const float2 gsum_outK = mul2(pf(-c.dt), garg), gsum_out = mul2(gsum_outK, fw.K);
    float2 gK = mul2(gsum_outK, fw.sum_out);
#pragma unroll
    for (int d = 0; d < 4; ++d) gK = add2(gK, mul2(Af[d], fw.g[d]));
    // K = depth / outflow where it scales (thinner films: locally constant)
    const bool kx = fw.scaled_x & (d1.x >= FILM_DEPTH), ky = fw.scaled_y & (d1.y >= FILM_DEPTH);
    float2 gden = z;
    if (kx | ky) {
        const float2 rd = fw.rden, g1 = mul2(gK, rd);
        gden = sel(kx, ky, mul2(mul2(mul2(mul2(make_float2(-gK.x, -gK.y), d1), rd), rd), pf(c.dt)), z);
        gd1 = sel(kx, ky, add2(gd1, g1), gd1);
    }
    const float2 wd = pf(c.dt * c.G);
    float2 gw = z;
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        float2 gg = add2(mul2(Af[d], fw.K), gsum_out);
        gg = sel(kx, ky, add2(gg, gden), gg);
        gg = sel(fw.g[d].x > 0.0f, fw.g[d].y > 0.0f, gg, z);
        st2(a.R.h[d] + i, gg);
        gw = add2(gw, mul2(wd, gg));
    }
    st2(a.R.b + i, add2(gb, gw));
    st2(a.R.d + i, add2(gw, gd1));
    // ---- sediment_transport of step j - 1 reversed ----------------------
    if (a.scatter_prev) {
        const float* const se[1] = {a.prev.se};
        Taps<1> q;
        load_taps<1>(c, se, x, y, own[O_PU * NTH], own[O_PV * NTH], q);
        sediment_adjoint(c, q, i, gs, a.dse_prev, a.du, a.dv);
    } else {
        st2(a.R.s + i, gs);
    }
    if (ks_any) st2(a.dks + i, add2(dks, mul2(gKs, pf(c.dt))));
}

constexpr size_t ADJ_SMEM = X_N * H_RC * sizeof(float) + O_N * NTH * sizeof(float2);

__global__ void __launch_bounds__(NTH, 3) k_adj_cell(const __grid_constant__ AdjCellArgs a, int* err) {
    extern __shared__ __align__(128) float sm[];  // staged tile, then the pairs' own inputs
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    const int n = a.c.n;
    const int tx0 = blockIdx.x * TW, ty0 = blockIdx.y * TH;
    const bool inner = tx0 - HX >= 0 && tx0 + TW + HX <= n && ty0 - 1 >= 0 && ty0 + TH + 1 <= n;
    if (inner) adj_tile<false>(a, sm, &bar, tx0, ty0, err);
    else adj_tile<true>(a, sm, &bar, tx0, ty0, err);
}

// ---- k_adj_final -----------------------------------------------------------------
template <bool EDGE>
__device__ __forceinline__ float2 adj_rock_pair(const StepConsts1& c, const AdjState& A, int x, int y) {
    const size_t i = at(c.n, x, y);
    const float2 nbw = adj_nbw<EDGE>(c, A, x, y, i, ldg2(A.h[0] + i), ldg2(A.h[1] + i));
    return add2(sub2(ldg2(A.b + i), nbw), adj_normal<EDGE>(A, c.n, x, y, i));
}
__global__ void k_adj_final(StepConsts c, AdjState A, float* __restrict__ out_b) {
    const int x = 2 * (blockIdx.x * BX + threadIdx.x), y = blockIdx.y * BY + threadIdx.y;
    const float2 v = adj_rock_pair<true>(c, A, x, y);
    float* o = out_b + at(c.n, x, y);  // the caller's buffer: on any float's boundary
    o[0] = v.x;
    o[1] = v.y;
}

// ---- k_adj_thermal ---------------------------------------------------------------
// Reverse of thermal_erosion + thermal_transport (layer 0): from the adjoint
// A of the rock after the talus passes to the adjoint G of the eroded rock.
// rock' = b + sum_k in_k - sum_k o_k, o_k = S dh_k / bk for the marked
// directions, S = dt Kspeed sharp^3 H / 2.  With g_k = A(neighbour k) - A(c):
//   dL/ddh_j = S/bk (g_j - gbar) for marked j, gbar = sum_k g_k dh_k / bk
//   dL/dS = gbar; H = min(b, max dh) and the steepest marked slope pass
//   their derivative to the direction that attains them (the first one in
//   direction order); the marks themselves are locally constant.
// dh_j = b(c) - b(neighbour j): +dL/ddh_j to the cell, - to the neighbour.
// 64 x 8 tiles of 256 threads; the per-cell terms of the tile and its one-cell
// ring go through shared memory (dynamic), from a TMA box of the eroded rock
// and the gathered A, both with a two-cell halo.  Bound by issue slots and the
// barriers between its phases.  Marks are 1 / 0 factors, the directions that
// attain a maximum are found by equality, and quotients are the Newton forms:
// 310 instructions per cell against 445 for the one with an argmax chain and
// built-in division, 20 us against 23 at 1024² with talus.  2048² with talus,
// 12 steps forward and backward: 3287 us; 64 x 16 tiles of 512 threads at 64
// registers 3332, at 40 (spills) 3423; five blocks per SM 3437; a row per warp
// in pairs as the forward's talus pass 3545 (27 to 30 us a launch: a chain of
// staging, gather and exchange per row, too few warps to hide it).
constexpr int TT_H = 8, TT_NTH = 256;
constexpr int TT_RW = TW + 2 * HX, TT_BH = TT_H + 4, TT_BOX = TT_RW * TT_BH;
constexpr int TT_BRC = ((TT_BOX + 31) / 32) * 32;
constexpr int TT_CW = TW + 2, TT_CH = TT_H + 2, TT_NC = TT_CW * TT_CH;  // tile + ring
// direction k = L, R, T, B, LT, RT, LB, RB -> offset
__host__ __device__ constexpr int tt_ox(int k) { return (k == 0 || k == 4 || k == 6) ? -1 : (k == 1 || k == 5 || k == 7) ? 1 : 0; }
__host__ __device__ constexpr int tt_oy(int k) { return (k == 2 || k == 4 || k == 5) ? 1 : (k == 3 || k == 6 || k == 7) ? -1 : 0; }

struct ThermalArgs {
    CUtensorMap map_b;  // eroded rock of the step (box TT_RW x TT_BH)
    AdjState A;         // adjoint of the step's output
    StepConsts c;
    float* g;           // out: adjoint of the eroded rock
};

// The derivatives of one cell's outflows: gdh[k] = dL/ddh_k, and the cell's own
// term (dL/db through H, plus sum_k dL/ddh_k).  dh: its drops, a: A at its
// neighbours, ac: at the cell.  Any operands; the kernel leaves ties,
// infinities and what the Newton forms do not take to it.
__device__ __noinline__ void thermal_lane(const StepConsts& c, float b, const float dh[8], const float a[8], float ac,
                                          float gdh[8], float& own) {
    float Hmax = 0.0f;
    int jh = -1;
    own = 0.0f;
    for (int k = 0; k < 8; ++k) {
        gdh[k] = 0.0f;
        if (dh[k] > Hmax) { Hmax = dh[k]; jh = k; }
    }
    const float H = gmin(b, Hmax);
    float bk = 0.0f, max_cross = 0.0f, max_diag = 0.0f;
    int jc = -1, jd = -1;
    auto marked = [&](int k) { return dh[k] >= (k < 4 ? c.talus_x_cross : c.talus_b_diag); };
    for (int k = 0; k < 8; ++k) {
        if (!marked(k)) continue;
        bk += dh[k];
        if (k < 4) { if (dh[k] > max_cross) { max_cross = dh[k]; jc = k; } }
        else if (dh[k] > max_diag) { max_diag = dh[k]; jd = k; }
    }
    if (!(bk > 0.0f)) return;
    const float sd = max_diag / SQRT2_F;
    const float slope = fmaxf(max_cross, sd);
    const int js = (jd >= 0 && sd > max_cross) ? jd : jc;
    float s1 = 1.0f;
    const float newsh = 1.0f + poly_atanf(slope) - c.Kalpha0;
    const bool taken = newsh > s1;
    if (taken) s1 = newsh;
    const float sh3 = s1 * (s1 * s1);
    const float S = c.dt * c.Kspeed0 * sh3 * H / 2.0f;
    const float rbk = __frcp_rn(bk);
    float gbar = 0.0f;
    for (int k = 0; k < 8; ++k)
        if (marked(k)) gbar += (a[k] - ac) * dh[k];
    gbar *= rbk;
    const float sb = S * rbk;
    for (int k = 0; k < 8; ++k)
        if (marked(k)) gdh[k] = sb * ((a[k] - ac) - gbar);
    const float dH = gbar * (c.dt * c.Kspeed0 * sh3 * 0.5f);
    if (taken && js >= 0) {
        const float ds1 = gbar * (c.dt * c.Kspeed0 * H * 0.5f) * 3.0f * s1 * s1;
        const float dslope = ds1 * __frcp_rn(1.0f + slope * slope);
        gdh[js] += js < 4 ? dslope : dslope * RCP_SQRT2_F;
    }
    if (Hmax < b) gdh[jh] += dH;
    else own += dH;
    for (int k = 0; k < 8; ++k) own += gdh[k];
}


template <bool EDGE>
__device__ __forceinline__ void thermal_tile(const ThermalArgs& ta, float* bs, float* as, float* gd, uint64_t* bar,
                                             int tx0, int ty0, int* err) {
    const StepConsts& c = ta.c;
    const int n = c.n, tid = threadIdx.x;
    const int gx0 = tx0 - HX, gy0 = ty0 - 2;
    if (tid == 0) {
        mbar_arrive_expect_tx(bar, TT_BOX * sizeof(float));
        tma_load_2d(bs, &ta.map_b, gx0, gy0, bar);
    }
    // while the eroded rock flies: the gathered adjoint A of the output rock
    // over the region's columns 2 .. TT_RW - 3 (the tile, its ring and their
    // neighbours), 0 outside the grid
    constexpr int GP = (TT_RW - 4) / 2;  // pairs per row
#pragma unroll 1
    for (int q = tid; q < GP * TT_BH; q += TT_NTH) {
        const int rx = 2 + 2 * (q % GP), ry = q / GP;
        const int x = gx0 + rx, y = gy0 + ry;
        float2 v = pf(0.0f);
        if (!EDGE || (x >= 0 && x < n && y >= 0 && y < n)) v = adj_rock_pair<EDGE>(c, ta.A, x, y);
        st2(as + ry * TT_RW + rx, v);
    }
    bool ok = __syncthreads_and(mbar_wait(bar, 0));
    if (!ok) {
        if (tid == 0) atomicExch(err, 1);
        mbar_wait(bar, 0);
        return;
    }
    // per-cell terms of the tile and its ring: gd[k * TT_NC + q] = dL/ddh_k,
    // gd[8 * TT_NC + q] = the cell's own term (dL/db through H, plus sum_k dL/ddh_k)
#pragma unroll 1
    for (int q = tid; q < TT_NC; q += TT_NTH) {
        const int rx = q % TT_CW - 1, ry = q / TT_CW - 1;
        const int x = tx0 + rx, y = ty0 + ry;
        float gdh[8] = {0, 0, 0, 0, 0, 0, 0, 0}, own = 0.0f;
        if (!EDGE || (x >= 0 && x < n && y >= 0 && y < n)) {
            const int si = (ry + 2) * TT_RW + HX + rx;
            const float b = bs[si];
            auto nb = [&](const float* p, int k) { return p[si + tt_oy(k) * TT_RW + tt_ox(k)]; };
            float dh[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                bool out = EDGE && (x + tt_ox(k) < 0 || x + tt_ox(k) >= n || y + tt_oy(k) < 0 || y + tt_oy(k) >= n);
                dh[k] = b - (out ? FAR_HEIGHT : nb(bs, k));
            }
            float mc = fmaxf(fmax3(dh[0], dh[1], dh[2]), dh[3]), md = fmaxf(fmax3(dh[4], dh[5], dh[6]), dh[7]);
            if ((mc >= c.talus_x_cross) | (md >= c.talus_b_diag)) {
                // the forward's values (cell_thermal_outflows_dh2)
                const float Hmax = fmax3(mc, md, 0.0f), H = fminf(b, Hmax);
                mc = mc >= c.talus_x_cross ? mc : 0.0f;
                md = md >= c.talus_b_diag ? md : 0.0f;
                float m[8], bk = 0.0f;  // 1 where marked
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    m[k] = set_ge(dh[k], k < 4 ? c.talus_x_cross : c.talus_b_diag);
                    bk = __fmaf_rn(dh[k], m[k], bk);  // (the product is exact)
                }
                const float sd = div_recip(md, SQRT2_F, RCP_SQRT2_F);
                const float slope = fmaxf(mc, sd);
                const float newsh = 1.0f + poly_atanf(slope) - c.Kalpha0, s1 = fmaxf(newsh, 1.0f);
                const float sh3 = s1 * (s1 * s1), dtK = c.dt * c.Kspeed0;
                const float S = dtK * sh3 * H * 0.5f;
                // reverse: differences of A in the marked directions
                const float ac = as[si];
                const float rbk = rcp_newton(bk);
                float gbar = 0.0f;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    gdh[k] = (nb(as, k) - ac) * m[k];
                    gbar += gdh[k] * dh[k];
                }
                gbar *= rbk;
                const float sb = S * rbk;
                const float dH = gbar * (dtK * sh3 * 0.5f), dHn = Hmax < b ? dH : 0.0f;
                // the steepest marked slope's direction, where it sets the sharpness
                const float ds1 = gbar * (dtK * H * 0.5f) * 3.0f * s1 * s1;
                const float ds = newsh > 1.0f ? ds1 * rcp_newton(1.0f + slope * slope) : 0.0f;
                const float dsd = ds * RCP_SQRT2_F;
                const float NONE = __int_as_float(0x7fc00000);  // equal to nothing
                const float kc = sd > mc ? NONE : mc, kd = sd > mc ? md : NONE;
                float hits = 0.0f;  // directions that attain the two maxima: 2, more in a tie
                own = Hmax < b ? 0.0f : dH;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float ts = set_eq(dh[k], k < 4 ? kc : kd), th = set_eq(dh[k], Hmax);
                    hits += ts + th;
                    const float v = sb * (gdh[k] - gbar) * m[k];
                    gdh[k] = __fmaf_rn(th, dHn, __fmaf_rn(ts, k < 4 ? ds : dsd, v));  // (products with 0 and 1 are exact)
                    own += gdh[k];
                }
                // else: outside the Newton forms' range, several directions at a maximum, sums not finite
                if (!((c.fast_div != 0) & (bk <= 0x1p40f) & (S >= 0x1p-50f) & (S <= 0x1p40f) & (hits == 2.0f) &
                      (fabsf(own) < 0x1p126f))) {
                    float al[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) al[k] = nb(as, k);
                    float dl[8], gl[8], ol;
#pragma unroll
                    for (int k = 0; k < 8; ++k) dl[k] = dh[k];
                    thermal_lane(c, b, dl, al, ac, gl, ol);
#pragma unroll
                    for (int k = 0; k < 8; ++k) gdh[k] = gl[k];
                    own = ol;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) gd[k * TT_NC + q] = gdh[k];
        gd[8 * TT_NC + q] = own;
    }
    __syncthreads();
    // G(c) = A(c) + own(c) - sum over neighbours m of m's dL/ddh toward c
#pragma unroll 1
    for (int q = tid; q < TW * TT_H; q += TT_NTH) {
        const int ix = q % TW, iy = q / TW;
        const int x = tx0 + ix, y = ty0 + iy;
        const int rq = (iy + 1) * TT_CW + ix + 1;
        float gsum = as[(iy + 2) * TT_RW + HX + ix] + gd[8 * TT_NC + rq];  // A(c), from the staged box
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int xx = x + tt_ox(k), yy = y + tt_oy(k);
            if (EDGE && (xx < 0 || xx >= n || yy < 0 || yy >= n)) continue;
            gsum -= gd[(k ^ (k < 4 ? 1 : 3)) * TT_NC + rq + tt_oy(k) * TT_CW + tt_ox(k)];  // opposite direction
        }
        ta.g[(size_t)y * n + x] = gsum;
    }
}

constexpr size_t TT_SMEM = (2 * TT_BRC + 9 * TT_NC) * sizeof(float) + 8;

__global__ void __launch_bounds__(TT_NTH, 4) k_adj_thermal(const __grid_constant__ ThermalArgs ta, int* err) {
    extern __shared__ __align__(128) float tdyn[];
    float* bs = tdyn;
    float* as = tdyn + TT_BRC;
    float* gd = tdyn + 2 * TT_BRC;
    uint64_t& bar = *reinterpret_cast<uint64_t*>(tdyn + 2 * TT_BRC + 9 * TT_NC);
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    const int n = ta.c.n;
    const int tiles_x = n / TW;
    const int tx0 = (blockIdx.x % tiles_x) * TW, ty0 = (blockIdx.x / tiles_x) * TT_H;
    bool inner = tx0 - HX >= 0 && tx0 + TW + HX <= n && ty0 - 2 >= 0 && ty0 + TT_H + 2 <= n;
    if (inner) thermal_tile<false>(ta, bs, as, gd, &bar, tx0, ty0, err);
    else thermal_tile<true>(ta, bs, as, gd, &bar, tx0, ty0, err);
}

// d(mean((rock - target)^2))/d rock, and the loss partials
__global__ void k_mse_grad(const float* __restrict__ b, const float* __restrict__ target, size_t count,
                           float* __restrict__ grad, double* __restrict__ part) {
    __shared__ double sh[256 / 32];
    double acc = 0.0;
    const double inv = 1.0 / (double)count;
    const double twice = 2.0 * inv;
    const size_t step = (size_t)gridDim.x * blockDim.x;
    auto one = [&](size_t i, float e) {
        const double d = (double)e;
        acc = fma(d, d, acc);
        if (grad) grad[i] = (float)(d * twice);  // (in two floats 9 us less at 1024², but inf - inf and fewer bits)
    };
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + 3 * step < count; i += 4 * step) {
        float e[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) e[k] = b[i + k * step] - target[i + k * step];
#pragma unroll
        for (int k = 0; k < 4; ++k) one(i + k * step, e[k]);
    }
    for (; i < count; i += step) one(i, b[i] - target[i]);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += sh[k];
        part[blockIdx.x] = t * inv;
    }
}

// the partials' sum, in a fixed order: each lane its share, then the lanes'
// (one lane alone took 22 us for 304 partials, so 5)
__device__ __forceinline__ double sum_parts(const double* __restrict__ part, int nparts) {
    double t = 0.0;
#pragma unroll 4
    for (int k = threadIdx.x; k < nparts; k += 32) t += part[k];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}
__global__ void k_sum_parts(const double* __restrict__ part, int nparts, double* __restrict__ out) {
    const double t = sum_parts(part, nparts);
    if (threadIdx.x == 0) *out = t;
}

// per-block sums of g^2 in FP64 (the gradient norm's accumulation)
__global__ void k_sumsq_part(const float* __restrict__ g, size_t count, double* __restrict__ part) {
    __shared__ double sh[256 / 32];
    double acc = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x)
        acc += (double)g[i] * (double)g[i];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += sh[k];
        part[blockIdx.x] = t;
    }
}

// *out += sum of the partials (fixed order)
__global__ void k_add_parts(const double* __restrict__ part, int nparts, double* __restrict__ out) {
    const double t = sum_parts(part, nparts);
    if (threadIdx.x == 0) *out += t;
}

// per-block max |g| (max is order-free, so the result does not depend on the split)
__global__ void k_absmax_part(const float* __restrict__ g, size_t count, float* __restrict__ part) {
    __shared__ float sh[256 / 32];
    float m = 0.0f;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x)
        m = fmaxf(m, fabsf(g[i]));
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t = fmaxf(t, sh[k]);
        part[blockIdx.x] = t;
    }
}

// x <- clamp(x - (step / max|g|) g, lo, hi): the largest change of any cell is `step`
__global__ void k_descend(float* __restrict__ x, const float* __restrict__ g, size_t count,
                          const float* __restrict__ part, int nparts, float step, float lo, float hi) {
    __shared__ float a_sh;
    if (threadIdx.x < 32) {
        float m = 0.0f;
        for (int k = threadIdx.x; k < nparts; k += 32) m = fmaxf(m, part[k]);
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) a_sh = step / fmaxf(m, 1e-30f);
    }
    __syncthreads();
    const float a = a_sh;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x)
        x[i] = fminf(fmaxf(x[i] - a * g[i], lo), hi);
}

dim3 grid_for(int n) { return dim3(n / (2 * BX), n / BY); }  // n % 64 == 0: every thread has a pair

}  // namespace

bool adjoint_tile_ok(int n) { return n % TW == 0 && n % TH == 0; }

int adjoint_box_rows() { return H_RH; }

void launch_adjoint_sediment(const StepConsts& c, const AdjSlot& slot, const float* as, float* dse, float* du,
                             float* dv, cudaStream_t st) {
    k_adj_sediment<<<grid_for(c.n), dim3(BX, BY), 0, st>>>(c, slot, as, dse, du, dv);
    count_launch();
}

void launch_adjoint_cell(const AdjCellArgs& args, int* err, cudaStream_t st) {
    const int n = args.c.n;
    cudaFuncSetAttribute(k_adj_cell, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ADJ_SMEM);
    k_adj_cell<<<dim3(n / TW, n / TH), NTH, ADJ_SMEM, st>>>(args, err);
    count_launch();
}

void launch_adjoint_final(const StepConsts& c, const AdjState& A, float* out_b, cudaStream_t st) {
    k_adj_final<<<grid_for(c.n), dim3(BX, BY), 0, st>>>(c, A, out_b);
    count_launch();
}

int adjoint_thermal_box_rows() { return TT_BH; }

void launch_adjoint_thermal(const StepConsts& c, const CUtensorMap& map_b, const AdjState& A, float* g, int* err,
                            cudaStream_t st) {
    ThermalArgs ta;
    ta.map_b = map_b;
    ta.A = A;
    ta.c = c;
    ta.g = g;
    cudaFuncSetAttribute(k_adj_thermal, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TT_SMEM);
    k_adj_thermal<<<(c.n / TW) * (c.n / TT_H), TT_NTH, TT_SMEM, st>>>(ta, err);
    count_launch();
}

void launch_mse(const float* b, const float* target, size_t count, float* grad, double* part, int nparts,
                double* out, cudaStream_t st) {
    k_mse_grad<<<nparts, 256, 0, st>>>(b, target, count, grad, part);
    k_sum_parts<<<1, 32, 0, st>>>(part, nparts, out);
    count_launch(2);
}

void launch_add_sumsq(const float* g, size_t count, double* part, int nparts, double* out, cudaStream_t st) {
    k_sumsq_part<<<nparts, 256, 0, st>>>(g, count, part);
    k_add_parts<<<1, 32, 0, st>>>(part, nparts, out);
    count_launch(2);
}

void launch_descend(float* x, const float* g, size_t count, float step, float lo, float hi, float* part, int nparts,
                    cudaStream_t st) {
    k_absmax_part<<<nparts, 256, 0, st>>>(g, count, part);
    k_descend<<<nparts * 4, 256, 0, st>>>(x, g, count, part, nparts, step, lo, hi);
    count_launch(2);
}

}  // namespace hg
