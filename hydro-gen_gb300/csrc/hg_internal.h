// Internal declarations shared by the library's translation units.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <atomic>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/hydrogen.h"
#include "hg_device.cuh"

namespace hg {

// Carried state fields, in the order of the HG_FIELD_* ids 0..6.
enum { S_ROCK = 0, S_WATER, S_SED, S_FL, S_FR, S_FT, S_FB, S_COUNT };

struct StateBufs {
    float* f[S_COUNT];
};

extern std::atomic<uint64_t> g_launches;
inline void count_launch(uint64_t k = 1) { g_launches.fetch_add(k, std::memory_order_relaxed); }

// ---- per-pass kernels (hg_plain.cu) --------------------------------------------
void launch_rain(const StepConsts& c, const RainStep& r, float* water, cudaStream_t st);
void launch_flux(const StepConsts& c, const float* rock, const float* water, const float* fl, const float* fr,
                 const float* ft, const float* fb, float* water_o, float* fl_o, float* fr_o, float* ft_o,
                 float* fb_o, float* u, float* v, float* vz, cudaStream_t st);
// launch_flux and launch_erosion of the state `in` in one kernel, after `rain`
// on every cell (-0: none) and with the evaporation; sed in place
void launch_flux_erosion(const StepConsts& c, float rain, const float* const in[S_COUNT], float* const out[S_COUNT], float* sed,
                         float* u, float* v, float* vz, cudaStream_t st);
// sediment transport without the evaporation
void launch_gather(const StepConsts& c, const float* u, const float* v, const float* sed, float* sed_o,
                   cudaStream_t st);
// both talus passes of a whole map's layer 0
void launch_talus(const StepConsts& c, const float* rock, float* rock_o, cudaStream_t st);
// the same by k_transport's marching warps (hg_fused.cu)
void launch_talus_march(const StepConsts& c, const float* rock, float* rock_o, cudaStream_t st);
// sediment transport without the evaporation and both talus passes of a whole
// map's layer 0
void launch_gather_talus(const StepConsts& c, const float* rock, float* rock_o, const float* u, const float* v,
                  const float* sed, float* sed_o, cudaStream_t st);
void launch_erosion(const StepConsts& c, const float* u, const float* v, const float* vz, const float* rock,
                    float* rock_o, float* sed_inout, cudaStream_t st);
void launch_sediment(const StepConsts& c, const float* u, const float* v, const float* sed, float* sed_o,
                     float* water_inout, cudaStream_t st);
void launch_thermal_out(const StepConsts& c, const float* rock, float4* tc, float4* td, cudaStream_t st);
void launch_thermal_in(const StepConsts& c, const float* rock, const float4* tc, const float4* td,
                       float* rock_o, cudaStream_t st);
// smoothing pass on rock (run when c.smooth_m != 0)
void launch_smooth(const StepConsts& c, const float* rock, float* rock_o, cudaStream_t st);

// ---- the reference's terrain generator and rain (hg_terrain.cu) --------------------
// (zero: up to 20 fields to clear in the same launch)
void launch_ref_heightmap(const hg_map_settings& cfg, int n, float* rock, float* dirt, float* const* zero, int nzero,
                          cudaStream_t st);
// water += the reference's rain at frame time `time`; dirt may be nullptr (one layer)
void launch_ref_rain(const hg_rain_settings& rs, const hg_map_settings& map, float time, int n, const float* rock,
                     const float* dirt, float* water, cudaStream_t st);

// ---- two-layer per-pass kernels (hg_layers.cu) -----------------------------------
// flux, erosion of both layers and evaporation of the state (in, dirt); sediments in place
void launch_flux_erosion2(const StepConsts& c, const float* const in[S_COUNT], const float* dirt,
                          float* const out[S_COUNT], float* dirt_o, float* s0, float* s1, float* u, float* v, float* vz,
                          cudaStream_t st);
// sediment transport of both channels without the evaporation
void launch_gather2(const StepConsts& c, const float* u, const float* v, const float* s0, const float* s1, float* s0_o,
                    float* s1_o, cudaStream_t st);
// both talus passes of layer 1 (dirt)
void launch_talus1(const StepConsts& c, const Talus1& t1, const float* rock, const float* dirt, float* dirt_o,
                   cudaStream_t st);
void launch_smooth2(const StepConsts& c, const float* rock, const float* dirt, float* rock_o, float* dirt_o,
                    cudaStream_t st);

// ---- headless ray-marcher (hg_render.cu) ------------------------------------------
struct RenderInput {
    int n;
    float max_height;  // map settings: the shadow rays' ceiling
    int hmap_dim_x;    // map settings: alpha of the low-resolution form
    const float* rock;
    const float* dirt;   // nullptr: one-layer world
    const float* water;
    const float* sed0;
    const float* sed1;   // nullptr: one-layer world
    float4* hm;          // n*n packed heightmap texels (written)
    float* total;        // n*n totals (written)
    float2* ground;      // n*n (rock, dirt) (written)
    float2* sed;         // n*n packed sediment texels (written when displayed)
};
// packs the heightmap and renders width x height pixels into rgba_dev
// (and the float colour into rgb_dev when not null); HG_ERR_INVALID for a
// singular view or perspective matrix
int render_image(const RenderInput& in, const hg_camera& cam, int width, int height, uint8_t* rgba_dev,
                 float* rgb_dev, cudaStream_t st);

// ---- fused two-layer step (hg_fused2.cu) ------------------------------------------
// Inputs and outputs of one fused two-layer step (out of place) and its
// scratch fields.
struct Fused2Bufs {
    const float *rock, *dirt, *water, *s0, *s1, *fl, *fr, *ft, *fb;
    float *rock_o, *dirt_o, *water_o, *s0_o, *s1_o, *fl_o, *fr_o, *ft_o, *fb_o;
    float *u, *v;
    float *s0_ero, *s1_ero;  // eroded sediment (rock, dirt)
    const float *s0_prev, *s1_prev;  // the previous step's, in a chain
    float *b_ero;            // eroded rock (input of the rock talus pass)
    float *rock_mid;         // rock after the rock talus pass (input of the dirt pass)
    float *g_ero;            // eroded dirt (input of the dirt pass)
};
struct TmaCache;
bool fused2_ok(int n);
// ---- particle erosion (hg_particles.cu) --------------------------------------------
// Droplets as structure of arrays (Particle, glsl/bindings.glsl:101-110).
struct Drops {
    int count;
    float *px, *py, *vx, *vy, *vol;
    float *s0, *s1;  // sediment of the rock / dirt layer
    float* sc;       // sediment capacity
    uint32_t* iters;
    int32_t* kill;
};
// Bucket and per-record buffers of one particle world.
struct ParticleBufs {
    Drops d;
    uint32_t* cnt;      // n*n records per texel, then particle_counters() counters
    uint32_t* offs;     // n*n: where a texel's bucket begins
    uint32_t* keys;     // 4*count records (droplet * 4 + corner), bucketed by texel
    uint32_t* sorted;   // 4*count: the largest buckets' chunks in droplet-id order
    uint32_t* list[4];  // texels by record count, particle_list_capacity() each
    uint4* rank;        // count: the places of a droplet's records in their buckets
    float4* pack;       // 2*count: what a record reads of its droplet
    float2* rec;        // 4*count: what a record left for its droplet
};
// The fields a particle pass reads or writes; mom = momentum (x, y, z, w).
struct PWorld {
    float* rock;
    float* dirt;
    float* water;
    float* mom[4];
};
size_t particle_counters();
int particle_lists();
size_t particle_list_capacity(int list, size_t cells, int count);
// movement, counting sort, erosion in droplet-id order, sediment replay
void launch_particle_step(const StepConsts& c, const hg_erosion_settings& es, const ParticleBufs& pb,
                          const PWorld& pw, uint32_t step1, uint64_t seed, bool should_rain, cudaStream_t st);
// smoothing with the particle branch: in -> out (all of rock, dirt, water, momentum)
void launch_particle_smooth(const StepConsts& c, float count, const PWorld& in, const PWorld& out, cudaStream_t st);
struct Talus1;
// the particle step's talus passes (rock, then dirt) and smoothing with the
// particle branch as fused kernels (hg_fused2.cu, n a multiple of 64):
// in -> out, the rock after its talus pass in rock_mid
struct TmaCache;
int launch_particle_thermal_smooth(const StepConsts& c, const Talus1& t1, float count, const PWorld& in,
                                   const PWorld& out, float* rock_mid, TmaCache& tma, int* err, cudaStream_t st);

// ---- fused step (hg_fused.cu) ---------------------------------------------------
// Rain settings without the step number (the kernels add the step).
struct RainBase {
    int mode;  // HG_RAIN_*
    int period;
    float amount;
    uint32_t threshold;
    uint32_t seed_lo, seed_hi, terrain_id;
};

// One terrain (world) of a fused launch, without its tensor maps.
struct TerrainHot {
    StepConsts1 c;
    RainBase rain;
    float* out[S_COUNT];
    float* u;
    float* v;
    float* s_ero;  // eroded sediment of every cell (k_hydro -> the next gather)
    float* b_ero;  // eroded rock of every cell (k_hydro -> k_transport, thermal on)
    const float* s_prev;  // the previous step's s_ero (a chained k_hydro gathers from it)
    float* s_keep;        // where a chained k_hydro leaves the gathered sediment, or nullptr
    ptrdiff_t uv_prev;    // the previous step's u and v lie this many floats from u and v
    unsigned long long* step;  // device step counter (steps completed)
    int tiles_x;
    int t_rows;  // k_transport: rows a warp marches
};
// maps[0..6]: TMA boxes of the step's input rock, water, sediment, fL, fR,
// fT, fB.  (CUtensorMap makes it 64-byte aligned.)
constexpr int MAPS_PER_TERRAIN = 7;
struct TerrainDesc {
    CUtensorMap maps[MAPS_PER_TERRAIN];
    TerrainHot h;
    int row_lo, row_hi;  // rows to do (a row slab's; all of the world otherwise)
};
// A batch launch's terrain records travel as one kernel parameter (read
// through the constant bank); the tensor maps stay in global memory.
constexpr int MAX_BATCH = 128;
struct BatchParams {
    int nterr;
    int tasks;              // k_transport's warps over all terrains
    int tile0[MAX_BATCH];   // k_hydro: first tile of each terrain
    int task0[MAX_BATCH];   // k_transport: first warp of each terrain
    TerrainHot t[MAX_BATCH];
};
static_assert(sizeof(BatchParams) + 2 * sizeof(void*) <= 32764, "kernel parameter space");

// Host view of one terrain for one step direction (inputs -> outputs).
struct TerrainSrc {
    StepConsts c;
    RainBase rain;
    const float* in[S_COUNT];
    float* out[S_COUNT];
    float* u;
    float* v;
    float* s_ero;
    float* b_ero;
    const float* s_prev;
    float* s_keep;
    ptrdiff_t uv_prev;
    unsigned long long* step;
};

// A step's place in a run of steps launched together (a chain).  Within a
// chain a step's sediment gather runs in the next step's k_hydro, and the
// device step counter stays at the chain's start until its end.
struct ChainPos {
    int index;  // steps of the chain before this one
    bool last;  // the step's results become the state
};

// One fused two-layer step (hg_fused2.cu).
struct TmaCache;
int launch_fused2_step(const StepConsts& c, const Talus1& t1, const RainStep& r, const Fused2Bufs& b, ChainPos pos,
                       TmaCache& tma, int* err, cudaStream_t st);

// Tensor maps encoded once per (buffer, box) and reused.
struct TmaCache {
    struct Entry {
        const float* base;
        int n, box_h;
        CUtensorMap map;
    };
    std::vector<Entry> entries;
    bool get(const float* base, int n, int box_h, CUtensorMap* out);
};

// Tile height th (16 or 8) divides n and 64 divides n.
bool fused_tile_ok(int n, int th);
int fused_tiles(int n, int th);
// Fills a descriptor (tensor maps from the cache); false if a map cannot be encoded.
bool fill_desc(TerrainDesc& d, const TerrainSrc& s, int th, TmaCache& cache);
// Rows a warp of k_transport marches in a launch over rows[i] rows of each terrain
// of side sides[i].
int chunk_rows(const int* sides, const int* rows, int count);
// Warps it runs for `rows` rows of an n x n terrain.
int transport_tasks(int n, int rows, int t_rows);
// One fused step (k_hydro, k_transport) over every tile of the batch's
// terrains; maps holds MAPS_PER_TERRAIN tensor maps per terrain (device
// memory); thermal: some terrain has talus passes.
void launch_fused_table(const BatchParams& bp, const CUtensorMap* maps, int total_tiles, int th, bool thermal,
                        ChainPos pos, int* err, cudaStream_t st);
// Same for one terrain whose descriptor travels as a kernel parameter.
void launch_fused_one(const TerrainDesc& td, int th, ChainPos pos, int* err, cudaStream_t st);
// One kernel of an unchained fused step (which 0: k_hydro, 1: k_transport)
// over the descriptor's rows (whole tile rows) of a single world.
void launch_fused_half(const TerrainDesc& td, int th, int which, int* err, cudaStream_t st);

// ---- adjoint (hg_adjoint.cu) ----------------------------------------------------------
// Forward intermediates of one step kept by the segment recompute.
struct AdjSlot {
    const float* u;
    const float* v;
    const float* se;  // eroded sediment
};
// Adjoint of a state, as twelve fields per cell.  b, d, s: what the cell passes
// to its own rock, water and sediment.  h: the adjoint of its four outflows
// before scaling, 0 where nothing flows (L, R, T, B); p: of its inflows' sum;
// gu, gv: of its velocity times its depth; nx, nz: of the terrain normal's
// height differences.  A reader adds what a cell's neighbours pass to it: with
// these terms that needs 12 fields against 17 when every neighbour's share is
// stored by itself.
struct AdjState {
    float *b, *d, *s;
    float* h[4];
    float *p, *gu, *gv, *nx, *nz;
};
constexpr int ADJ_FIELDS = 12;
// Arguments of k_adj_cell (one kernel parameter).
struct AdjCellArgs {
    // X: rock, water, sediment, fL, fR, fT, fB; A: h (4), p, gu, gv (64-wide tiles, 1-row halo)
    CUtensorMap maps[14];
    StepConsts c;
    RainStep rain;
    AdjState A;           // adjoint of the step's output
    float* dse;           // this step's sediment adjoint (read, then cleared)
    float* dse_prev;      // step j - 1's sediment adjoint (scatter target)
    float* du;            // back-trace velocity adjoint: read for step j, written for step j - 1
    float* dv;
    const float* gbe;     // thermal on: adjoint of the eroded rock (replaces A's rock), else nullptr
    AdjSlot prev;         // step j - 1's intermediates
    int scatter_prev;     // reverse step j - 1's sediment pass here (its intermediates exist)
    AdjState R;           // out: adjoint of the step's input (s only without scatter_prev)
    float* dks;           // per-cell Ks gradient (accumulated)
};
bool adjoint_tile_ok(int n);
// Rows of the TMA box k_adj_cell stages per field (tile rows plus halo);
// AdjCellArgs::maps must be encoded with this box height.
int adjoint_box_rows();
void launch_adjoint_sediment(const StepConsts& c, const AdjSlot& slot, const float* as, float* dse, float* du,
                             float* dv, cudaStream_t st);
void launch_adjoint_cell(const AdjCellArgs& args, int* err, cudaStream_t st);
// gathered rock adjoint of a state into out_b
void launch_adjoint_final(const StepConsts& c, const AdjState& A, float* out_b, cudaStream_t st);
// reverse of the talus passes: A (adjoint of the step's output; its rock part
// is gathered in the kernel) -> g (adjoint of the
// eroded rock); map_b: boxes 72 x adjoint_thermal_box_rows() of the eroded rock
int adjoint_thermal_box_rows();
void launch_adjoint_thermal(const StepConsts& c, const CUtensorMap& map_b, const AdjState& A, float* g, int* err,
                            cudaStream_t st);
// loss = mean((b - target)^2) into *out (device), grad = dloss/db (optional).
void launch_mse(const float* b, const float* target, size_t count, float* grad, double* part, int nparts,
                double* out, cudaStream_t st);
// *out += the count of NaN and infinite values of x
void launch_count_nonfinite(const float* x, size_t count, unsigned long long* out, cudaStream_t st);
// *out += sum of g^2 in FP64 (fixed order); part holds nparts doubles
void launch_add_sumsq(const float* g, size_t count, double* part, int nparts, double* out, cudaStream_t st);
// x <- clamp(x - step * g / max|g|, lo, hi); part holds nparts floats
void launch_descend(float* x, const float* g, size_t count, float step, float lo, float hi, float* part, int nparts,
                    cudaStream_t st);

// ---- init and reductions (hg_init.cu) ---------------------------------------------
void launch_fbm_raw(float* out, int n, const hg_noise_settings& s, cudaStream_t st);
// min and max of a device array into two floats of `minmax` (device).
void launch_minmax(const float* x, size_t count, float* partial, int nparts, float* minmax, cudaStream_t st);
void launch_scale(float* x, size_t count, const float* minmax, float lo, float hi, cudaStream_t st);
void launch_ks_from_fbm(float* x, size_t count, float base, float k_over_amp, cudaStream_t st);
// Deterministic FP64 sum of up to 8 arrays: out[i] = sum of field i.
struct PtrList8 { const float* p[8]; };
void launch_sum_f64(const PtrList8& fields, int nfields, size_t count, double* partial, int nparts,
                    double* out, cudaStream_t st);
int reduction_parts();

// host copy of the polynomial arctangent (same operations as poly_atanf)
float host_poly_atanf(float x);

// Records msg as this thread's hg_last_error() and returns code.
int hg_report_error(int code, const char* msg);

}  // namespace hg
