// Kernels of one SPH time step (Geoflow-SPH RK45, SPH_MAIN_2019.f90:746-1005)
// on sm_100a.  Particles live in HBM as structure-of-arrays, re-sorted by cell
// every step (counting sort); the neighbour table is built once per step and
// reused by the density, force and XSPH passes, as the reference reuses its
// pair list (w and dW frozen at the start of the step).
//
// Cell grids: while every level's grid over the bounding box fits the dense
// budget (4M cells, or 8 per particle), the cell keys are row-major over each
// level (dense mode).  Beyond it (separated releases on a large DEM with
// small smoothing lengths) the grids are block-sparse: cut into blocks of
// 32 x 8 cells, a dense block map over the box marks the blocks that hold
// particles, and only those blocks get cells, so the cell count follows the
// area the flow covers.  The occupied blocks of one block row share their
// keys row by row (sparse_key), so that a row of cells is one key range in
// either layout, across block edges too.
#pragma once
#include <climits>

#include "gfsph_device.cuh"

namespace gfsph {

constexpr int kScanTile = 2048;  // cells per scan tile (256 threads x 8)
constexpr int kScanThreads = 256;
constexpr float kBigFactor = 1.5f;  // default level-0 bound Hc = kBigFactor * mean(hsml)
constexpr float kCellDiv = 3.f;     // default cell width of level k: Hc * 2^k / kCellDiv
constexpr float kCellAspect = 1.5f;  // cell height over width: a stencil row is one slot range whatever its width,
                                     // so fewer, higher rows cost less than the candidates they add
constexpr int kRegLevels = 2;       // default regular levels: their particles take a thread and the table
constexpr int kMaxLevels = 24;      // level k cell size Hc * 2^(k-1)
constexpr int kBlkX = 32;           // cells per block along x
constexpr int kBlkY = 8;            // cells per block along y
constexpr int kBlockCells = kBlkX * kBlkY;
constexpr long long kDenseCells = 1LL << 22;  // dense-mode budget (or 8 cells per particle)
constexpr int kThreadsBounds = 256;
constexpr int kBoundsBlocks = 148 * 4;  // at most; k_grid reduces their partials

// error bits in StepScalars::err
constexpr int kErrCells = 1;
constexpr int kErrNbr = 2;
constexpr int kErrNonFinite = 4;
constexpr int kErrEmpty = 8;
constexpr int kErrBlocks = 16;

// Device-resident scalars of the step (one per handle).
struct StepScalars {
    double time;      // time_sph
    double t_end;
    double hsum;      // sum of hsml over the particles inside the DEM box
    float dt;         // dt_sph, committed at the end of a completed step
    float dt_step;    // dt of the step in flight (a step stopped by a capacity error leaves dt unchanged)
    int skip;         // this step does nothing (time >= t_end or an error)
    int err;          // sticky error bits
    int steps_done;
    unsigned int xmin_o, xmax_o, ymin_o, ymax_o, hmax_o, dtmin_o;  // reductions (ordered uint)
    int hcount;
    int bad;          // non-finite state seen by k_bounds
    float hc;         // regular-hsml bound Hc: level k holds hsml in (Hc*2^(k-1), Hc*2^k], level 0 hsml <= Hc
    int nlev;         // number of grid levels
    float lev_gx0[kMaxLevels], lev_gy0[kMaxLevels], lev_c[kMaxLevels];  // origin and cell width per level
    int lev_ndx[kMaxLevels], lev_ndy[kMaxLevels];  // cells per level along x and y
    int lev_off[kMaxLevels + 1];  // dense mode: first cell key of each level
    int lev_nbx[kMaxLevels], lev_boff[kMaxLevels + 1];  // sparse mode: blocks per level along x, first block-map entry
    int sparse;       // 1: block-sparse cell keys this step
    unsigned int lev_hmax_o[kMaxLevels];  // max hsml of the particles of each level (ordered uint, 0 = empty)
    int nblocks;      // block-map entries (all levels)
    int ncells;       // cells of the occupied blocks
    int nreg, nbig, nactive, nout;
    int need_cells, need_nbr, need_big, need_blocks;
    int ex0, ex1, ey0, ey1;  // DEM node box touched by erosion this step
    unsigned int scan_ticket[2];  // tiles of k_scan_tiles done: cells, block map
    unsigned int end_ticket;      // blocks of k_dem_erode done
    int reg_levels;   // levels 0 .. reg_levels-1 are regular (thread + neighbour table)
    // the reference's own grid of grid_find_NEW_tools (skf 2, 3): origin, cell, cells
    float ref_xmin, ref_ymin, ref_delt;
    int ref_ndx, ref_ndy;
    int advance;      // 1 inside gfsph_step, 0 for search-only passes
    int irregular;    // some step since the host cleared it had a particle outside the DEM or on a coarse level
};

// Particle state, structure of arrays, one buffer set per ordering.
struct PState {
    float2* pos;
    float2* vel;
    float* rho;
    float* mass;
    float* hsml;
    int* flag;
    int* id;
    float* pwp;  // basal pore-water pressure Uaux(1,:) (icpwp = 3)
};

// Programmatic dependent launch: every kernel of the step is launched with
// programmatic stream serialisation, so the next kernel's launch and block
// set-up overlap this one's tail.  Each kernel first waits for the kernels
// before it to finish and their writes to be visible (griddepcontrol.wait,
// a no-op for an ordinary launch), then lets its dependents launch (a block that
// ends without that does so by ending).
#define PDL_WAIT() asm volatile("griddepcontrol.wait;" ::: "memory")
#define PDL_NEXT() asm volatile("griddepcontrol.launch_dependents;" :::)
#define PDL_ENTRY() \
    do {            \
        PDL_WAIT(); \
        PDL_NEXT(); \
    } while (0)

// Scratch of the neighbour search (sorted order).
struct Search {
    const int* bstart;   // block-map entry -> slot of its block (exclusive scan of the marks), nblocks+1
    const int* start;    // cell key -> first particle slot (exclusive scan), ncells+1
    const float4* xhm;   // slot -> (x, y, hsml, mass) at the start of the step
    // neighbour table of the regular particles (layout: tab_base): per entry
    // j, W_ij and its gradient, computed once per pair by the search, as
    // grid_find stores w and dwdx.  Three arrays, since the internal force
    // reads j and the gradient, av_vel and the normalisation j and W.  With
    // skf 1 the gradient is spline_pair's one factor (the internal force, which
    // waits for the table, has the arithmetic for the rest to spare); else a
    // float2.
    int* nj;
    float* nw;
    float* ng;
    int* ncount;
    float* pterm;        // p/h^2 (pa_sph 2) or p (pa_sph 1)
    float2* indv;        // internal acceleration of every active particle (slot order)
    float* rho0;         // depth at the start of the step, after Adaptive_dt's h_inf clamp (icpwp = 3)
    const int2* rcell;   // slot -> cell of the reference's own grid (skf 2, 3), else null
    float4* xsv;         // slot -> (vx, vy, h, m) after the RK update: what av_vel gathers
    // ic_ws_Interact = 1: slot -> material (1 soil, 2 water); at the water
    // particles Z + hs of the current stage and its gradient; per particle the
    // sum of its soil-water pair terms.  A soil-water pair is kept in the
    // neighbour table with the sign bit of j set (type 1 of
    // Pint_Update_SW_tools): the density, the internal force and av_vel skip it.
    const unsigned char* spec;
    float* zpw;
    float2* gzw;
    float2* bxy;
    const float* mass0;  // caller index -> mass at upload (nfric 3), else null
    // nor_density: m/h per slot with the depth of the previous
    // sum_density_Tools call, for the next one to gather; call k reads
    // ratio[k & 1] and writes the other
    float* ratio[2];
    int kcap;
};

// nsoilB = (m - m0)/m of basal_friction_Ext_SW (SPH_SW_2019.f90:9449-9451),
// the share of a particle's mass gained by erosion; 0 unless nfric = 3.
__device__ __forceinline__ float soil_fraction(const Rheo& c, const Search& Q, const PState& A, int i) {
    if (c.nfric != 3) return 0.f;
    const float m = A.mass[i];
    return (m - Q.mass0[A.id[i]]) / m;
}
constexpr int kCrossBit = (int)0x80000000;

__device__ __forceinline__ bool step_skipped(const StepScalars* S) { return S->skip != 0; }

// The step scalars in shared memory for the serial set-up code that one
// thread runs at the end of a kernel (grid set-up, step end): the block
// copies the struct in and out in one parallel pass each, so the set-up does
// not wait for a global round trip per field it reads.  Every thread of the
// block calls both, and nothing else writes S meanwhile.
static_assert(sizeof(StepScalars) % 4 == 0, "StepScalars is copied as 32-bit words");
__device__ __forceinline__ StepScalars* scalars_to_smem(const StepScalars* S) {
    __shared__ __align__(16) StepScalars sS;
    const int nw = (int)(sizeof(StepScalars) / 4);
    const unsigned int* src = reinterpret_cast<const unsigned int*>(S);
    unsigned int* dst = reinterpret_cast<unsigned int*>(&sS);
    for (int k = threadIdx.x; k < nw; k += blockDim.x) dst[k] = __ldcg(src + k);
    __syncthreads();
    return &sS;
}
__device__ __forceinline__ void scalars_from_smem(StepScalars* S, const StepScalars* L) {
    __syncthreads();
    const int nw = (int)(sizeof(StepScalars) / 4);
    const unsigned int* src = reinterpret_cast<const unsigned int*>(L);
    unsigned int* dst = reinterpret_cast<unsigned int*>(S);
    for (int k = threadIdx.x; k < nw; k += blockDim.x) dst[k] = src[k];
}

// Neighbour-table layout, blocked by warps of 32 particles: entry k of
// particle i is at tab_base(i, kcap) + 32 k.  The lanes of a warp read entry k
// of their particles as one 128-byte run, and the entries a
// warp appends while its lanes are at different k stay within its own
// 32 kcap entries.
__host__ __device__ __forceinline__ size_t tab_base(int i, int kcap) {
    return (size_t)(i >> 5) * ((size_t)kcap << 5) + (size_t)(i & 31);
}
constexpr int kTabStride = 32;

// Asks for the first rows entries of one table array of a warp's particles
// (contiguous, tab_base) into L2, one instruction of one lane; at: the
// warp's first entry.
__device__ __forceinline__ void prefetch_rows(const void* at, int rows) {
    if (rows > 0)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(at), "r"(rows * kTabStride * 4) : "memory");
}

// Whether every pair of a particle with smoothing length hi, in a step whose
// largest is hmax, has a mean within kQuotMin .. kQuotMax.
__device__ __forceinline__ bool quot_safe(float hi, float hmax) { return hi >= 2.f * kQuotMin && hmax <= kQuotMax; }

// The gradient of table entry `at` of particle i (at xi) with neighbour j (at
// xj): load, then grad.
template <int SKF>
struct TabGrad {
    float g0, g1;
    __device__ __forceinline__ void load(const Search& Q, size_t at) {
        if (SKF == 1) {
            g0 = __ldg(Q.ng + at);
        } else {
            const float2 g = __ldg(reinterpret_cast<const float2*>(Q.ng) + at);
            g0 = g.x;
            g1 = g.y;
        }
    }
    __device__ __forceinline__ void grad(float2 xi, float4 xj, bool safe, float& d0, float& d1) const {
        if (SKF == 1) {
            spline_grad(g0, xi.x - xj.x, xi.y - xj.y, safe, d0, d1);
        } else {
            d0 = g0;
            d1 = g1;
        }
    }
};

// ---------------------------------------------------------------- prologue
// Decides whether the coming step runs and resets its reductions; run at the
// start of a batch (k_prep) and at the end of every step for the next one
// (k_step_end).
__device__ __forceinline__ void prepare_step(StepScalars* S, int advance) {
    S->advance = advance;
    S->skip = (S->err != 0) || (advance && S->time >= S->t_end);
    S->xmin_o = 0xffffffffu; S->ymin_o = 0xffffffffu;
    S->xmax_o = 0u; S->ymax_o = 0u; S->hmax_o = 0u;
    S->dtmin_o = 0xffffffffu;
    S->hsum = 0.0;
    S->hcount = 0;
    S->bad = 0;
    S->nout = 0;
    S->nbig = 0;
    S->ex0 = 0x7fffffff; S->ey0 = 0x7fffffff; S->ex1 = -1; S->ey1 = -1;
    for (int k = 0; k < kMaxLevels; k++) S->lev_hmax_o[k] = 0u;
}

// advance: the start of a batch of steps up to t_end.
__global__ void k_prep(StepScalars* S, int advance, double t_end) {
    PDL_ENTRY();
    StepScalars* L = scalars_to_smem(S);
    if (threadIdx.x == 0) {
        if (advance) { L->t_end = t_end; L->steps_done = 0; }
        prepare_step(L, advance);
    }
    scalars_from_smem(S, L);
}

__global__ void k_set_time(StepScalars* S, double t, float dt) {
    S->time = t;
    S->dt = dt;
}

__device__ __forceinline__ float warp_min(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ int warp_sum(int v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The stability time step of Adaptive_dt_sph_SW (SPH_SW_2019.f90:6537-6567,
// min hsml/(3 max(1e-6, sqrt(g h))) [+|v|]) over the particles not yet
// flagged; then the Check_Out_Domain at the start of time_integration_sph
// (SPH_MAIN_2019.f90:232, :1764-1788) and, over the particles still inside,
// the bounds, max and mean of hsml for the cell grid.
// k_bounds: the per-particle part and block partials; k_grid, one block: the
// global bounds and grid_setup.
struct BoundsPart {
    float xmn, xmx, ymn, ymx, hmx, dtm;
    double hsum;
    int hcnt, bad;
};

__device__ __forceinline__ void bounds_merge(BoundsPart& a, const BoundsPart& b) {
    a.xmn = fminf(a.xmn, b.xmn); a.xmx = fmaxf(a.xmx, b.xmx);
    a.ymn = fminf(a.ymn, b.ymn); a.ymx = fmaxf(a.ymx, b.ymx);
    a.hmx = fmaxf(a.hmx, b.hmx); a.dtm = fminf(a.dtm, b.dtm);
    a.hsum += b.hsum; a.hcnt += b.hcnt; a.bad |= b.bad;
}

// Capacities and search tunables handed to grid_setup.
struct GridArgs {
    int cap_blocks, cap_cells, max_cells;
    float level_factor, cell_div;
    int reg_levels;
};

__device__ void grid_setup(const Rheo& c, StepScalars* S, const GridArgs ga);

__global__ void __launch_bounds__(kThreadsBounds) k_bounds(PState B, int n, Rheo c, DemView dem, const StepScalars* S,
                                                           BoundsPart* part) {
    PDL_ENTRY();
    if (step_skipped(S)) return;
    float xmn = 3.4e38f, xmx = -3.4e38f, ymn = 3.4e38f, ymx = -3.4e38f, hmx = 0.f, dtm = 1.e10f;
    double hs_sum = 0.0;
    int hs_cnt = 0;
    int bad = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        // every load issued before the flag test, so that they overlap
        const int fl = B.flag[i];
        float2 p = B.pos[i];
        float hs = B.hsml[i];
        float h = B.rho[i];
        float2 v = B.vel[i];
        if (fl) continue;
        if (!(isfinite(p.x) && isfinite(p.y) && isfinite(hs) && isfinite(h) && isfinite(v.x) && isfinite(v.y))) bad = 1;
        bool out = out_of_box(dem, p.x, p.y);
        if (out && S->advance) B.flag[i] = 1;
        if (!out) {
            xmn = fminf(xmn, p.x); xmx = fmaxf(xmx, p.x);
            ymn = fminf(ymn, p.y); ymx = fmaxf(ymx, p.y);
            hmx = fmaxf(hmx, hs);
            hs_sum += (double)hs;
            hs_cnt += 1;
        }
        if (c.ic_adapt != 0) {
            float vv = 0.f;
            if (c.ic_adapt != 1) vv = sqrtf(v.x * v.x + v.y * v.y);
            if (c.ic_adapt != 4) {  // modes 1, 2, 10: hsml / (3 (c [+ |v|])) with h clamped to h_inf
                float hh = (h < c.h_inf) ? c.h_inf : h;
                float cs = sqrtf(c.g * hh);
                float cc = (1.e-6f > cs) ? 1.e-6f : cs;
                if (c.ic_adapt == 2) cc = cc + vv;
                cc = hs / (3.f * cc);
                dtm = fminf(dtm, cc);
            }
            if (c.ic_adapt == 4 || c.ic_adapt == 10)  // |DEM cell diagonal| / |v|, +inf at rest
                dtm = fminf(dtm, sqrtf(dem.dx * dem.dx + dem.dy * dem.dy) / vv);
        }
    }
    __shared__ BoundsPart wp[kThreadsBounds / 32];
    BoundsPart q{warp_min(xmn), warp_max(xmx), warp_min(ymn), warp_max(ymx), warp_max(hmx), warp_min(dtm),
                 warp_sum(hs_sum), warp_sum(hs_cnt), __any_sync(0xffffffffu, bad) ? 1 : 0};
    if ((threadIdx.x & 31) == 0) wp[threadIdx.x >> 5] = q;
    __syncthreads();
    if (threadIdx.x == 0) {
        BoundsPart b = wp[0];
        for (int k = 1; k < kThreadsBounds / 32; k++) bounds_merge(b, wp[k]);
        part[blockIdx.x] = b;
    }
}

// The partials in a fixed order (deterministic FP64 sum, no same-address
// atomics), then the grids.
__global__ void __launch_bounds__(kThreadsBounds) k_grid(Rheo c, StepScalars* S, const BoundsPart* part, int nparts,
                                                         GridArgs ga) {
    PDL_ENTRY();
    if (step_skipped(S)) return;
    __shared__ BoundsPart wp[kThreadsBounds / 32];
    StepScalars* L = scalars_to_smem(S);
    BoundsPart b{3.4e38f, -3.4e38f, 3.4e38f, -3.4e38f, 0.f, 1.e10f, 0.0, 0, 0};
    for (int k = threadIdx.x; k < nparts; k += kThreadsBounds) bounds_merge(b, part[k]);
    b.xmn = warp_min(b.xmn); b.xmx = warp_max(b.xmx); b.ymn = warp_min(b.ymn); b.ymx = warp_max(b.ymx);
    b.hmx = warp_max(b.hmx); b.dtm = warp_min(b.dtm); b.hsum = warp_sum(b.hsum); b.hcnt = warp_sum(b.hcnt);
    b.bad = __any_sync(0xffffffffu, b.bad) ? 1 : 0;
    if ((threadIdx.x & 31) == 0) wp[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x < 32) {
        BoundsPart t = wp[0];
        for (int k = 1; k < kThreadsBounds / 32; k++) bounds_merge(t, wp[k]);
        if (threadIdx.x == 0) {
            L->xmin_o = f2o(t.xmn); L->xmax_o = f2o(t.xmx); L->ymin_o = f2o(t.ymn); L->ymax_o = f2o(t.ymx);
            L->hmax_o = f2o(t.hmx); L->dtmin_o = f2o(t.dtm);
            L->hsum = t.hsum; L->hcount = t.hcnt; L->bad = t.bad;
        }
        __syncwarp();
        grid_setup(c, L, ga);
    }
    scalars_from_smem(S, L);
}

// dt update (Adaptive_dt_sph_SW :6658-6662) and the cell grids.  The
// reference sizes its single grid by 2*max(hsml) (grid_find :906-919), so one
// thin-front particle whose hsml keeps growing inflates every cell.  Here
// particles are split by smoothing length into levels: level 0 holds
// hsml <= Hc = min(max, level_factor*mean), level k >= 1 holds hsml in
// (Hc*2^(k-1), Hc*2^k]; level k has its own grid of cell size
// Hc*2^k/cell_div over the same box, and one cell-key space covers all
// levels.  The particles of the first reg_levels levels ("regular") take a
// thread each and the neighbour table; those of the coarser levels, few and
// with long neighbour lists, a block or a warp each.  A particle
// searches each level within hsml_i + (that level's hsml bound), so the
// neighbour set is the reference's {j : r_ij < 2*(h_i+h_j)/2} exactly.
// level_factor and cell_div are the search's tunables (gfsph_set_search):
// Hc = min(max, level_factor * mean hsml) and level k's cell size is
// Hc * 2^k / cell_div; neither changes the neighbour sets.
// Run by one warp on the shared copy of the scalars: the scalars by all lanes
// alike (lane 0 writes), level k by lane k.
__device__ void grid_setup(const Rheo& c, StepScalars* S, const GridArgs ga) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool first = lane == 0;
    if (first) S->reg_levels = ga.reg_levels;
    if (S->skip) return;
    auto stop = [&](int bits) {
        if (first) { S->err |= bits; S->skip = 1; }
    };
    if (S->bad) return stop(kErrNonFinite);
    const float xmn = o2f(S->xmin_o), xmx = o2f(S->xmax_o), ymn = o2f(S->ymin_o), ymx = o2f(S->ymax_o);
    const float hmx = o2f(S->hmax_o);
    if (S->xmin_o == 0xffffffffu || !(hmx > 0.f) || S->hcount == 0) return stop(kErrEmpty);
    float dt = S->dt;
    if (S->advance) {
        float dtmin = (c.ic_adapt != 0) ? o2f(S->dtmin_o) : 1.e10f;
        if (dtmin < dt) dt = dtmin;
        else if (c.ic_adapt != 0) dt = fminf(1.1f * dt, dtmin);
    }
    const float lx = xmx - xmn, ly = ymx - ymn;
    if (first) {
        S->dt_step = dt;
        // the reference's grid: cells of 2*max(hsml) (grid_find_NEW_tools My_SPH_Tools_2019.f90:1168-1181)
        const float delt = hmx * 2.f;
        int nd = (int)(lx / delt + 1.f);
        S->ref_ndx = nd;
        S->ref_xmin = (xmn - ((float)nd * delt - lx) / 2.f) - 0.001f * lx;
        nd = (int)(ly / delt + 1.f);
        S->ref_ndy = nd;
        S->ref_ymin = (ymn - ((float)nd * delt - ly) / 2.f) - 0.001f * ly;
        S->ref_delt = delt;
    }
    const float mean = (float)(S->hsum / (double)S->hcount);
    const float hc = fminf(hmx, ga.level_factor * mean);
    int nlev = 1;
    while (nlev < kMaxLevels && ldexpf(hc, nlev - 1) < hmx) nlev++;
    const int k = lane;
    float cell = 0.f, cellh = 0.f, fx = 1.f, fy = 1.f;
    if (k < nlev) {
        cell = ldexpf(hc, k) / ga.cell_div;
        cellh = cell * kCellAspect;
        fx = lx / cell + 1.f;
        fy = ly / cellh + 1.f;
    }
    const bool far = !(fx < 1.0e8f) || !(fy < 1.0e8f) || !(fx * fy < 2.0e9f);  // far beyond any capacity
    if (__any_sync(full, far) || ldexpf(hc, nlev - 1) < hmx) {
        if (first) S->need_cells = 0x3fffffff;
        return stop(kErrCells);
    }
    const int ndx = (int)fx, ndy = (int)fy;
    const int nbx = (ndx + kBlkX - 1) / kBlkX, nby = (ndy + kBlkY - 1) / kBlkY;
    long long off = (k < nlev) ? (long long)nbx * nby : 0, doff = (k < nlev) ? (long long)ndx * ndy : 0;
    for (int o = 1; o < 32; o <<= 1) {  // the levels' blocks and cells up to and with level k
        const long long t = __shfl_up_sync(full, off, o), u = __shfl_up_sync(full, doff, o);
        if (lane >= o) { off += t; doff += u; }
    }
    if (k < nlev) {
        const float lxn = (float)ndx * cell, lyn = (float)ndy * cellh;
        S->lev_gx0[k] = (xmn - (lxn - lx) / 2.f) - 0.001f * lx;
        S->lev_gy0[k] = (ymn - (lyn - ly) / 2.f) - 0.001f * ly;
        S->lev_c[k] = cell;
        S->lev_ndx[k] = ndx;
        S->lev_ndy[k] = ndy;
        S->lev_nbx[k] = nbx;
        S->lev_boff[k + 1] = (int)min(off, 0x7fffffffLL);
        S->lev_off[k + 1] = (int)min(doff, 0x7fffffffLL);
    }
    off = __shfl_sync(full, off, nlev - 1);
    doff = __shfl_sync(full, doff, nlev - 1);
    if (!first) return;
    S->lev_boff[0] = 0;
    S->lev_off[0] = 0;
    S->hc = hc;
    S->nlev = nlev;
    const long long budget = min((long long)ga.max_cells, max(kDenseCells, 8LL * S->hcount));
    S->sparse = (doff + 1 > budget) ? 1 : 0;
    if (!S->sparse) {
        if (doff + 1 > (long long)ga.cap_cells) {
            S->need_cells = (int)(doff + 1);
            return stop(kErrCells);
        }
        S->ncells = (int)doff;
        return;
    }
    if (off + 1 > (long long)ga.cap_blocks) {
        S->need_blocks = (off + 1 > 0x3fffffffLL) ? 0x3fffffff : (int)(off + 1);
        return stop(kErrBlocks);
    }
    S->nblocks = (int)off;
}

__device__ __forceinline__ void cell_of(float2 p, const StepScalars* S, int k, int& cx, int& cy) {
    float gd = S->lev_c[k];
    int ix = (int)((p.x - S->lev_gx0[k]) / gd + 1.f);
    int iy = (int)((p.y - S->lev_gy0[k]) / (gd * kCellAspect) + 1.f);
    cx = min(max(ix, 1), S->lev_ndx[k]) - 1;
    cy = min(max(iy, 1), S->lev_ndy[k]) - 1;
}

__device__ __forceinline__ int level_of(float hs, const StepScalars* S) {
    int k = 0;
    while (k + 1 < S->nlev && hs > ldexpf(S->hc, k)) k++;
    return k;
}

// Cell coordinates are never negative: unsigned division and remainder by
// the block sides compile to shifts and masks.
__device__ __forceinline__ int block_of(const StepScalars* S, int k, int cx, int cy) {
    return S->lev_boff[k] + (int)((unsigned)cy / kBlkY) * S->lev_nbx[k] + (int)((unsigned)cx / kBlkX);
}

// An exclusive scan before its tile offsets are added in (k_scan_tiles leaves
// the scan of each tile and the scanned tile sums): entry i.
struct TileScan {
    const int* part;
    const int* tile;
    __device__ __forceinline__ int operator[](int i) const { return part[i] + tile[(unsigned)i / kScanTile]; }
};

// Sparse layout: the key of cell (cx, cy) of level k, block b.  The occupied
// blocks of its block row (block-map entries rb .. rb + nbx - 1, slots f ..
// f + nocc - 1) take 256 nocc keys from 256 f, cell row by cell row, 32 keys a
// block in each.
__device__ __forceinline__ int sparse_key(const StepScalars* S, TileScan bstart, int k, int cx, int cy, int b) {
    const int nbx = S->lev_nbx[k], rb = S->lev_boff[k] + (int)((unsigned)cy / kBlkY) * nbx;
    const int f = bstart[rb], nocc = bstart[rb + nbx] - f;
    return f * kBlockCells + (int)((unsigned)cy % kBlkY) * (nocc * kBlkX) + (bstart[b] - f) * kBlkX +
           (int)((unsigned)cx % kBlkX);
}

// Marks the blocks that hold particles (block map, all levels; block-sparse
// layout only).
__global__ void k_mark(const PState B, int n, DemView dem, StepScalars* S, int* bmark) {
    PDL_ENTRY();
    if (S->skip || !S->sparse) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (B.flag[i]) continue;
        float2 p = B.pos[i];
        if (out_of_box(dem, p.x, p.y)) continue;
        int k = level_of(B.hsml[i], S);
        int cx, cy;
        cell_of(p, S, k, cx, cy);
        int b = block_of(S, k, cx, cy);
        if (bmark[b] == 0) bmark[b] = 1;
    }
}

// Cell key (row-major in the dense layout, sparse_key in the sparse one) and
// within-cell arrival rank of each particle (counting sort histogram,
// grid_find :938-948); out-of-domain particles get key -1.  Also takes the
// largest smoothing length of every level, which bounds the stencils of the
// neighbour search more tightly than the level's upper limit.  If the
// occupied blocks need more cells than the histogram holds, nothing is
// counted and the step stops with kErrCells.
__global__ void k_hist(const PState B, int n, DemView dem, StepScalars* S, TileScan bstart, int* count, int2* keyrank,
                       int cap_cells) {
    PDL_ENTRY();
    if (S->skip) return;
    const bool sparse = S->sparse != 0;
    const long long ncells = sparse ? (long long)bstart[S->nblocks] * kBlockCells : (long long)S->ncells;
    const bool over = ncells + 1 > (long long)cap_cells;
    if (over && blockIdx.x == 0 && threadIdx.x == 0) {
        atomicOr(&S->err, kErrCells);
        S->need_cells = (ncells + 1 > 0x3fffffffLL) ? 0x3fffffff : (int)(ncells + 1);
    }
    if (sparse && !over && blockIdx.x == 0 && threadIdx.x == 0) S->ncells = (int)ncells;
    // per-level largest hsml, reduced in shared memory first: every particle
    // of a level would otherwise hit the same global word
    __shared__ unsigned int lmax[kMaxLevels];
    const int nlev = S->nlev;
    for (int k = threadIdx.x; k < nlev; k += blockDim.x) lmax[k] = 0u;
    __syncthreads();
    unsigned int h0 = 0u;  // largest level-0 hsml seen by this thread
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int2 kr = make_int2(-1, 0);
        const float2 p = B.pos[i];
        const float hs = B.hsml[i];
        if (!B.flag[i] && !out_of_box(dem, p.x, p.y)) {
            const int k = level_of(hs, S);
            if (k == 0) h0 = max(h0, f2o(hs));
            else atomicMax(&lmax[k], f2o(hs));
            int cx, cy;
            cell_of(p, S, k, cx, cy);
            const int key = sparse ? sparse_key(S, bstart, k, cx, cy, block_of(S, k, cx, cy))
                                   : S->lev_off[k] + cy * S->lev_ndx[k] + cx;
            if (!over) {
                kr.x = key;
                kr.y = atomicAdd(&count[key], 1);
            }
        }
        keyrank[i] = kr;
    }
    h0 = __reduce_max_sync(0xffffffffu, h0);
    if ((threadIdx.x & 31) == 0 && h0) atomicMax(&lmax[0], h0);
    __syncthreads();
    for (int k = threadIdx.x; k < nlev; k += blockDim.x)
        if (lmax[k]) atomicMax(&S->lev_hmax_o[k], lmax[k]);
}

// Exclusive prefix of the tile sums, by one block (1 <= ntiles <= kScanTops *
// blockDim.x): tile_sum[t] becomes the first index of tile t.
constexpr int kScanTops = 32;
__device__ void scan_tile_sums(int* tile_sum, int ntiles) {
    __shared__ int wsum[32];
    const int per = (ntiles + (int)blockDim.x - 1) / (int)blockDim.x;  // <= kScanTops
    int loc[kScanTops];
    int s = 0;
    for (int k = 0; k < kScanTops; k++) {
        if (k >= per) break;
        int g = threadIdx.x * per + k;
        int v = (g < ntiles) ? ((volatile int*)tile_sum)[g] : 0;
        loc[k] = s;
        s += v;
    }
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int incl = s;
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        int w = (lane < (int)(blockDim.x >> 5)) ? wsum[lane] : 0;
        int wi = w;
        for (int o = 1; o < 32; o <<= 1) {
            int t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < (int)(blockDim.x >> 5)) wsum[lane] = wi - w;
    }
    __syncthreads();
    int off = wsum[wid] + incl - s;
    for (int k = 0; k < kScanTops; k++) {
        if (k >= per) break;
        int g = threadIdx.x * per + k;
        if (g < ntiles) tile_sum[g] = off + loc[k];
    }
}

// Scan of count[0 .. *nptr] into start (exclusive), tile by tile; the last
// tile to finish also scans the tile sums.  The readers that come before
// k_reorder add the tile offsets themselves (TileScan), k_reorder adds them in
// for the rest of the step.  Zeroes the counts it has read, so that they start
// at zero in the next step without a clearing pass.
// which: 0 the cells, 1 the block map (only in the block-sparse layout).  A
// step whose earlier kernels raised an error is stopped here.
__global__ void k_scan_tiles(int* count, int* start, int* tile_sum, const int* nptr, StepScalars* S,
                             int which) {
    PDL_ENTRY();
    if (S->skip || (which == 1 && !S->sparse)) return;
    if (S->err) {
        if (blockIdx.x == 0 && threadIdx.x == 0) S->skip = 1;
        return;
    }
    int m = *nptr + 1;
    const int ntiles = (m + kScanTile - 1) / kScanTile;
    int base = blockIdx.x * kScanTile;
    if (base >= m) return;
    __shared__ int sh[kScanTile];
    __shared__ int wsum[kScanThreads / 32];
    __shared__ bool last;
    constexpr int per = kScanTile / kScanThreads;
    int v[per];  // all loads before the stores
#pragma unroll
    for (int k = 0; k < per; k++) {
        const int g = base + k * kScanThreads + threadIdx.x;
        v[k] = (g < m) ? count[g] : 0;
    }
#pragma unroll
    for (int k = 0; k < per; k++) {
        const int g = base + k * kScanThreads + threadIdx.x;
        sh[k * kScanThreads + threadIdx.x] = v[k];
        if (g < m) count[g] = 0;
    }
    __syncthreads();
    int loc[per];
    int s = 0;
    for (int k = 0; k < per; k++) { loc[k] = s; s += sh[threadIdx.x * per + k]; }
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int incl = s;
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        int w = (lane < kScanThreads / 32) ? wsum[lane] : 0;
        int wi = w;
        for (int o = 1; o < 32; o <<= 1) {
            int t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < kScanThreads / 32) wsum[lane] = wi - w;
        if (lane == kScanThreads / 32 - 1) tile_sum[blockIdx.x] = wi;
    }
    __syncthreads();
    int off = wsum[wid] + incl - s;
    for (int k = 0; k < per; k++) sh[threadIdx.x * per + k] = off + loc[k];
    __syncthreads();
    for (int k = threadIdx.x; k < kScanTile; k += kScanThreads) {
        int g = base + k;
        if (g < m) start[g] = sh[k];
    }
    if (ntiles == 1) {
        if (threadIdx.x == 0) tile_sum[0] = 0;
        return;
    }
    if (threadIdx.x == 0) {
        __threadfence();
        last = (atomicAdd(&S->scan_ticket[which], 1u) == (unsigned)ntiles - 1u);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    scan_tile_sums(tile_sum, ntiles);
    if (threadIdx.x == 0) S->scan_ticket[which] = 0u;
}

// Scatter (grid_find :952-958): particles to start[cell] + rank (level 0
// first, then the higher levels), out-of-domain particles behind them.
__global__ void k_scatter(const int2* keyrank, int n, TileScan start, TileScan bstart, StepScalars* S, int* perm) {
    PDL_ENTRY();
    if (S->skip) return;
    int nact = start[S->ncells];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int2 kr = keyrank[i];
        int slot = (kr.x >= 0) ? start[kr.x] + kr.y : nact + atomicAdd(&S->nout, 1);
        perm[slot] = i;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // regular particles: levels 0 .. reg_levels-1 (slots before the first
        // key of level reg_levels; lev_off[nlev] ends the key space)
        const int r = min(S->nlev, S->reg_levels);
        int first = S->sparse ? bstart[S->lev_boff[r]] * kBlockCells : S->lev_off[r];
        int nreg = start[first];
        S->nreg = nreg;
        S->nbig = nact - nreg;
        S->nactive = nact;
        if (nreg != n) S->irregular = 1;
    }
}

// Gathers the state into the new (cell-sorted) order, each cell's particles
// ordered by original index, so that the within-cell order, hence every
// neighbour-sum order, is independent of the atomics' arrival order: a
// particle counts the members of its cell with a smaller index (a cell holds
// one or two).  With icpwp = 3 also the pore-water pressure; with icpwp = 3 or
// nor_density rho0, the depth RK45 keeps at its start (after the h_inf clamp
// of Adaptive_dt_sph_SW :6540, modes 1, 2 and 10).  Also adds the tile offsets
// into the cell starts (to startF, since other threads still read start) and
// the block starts.
__global__ void k_reorder(const PState B, int n, const int* perm, const int2* keyrank, PState A,
                          float4* xhm, const StepScalars* S, Rheo c, float* rho0, float* ratio0, int2* rcell,
                          const unsigned char* spec_u, unsigned char* spec_a, TileScan start, int* startF, int* bstart,
                          const int* btile) {
    PDL_ENTRY();
    if (S->skip) return;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    const int nact = S->nactive;
    for (int s0 = tid; s0 < n; s0 += nt) {
        const int o = perm[s0];
        int s = s0;
        if (s0 < nact) {
            const int key = keyrank[o].x, a = start[key], b = start[key + 1];
            if (b - a > 1) {
                const int me = B.id[o];
                s = a;
                for (int m = a; m < b; m++) s += (B.id[perm[m]] < me) ? 1 : 0;
            }
        }
        float2 p = B.pos[o];
        float hs = B.hsml[o], m = B.mass[o];
        float r = B.rho[o];
        A.pos[s] = p;
        A.vel[s] = B.vel[o];
        A.rho[s] = r;
        if (c.icpwp != 0) A.pwp[s] = B.pwp[o];
        if (c.icpwp != 0 || c.nor_density)
            rho0[s] = ((c.ic_adapt == 1 || c.ic_adapt == 2 || c.ic_adapt == 10) && r < c.h_inf) ? c.h_inf : r;
        if (c.nor_density) ratio0[s] = m / rho0[s];
        A.mass[s] = m;
        A.hsml[s] = hs;
        A.flag[s] = B.flag[o];
        A.id[s] = B.id[o];
        if (c.ws) spec_a[s] = spec_u[B.id[o]];
        xhm[s] = make_float4(p.x, p.y, hs, m);
        if (rcell && !B.flag[o]) {  // cell of the reference's grid (:1203-1204)
            int ix = (int)((p.x - S->ref_xmin) / S->ref_delt + 1.f);
            int iy = (int)((p.y - S->ref_ymin) / S->ref_delt + 1.f);
            rcell[s] = make_int2(min(ix, S->ref_ndx), min(iy, S->ref_ndy));
        }
    }
    const int nc = S->ncells, nb = S->sparse ? S->nblocks : -1;
    for (int k = tid; k <= nc; k += nt) startF[k] = start[k];
    for (int k = tid; k <= nb; k += nt) bstart[k] += btile[(unsigned)k / kScanTile];
}

// Largest neighbour distance against a level whose hsml <= Hk:
// r < SK*(hi + hj)/2 <= SK/2 (hi + Hk).
template <int SK>
__device__ __forceinline__ float support_span(float hi, float hk) {
    return (SK == 2) ? hi + hk : 1.5f * (hi + hk);
}

// The reference's own cell test, needed for supports of 3 h (skf 2, 3):
// grid_find pairs only particles in the same or adjacent cells of its grid
// of 2*max(hsml) (My_SPH_Tools_2019.f90:1257-1264), so pairs up to 3 h apart
// are kept or dropped by where that grid falls.  (With 2 h supports every
// pair lies within one cell and the test is implied.)
template <int SK>
__device__ __forceinline__ bool ref_adjacent(const Search& Q, int2 ci, int j) {
    if (SK == 2) return true;
    const int2 cj = Q.rcell[j];
    return abs(cj.x - ci.x) <= 1 && abs(cj.y - ci.y) <= 1;
}

// Neighbour search and summation density of the regular particles, fused:
// every j with r < 2*(hi+hj)/2 (the pair set of grid_find, :987-1060) is
// entered in the neighbour table (tab_base) with the pair's kernel value and
// gradient, and h_i = W(0,h_i) m_i + sum_j m_j W_ij (sum_density_Tools
// :1796-1836) is accumulated in FP64.  Also stores the pressure term of
// IntForces_SW with h clamped to h_inf (:6769, :6797): p/h^2 (pa_sph 2) or p
// (pa_sph 1).
//
// G lanes share a particle.  Two phases: (1) each lane scans every G-th row
// of the stencil and lists the neighbours it finds in shared memory (the test
// alone, ~12 instructions a candidate, half of which are kept); (2) the
// lanes share out the listed pairs evenly and evaluate them, every lane busy,
// the table entries of a warp in whole sectors.  One pass over the candidates
// that evaluated a pair wherever one lane of the warp kept it ran the ~130
// instructions of a pair at a third of its lanes and, with one thread per
// particle, as one chain of 100 dependent gathers: 57 us even for 850
// particles.  A lane whose list is full counts on; the scan is then repeated
// for the next kDenList of each lane.
constexpr int kDenThreads = 128;
constexpr int kDenBlocks = 7;  // resident blocks asked for
constexpr int kScanStep = 4;  // candidates loaded at a time
template <int G> struct DenList { static constexpr int value = (G == 2) ? 40 : (G == 4 ? 24 : 16); };  // ~1.5x a lane's share of 50
// The particles of the coarse levels, few, are not searched through their
// mostly empty grids: each block picks those that reach its particles' box
// and its lanes test these alone.  Beyond kBigScan of them, when every block
// reads as many more, the grids are walked as well: us a launch for 200k
// particles, direct and walked, 1000 coarse ones 107 and 96, 3000 172 and 128,
// 4000 214 and 146 (300: 86 direct).
constexpr int kBigScan = 512;

// The rows of level k's cells that the support of particle i (position xi,
// smoothing length hi) can touch: every j of the level has hsml_j <= Hk (the
// level's largest), so |x_i - x_j| < SK/2 (hi + Hk).  In units of the cell
// width, with i at (u, v): row jy lies dy away from it, and j within
// sqrt(s^2 - dy^2) of u in that row, taken from i's place inside its cell (the
// cell numbers alone would cost a cell on each side: 102 candidates for 46
// neighbours on the lattice, 66 with the place).  ex, ey (cells) cover the
// rounding of u, v and of j's own cell numbers, 2^-21 of the grid's extent and
// more.  Either layout keeps a row's cells in order, so each row is one slot
// range.
template <bool SPARSE>
struct LevelRows {
    float u, v, s2, ex, ey, reach;  // reach: SK/2 (hi + Hk)
    int y0, nrow, ndx, base, nbx;  // base: the level's first key (dense) or block-map entry (sparse)

    // false for an empty level
    template <int SK>
    __device__ __forceinline__ bool open(const StepScalars* S, int k, float2 xi, float hi) {
        const unsigned int hk = S->lev_hmax_o[k];
        if (hk == 0u) return false;
        const float rc = 1.f / S->lev_c[k];
        ndx = S->lev_ndx[k];
        const int ndy = S->lev_ndy[k];
        // clamped as the cell numbers are: that brings no two particles further apart
        u = fminf(fmaxf((xi.x - S->lev_gx0[k]) * rc, 0.f), (float)ndx);
        v = fminf(fmaxf((xi.y - S->lev_gy0[k]) * (rc * (1.f / kCellAspect)), 0.f), (float)ndy);
        reach = support_span<SK>(hi, o2f(hk));
        const float s = reach * rc;
        s2 = s * s;
        ex = 0.01f + (float)ndx * 1.e-6f;
        ey = 0.01f + (float)ndy * 1.e-6f;
        const float sy = s * (1.f / kCellAspect) + ey;
        y0 = min(max((int)(v - sy), 0), ndy - 1);
        nrow = min((int)fminf(v + sy, 1.e9f), ndy - 1) - y0 + 1;
        base = SPARSE ? S->lev_boff[k] : S->lev_off[k];
        nbx = SPARSE ? S->lev_nbx[k] : 0;
        return true;
    }

    // slots ja .. jb-1 of the row-th row (empty: ja >= jb)
    __device__ __forceinline__ void range(const Search& Q, int row, int& ja, int& jb) const {
        ja = jb = 0;
        const int jy = y0 + row;
        const float dy = fmaxf(fmaxf((float)jy - v, v - (float)(jy + 1)) - ey, 0.f) * kCellAspect;
        const float q = s2 - dy * dy;
        if (!(q > 0.f)) return;
        const float hw = q * rsqrtf(q) + ex;
        const int x0 = min(max((int)(u - hw), 0), ndx - 1), x1 = min((int)fminf(u + hw, 1.e9f), ndx - 1);
        if (!SPARSE) {
            const int key = base + jy * ndx;
            ja = Q.start[key + x0];
            jb = Q.start[key + x1 + 1];
            return;
        }
        const int rb = base + (int)((unsigned)jy / kBlkY) * nbx;
        const int f = Q.bstart[rb], nocc = Q.bstart[rb + nbx] - f;
        if (nocc == 0) return;
        const int c0 = (int)((unsigned)x0 / kBlkX), c1 = (int)((unsigned)x1 / kBlkX);
        const int s0 = Q.bstart[rb + c0], s1 = Q.bstart[rb + c1];
        // an empty block at either end adds no keys
        const int o0 = (Q.bstart[rb + c0 + 1] != s0) ? (int)((unsigned)x0 % kBlkX) : 0;
        const int o1 = (Q.bstart[rb + c1 + 1] != s1) ? (int)((unsigned)x1 % kBlkX) + 1 : 0;
        const int key = f * kBlockCells + (int)((unsigned)jy % kBlkY) * (nocc * kBlkX) - f * kBlkX;
        ja = Q.start[key + s0 * kBlkX + o0];
        jb = Q.start[key + s1 * kBlkX + o1];
    }
};

// The coarse-level particles, with up to every particle in their support, have
// blocks of their own in the pair kernels (of kBigThreads, k_density of
// kDenThreads): the first kBigBlocks, which take the usual few, up to kBigRounds
// each, beside the regular ones, and with more of them also the last half of the
// others.  All warps of a block share a particle (with one warp each, the one
// with the longest list took 38 us of the 200k flow's step in each of the three
// passes), until there are more than four a block: then a warp takes a particle,
// since there are warps enough and the block's barriers and short rows count.
// us a step of 200k particles with 0, 300, 1000, 5000 and 20,000 coarse ones of
// 8 times the smoothing length: 181, 208, 230, 374 and 870; with the first
// kBigBlocks blocks alone 180, 207, 255, 760 and 2790; with one warp each and the
// kernels of a thread per particle 246, 321, 342, 432 and 1000.  (Blocks that
// take regular and coarse particles in turn, or more blocks behind the regular
// ones, cost every step 1 to 3 %.)
constexpr int kBigThreads = 256;
constexpr int kBigBlocks = 148;
constexpr int kBigRounds = 4;
// What the pair kernels read of the scalars first, in one trip to memory, and
// the blocks of the coarse particles: the first kBigBlocks and those from tail on.
struct PairWork {
    int skip, nreg, nbig, tail;
    __device__ __forceinline__ explicit PairWork(const StepScalars* S) : skip(S->skip), nreg(S->nreg), nbig(S->nbig) {
        const int grid = (int)gridDim.x;
        tail = nbig > kBigRounds * kBigBlocks ? kBigBlocks + (grid - kBigBlocks + 1) / 2 : grid;
    }
    __device__ __forceinline__ bool coarse() const { return blockIdx.x < kBigBlocks || (int)blockIdx.x >= tail; }
};
// Calls f(i, lw) for the coarse particles of this block or warp; 1 << lw warps share one.
template <int T, class F>
__device__ __forceinline__ void coarse_particles(int nreg, int nbig, int tail, F&& f) {
    constexpr int LW = T == 256 ? 3 : 2;
    static_assert(T == 32 << LW, "T is 128 or 256");
    const int nc = kBigBlocks + (int)gridDim.x - tail;
    const int cb = blockIdx.x < kBigBlocks ? blockIdx.x : kBigBlocks + (int)blockIdx.x - tail;
    const bool alone = nbig > 4 * nc;
    const int lw = alone ? 0 : LW, step = nc << (LW - lw);
    for (int b = alone ? (cb << LW) + (threadIdx.x >> 5) : cb; b < nbig; b += step) f(nreg + b, lw);
}

// The neighbours of coarse particle i: the sharing warps take the rows of a
// level's stencil in turn, the lanes fetch the slot ranges of up to 32 rows at
// once, then share each row's candidates.
template <bool SPARSE, int SK, class F>
__device__ __forceinline__ void coarse_rows(const Search& Q, const StepScalars* S, int i, int lw, F& f) {
    const int lane = threadIdx.x & 31, wid = (threadIdx.x >> 5) & ((1 << lw) - 1);
    const float4 me = Q.xhm[i];
    const float2 xi = make_float2(me.x, me.y);
    const float hi = me.z;
    const int2 ci = (SK == 2) ? make_int2(0, 0) : Q.rcell[i];
    for (int k = 0; k < S->nlev; k++) {
        LevelRows<SPARSE> rows;
        if (!rows.template open<SK>(S, k, xi, hi)) continue;
        for (int rb = 0; rb < rows.nrow; rb += 32 << lw) {
            const int row = rb + (lane << lw) + wid;
            int ja = 0, jb = 0;
            if (row < rows.nrow) rows.range(Q, row, ja, jb);
            const int nr = min(32, (rows.nrow - rb - wid + (1 << lw) - 1) >> lw);
            for (int r = 0; r < nr; r++) {
                const int a = __shfl_sync(0xffffffffu, ja, r), e = __shfl_sync(0xffffffffu, jb, r);
                for (int j = a + lane; j < e; j += 32) {
                    if (j == i) continue;
                    const float4 o = Q.xhm[j];
                    PairGeom g;
                    if (pair_search<SK>(xi, make_float2(o.x, o.y), hi, o.z, g) && ref_adjacent<SK>(Q, ci, j))
                        f(j, o, g);
                }
            }
        }
    }
}
template <int SK, class F>
__device__ __forceinline__ void coarse_neighbours(const Search& Q, const StepScalars* S, int i, int lw, F&& f) {
    if (S->sparse) coarse_rows<true, SK>(Q, S, i, lw, f);
    else coarse_rows<false, SK>(Q, S, i, lw, f);
}
// Sum over the warps that share a particle, in a fixed order, in the first lane
// of the first; every thread of them calls it.
__device__ __forceinline__ double coarse_sum(double v, int lw) {
    v = warp_sum(v);
    if (lw == 0) return v;
    __shared__ double part[kBigThreads / 32];
    __syncthreads();
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += part[w];
    return t;
}
__device__ __forceinline__ bool coarse_first(int lw) { return (threadIdx.x & (lw ? ~0u : 31u)) == 0; }

// Summation density of the coarse-level particles.
template <int SKF, bool WS>
__device__ __forceinline__ void density_big(const PState& A, const Search& Q, const StepScalars* S, const Rheo& c, const PairWork& pw) {
    constexpr int SK = SupportScale<SKF>::value;
    coarse_particles<kDenThreads>(pw.nreg, pw.nbig, pw.tail, [&](int i, int lw) {
        double acc = 0.0;
        const unsigned char si = WS ? Q.spec[i] : 0;
        coarse_neighbours<SK>(Q, S, i, lw, [&](int j, float4 o, const PairGeom& g) {
            if (WS && Q.spec[j] != si) return;  // type 1: not in the density (:1829)
            acc += (double)(o.w * sph_kernel_w<SKF>(g.r, g.mh));
        });
        acc = coarse_sum(acc, lw);
        if (coarse_first(lw)) {
            float4 me = Q.xhm[i];
            float h = (float)((double)(sph_kernel_w<SKF>(0.f, me.z) * me.w) + acc);
            A.rho[i] = h;
            float hc = (h < c.h_inf) ? c.h_inf : h;
            float p = (c.cgra05 * hc) * hc;
            Q.pterm[i] = (c.pa_sph == 1) ? p : p / (hc * hc);
        }
    });
}

// Bound by FP32 issue and the latency of the gathers: 200k particles (release,
// two lanes) 78 us a launch (89 before the pairs were evaluated two at a time)
// where one thread per particle, evaluating each pair as it was found, took
// 115; the flow with coarse levels 94 (106) against 190; 1M particles 350 (390)
// against 480.  Instantiated for both cell layouts; the
// launch whose layout this step does not use returns at once.
template <bool SPARSE, int SKF, bool WS, int G>
__global__ void __launch_bounds__(kDenThreads, kDenBlocks) k_density(PState A, Search Q, StepScalars* S, Rheo c, int n) {
    PDL_WAIT();
    // Behind the dense launch comes the sparse one.  Let in at once, its blocks wait here for all of the dense ones with
    // their registers held, which other streams' kernels could use: beyond two blocks an SM they come in as this
    // launch's blocks end (ten members of 2k to 24k particles side by side, a pass of 16 steps 4808 -> 4608 us; a
    // run alone, when nothing else wants the places: within 0.3 % from 2k particles on, 850 1.4 % slower).
    if (SPARSE || gridDim.x <= 2 * kBigBlocks) PDL_NEXT();
    if ((S->sparse != 0) != SPARSE) return;
    const PairWork pw(S);
    if (__syncthreads_or(pw.skip)) return;  // another block may set it meanwhile: one decision per block
    if (pw.coarse()) {
        density_big<SKF, WS>(A, Q, S, c, pw);
        return;
    }
    constexpr int SK = SupportScale<SKF>::value;
    constexpr int L = DenList<G>::value, P = kDenThreads / G;
    constexpr unsigned full = 0xffffffffu;
    __shared__ int list[L * kDenThreads];  // entry e of thread t at e * kDenThreads + t
    __shared__ float4 bigs[kDenThreads];
    __shared__ int bigj[kDenThreads];
    __shared__ float wbox[kDenThreads / 32][5];
    __shared__ int wcnt[kDenThreads / 32];
    const int tid = threadIdx.x, gl = tid % G, lane = tid & 31, wid = tid >> 5;
    const int nreg = pw.nreg, nbig = pw.nbig;
    const bool scan_big = nbig > 0 && nbig <= kBigScan;
    const int nlev = (nbig > 0 && !scan_big) ? S->nlev : min(S->nlev, S->reg_levels);
    const float hmax = o2f(S->hmax_o);
    const int bid = blockIdx.x - kBigBlocks, nb = pw.tail - kBigBlocks;
    for (int base = bid * P; base < nreg; base += nb * P) {  // the same trips for the whole block
        const int i = base + tid / G;
        const bool act = i < nreg;
        const float4 me = Q.xhm[act ? i : base];
        const float2 xi = make_float2(me.x, me.y);
        const float hi = me.z;
        const int2 ci = (SK == 2) ? make_int2(0, 0) : Q.rcell[act ? i : base];
        const unsigned char si = WS ? Q.spec[act ? i : base] : 0;
        const bool safe = quot_safe(hi, hmax);
        const size_t tab = tab_base(act ? i : base, Q.kcap);
        float bx0 = 0.f, bx1 = 0.f, by0 = 0.f, by1 = 0.f, bh = 0.f;  // the block's box and largest hsml
        if (scan_big) {
            bx0 = warp_min(me.x); bx1 = warp_max(me.x);
            by0 = warp_min(me.y); by1 = warp_max(me.y);
            bh = warp_max(hi);
            if (lane == 0) {
                wbox[wid][0] = bx0; wbox[wid][1] = bx1; wbox[wid][2] = by0; wbox[wid][3] = by1; wbox[wid][4] = bh;
            }
            __syncthreads();
            for (int w = 0; w < kDenThreads / 32; w++) {
                bx0 = fminf(bx0, wbox[w][0]); bx1 = fmaxf(bx1, wbox[w][1]);
                by0 = fminf(by0, wbox[w][2]); by1 = fmaxf(by1, wbox[w][3]);
                bh = fmaxf(bh, wbox[w][4]);
            }
        }
        double acc = 0.0;
        int found = 0;  // entries of this particle in the table
        for (int skip = 0;; skip += L) {
            // phase 1: the neighbours this lane finds, from the skip-th on, go into its list; at is the next place,
            // before the list while the first skip ones pass
            int at = tid - skip * kDenThreads;
            auto keep = [&](int j, bool ok) {
                if (ok && (unsigned)at < (unsigned)(L * kDenThreads)) list[at] = j;
                at += ok ? kDenThreads : 0;
            };
            int first = gl;  // this lane's first row of the next level
            for (int k = 0; k < nlev; k++) {
                LevelRows<SPARSE> rows;
                if (!rows.template open<SK>(S, k, xi, hi)) continue;
                const float edge = kEdge * rows.reach * rows.reach;
                if (act)
                    for (int s = first; s < rows.nrow; s += G) {
                        int ja, jb;
                        rows.range(Q, s, ja, jb);
                        for (int j = ja; j < jb; j += kScanStep) {
                            float4 o[kScanStep];  // xhm is padded by kScanStep entries
                            float v[kScanStep];
                            bool near = false;
#pragma unroll
                            for (int u = 0; u < kScanStep; u++) o[u] = Q.xhm[j + u];
#pragma unroll
                            for (int u = 0; u < kScanStep; u++) {
                                v[u] = pair_gap<SK>(xi, o[u], hi);
                                near |= fabsf(v[u]) <= edge;
                            }
                            if (near) {
#pragma unroll
                                for (int u = 0; u < kScanStep; u++)
                                    if (fabsf(v[u]) <= edge) v[u] = pair_exact<SK>(xi, o[u], hi) ? -1.f : 1.f;
                            }
#pragma unroll
                            for (int u = 0; u < kScanStep; u++)
                                keep(j + u, (v[u] < 0.f) & (j + u < jb) & (j + u != i) && ref_adjacent<SK>(Q, ci, j + u));
                        }
                    }
                first = (first + G - rows.nrow % G) % G;
            }
            if (scan_big)
                for (int b0 = 0; b0 < nbig; b0 += kDenThreads) {
                    const int b = nreg + b0 + tid;
                    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
                    bool near = false;
                    if (b0 + tid < nbig) {
                        o = Q.xhm[b];
                        // distance to the box, with a margin for the rounding of both sides
                        const float dx = fmaxf(0.f, fmaxf(bx0 - o.x, o.x - bx1)), dy = fmaxf(0.f, fmaxf(by0 - o.y, o.y - by1));
                        const float t = support_span<SK>(bh, o.z);
                        near = dx * dx + dy * dy <= (t * t) * 1.0001f;
                    }
                    const unsigned m = __ballot_sync(full, near);
                    __syncthreads();  // the last chunk has been read
                    if (lane == 0) wcnt[wid] = __popc(m);
                    __syncthreads();
                    int put = __popc(m & ((1u << lane) - 1u)), tot = 0;
                    for (int w = 0; w < kDenThreads / 32; w++) {
                        if (w < wid) put += wcnt[w];
                        tot += wcnt[w];
                    }
                    if (near) { bigs[put] = o; bigj[put] = b; }
                    __syncthreads();
                    if (act)
                        for (int e = gl; e < tot; e += G) {
                            const int j = bigj[e];
                            keep(j, pair_exact<SK>(xi, bigs[e], hi) && ref_adjacent<SK>(Q, ci, j));
                        }
                }
            // phase 2: the group's listed pairs in lane order, shared out evenly
            const int mine = min(max((at - tid) / kDenThreads, 0), L);
            int pre = mine;  // exclusive prefix over the lanes of the group
#pragma unroll
            for (int o = 1; o < G; o <<= 1) {
                const int t = __shfl_up_sync(full, pre, o, G);
                if (gl >= o) pre += t;
            }
            const int tot = __shfl_sync(full, pre, G - 1, G);
            pre -= mine;
            int from[G];  // the lanes' first entries
#pragma unroll
            for (int o = 0; o < G; o++) from[o] = __shfl_sync(full, pre, o, G);
            __syncwarp();
            auto entry = [&](int t) {  // the neighbour at place t of the group's lists
                int own = 0, f = 0;
#pragma unroll
                for (int o = 1; o < G; o++)
                    if (t >= from[o]) { own = o; f = from[o]; }
                return list[(t - f) * kDenThreads + tid - gl + own];
            };
            auto store = [&](int t, int j, const float4& o, float w, float d0, float d1) {
                const bool cross = WS && Q.spec[j] != si;
                if (found + t < Q.kcap) {
                    const size_t to = tab + (size_t)(found + t) * kTabStride;
                    Q.nj[to] = cross ? (j | kCrossBit) : j;
                    Q.nw[to] = w;
                    if (SKF == 1) Q.ng[to] = d0;
                    else reinterpret_cast<float2*>(Q.ng)[to] = make_float2(d0, d1);
                }
                if (!cross) acc += (double)(o.w * w);
            };
            auto pair = [&](int t, int j, const float4& o) {
                const float dx0 = xi.x - o.x, dx1 = xi.y - o.y;
                const float dr = dx0 * dx0 + dx1 * dx1;
                const float mh = (hi + o.z) / 2.f;
                float w, d0, d1 = 0.f;
                if (SKF == 1) spline_pair(dr, mh, safe, w, d0);
                else sph_kernel<SKF>(sqrtf(dr), dx0, dx1, mh, w, d0, d1);
                store(t, j, o, w, d0, d1);
            };
            int t = gl;
            for (; t + G < tot; t += 2 * G) {  // two independent pairs at a time
                const int ja = entry(t), jb = entry(t + G);
                const float4 oa = Q.xhm[ja], ob = Q.xhm[jb];
                if (SKF == 1 && safe) {
                    const F2 da = f2(xi.x, xi.y) - f2(oa.x, oa.y), db = f2(xi.x, xi.y) - f2(ob.x, ob.y);
                    float a0, a1, b0, b1;
                    split(da * da, a0, a1);
                    split(db * db, b0, b1);
                    F2 w, g;
                    spline_pair2(f2(a0 + a1, b0 + b1), (f2(hi) + f2(oa.z, ob.z)) * f2(0.5f), w, g);
                    float wa, wb, ga, gb;
                    split(w, wa, wb);
                    split(g, ga, gb);
                    store(t, ja, oa, wa, ga, 0.f);
                    store(t + G, jb, ob, wb, gb, 0.f);
                } else {
                    pair(t, ja, oa);
                    pair(t + G, jb, ob);
                }
            }
            if (t < tot) {
                const int j = entry(t);
                pair(t, j, Q.xhm[j]);
            }
            found += tot;
            const bool more = at - tid > L * kDenThreads;
            if (scan_big ? !__syncthreads_or(more) : !__any_sync(full, more)) break;
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(full, acc, o);
        if (act && gl == 0) {
            Q.ncount[i] = found;
            if (found > Q.kcap) {  // table too small: stop this step before any state is written
                atomicOr(&S->err, kErrNbr);
                atomicMax(&S->need_nbr, found);
                atomicExch(&S->skip, 1);
            }
            const float h = (float)((double)(sph_kernel_w<SKF>(0.f, hi) * me.w) + acc);
            A.rho[i] = h;
            const float hc = (h < c.h_inf) ? c.h_inf : h;
            const float p = (c.cgra05 * hc) * hc;
            const float pt = (c.pa_sph == 1) ? p : p / (hc * hc);
            Q.pterm[i] = pt;
        }
        if (scan_big) __syncthreads();  // the box is rewritten
    }
}
// One pair term of IntForces_SW (SPH_SW_2019.f90:6905-6920) for particle i,
// from the pair's kernel gradient (d0, d1).
__device__ __forceinline__ void pressure_terms(const Rheo& c, float pi_, float rhoi, float pj, float rhoj, float mj,
                                               float d0, float d1, double& a0, double& a1) {
    float h0, h1;
    if (c.pa_sph == 1) {
        rhoi = (rhoi < c.h_inf) ? c.h_inf : rhoi;
        rhoj = (rhoj < c.h_inf) ? c.h_inf : rhoj;
        float rij = 1.f / (rhoi * rhoj);
        h0 = (-(pi_ + pj) * d0) * rij;
        h1 = (-(pi_ + pj) * d1) * rij;
    } else {
        h0 = -(pi_ + pj) * d0;
        h1 = -(pi_ + pj) * d1;
    }
    a0 += (double)(mj * h0);
    a1 += (double)(mj * h1);
}

// The same with the pair geometry: the kernel gradient evaluated here.
template <int SKF>
__device__ __forceinline__ void pressure_pair(const Rheo& c, float pi_, float rhoi, float pj, float rhoj, float mj,
                                              const PairGeom& g, double& a0, double& a1) {
    float w, d0, d1;
    sph_kernel<SKF>(g.r, g.dx0, g.dx1, g.mh, w, d0, d1);
    pressure_terms(c, pi_, rhoi, pj, rhoj, mj, d0, d1, a0, a1);
}

// One soil-water pair term of ExtForces_SW (:8502-8521) for particle i from
// its table entry (gradient d of W_ij with x_i - x_j): a soil particle gets
// -dens_ws g m_j grad W; a water particle, with ic_SWalg = 0, +g m_j grad W
// of the pair taken from the soil side (-d here).
__device__ __forceinline__ void wir_pair_term(const Rheo& c, bool water, float mj, float d0, float d1, double& b0,
                                              double& b1) {
    if (!water) {
        b0 -= (double)(((c.dens_ws * c.g) * mj) * d0);
        b1 -= (double)(((c.dens_ws * c.g) * mj) * d1);
    } else if (c.swalg == 0) {
        b0 += (double)(-((c.g * mj) * d0));
        b1 += (double)(-((c.g * mj) * d1));
    }
}

// Internal acceleration of the coarse-level particles.
template <int SKF, bool WS>
__device__ __forceinline__ void force_big(const PState& A, const Search& Q, const StepScalars* S, const Rheo& c,
                                          bool cross, const PairWork& pw) {
    constexpr int SK = SupportScale<SKF>::value;
    coarse_particles<kBigThreads>(pw.nreg, pw.nbig, pw.tail, [&](int i, int lw) {
        const float pi_ = Q.pterm[i], rhoi = A.rho[i];
        double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0;
        const unsigned char si = WS ? Q.spec[i] : 0;
        coarse_neighbours<SK>(Q, S, i, lw, [&](int j, float4 o, const PairGeom& g) {
            if (WS && Q.spec[j] != si) {  // type 0 only (:6899)
                if (cross) {
                    float w, d0, d1;
                    sph_kernel<SKF>(g.r, g.dx0, g.dx1, g.mh, w, d0, d1);
                    wir_pair_term(c, si == 2, o.w, d0, d1, b0, b1);
                }
                return;
            }
            pressure_pair<SKF>(c, pi_, rhoi, Q.pterm[j], A.rho[j], o.w, g, a0, a1);
        });
        a0 = coarse_sum(a0, lw);
        a1 = coarse_sum(a1, lw);
        if (coarse_first(lw)) Q.indv[i] = make_float2((float)a0, (float)a1);
        if (WS && cross) {
            b0 = coarse_sum(b0, lw);
            b1 = coarse_sum(b1, lw);
            if (coarse_first(lw)) Q.bxy[i] = make_float2((float)b0, (float)b1);
        }
    });
}

// With 4 or 8 lanes a particle a lane has some 6 to 12 entries and the one by
// one rest of a loop over fours is up to half of its chain of loads: there
// the rest goes together, with the registers of fewer resident blocks (the
// few particles leave room).  us with ~6 of the event, k_iforce / k_xsph: 850
// particles 10.6 / 10.5 -> 8.9 / 8.6; a step of 13k 79 -> 75, of 23k 91 -> 88.
// With 1 or 2 lanes occupancy hides the rest and the registers spill (1M
// particles 142 -> 210).  Soil and water with 2 lanes spill 52 B at 4 blocks and
// nothing at 3, a step of 60k 263 and 254 us, but of 120k 334 and 344, of 250k 608
// and 629 (1 lane, 560k: equal).  k_iforce for one material with 2 lanes spills
// 20 B; its warps counted down instead spill nothing and are slower, 200k
// particles 43 and 45 us.
template <int G>
constexpr bool kFewPerLane = G >= 4;
template <int G>
constexpr int kPairBlocks = G == 8 ? 2 : G == 4 ? 3 : 4;

// Internal acceleration of a regular particle over its neighbour table, by G
// lanes: lane gl takes every G-th entry.  Per entry the stored gradient and
// the gathers of (x, m) and the pressure term of the neighbour (its depth too
// with pa_sph 1).  The table is read four entries at a time so that the
// gathers of four pairs are in flight per thread.  The sums over the lanes are
// valid in all of them.
template <int SKF, bool WS, int G>
__device__ __forceinline__ void internal_force(const Search& Q, const Rheo& c, const float* rho, float hmax, int i,
                                               int gl, bool cross, float& in0, float& in1, float2& bxy) {
    const float4 me = __ldg(&Q.xhm[i]);
    const float2 xi = make_float2(me.x, me.y);
    const bool safe = quot_safe(me.z, hmax);
    const float pi_ = __ldg(&Q.pterm[i]), rhoi = rho[i];
    double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0;
    const bool water = WS && Q.spec[i] == 2;
    const int cnt = Q.ncount[i];
    const size_t tab = tab_base(i, Q.kcap);
    // an entry of the particle's own material (type 0, :6899) or, with cross, of the other
    auto term = [&](int e, const TabGrad<SKF>& g, const float4& o, float pj) {
        if (WS && e < 0 && !cross) return;
        float d0, d1;
        g.grad(xi, o, safe, d0, d1);
        if (WS && e < 0) wir_pair_term(c, water, o.w, d0, d1, b0, b1);
        else pressure_terms(c, pi_, rhoi, pj, c.pa_sph == 1 ? rho[e] : 0.f, o.w, d0, d1, a0, a1);
    };
    // four entries at a time, the next four on their way meanwhile
    constexpr bool few = kFewPerLane<G>;  // the last ones, up to three, together as well
    int k = gl;
    int e[4];
    TabGrad<SKF> g[4];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (!few || k0 + u * G < cnt) {
                e[u] = __ldg(Q.nj + tab + (size_t)(k0 + u * G) * kTabStride);
                g[u].load(Q, tab + (size_t)(k0 + u * G) * kTabStride);
            }
    };
    if (few || k + 3 * G < cnt) fetch(k);
    for (; k + 3 * G < cnt; k += 4 * G) {
        int je[4];
        TabGrad<SKF> gg[4];
        float4 o[4];
        float pj[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            je[u] = e[u];
            gg[u] = g[u];
            const int j = WS ? (e[u] & ~kCrossBit) : e[u];
            o[u] = __ldg(&Q.xhm[j]);
            pj[u] = __ldg(&Q.pterm[j]);
        }
        if (few || k + 7 * G < cnt) fetch(k + 4 * G);
#pragma unroll
        for (int u = 0; u < 4; u++) term(je[u], gg[u], o[u], pj[u]);
    }
    if (few) {
        float4 o[3];
        float pj[3];
#pragma unroll
        for (int u = 0; u < 3; u++)
            if (k + u * G < cnt) {
                const int j = WS ? (e[u] & ~kCrossBit) : e[u];
                o[u] = __ldg(&Q.xhm[j]);
                pj[u] = __ldg(&Q.pterm[j]);
            }
#pragma unroll
        for (int u = 0; u < 3; u++)
            if (k + u * G < cnt) term(e[u], g[u], o[u], pj[u]);
    }
    for (; !few && k < cnt; k += G) {
        const int ek = __ldg(Q.nj + tab + (size_t)k * kTabStride), j = WS ? (ek & ~kCrossBit) : ek;
        TabGrad<SKF> gk;
        gk.load(Q, tab + (size_t)k * kTabStride);
        term(ek, gk, __ldg(&Q.xhm[j]), __ldg(&Q.pterm[j]));
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        a0 += __shfl_xor_sync(0xffffffffu, a0, o);
        a1 += __shfl_xor_sync(0xffffffffu, a1, o);
        if (WS && cross) {
            b0 += __shfl_xor_sync(0xffffffffu, b0, o);
            b1 += __shfl_xor_sync(0xffffffffu, b1, o);
        }
    }
    in0 = (float)a0;
    in1 = (float)a1;
    bxy = make_float2((float)b0, (float)b1);
}

// DEM node box touched by the erosion scatter, kept per thread and reduced
// per block before the four atomics on the step scalars (same-address
// atomics from every warp serialise).
struct NodeBox {
    int x0, x1, y0, y1;
};
__device__ __forceinline__ NodeBox empty_node_box() { return NodeBox{INT_MAX, INT_MIN, INT_MAX, INT_MIN}; }

// Every thread of the block must call it (one __syncthreads).
__device__ __forceinline__ void flush_node_box(StepScalars* S, NodeBox b) {
    __shared__ NodeBox wb[32];
    const unsigned full = 0xffffffffu;
    b.x0 = __reduce_min_sync(full, b.x0); b.x1 = __reduce_max_sync(full, b.x1);
    b.y0 = __reduce_min_sync(full, b.y0); b.y1 = __reduce_max_sync(full, b.y1);
    if ((threadIdx.x & 31) == 0) wb[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x == 0) {
        NodeBox t = wb[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) {
            t.x0 = min(t.x0, wb[w].x0); t.x1 = max(t.x1, wb[w].x1);
            t.y0 = min(t.y0, wb[w].y0); t.y1 = max(t.y1, wb[w].y1);
        }
        if (t.x1 >= t.x0) {
            atomicMin(&S->ex0, t.x0); atomicMax(&S->ex1, t.x1);
            atomicMin(&S->ey0, t.y0); atomicMax(&S->ey1, t.y1);
        }
    }
}

// DEM scatter of ExtForces_SW(1) (SPH_SW_2019.f90:8731-8750): the particle
// adds base/dist and 1/dist to the 4x4 DEM nodes around its DEM cell.
// Consecutive particles of the cell-sorted order mostly share a DEM cell, so
// within a warp the lanes form runs of equal DEM cell.  Each lane writes its
// 32 FP32 terms (16 nodes x {base/dist, 1/dist}) to shared memory, and
// add_node_runs sums them.  Lanes with part == false take no part; every lane
// of the warp must call this, in blocks of at most kScatterWarps warps.
__device__ __forceinline__ void erosion_scatter(const DemView& dem, float xx, float xy, float base, bool part,
                                                double2* auxv, NodeBox& box) {
    __shared__ NodeRuns runs[kScatterWarps];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    NodeRuns& R = runs[threadIdx.x >> 5];
    int ipx = 0, ipy = 0, key = -1 - lane;  // non-participants: singleton runs with zero terms
    if (part) {
        ipx = dem_node_x(dem, xx);
        ipy = dem_node_y(dem, xy);
        key = ipy * (dem.nx + 2) + ipx;
    }
    if (!__any_sync(full, part)) return;
    // the 4x4 nodes (ipx-1..ipx+2) x (ipy-1..ipy+2); nodes outside the DEM add zero
    float dx2[4], dy2[4];
#pragma unroll
    for (int o = 0; o < 4; o++) {
        const float ddx = xx - (dem.xmin + (float)(ipx + o - 2) * dem.dx), ddy = xy - (dem.ymin + (float)(ipy + o - 2) * dem.dy);
        dx2[o] = ddx * ddx;
        dy2[o] = ddy * ddy;
    }
#pragma unroll
    for (int o = 0; o < 16; o++) {
        const int ix = ipx + (o >> 2) - 1, iy = ipy + (o & 3) - 1;
        const bool inside = part && ix >= 1 && ix <= dem.nx && iy >= 1 && iy <= dem.ny;
        // max(1e-6, distance); the root is kept off 0
        const float dist = fmaxf(root(fmaxf(dx2[o >> 2] + dy2[o & 3], 1.e-30f)), 1.e-6f);
        const float y = recip(dist);
        R.term[o][lane] = inside ? quot(base, dist, y) : 0.f;
        R.term[16 + o][lane] = inside ? y : 0.f;
    }
    if (part && !quot_fits(base)) {  // beyond quot: an infinite rate, or next to none
#pragma unroll 1
        for (int o = 0; o < 16; o++) {
            const int ix = ipx + (o >> 2) - 1, iy = ipy + (o & 3) - 1;
            const float ddx = xx - (dem.xmin + (float)(ix - 1) * dem.dx), ddy = xy - (dem.ymin + (float)(iy - 1) * dem.dy);
            if (ix >= 1 && ix <= dem.nx && iy >= 1 && iy <= dem.ny)
                R.term[o][lane] = base / fmaxf(sqrtf(ddx * ddx + ddy * ddy), 1.e-6f);
        }
    }
    add_node_runs(R, lane, key, ipx, ipy, dem.nx, dem.ny, auxv);
    if (part) {
        box.x0 = min(box.x0, max(1, ipx - 1)); box.x1 = max(box.x1, min(dem.nx, ipx + 2));
        box.y0 = min(box.y0, max(1, ipy - 1)); box.y1 = max(box.y1, min(dem.ny, ipy + 2));
    }
}

// A particle out of the domain at the start of the step: copied through.
__device__ __forceinline__ void rk_carry(const PState& A, const Rheo& c, const PState& B, float2* velfin, float4* xsv,
                                         int i) {
    B.pos[i] = A.pos[i]; B.vel[i] = A.vel[i]; velfin[i] = A.vel[i];
    xsv[i] = make_float4(A.vel[i].x, A.vel[i].y, A.rho[i], A.mass[i]);
    B.rho[i] = A.rho[i]; B.mass[i] = A.mass[i]; B.hsml[i] = A.hsml[i];
    B.flag[i] = A.flag[i]; B.id[i] = A.id[i];
    if (c.icpwp == 3) B.pwp[i] = 0.f;  // Get_Pwp_SW zeroes out-of-domain particles
    if (c.icpwp == 1) B.pwp[i] = A.pwp[i];  // u of a frozen particle stays
}

// The end of the RK45 body of an active particle: the final update
// (SPH_MAIN_2019.f90:908-922), Check_Out_Domain, Hungr erosion of the mass
// and the DEM scatter of ExtForces_SW(1) (SPH_SW_2019.f90:8717-8760),
// h_upgrade (:2925-2931) and the pore-pressure update, written to B.  h is
// the step's final depth; (xx, xy, vx, vy) the last stage's state, kept as
// the result when the particle left the domain in a stage (out).  Every lane
// of the warp must call it (erosion_scatter).
template <bool GEN = true>
__device__ __forceinline__ void rk_finish(const PState& A, const Search& Q, StepScalars* S, const Rheo& c,
                                          const DemView& dem, const PState& B, float2* velfin, double2* auxv, int i,
                                          float dt, float2 x0, float2 v0, float Dx0, float Dx1, float Dv0, float Dv1,
                                          float xx, float xy, float vx, float vy, bool out, float h, float pwp,
                                          float u0, float Du, float acc0, float acc1, NodeBox& box) {
    float m = A.mass[i];
    float hs = A.hsml[i];
    if (!out) {
        float dt6 = dt / 6.f;
        xx = x0.x + dt6 * Dx0;
        xy = x0.y + dt6 * Dx1;
        vx = v0.x + dt6 * Dv0;
        vy = v0.y + dt6 * Dv1;
        if (c.icpwp == 1) pwp = u0 + dt6 * Du;  // u of icpwp 1 (:921); else pwp is the stage's u
        out = out_of_box(dem, xx, xy);
    }
    float er = 0.f;
    if (!out && c.erosion)
        er = erosion_rate_final<GEN>(c, dem, xx, xy, vx, vy, h, pwp, soil_fraction(c, Q, A, i), acc0, acc1, dt);
    if (c.erosion) erosion_scatter(dem, xx, xy, dt * er, !out, auxv, box);
    if (!out) {
        if (c.erosion) m = m + ((dt * er) * m) / h;
        if (c.sle == 1) hs = 2.f * sqrtf(m / h);
    }
    B.pos[i] = make_float2(xx, xy);
    velfin[i] = make_float2(vx, vy);
    Q.xsv[i] = make_float4(vx, vy, h, m);
    B.vel[i] = make_float2(vx, vy);
    B.rho[i] = h;
    B.mass[i] = m;
    B.hsml[i] = hs;
    B.flag[i] = out ? 1 : 0;
    B.id[i] = A.id[i];
    if (c.icpwp == 3) B.pwp[i] = out ? 0.f : pwp_update(c, pwp, h, h - Q.rho0[i], dt);
    if (c.icpwp == 1) {  // bounded by the depth after ExtForces_SW(1), RK45 :974-979
        if (!out) {
            if (pwp > h) pwp = h;
            if (pwp < 0.f) pwp = 0.f;
        }
        B.pwp[i] = pwp;
    }
}

// Internal acceleration: the coarse-level particles in their own blocks, the
// regular ones, G lanes each, in the others.  The
// warps take the particles from the last to the first: the neighbour search
// has just written the table front to back, so its last-written part (still
// in L2) is read first, and av_vel, which walks the table front to back after
// this pass, starts on the part this pass read last.
// cross (soil and water, first stage): also the sums over the soil-water
// pairs, from the same walk.
template <int SKF, bool WS, int G>
__global__ void __launch_bounds__(kBigThreads, kPairBlocks<G>) k_iforce(PState A, Search Q, StepScalars* S, Rheo c, int n, int cross) {
    PDL_ENTRY();
    const PairWork pw(S);
    if (pw.skip) return;
    if (pw.coarse()) {
        force_big<SKF, WS>(A, Q, S, c, cross != 0, pw);
        return;
    }
    constexpr int P = 32 / G;  // particles per warp
    const int nreg = pw.nreg;
    const float hmax = o2f(S->hmax_o);
    const int nw = (nreg + P - 1) / P;
    const int lane = threadIdx.x & 31, bid = blockIdx.x - kBigBlocks, nb = pw.tail - kBigBlocks;
    for (int w = (bid * kBigThreads + threadIdx.x) >> 5; w < nw; w += (nb * kBigThreads) >> 5) {
        const int i = (nw - 1 - w) * P + lane / G;
        if (G == 1) {
            const int rows = __reduce_max_sync(0xffffffffu, Q.ncount[min(i, nreg - 1)]);
            const size_t at = tab_base(i - lane, Q.kcap);
            if (lane == 0 && rows <= Q.kcap) prefetch_rows(Q.nj + at, rows);
            if (lane == 1 && rows <= Q.kcap) prefetch_rows(Q.ng + (SKF == 1 ? at : 2 * at), SKF == 1 ? rows : 2 * rows);
        }
        float in0, in1;
        float2 b;
        internal_force<SKF, WS, G>(Q, c, A.rho, hmax, min(i, nreg - 1), lane % G, cross != 0, in0, in1, b);
        if (i < nreg && lane % G == 0) {
            Q.indv[i] = make_float2(in0, in1);
            if (WS && cross) Q.bxy[i] = b;
        }
    }
}

// The RK45 body for each active particle, entirely in registers: the
// internal acceleration (stage-invariant, see below; from k_iforce), four stages of
// x = x0 + c_i dt v, v = v0 + c_i dt (ex + in) with ExtForces_SW(0) at each
// stage (SPH_MAIN_2019.f90:808-906), the final update (:908-922), the
// out-of-domain freeze (Check_Out_Domain), Hungr erosion of mass and the DEM
// scatter of ExtForces_SW(1) (:8717-8760), and h_upgrade (:2925-2931).
//
// Why the internal force is computed once: with summation density the stage
// density depends only on masses, hsml and the frozen W_ij, none of which
// change inside the step, so IntForces_SW returns the same value in all four
// stages.  (A particle that leaves the DEM box mid-step is frozen; the
// reference then keeps scattering its stale pressure into its neighbours for
// the remaining stages, which is not reproduced.)
// PWP1 (icpwp = 1) carries u through the stages; GEN compiles every basal
// law and erosion law (else only nfric 4-8, 26, 27 and erosion law 1).  The
// other runs are compiled without them, so their stage loop keeps its
// registers and its code small.
template <bool PWP1, bool GEN>
__global__ void __launch_bounds__(128, 6) k_force_rk(PState A, Search Q, StepScalars* S, Rheo c, DemView dem, int n,
                                                   PState B, float2* velfin, double2* auxv, int forces_only,
                                                   float2* indv_out) {
    PDL_ENTRY();
    if (S->skip) return;
    const int nact = S->nactive;
    const float dt = S->dt_step;
    if (forces_only) {
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nact; i += gridDim.x * blockDim.x)
            indv_out[i] = Q.indv[i];
        return;
    }
    // block-uniform trip count: every lane of a warp reaches erosion_scatter,
    // every thread the box flush
    NodeBox box = empty_node_box();
    for (int i0 = blockIdx.x * blockDim.x; i0 < n; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + threadIdx.x;
        if (i >= n) {
            if (c.erosion) erosion_scatter(dem, 0.f, 0.f, 0.f, false, auxv, box);
            continue;
        }
        if (i >= nact) {  // carried particles (out of the domain at step start)
            rk_carry(A, c, B, velfin, Q.xsv, i);
            if (c.erosion) erosion_scatter(dem, 0.f, 0.f, 0.f, false, auxv, box);
            continue;
        }
        const float2 fin = Q.indv[i];
        const float in0 = fin.x, in1 = fin.y;
        const float h = A.rho[i];
        const float hc = (h < c.h_inf) ? c.h_inf : h;  // IntForces_SW clamp, seen by ExtForces_SW(0)
        const float2 x0 = A.pos[i], v0 = A.vel[i];
        // icpwp 3: Uaux(1) of the step start; icpwp 1: u0, then u of each stage
        const float u0 = (c.icpwp != 0) ? A.pwp[i] : 0.f;
        float pwp = u0, du = 0.f, Du = 0.f;
        const float nsoil = soil_fraction(c, Q, A, i);
        float xx = x0.x, xy = x0.y, vx = v0.x, vy = v0.y;
        float ex0 = 0.f, ex1 = 0.f;
        float Dx0 = 0.f, Dx1 = 0.f, Dv0 = 0.f, Dv1 = 0.f;
        bool out = false;
#pragma unroll 1  // one copy of ExtForces_SW(0): the unrolled body overflows the instruction cache
        for (int s = 0; s < 4; s++) {
            const float f1 = (s == 0) ? 0.f : (s == 3 ? 1.f : 0.5f);
            const float f2 = (s == 0 || s == 3) ? 1.f : 2.f;
            if (!out) {
                float fdt = f1 * dt;
                float nxx = x0.x + fdt * vx;
                float nxy = x0.y + fdt * vy;
                float nvx = v0.x + fdt * (ex0 + in0);
                float nvy = v0.y + fdt * (ex1 + in1);
                xx = nxx; xy = nxy; vx = nvx; vy = nvy;
                if (PWP1) {  // RK45 :823-830, bounded by the depth as the stage finds it
                    pwp = u0 + fdt * du;
                    const float rc = (s == 0) ? Q.rho0[i] : hc;
                    if (pwp > rc) pwp = rc;
                    else if (pwp < 0.f) pwp = 0.f;
                }
                if (out_of_box(dem, xx, xy)) {
                    out = true;
                } else {
                    ext_accel<false, GEN>(c, dem, dt, xx, xy, vx, vy, hc, pwp, nsoil, in0, in1, ex0, ex1);
                    if (PWP1) {
                        du = pwp1_rate(c, hc, pwp, dt);
                        Du = Du + f2 * du;
                    }
                    Dv0 = Dv0 + f2 * (ex0 + in0);
                    Dv1 = Dv1 + f2 * (ex1 + in1);
                    Dx0 = Dx0 + f2 * vx;
                    Dx1 = Dx1 + f2 * vy;
                }
            }
        }
        rk_finish<GEN>(A, Q, S, c, dem, B, velfin, auxv, i, dt, x0, v0, Dx0, Dx1, Dv0, Dv1, xx, xy, vx, vy, out, h, pwp,
                       u0, Du, GEN ? ex0 + in0 : 0.f, GEN ? ex1 + in1 : 0.f, box);
    }
    if (c.erosion) flush_node_box(S, box);
}

// ---------------------------------------------------------------- staged RK45
// With nor_density or ic_cosTheta = 1 the pressure changes from stage to
// stage: each sum_density_Tools call divides the plain sum by
// sum_j (m_j/h_j) W_ij taken with the depths of the call before it
// (My_SPH_Tools_2019.f90:1790-1846), and ic_cosTheta = 1 takes g/deng at each
// stage's position (IntForces_SW :6775-6783).  The step then runs stage by
// stage.  The five depths of the step (four stages and the sum after the
// final update) depend only on the frozen W_ij, the masses and the depths
// before them, so they are computed first (k_norm); then each stage runs the
// internal force over the neighbour table with that stage's pressure term
// and the RK stage of every particle (k_stage), whose state is carried in
// HBM between the launches; the last stage also finishes the step
// (k_stage_final).  The pressure term of stage s+1 is written by stage s,
// once the particle's stage position is known.

// RK45 state carried between the stage launches (slot order).
struct StageCarry {
    float2* v;    // velocity of the last stage
    float2* acc;  // ex + in of the last stage
    float2* dx;   // Dx_RK
    float2* dv;   // Dvx_RK
    float2* xo;   // stage position of a particle that left the DEM box
    int* out;     // 1 once it has (it is frozen for the rest of the step)
    // icpwp = 1: u of the last stage (kept by a particle that left), its
    // rate du and Du_RK
    float* u;
    float* du;
    float* Du;
};

// The stage value of icpwp 1's u (RK45 :823-830): u0 + f1 dt du of the
// previous stage, bounded by the depth that stage left (the step start's,
// after Adaptive_dt's clamp, in stage 0; else IntForces_SW's clamp to h_inf).
__device__ __forceinline__ float pwp1_stage(const Rheo& c, const PState& A, const Search& Q, const StageCarry& C,
                                            int s, int i, float fdt, const float* hprev) {
    float u = A.pwp[i] + fdt * ((s > 0) ? C.du[i] : 0.f);
    float rc = Q.rho0[i];
    if (s > 0) {
        rc = hprev[i];
        if (rc < c.h_inf) rc = c.h_inf;
    }
    if (u > rc) u = rc;
    else if (u < 0.f) u = 0.f;
    C.u[i] = u;
    return u;
}

// Its rate of this stage and the running Du_RK.
__device__ __forceinline__ void pwp1_accumulate(const Rheo& c, const StageCarry& C, int s, int i, float hc, float u,
                                                float dt, float f2) {
    const float du = pwp1_rate(c, hc, u, dt);
    C.du[i] = du;
    C.Du[i] = ((s > 0) ? C.Du[i] : 0.f) + f2 * du;
}

// Depth of the previous sum_density_Tools call as the next one reads it:
// clamped to h_inf when IntForces_SW (:6769) has run in between.
__device__ __forceinline__ float prev_depth(const Rheo& c, const float* hp, int j, int clamp_prev) {
    float h = __ldg(hp + j);
    return (clamp_prev && h < c.h_inf) ? c.h_inf : h;
}
// The end of a normalised sum for particle i: its depth, and m/h as the next
// call gathers it (IntForces_SW has clamped the depth by then).
__device__ __forceinline__ void norm_store(const PState& A, const Rheo& c, int i, float mass, double den, float* hout,
                                           float* next) {
    const float h = A.rho[i] / (float)den;
    hout[i] = h;
    next[i] = mass / ((h < c.h_inf) ? c.h_inf : h);
}

// A normalised sum of the coarse-level particles.
template <int SKF>
__device__ __forceinline__ void norm_big(const PState& A, const Search& Q, const StepScalars* S, const Rheo& c,
                                         const float* hp, int clamp_prev, float* hout, const float* ratio,
                                         float* next, const PairWork& pw) {
    constexpr int SK = SupportScale<SKF>::value;
    coarse_particles<kBigThreads>(pw.nreg, pw.nbig, pw.tail, [&](int i, int lw) {
        double den = 0.0;
        coarse_neighbours<SK>(Q, S, i, lw, [&](int j, float4 o, const PairGeom& g) {
            den += (double)(__ldg(ratio + j) * sph_kernel_w<SKF>(g.r, g.mh));
        });
        den = coarse_sum(den, lw);
        if (coarse_first(lw)) {
            const float4 me = Q.xhm[i];
            den = (double)((sph_kernel_w<SKF>(0.f, me.z) * me.w) / prev_depth(c, hp, i, clamp_prev)) + den;
            norm_store(A, c, i, me.w, den, hout, next);
        }
    });
}

// One normalised sum_density_Tools call: h_i = num_i / (W(0,h_i) m_i/hp_i +
// sum_j (m_j/hp_j) W_ij), num_i the plain sum of k_density (in A.rho), hp the
// previous call's depths; m_j/hp_j is gathered as the quotient that call left
// (one division per particle instead of one per pair: 23 -> 9 us a call for
// 60k particles, with four lanes a particle).  The coarse-level particles in
// their own blocks, the regular ones over the table in the others.
template <int SKF, int G>
__global__ void __launch_bounds__(kBigThreads, 5) k_norm(PState A, Search Q, StepScalars* S, Rheo c, int n, const float* hp,
                                                      int clamp_prev, float* hout, const float* ratio, float* next) {
    PDL_ENTRY();
    const PairWork pw(S);
    if (pw.skip) return;
    const int nreg = pw.nreg;
    if (pw.coarse()) {
        norm_big<SKF>(A, Q, S, c, hp, clamp_prev, hout, ratio, next, pw);
        return;
    }
    constexpr int P = 32 / G;  // particles per warp
    const int lane = threadIdx.x & 31, gl = lane % G, bid = blockIdx.x - kBigBlocks, nb = pw.tail - kBigBlocks;
    const int nw = (nreg + P - 1) / P;
    for (int wp = (bid * kBigThreads + threadIdx.x) >> 5; wp < nw; wp += (nb * kBigThreads) >> 5) {
        const int i0 = wp * P + lane / G, i = min(i0, nreg - 1);
        const int cnt = Q.ncount[i];
        const size_t tab = tab_base(i, Q.kcap);
        double den = 0.0;
        int k = gl;
        for (; k + 3 * G < cnt; k += 4 * G) {
            int e[4];
            float w[4], q[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                e[u] = __ldg(Q.nj + tab + (size_t)(k + u * G) * kTabStride);
                w[u] = __ldg(Q.nw + tab + (size_t)(k + u * G) * kTabStride);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) q[u] = __ldg(ratio + e[u]);
#pragma unroll
            for (int u = 0; u < 4; u++) den += (double)(q[u] * w[u]);
        }
        for (; k < cnt; k += G)
            den += (double)(__ldg(ratio + __ldg(Q.nj + tab + (size_t)k * kTabStride)) *
                            __ldg(Q.nw + tab + (size_t)k * kTabStride));
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
        if (i0 < nreg && gl == 0) {
            const float4 me = Q.xhm[i];
            den = (double)((sph_kernel_w<SKF>(0.f, me.z) * me.w) / prev_depth(c, hp, i, clamp_prev)) + den;
            norm_store(A, c, i, me.w, den, hout, next);
        }
    }
}

// Pressure term of IntForces_SW for depth h at (xx, yy): h clamped to h_inf
// (:6769), p = (g_z/2) h^2 (:6797) with g_z = g/deng there when COS
// (:6775-6783); p/h^2 for pa_sph 2, p for pa_sph 1.
template <bool COS>
__device__ __forceinline__ float stage_pterm(const Rheo& c, const DemView& dem, float h, float xx, float yy) {
    const float hc = (h < c.h_inf) ? c.h_inf : h;
    float cg05 = c.cgra05;
    if (COS) {
        float zpx, zpy, top[6];
        dem_lookup(dem, xx, yy, zpx, zpy, false, top);
        cg05 = 0.5f * (c.g / terrain_deng(zpx, zpy));
    }
    const float p = (cg05 * hc) * hc;
    return (c.pa_sph == 1) ? p : p / (hc * hc);
}

// Pressure term of the first stage (positions of the step start).
template <bool COS>
__global__ void __launch_bounds__(128) k_stage_begin(PState A, Search Q, StepScalars* S, Rheo c, DemView dem,
                                                     const float* h1) {
    PDL_ENTRY();
    if (S->skip) return;
    const int nact = S->nactive;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nact; i += gridDim.x * blockDim.x) {
        const float2 p = A.pos[i];
        Q.pterm[i] = stage_pterm<COS>(c, dem, h1[i], p.x, p.y);
    }
}

// ---------------------------------------------------- soil and water (ic_ws_Interact = 1)
// Position of an active particle in RK45 stage s (s = 0: the step start; a
// frozen particle has none).  The same arithmetic as k_stage's.
__device__ __forceinline__ bool wir_stage_pos(const PState& A, const StageCarry& C, int s, float dt, int i,
                                              float2& p) {
    if (s == 0) {
        p = A.pos[i];
        return true;
    }
    if (C.out[i]) return false;
    const float f1 = (s == 3) ? 1.f : 0.5f;
    const float2 x0 = A.pos[i], vp = C.v[i];
    const float fdt = f1 * dt;
    p = make_float2(x0.x + fdt * vp.x, x0.y + fdt * vp.y);
    return true;
}

// Get_hs_at_w_SW (SPH_SW_2019.f90:17789-17857): each soil particle's depth
// spread over the 4 x 4 DEM nodes around it with weights 1/max(1e-6, dist),
// summed in FP64.
__global__ void __launch_bounds__(128) k_wir_scatter(PState A, Search Q, StepScalars* S, Rheo c, DemView dem,
                                                     StageCarry C, int s, const float* hdep, double2* acc) {
    PDL_ENTRY();
    if (S->skip) return;
    const int nact = S->nactive;
    const float dt = S->dt_step;
    // the same terms h/dist and 1/dist as the erosion scatter, combined over
    // runs of lanes with equal DEM cells before one FP64 atomic per run;
    // block-uniform trip count: every lane of a warp reaches the scatter
    NodeBox box = empty_node_box();
    for (int i0 = blockIdx.x * blockDim.x; i0 < nact; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + threadIdx.x;
        float2 p = make_float2(0.f, 0.f);
        float h = 0.f;
        bool part = false;
        if (i < nact && Q.spec[i] == 1 && wir_stage_pos(A, C, s, dt, i, p) && !out_of_box(dem, p.x, p.y)) {
            h = hdep[i];
            part = true;
        }
        erosion_scatter(dem, p.x, p.y, h, part, acc, box);
    }
}

// Z + hs at the DEM nodes (:17861-17867); the accumulators are left zeroed
// for the next stage.
__global__ void k_wir_nodes(double2* acc, const float* z, float* hsz, int np, const StepScalars* S) {
    PDL_ENTRY();
    if (S->skip) return;
    for (int ip = blockIdx.x * blockDim.x + threadIdx.x; ip < np; ip += gridDim.x * blockDim.x) {
        const double2 a = acc[ip];
        hsz[ip] = (a.y > (double)1.e-6f) ? z[ip] + (float)(a.x / a.y) : z[ip];
        acc[ip] = make_double2(0.0, 0.0);
    }
}

// Per active particle in stage s: at a water particle Z + hs of the soil
// and its gradient, bilinear on its DEM cell (:17869-17933; a particle on the
// far edge of the DEM takes the last cell); then the pressure term of the
// stage (IntForces_SW :6793-6828): g/2 (h^2 - Zp^2) for the water with
// ic_SWalg = 1, g/2 h^2 otherwise, h clamped to h_inf.
__global__ void __launch_bounds__(128) k_wir_press(PState A, Search Q, StepScalars* S, Rheo c, DemView dem,
                                                   StageCarry C, int s, const float* hdep, const float* hsz) {
    PDL_ENTRY();
    if (S->skip) return;
    const int nact = S->nactive;
    const float dt = S->dt_step;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nact; i += gridDim.x * blockDim.x) {
        const bool water = Q.spec[i] == 2;
        float2 p;
        if (!wir_stage_pos(A, C, s, dt, i, p) || out_of_box(dem, p.x, p.y)) continue;  // keeps its term
        float zp = 0.f;
        if (water) {
            const int ipx = min(max(dem_node_x(dem, p.x), 1), dem.nx - 1);
            const int ipy = min(max(dem_node_y(dem, p.y), 1), dem.ny - 1);
            const int n1 = (ipy - 1) * dem.nx + (ipx - 1), n2 = n1 + 1, n3 = n1 + 1 + dem.nx, n4 = n3 - 1;
            const float xref = dem.xmin + (float)(ipx - 1) * dem.dx, yref = dem.ymin + (float)(ipy - 1) * dem.dy;
            const float xi = quot(p.x - xref, dem.dx, dem.rdx), eta = quot(p.y - yref, dem.dy, dem.rdy);
            const float sh1 = (1.f - xi) * (1.f - eta), sh2 = xi * (1.f - eta), sh3 = xi * eta, sh4 = (1.f - xi) * eta;
            const float d1x = (-1.f + eta) / dem.dx, d2x = (1.f - eta) / dem.dx, d3x = eta / dem.dx, d4x = (-eta) / dem.dx;
            const float d1y = (-1.f + xi) / dem.dy, d2y = (-xi) / dem.dy, d3y = xi / dem.dy, d4y = (1.f - xi) / dem.dy;
            const float h1 = hsz[n1], h2 = hsz[n2], h3 = hsz[n3], h4 = hsz[n4];
            zp = ((sh1 * h1 + sh2 * h2) + sh3 * h3) + sh4 * h4;
            Q.zpw[i] = zp;
            Q.gzw[i] = make_float2(((h1 * d1x + h2 * d2x) + h3 * d3x) + h4 * d4x,
                                   ((h1 * d1y + h2 * d2y) + h3 * d3y) + h4 * d4y);
        }
        const float h = hdep[i];
        const float hc = (h < c.h_inf) ? c.h_inf : h;
        const float p_ = (water && c.swalg == 1) ? c.cgra05 * (hc * hc - zp * zp) : (c.cgra05 * hc) * hc;
        Q.pterm[i] = (c.pa_sph == 1) ? p_ : p_ / (hc * hc);
    }
}

// RK45 stage s = 0, 1, 2 of every active particle (SPH_MAIN_2019.f90:808-906):
// x = x0 + c_s dt v, v = v0 + c_s dt (ex + in), the out-of-domain check,
// ExtForces_SW(0) with the stage depth hs_ (clamped as IntForces_SW leaves
// it) and the internal acceleration of this stage, the Dx/Dv sums; then the
// pressure term of stage s+1 at its position with depth hnext.  A particle
// that will leave the domain in stage s+1 keeps its old term, as IntForces_SW
// skips it.
template <bool COS>
__global__ void __launch_bounds__(128) k_stage(PState A, Search Q, StepScalars* S, Rheo c, DemView dem,
                                               StageCarry C, int s, const float* hs_, const float* hnext,
                                               const float* hprev) {
    PDL_ENTRY();
    if (S->skip) return;
    const int nact = S->nactive;
    const float dt = S->dt_step;
    const float f1 = (s == 0) ? 0.f : 0.5f, f2 = (s == 0) ? 1.f : 2.f;
    const float f1n = (s == 2) ? 1.f : 0.5f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nact; i += gridDim.x * blockDim.x) {
        if (s > 0 && C.out[i]) continue;  // frozen: its pressure term stays
        const float2 x0 = A.pos[i], v0 = A.vel[i];
        float2 vp = v0, ap = make_float2(0.f, 0.f), dx = make_float2(0.f, 0.f), dv = make_float2(0.f, 0.f);
        if (s > 0) { vp = C.v[i]; ap = C.acc[i]; dx = C.dx[i]; dv = C.dv[i]; }
        const float fdt = f1 * dt;
        const float xx = x0.x + fdt * vp.x, xy = x0.y + fdt * vp.y;
        const float vx = v0.x + fdt * ap.x, vy = v0.y + fdt * ap.y;
        const float u1 = (c.icpwp == 1) ? pwp1_stage(c, A, Q, C, s, i, fdt, hprev) : 0.f;
        if (out_of_box(dem, xx, xy)) {
            C.out[i] = 1;
            C.xo[i] = make_float2(xx, xy);
            C.v[i] = make_float2(vx, vy);
            continue;
        }
        if (s == 0) C.out[i] = 0;
        const float h = hs_[i];
        const float hc = (h < c.h_inf) ? c.h_inf : h;
        const float2 fin = Q.indv[i];
        const float pwp = (c.icpwp == 3) ? A.pwp[i] : u1;
        float ex0, ex1;
        if (c.ws)
            ext_accel_wir(c, dem, dt, xx, xy, vx, vy, hc, fin.x, fin.y, Q.spec[i] == 2, Q.zpw[i], Q.gzw[i], Q.bxy[i],
                          ex0, ex1);
        else
            ext_accel<COS>(c, dem, dt, xx, xy, vx, vy, hc, pwp, soil_fraction(c, Q, A, i), fin.x, fin.y, ex0, ex1);
        if (c.icpwp == 1) pwp1_accumulate(c, C, s, i, hc, u1, dt, f2);
        const float a0 = ex0 + fin.x, a1 = ex1 + fin.y;
        dv.x = dv.x + f2 * a0;
        dv.y = dv.y + f2 * a1;
        dx.x = dx.x + f2 * vx;
        dx.y = dx.y + f2 * vy;
        C.v[i] = make_float2(vx, vy);
        C.acc[i] = make_float2(a0, a1);
        C.dx[i] = dx;
        C.dv[i] = dv;
        if (c.ws) continue;  // the next stage's pressure needs its soil surface: k_wir_press
        const float fdn = f1n * dt;
        const float nx_ = x0.x + fdn * vx, ny_ = x0.y + fdn * vy;
        if (!out_of_box(dem, nx_, ny_)) Q.pterm[i] = stage_pterm<COS>(c, dem, hnext[i], nx_, ny_);
    }
}

// The last stage (s = 3) and the end of the step (rk_finish) with the final
// depth hfin.
template <bool COS>
__global__ void __launch_bounds__(128) k_stage_final(PState A, Search Q, StepScalars* S, Rheo c, DemView dem, int n,
                                                     PState B, float2* velfin, double2* auxv, StageCarry C,
                                                     const float* h4, const float* hfin, const float* h3) {
    PDL_ENTRY();
    if (S->skip) return;
    const int nact = S->nactive;
    const float dt = S->dt_step;
    // block-uniform trip count: every lane of a warp reaches erosion_scatter,
    // every thread the box flush
    NodeBox box = empty_node_box();
    for (int i0 = blockIdx.x * blockDim.x; i0 < n; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + threadIdx.x;
        if (i >= n) {
            if (c.erosion) erosion_scatter(dem, 0.f, 0.f, 0.f, false, auxv, box);
            continue;
        }
        if (i >= nact) {
            rk_carry(A, c, B, velfin, Q.xsv, i);
            if (c.erosion) erosion_scatter(dem, 0.f, 0.f, 0.f, false, auxv, box);
            continue;
        }
        const float2 x0 = A.pos[i], v0 = A.vel[i];
        float pwp = (c.icpwp == 3) ? A.pwp[i] : 0.f;
        bool out = C.out[i] != 0;
        float xx, xy, vx, vy;
        float2 dx = make_float2(0.f, 0.f), dv = make_float2(0.f, 0.f);
        float2 acc = make_float2(0.f, 0.f);  // ex + in of the last stage
        if (out) {
            const float2 xo = C.xo[i], vo = C.v[i];
            xx = xo.x; xy = xo.y; vx = vo.x; vy = vo.y;
            if (c.icpwp == 1) pwp = C.u[i];  // u of the stage it left in
        } else {
            const float2 vp = C.v[i], ap = C.acc[i];
            dx = C.dx[i];
            dv = C.dv[i];
            const float fdt = 1.f * dt;
            xx = x0.x + fdt * vp.x; xy = x0.y + fdt * vp.y;
            vx = v0.x + fdt * ap.x; vy = v0.y + fdt * ap.y;
            if (c.icpwp == 1) pwp = pwp1_stage(c, A, Q, C, 3, i, fdt, h3);
            if (out_of_box(dem, xx, xy)) {
                out = true;
            } else {
                const float h = h4[i];
                const float hc = (h < c.h_inf) ? c.h_inf : h;
                const float2 fin = Q.indv[i];
                float ex0, ex1;
                if (c.ws)
                    ext_accel_wir(c, dem, dt, xx, xy, vx, vy, hc, fin.x, fin.y, Q.spec[i] == 2, Q.zpw[i], Q.gzw[i],
                                  Q.bxy[i], ex0, ex1);
                else
                    ext_accel<COS>(c, dem, dt, xx, xy, vx, vy, hc, pwp, soil_fraction(c, Q, A, i), fin.x, fin.y,
                                   ex0, ex1);
                if (c.icpwp == 1) pwp1_accumulate(c, C, 3, i, hc, pwp, dt, 1.f);
                acc = make_float2(ex0 + fin.x, ex1 + fin.y);
                dv.x = dv.x + 1.f * acc.x;
                dv.y = dv.y + 1.f * acc.y;
                dx.x = dx.x + 1.f * vx;
                dx.y = dx.y + 1.f * vy;
            }
        }
        const float u0 = (c.icpwp == 1) ? A.pwp[i] : 0.f;
        const float Du = (c.icpwp == 1 && !out) ? C.Du[i] : 0.f;
        rk_finish(A, Q, S, c, dem, B, velfin, auxv, i, dt, x0, v0, dx.x, dx.y, dv.x, dv.y, xx, xy, vx, vy, out,
                  hfin[i], pwp, u0, Du, acc.x, acc.y, box);
    }
    if (c.erosion) flush_node_box(S, box);
}

// One pair term of av_vel (SPH_MAIN_2019.f90:3072-3080) for particle i with
// the pair's kernel value w.
__device__ __forceinline__ void xsph_terms(float2 vi, float rhoi, float2 vj, float rhoj, float mj, float w, double& a0,
                                           double& a1) {
    const float den = rhoi + rhoj;
    const float n0 = (2.f * mj) * (vi.x - vj.x), n1 = (2.f * mj) * (vi.y - vj.y);
    float q0, q1;
    quot2_in(n0, n1, den, q0, q1);
    a0 -= (double)(q0 * w);
    a1 -= (double)(q1 * w);
}

// The same with the pair geometry: the kernel value evaluated here.
template <int SKF>
__device__ __forceinline__ void xsph_pair(float2 vi, float rhoi, float2 vj, float rhoj, float mj, const PairGeom& g,
                                          double& a0, double& a1) {
    xsph_terms(vi, rhoi, vj, rhoj, mj, sph_kernel_w<SKF>(g.r, g.mh), a0, a1);
}

// av_vel (SPH_MAIN_2019.f90:3042-3099) with the start-of-step W_ij, then
// v += 0.3*av for particles still inside the domain (:987-993); the coarse
// particles in their own blocks, the regular ones, G lanes each as in k_iforce,
// in the others.
template <int SKF, bool WS>
__device__ __forceinline__ void xsph_big(const Search& Q, const StepScalars* S, const PState& B, const PairWork& pw) {
    constexpr int SK = SupportScale<SKF>::value;
    coarse_particles<kBigThreads>(pw.nreg, pw.nbig, pw.tail, [&](int i, int lw) {
        if (B.flag[i]) return;  // uniform over the warps that share i
        const float4 si = Q.xsv[i];
        const float2 vi = make_float2(si.x, si.y);
        const float rhoi = si.z;
        double a0 = 0.0, a1 = 0.0;
        const unsigned char own = WS ? Q.spec[i] : 0;
        coarse_neighbours<SK>(Q, S, i, lw, [&](int j, float4 o, const PairGeom& g) {
            if (WS && Q.spec[j] != own) return;  // type 0 only (SPH_MAIN_2019.f90:3071)
            const float4 sj = Q.xsv[j];
            xsph_pair<SKF>(vi, rhoi, make_float2(sj.x, sj.y), sj.z, sj.w, g, a0, a1);
        });
        a0 = coarse_sum(a0, lw);
        a1 = coarse_sum(a1, lw);
        if (coarse_first(lw)) {
            const float av0 = 0.3f * (float)a0, av1 = 0.3f * (float)a1;
            B.vel[i] = make_float2(vi.x + av0, vi.y + av1);
        }
    });
}

template <int SKF, bool WS, int G>
__global__ void __launch_bounds__(kBigThreads, kPairBlocks<G>) k_xsph(PState A, Search Q, StepScalars* S, Rheo c, int n, PState B) {
    PDL_ENTRY();
    const PairWork pw(S);
    if (pw.skip || !c.av_vel) return;
    if (pw.coarse()) {
        xsph_big<SKF, WS>(Q, S, B, pw);
        return;
    }
    constexpr int P = 32 / G;     // particles per warp
    constexpr bool few = kFewPerLane<G>;
    const int nreg = pw.nreg;
    const int lane = threadIdx.x & 31, gl = lane % G, bid = blockIdx.x - kBigBlocks, nb = pw.tail - kBigBlocks;
    const int nw = (nreg + P - 1) / P;
    for (int wp = (bid * kBigThreads + threadIdx.x) >> 5; wp < nw; wp += (nb * kBigThreads) >> 5) {
        const int i0 = wp * P + lane / G, i = min(i0, nreg - 1);
        const float4 si = Q.xsv[i];
        const float2 vi = make_float2(si.x, si.y);
        const float rhoi = si.z;
        const bool go = i0 < nreg && !B.flag[i];
        const int cnt = go ? Q.ncount[i] : 0;
        const size_t tab = tab_base(i, Q.kcap);
        if (G == 1) {
            const int rows = __reduce_max_sync(0xffffffffu, cnt);
            const size_t at = tab_base(i0 - lane, Q.kcap);
            if (lane == 0) prefetch_rows(Q.nj + at, rows);
            if (lane == 1) prefetch_rows(Q.nw + at, rows);
        }
        double a0 = 0.0, a1 = 0.0;
        int k = gl;
        int e[4];
        float w[4];
        auto fetch = [&](int k0) {
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (!few || k0 + u * G < cnt) {
                    e[u] = __ldcs(Q.nj + tab + (size_t)(k0 + u * G) * kTabStride);
                    w[u] = __ldcs(Q.nw + tab + (size_t)(k0 + u * G) * kTabStride);
                }
        };
        if (few || k + 3 * G < cnt) fetch(k);
        for (; k + 3 * G < cnt; k += 4 * G) {
            int je[4];
            float ww[4];
            float4 sj[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                je[u] = e[u];
                ww[u] = w[u];
                sj[u] = Q.xsv[WS ? (e[u] & ~kCrossBit) : e[u]];
            }
            if (few || k + 7 * G < cnt) fetch(k + 4 * G);
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (!WS || je[u] >= 0)  // type 0 only (SPH_MAIN_2019.f90:3071)
                    xsph_terms(vi, rhoi, make_float2(sj[u].x, sj[u].y), sj[u].z, sj[u].w, ww[u], a0, a1);
        }
        if (few) {
            float4 sj[3];
#pragma unroll
            for (int u = 0; u < 3; u++)
                if (k + u * G < cnt) sj[u] = Q.xsv[WS ? (e[u] & ~kCrossBit) : e[u]];
#pragma unroll
            for (int u = 0; u < 3; u++)
                if (k + u * G < cnt && (!WS || e[u] >= 0))
                    xsph_terms(vi, rhoi, make_float2(sj[u].x, sj[u].y), sj[u].z, sj[u].w, w[u], a0, a1);
        }
        for (; !few && k < cnt; k += G) {
            const int e = __ldcs(Q.nj + tab + (size_t)k * kTabStride);
            const float w = __ldcs(Q.nw + tab + (size_t)k * kTabStride);
            const float4 sj = Q.xsv[WS ? (e & ~kCrossBit) : e];
            if (!WS || e >= 0) xsph_terms(vi, rhoi, make_float2(sj.x, sj.y), sj.z, sj.w, w, a0, a1);
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
            a0 += __shfl_xor_sync(0xffffffffu, a0, o);
            a1 += __shfl_xor_sync(0xffffffffu, a1, o);
        }
        const float av0 = 0.3f * (float)a0, av1 = 0.3f * (float)a1;
        if (go && gl == 0) B.vel[i] = make_float2(vi.x + av0, vi.y + av1);
    }
}

// DEM update of ExtForces_SW(1) (SPH_SW_2019.f90:8795-8807) over the node box
// touched this step; resets the scatter accumulators.

// DEM update over the touched node box, grid-stride.
__device__ __forceinline__ void erode_box(double2* auxv, float* z, float* eroded, float* avail, int nx, int x0, int x1,
                                          int y0, int y1) {
    int w = x1 - x0 + 1, hgt = y1 - y0 + 1;
    long long tot = (long long)w * hgt;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < tot; k += (long long)gridDim.x * blockDim.x) {
        int ix = x0 + (int)(k % w), iy = y0 + (int)(k / w);
        int ip = (iy - 1) * nx + (ix - 1);
        double2 a = auxv[ip];
        if ((float)a.y > 1.e-6f) {
            float xnum = (float)(a.x / a.y);
            float av = avail[ip];
            if (xnum > av) xnum = av;
            if (av > 0.f) {
                eroded[ip] = eroded[ip] + xnum;
                z[ip] = z[ip] - xnum;
                avail[ip] = av - xnum;
            }
        }
        auxv[ip] = make_double2(0.0, 0.0);
    }
}

// End of a step: time, dt and the counters; then the next step's decision
// (prepare_step).  One thread.
__device__ __forceinline__ void step_end(StepScalars* S) {
    if (!S->skip && S->advance) {
        S->dt = S->dt_step;
        S->time += (double)S->dt;
        S->steps_done += 1;
    }
    prepare_step(S, 1);
}

__global__ void k_step_end(StepScalars* S) {
    PDL_ENTRY();
    StepScalars* L = scalars_to_smem(S);
    if (threadIdx.x == 0) step_end(L);
    scalars_from_smem(S, L);
}

// DEM update of ExtForces_SW(1) (:8795-8807) over the node box touched this
// step, resetting the scatter accumulators; the last block to finish also
// ends the step (k_step_end), which saves a launch.
__global__ void k_dem_erode(double2* auxv, float* z, float* eroded, float* avail, int nx, StepScalars* S) {
    PDL_ENTRY();
    __shared__ bool last;
    const int x0 = S->ex0, x1 = S->ex1, y0 = S->ey0, y1 = S->ey1;
    if (!S->skip && x1 >= x0 && y1 >= y0) erode_box(auxv, z, eroded, avail, nx, x0, x1, y0, y1);
    // the last block to finish ends the step (k_step_end)
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = (atomicAdd(&S->end_ticket, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    StepScalars* L = scalars_to_smem(S);
    if (threadIdx.x == 0) {
        L->end_ticket = 0u;
        step_end(L);
    }
    scalars_from_smem(S, L);
}

// Neighbour pairs of the coarse-level particles, for the parity export: every
// (big i, j) pair with r < hi + hj, written as slot pairs.
template <int SKF>
__global__ void k_export_big(Search Q, StepScalars* S, int2* pairs, int* npairs, int cap) {
    constexpr int SK = SupportScale<SKF>::value;
    coarse_particles<kBigThreads>(S->nreg, S->nbig, kBigBlocks, [&](int i, int lw) {
        coarse_neighbours<SK>(Q, S, i, lw, [&](int j, float4 o, const PairGeom& g) {
            int k = atomicAdd(npairs, 1);
            if (k < cap) pairs[k] = make_int2(i, j);
        });
    });
}

// ---------------------------------------------------------------- outputs

// Depth raster: IDW of h onto the 4x4 DEM nodes around each particle
// (SPH_SW_2019.f90:14310-14400, auxv(1)/auxv(5)).
__global__ void __launch_bounds__(32 * kScatterWarps) k_raster_idw(const PState B, int n, DemView dem, double2* acc) {
    const float distg = sqrtf(dem.dx * dem.dx + dem.dy * dem.dy);
    // block-uniform trip count: every lane of a warp reaches idw_scatter
    for (int i0 = blockIdx.x * blockDim.x; i0 < n; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + threadIdx.x;
        const bool part = i < n && !B.flag[i];
        idw_scatter(dem.nx, dem.ny, dem.xmin, dem.ymin, dem.dx, dem.dy, distg, part ? B.pos[i] : make_float2(0.f, 0.f),
                    part ? B.rho[i] : 0.f, part, acc);
    }
}

__global__ void k_raster_idw_finish(const double2* acc, float* out, int np) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < np; k += gridDim.x * blockDim.x) {
        double2 a = acc[k];
        out[k] = ((float)a.y >= 1.e-6f) ? (float)(a.x / a.y) : (float)a.x;
    }
}

// Misfit of the depth raster against a target raster, L = sum_nodes (R - T)^2
// with R the IDW raster above, for back-analysis: per node lam = dL/dR =
// 2 (R - T) and the node's share of L, summed per block (the host adds the
// block sums in block order).
__global__ void k_misfit_nodes(const double2* acc, const float* target, int np, double* lam, double* part) {
    __shared__ double sh[32];
    double l = 0.0;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < np; k += gridDim.x * blockDim.x) {
        const double2 a = acc[k];
        const double R = ((float)a.y >= 1.e-6f) ? a.x / a.y : a.x;
        const double d = R - (double)target[k];
        lam[k] = 2.0 * d;
        l += d * d;
    }
    l = warp_sum(l);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[w];
        part[blockIdx.x] = t;
    }
}

// dL/dh and dL/dx of every particle inside the domain, through the IDW
// weights w = 1/dhat, dhat = max(dist, 1e-6)/distg, of its 4x4 nodes: with
// S = sum w and R = sum h w / S, dR/dh_i = w_i / S and dR/dw_i = (h_i - R)/S
// (where S < 1e-6 the raster is sum h w itself: w_i and h_i);
// dw/dp = -(distg / dist^2) (p - node)/dist.  Written in caller order.
__global__ void k_misfit_particles(const PState B, int n, DemView dem, const double2* acc, const double* lam,
                                   float2* gx, float* gh) {
    const float distg = sqrtf(dem.dx * dem.dx + dem.dy * dem.dy);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int o = B.id[i];
        if (B.flag[i]) {
            gx[o] = make_float2(0.f, 0.f);
            gh[o] = 0.f;
            continue;
        }
        const float2 p = B.pos[i];
        const double h = B.rho[i];
        const int ipx = (int)((p.x - dem.xmin) / dem.dx + 1.f);
        const int ipy = (int)((p.y - dem.ymin) / dem.dy + 1.f);
        const int ix0 = max(1, ipx - 1), iy0 = max(1, ipy - 1), ix1 = min(dem.nx, ipx + 2), iy1 = min(dem.ny, ipy + 2);
        double dh = 0.0, d0 = 0.0, d1 = 0.0;
        for (int ix = ix0; ix <= ix1; ix++)
            for (int iy = iy0; iy <= iy1; iy++) {
                const int ip = (iy - 1) * dem.nx + (ix - 1);
                const double ex = (double)p.x - (double)(dem.xmin + (float)(ix - 1) * dem.dx);
                const double ey = (double)p.y - (double)(dem.ymin + (float)(iy - 1) * dem.dy);
                const double dist = sqrt(ex * ex + ey * ey);
                const double dhat = fmax(dist, 1.e-6) / (double)distg;
                const double w = 1.0 / dhat;
                const double2 a = acc[ip];
                const double L = lam[ip];
                double dRdh, dRdw;
                if ((float)a.y >= 1.e-6f) {
                    dRdh = w / a.y;
                    dRdw = (h - a.x / a.y) / a.y;
                } else {
                    dRdh = w;
                    dRdw = h;
                }
                dh += L * dRdh;
                if (dist > 1.e-6) {
                    const double c = -L * dRdw * (double)distg / (dist * dist * dist);
                    d0 += c * ex;
                    d1 += c * ey;
                }
            }
        gx[o] = make_float2((float)d0, (float)d1);
        gh[o] = (float)dh;
    }
}

// Per-node hazard statistics of Get_MC_pixel_Vars_SW (SPH_SW_2019.f90:20739-20812):
// each particle adds h and |v| to the 4 nodes of its DEM cell.
__global__ void k_hazard(const PState B, int n, DemView dem, double* sum_h, double* sum_v, unsigned int* max_h,
                         unsigned int* max_v, int* cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (B.flag[i]) continue;
        float2 p = B.pos[i];
        int ipx = (int)((p.x - dem.xmin) / dem.dx + 1.f);
        int ipy = (int)((p.y - dem.ymin) / dem.dy + 1.f);
        ipx = min(max(ipx, 1), dem.nx - 1);
        ipy = min(max(ipy, 1), dem.ny - 1);
        int ip = (ipy - 1) * dem.nx + (ipx - 1);
        int nodes[4] = {ip, ip + 1, ip + 1 + dem.nx, ip + dem.nx};
        float hh = B.rho[i];
        float2 v = B.vel[i];
        float vv = sqrtf(v.x * v.x + v.y * v.y);
        for (int k = 0; k < 4; k++) {
            int q = nodes[k];
            atomicAdd(&cnt[q], 1);
            atomicAdd(&sum_h[q], (double)hh);
            atomicAdd(&sum_v[q], (double)vv);
            atomicMax(&max_h[q], f2o(hh));
            atomicMax(&max_v[q], f2o(vv));
        }
    }
}

}  // namespace gfsph
