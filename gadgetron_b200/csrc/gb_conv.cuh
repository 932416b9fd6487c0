// Arguments and launch configuration shared by the convolution kernels
// (gridding: gb_brick.cu; degridding and the trajectory gradient: gb_degrid.cu;
// the general kernels for other tiles, widths and 1D, and the launchers: gb_grid.cu).
#pragma once

#include "gb_internal.cuh"

namespace gb {

struct ConvArgs {
    KParams k;
    const float *pos;         // [D][Mtot] sorted positions
    const float *wtab;        // [Mtot][D][kWMax] tap weights of sorted samples
    const uint32_t *perm;     // sorted -> original
    const uint32_t *list;     // gridding list (sorted positions) or unused
    const WorkItem *items;
    int n_items;
    int64_t Mtot;
    int F;
    int nb;
    int layout;               // SampleLayout
    int il_stride;            // SORTED_IL: float2 per sample row (nb rounded up to even)
    const uint32_t *home_key; // sorted home keys (frame * ntiles_total + tile)
    const float *dcw;         // original order, may be null
    int dcw_pow;
    int sign_fold;
    int accumulate;
    // gridding split bookkeeping
    const SplitInfo *splits;
    float2 *partials;
    unsigned int *counters;
    int ncg;
    long long part_elems;     // float2 elements of one CTA's partial tile
    KLayout kl;               // k-space array layout
    const float *prows;       // gridding pair rows
    const uint2 *prng;        // footprint ranges of the gridding pairs
    int prow_floats;
    int lbx, lby, lbricks;    // brick kernel, log2: bricks per tile along x and y, in all,
    int lcta, lparts;         //   per CTA, warps per brick
};

// Taps of a sample at padded coordinate s along one dimension: first cell
// (unpadded) and count.  The same float expressions as the weight table's, which
// starts at that cell: from the unpadded coordinate s - pad/2, whose float grid is
// finer, the first cell can come out one further (W = 5.3, s just above a power of
// two), and every weight would sit one cell off.  The cell that rounding may add
// at an end lies beyond W/2 and has weight zero.
__device__ __forceinline__ int first_tap(const KParams &k, float s, int &n) {
    const int lo = (int)ceilf(s - k.radius);
    n = (int)floorf(s + k.radius) - lo + 1;
    return lo - k.hw;
}

__device__ __forceinline__ float sign_of(int g) { return (g & 1) ? -1.f : 1.f; }

// Which gridding kernel runs for a plan and batch count, with its coil group
// and the size of one CTA's partial tile (split tiles).
struct GridCfg {
    bool brick;       // k_grid_brick (else k_grid_nc2c)
    int cg;
    int nbricks;      // brick kernel: bricks per tile
    bool wide;        // brick kernel: the form for large launches
    int groups = 1;   // CTAs (split-tile counters) per tile
    int cpt;          // cell variant: cells per thread
    int ncg;
    int64_t part_elems;
};

// Coil group for nb batches: the requested one, halved while half of it
// still covers all of them.
int choose_cg(int requested, int nb);

// gb_brick.cu: fills cg and nbricks for this plan's tile; false when no brick
// shape divides the tile (1D plans, unusual tiles).
bool brick_config(const NufftPlan &p, int nb, GridCfg &c);
void launch_grid_brick(const GridCfg &c, const NufftPlan &p, const ConvArgs &a, const float2 *samples, float2 *grid,
                       cudaStream_t st);
// Samples [nb][Mtot] in the caller's order -> sorted coil-interleaved rows
// [Mtot][il] (padding zero), density weights folded in (dcw may be null).
void launch_samples_il(const NufftPlan &p, const float2 *samples, const float *dcw, int nb, float2 *rows,
                       cudaStream_t st);

// gb_degrid.cu: degridding and trajectory gradient from the weight table.
bool degrid_table_ok(const NufftPlan &p, int cg);
void launch_degrid_table(const NufftPlan &p, const ConvArgs &a, int cg, int ncg, bool comp, const float2 *grid,
                         float2 *out, cudaStream_t st);
bool grad_table_ok(const NufftPlan &p, int cg);
void launch_grad_table(const NufftPlan &p, const ConvArgs &a, int cg, const float2 *grid, const float2 *w, float *out,
                       cudaStream_t st);

}  // namespace gb
