// pcg_chip.h -- the Jacobi-PCG whose vectors stay on the chip (pcg_chip.cu): what pcg.cu needs.
#pragma once

#include "apply_tile.cuh"

namespace gbs {

// Designs of one cooperative launch.
constexpr int kChipMaxDesigns = 16;

// One design's share of a launch: its grid cut into Px x Py x Pz boxes of elements, one per CTA.
struct ChipGeom {
    int nx, ny, nz;
    int Px, Py, Pz;
    int G;         // pairs of x slabs a CTA's box is cut into (one warp task per row group and pair)
    int NYm, NZm;  // node strides of every box: the largest box's node extents along y and z
    int stride;    // nodes of the largest box (exchange packets per CTA)
    int q;         // node pairs of the largest box per thread
    int items;     // room for a box's packets to wait for, for its nodes of several neighbours and
    int multi;     // for the terms of those
    int terms;
};

// Where a solve starts: from x0 = 0 with the right-hand side b, or bdd ((h, l) pairs) scaled in
// FP32 by *bscale (fresh), or from the state in the workspace (r, w, s, p, x and the scalars in
// sc: a paused solve, or the setup kernels' iteration 0).
struct ChipItem {
    int nx, ny, nz;
    const float *E;      // element moduli
    const float *dinv;   // 1/diag on free DOFs, 0 on fixed ones
    float *u;            // the iterate (out; in too when not fresh)
    PcgScalars *sc;
    float *r, *w, *s, *p;  // state of a paused solve
    float4 *xch;           // exchange buffer; must not overlap the state when not fresh
    size_t xch_bytes;
    const float *b;
    const float2 *bdd;
    const double *bscale;
    double tol;
    int max_iter, fresh;
};

// Fewest CTAs that hold this solve (its grid, its packets), 0 when the chip does not. Host only.
int chip_min_blocks(const gbsimp_ctx *ctx, const ChipItem &it);
// Modelled SM cycles per iteration of n designs in one launch (of the slowest); 1e300 when they do not fit
// together. Host only.
double chip_cycles(const gbsimp_ctx *ctx, const ChipItem *items, int n);
// The cut that a single design takes on a GPU of `sms` SMs, and its bytes of shared memory; false when the
// chip does not hold the grid. Host only.
bool chip_plan(int nx, int ny, int nz, int sms, size_t xch_bytes, ChipGeom *g, size_t *smem);
// Runs the inner PCGs of n designs in one cooperative launch, CTAs shared so that the designs'
// modelled iteration times even out: at most `budget` iterations each (0: to the end). Returns
// kChipRefused, with nothing run, when they do not fit together or the launch is refused (a context
// that may use fewer SMs than the device has, for instance): the caller takes a streaming form.
constexpr int kChipRefused = -1;
int chip_run(const gbsimp_ctx *ctx, const ChipItem *items, int n, int budget, cudaStream_t st);

}  // namespace gbs
