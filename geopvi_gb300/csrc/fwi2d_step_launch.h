// fwi2d_step_launch.h -- shapes, parameters and launchers of the FD time step
// (kernels in fwi2d_step.cuh, one translation unit per FD half width).
#pragma once

#include "fwi2d_kernels.cuh"

namespace gbfwi {

// Rows per tile and resident blocks per SM the registers are capped for.
// The variants compute the same values bit for bit; step_variant_for chooses.
struct StepVariant {
    int rows, min_blocks;
};
constexpr StepVariant kStepVariants[] = {{16, 28}, {8, 28}, {4, 28}, {2, 28}};
constexpr int kNumStepVariants = sizeof(kStepVariants) / sizeof(kStepVariants[0]);

// Rows per tile of the top and bottom strips, whose rows cost about twice an
// interior row of 64 columns.
__host__ __device__ constexpr int strip_rows(int R) { return R == 16 ? 10 : R; }

constexpr int kWideUnroll = 2;  // rows per iteration of sweep_wide

// The staged p1 tile of a block: R rows and 32 (narrow) or 64 (wide) columns
// with H halo rows and 4 or 8 halo columns on each side (a TMA box starts on a
// 16-byte boundary).
template <int H, int R>
struct TileShape {
    static constexpr int kHaloX = H <= 4 ? 4 : 8;
    static constexpr int kNarrowX = kTileX + 2 * kHaloX;
    static constexpr int kWideX = 2 * kTileX + 2 * kHaloX;
    static constexpr int kRows = R + 2 * H;
    static constexpr int kNarrowBytes = 4 * kRows * kNarrowX;
    static constexpr int kWideBytes = 4 * kRows * kWideX;
    static constexpr int kSmem = kWideBytes + 16;  // + the mbarrier
};

// Tensor maps over the ring: the boxes of narrow and of wide tiles.
struct StepMaps {
    CUtensorMap narrow, wide;
};

// Fused launches over instances of different geometry (gb_fwi2d_run_instances).
constexpr int kMaxPieces = 16;  // pieces per k_step_multi launch

// One piece: consecutive solves of one instance -- its buffers (the ring and
// stored field of these solves), acquisition and time axis, and where its
// solves and blocks start.
struct PieceArgs {
    const float *vdt, *vel, *obs, *rik;
    float *syn, *ring, *psave, *gacc;
    int s_iz, r_iz, r_ix0, dr, nr, ds, s_ix0, ns, nt, nti, nt_save;
    int inst0;        // its first solve within the instance
    int tm_slot0;     // its first ring slot among the tensor map's fields
    Divisor by_ns;    // its Tiling::by_ns
    int nres;         // its solves
    int first_block;  // its first block in the launch
};

// Everything a k_step_multi launch reads about its pieces, passed by value
// as the kernel's parameter: the pieces share their grid (every Geom field
// but the acquisition and the time axis) and their rings lie back to back
// under one tensor map.  NP: the pieces it can hold (a launch's parameter
// bytes are part of its fixed cost, so small launches take a small table).
template <int NP>
struct MultiArgsN {
    StepMaps tm;
    Geom gc;
    const BlendCoef *coef;
    int *status;
    int blend_fp32, imaging, store, npieces;
    Tiling tl;          // of the launch's grid (by_ns, stored: each piece's)
    int first[NP + 1];  // first blocks, ascending; first[npieces] = the blocks of all pieces
    PieceArgs piece[NP];
};
using MultiArgs = MultiArgsN<kMaxPieces>;

// One step of `nres` resident solves (k_step).  `overlap`: the previous
// operation on the stream is the step before this one, and this step may be
// launched programmatically (its blocks become resident while that step
// drains; k_step waits for it before any access to what it writes).
template <int H>
cudaError_t launch_step_h(bool adj, const StepMaps &m, const Geom &g, const Batch &b, int nres, const StepArgs &sa,
                          cudaStream_t st, int variant, bool overlap);

// Step k of the first `nact` pieces of `args` (k_step_multi).
template <int H>
cudaError_t launch_multi_h(bool adj, const MultiArgs &args, int nact, int k, cudaStream_t st, int variant,
                           bool overlap);

// The bands of a solve's rows -- [tile_r0, pml), [pml, ntz - pml), [ntz - pml,
// tile_r1) -- in tiles of strip_rows(R), R and strip_rows(R) rows.
inline Tiling make_tiling(const Geom &g, int R, int levels, long long ninst)
{
    Tiling t;
    t.rows_s = strip_rows(R);
    t.top = (g.pml - g.tile_r0 + t.rows_s - 1) / t.rows_s;
    t.bottom = (g.tile_r1 - (g.ntz - g.pml) + t.rows_s - 1) / t.rows_s;
    t.strips = (t.top + t.bottom) * g.units;
    t.narrow = g.units - 2 * g.wides;
    t.left = g.wide0 - g.unit0;
    t.narrows = (g.nz + R - 1) / R * t.narrow;
    t.by_units = make_divisor(g.units);
    t.by_narrow = make_divisor(t.narrow);
    t.by_wides = make_divisor(g.wides);
    t.by_ns = make_divisor(ninst * g.ns < (1LL << 32) ? g.ns : 1);
    t.solve = (long long)levels * g.fstride;
    t.stored = (long long)g.nt_save * g.pstride;
    return t;
}

// Tiles per solve at R rows per tile.
inline int step_tiles(const Geom &g, int R)
{
    const Tiling t = make_tiling(g, R, 3, 1);
    return t.strips + t.narrows + (g.nz + R - 1) / R * g.wides;
}

// Widths of the staged boxes.
inline int step_box_x(int H, bool wide) { return (wide ? 2 : 1) * kTileX + 2 * (H <= 4 ? 4 : 8); }

}  // namespace gbfwi
