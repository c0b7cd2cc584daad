// fwi2d_kernels.cuh -- sm_103a kernels of the 2-D acoustic FWI engine.
//
// One fused kernel advances every (sample, shot) solve of a wave by one time
// step: the 2*(Lc-1)-order Laplacian stencil (fdtd_2d_calculate_p,
// geopvi/forward/fwi2d/fdtd2D_modelling.c:756-780), the hybrid one-way
// absorbing boundary (abc_for_p, :833-900), Ricker source injection and
// receiver sampling (forward_IO, :902-939) or residual injection and the
// zero-lag imaging/gradient term (backward_IO, :941-978).  updata_p's copies
// (:1053-1066) become a rotation of three buffers, so no step copies a field.
//
// The step kernels are in fwi2d_step.cuh; this file holds what they share
// with the other kernels: the geometry, the buffers of a wave and the exact
// boundary mix (the TMA and mbarrier helpers are in tma.cuh).
//
// Arithmetic of the forward pass follows the reference operation by
// operation: __fmul_rn / __fadd_rn / __fsub_rn never contract into FMA;
// divisions by the constant dx, dz use a correctly rounded quotient; the
// boundary blend is the value that the C expression's double arithmetic
// gives.  The forward data therefore match the reference bit for bit.
#pragma once

#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

#include "fd_weights.cuh"
#include "fwi2d_exact.h"
#include "tma.cuh"

namespace gbfwi {

constexpr int kTileX = 32;  // columns of a unit of tiling: one warp, a 128-byte line of a row

// Geometry shared by every solve of one launch (one parameter set).
struct Geom {
    int ntx, ntz;        // padded grid (fdtd2D_modelling.c:86-87)
    int pitch, xoff;     // row pitch in floats; memory column of padded ix = 0
    int nx, nz, ipitch;  // interior grid and the row pitch of interior arrays
    int ioff;            // memory column of interior ix = pml in interior arrays
    int pml, Lc, pml0;   // Lc here is the reference's Lc after Lc += 1
    int s_iz, r_iz, r_ix0, dr, nr;
    int ds, s_ix0;       // source column of shot is: s_ix0 + is*ds
    int ns, nt, nti, nt_save;
    // What the step's tiles cover: rows [tile_r0, tile_r1) and the 32-column
    // units [unit0, unit0 + units).  That is every cell but the rim (rows and
    // columns outside [Lc, n - Lc), which keep the ring's zeros), or the whole
    // grid when a source or receiver lies in the rim.  Units [wide0, wide0 + 2 *
    // wides) hold interior columns only and go in pairs, two columns a lane; the
    // others are narrow tiles.
    int tile_r0, tile_r1, unit0, units, wide0, wides;
    int fast_dx, fast_dz;  // the host proved div_const exact for this divisor
    int two;               // ... and div_two for both
    int pstd;            // laplace_solver = 1: pseudo-spectral Laplacian
    long long fstride;   // floats per padded field (ntz * pitch)
    long long pstride;   // floats per interior snapshot (nz * ipitch)
    float dx, dz, dt;
    float rdx, rdz;      // RN(1/dx), RN(1/dz)
    float rxh, rxl, rzh, rzl;      // div_two's 1/dx and 1/dz
    float x2h, x2l, z2h, z2l;      // 1/dx^2 and 1/dz^2 in two words (adjoint)
    float lo1, lo2;      // least dividends of div_two by dx and of div2_two (inf without such a quotient)
    float fd[8];
};

// Division by a launch constant d: n / d as the high word of n * (2^32 / d + 1),
// exact for 0 <= n with n * d < 2^32.
struct Divisor {
    uint32_t m;  // 0: d = 1
    __host__ __device__ __forceinline__ int quotient(int n) const
    {
#if defined(__CUDA_ARCH__)
        return m ? (int)__umulhi((uint32_t)n, m) : n;
#else
        return m ? (int)(((uint64_t)(uint32_t)n * m) >> 32) : n;
#endif
    }
};
inline Divisor make_divisor(int d) { return Divisor{d <= 1 ? 0u : (uint32_t)((1ull << 32) / (uint32_t)d + 1)}; }

// How a launch's ranks map to the tiles of a solve (fwi2d_step_tile.inc), worked
// out once per launch sequence by make_tiling.
struct Tiling {
    int top, bottom, rows_s;   // tiles of the top and of the bottom strip, and their rows
    int strips;                // ranks of the strips' tiles: (top + bottom) * units
    int narrow, left, narrows; // narrow units of an interior row of tiles, those left of the pairs; their ranks
    Divisor by_units, by_narrow, by_wides;
    Divisor by_ns;             // shots: solve -> sample (m = 0 with ns > 1: divide)
    long long solve;           // floats per resident solve of the ring
    long long stored;          // ... and of the stored field
};

// Where the solves of a wave live.  Solve `inst` = sample * ns + shot.
struct Batch {
    const float *vdt;    // [nsamples][fstride]   padded v*dt per sample
    const float *vel;    // [nsamples][nz*nx]      inner velocity per sample
    const float *obs;    // [ns][nt][nr]
    float *syn;          // [nsamples*ns][nt][nr]
    float *ring;         // [resident][levels][fstride]
    float *psave;        // [resident][nt_save][pstride]
    float *gacc;         // [nsamples*ns][pstride]
    const BlendCoef *coef;  // [pml0] boundary weight w, 1 - w split in floats and as double
    int blend_fp32;      // the host proved (1 - w) * q exact in double for every weight
    int *status;         // device error word (0 = ok), then k_prepare's flags
    int inst0;           // first solve of this wave
    int slot0;           // first resident slot of this launch (the wave's second half)
    int levels;          // fields per resident slot of `ring`: 3, or the levels of a stored segment
    int tm_slot0;        // resident slot of ring[0] in the tensor map's fields (a map over several rings)
    int imaging;         // run_fwi == 0
    int store;           // forward pass stores the wavefield for the adjoint
    double *spec;        // pseudo-spectral mode: [resident][ntz][ntx] real array, then the
                         // [resident][ntz][ntx/2+1] half spectrum right after it
    const float *kk;     // pseudo-spectral mode: |k|^2 per padded cell (wavenumber)
    int spec_resident;   // pseudo-spectral mode: solves the real array holds (the half
                         // spectrum starts after them)
    Tiling tl;           // the FD step's tiles
};

// Per-launch step data.
struct StepArgs {
    int k;        // step within the pass
    int l0, l1, l2;  // ring levels of p0, p1, p2: (k%3, (k+1)%3, (k+2)%3) in a 3-level ring
    int it;       // time index
    int snap;     // forward: snapshot index it/nt_interval, or -1 when it % nt_interval != 0
    float rik;    // Ricker value at it (forward)
    // adjoint: snapshots whose product with p0, p1 and p2 this step adds to the
    // gradient (-1: none); see adjoint_terms
    int acc0, acc1, acc2;
};

// The adjoint adds its imaging terms every third step, when the three fields
// of the ring hold the last three adjoint levels: one read and write of the
// accumulator for up to three terms, added in the order of the steps.
// `first` / `last`: the first and last step index k of the pass (or of a
// checkpointed segment), it = it_first - (k - first).
__host__ __device__ __forceinline__ void adjoint_terms(StepArgs &sa, int nti, int k, int first, int last, int snap0)
{
    sa.acc0 = sa.acc1 = sa.acc2 = -1;
    const int pos = (k - first) % 3;
    if (pos != 2 && k != last) return;
    if (sa.it % nti == 0) sa.acc2 = sa.it / nti - snap0;
    if (pos >= 1 && (sa.it + 1) % nti == 0) sa.acc1 = (sa.it + 1) / nti - snap0;
    if (pos == 2 && (sa.it + 2) % nti == 0) sa.acc0 = (sa.it + 2) / nti - snap0;
}

// StepArgs of step k of a pass over a 3-level ring.
__host__ __device__ __forceinline__ StepArgs ring_step(int k, int it, int snap, float rik)
{
    StepArgs sa;
    sa.k = k;
    sa.l0 = k % 3;
    sa.l1 = (k + 1) % 3;
    sa.l2 = (k + 2) % 3;
    sa.it = it;
    sa.snap = snap;
    sa.rik = rik;
    sa.acc0 = sa.acc1 = sa.acc2 = -1;
    return sa;
}

enum : int { kStatusOk = 0, kStatusTmaTimeout = 1 };
constexpr int kStatusWords = 2;  // the error word, and k_prepare's flags: no tile is skipped

__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }

// One blend of abc_for_p: a 2nd-order one-way extrapolation from the two
// previous levels along the inward direction, weighted by w against the
// current value (fdtd2D_modelling.c:843-849).  p1a..p1c = p1 at 0,1,2 steps
// inward; p0a..p0e = p0 at 0..4 steps inward.  The extrapolation is float;
// the final mix is the double expression w*ext + (1.0-w)*q, reproduced
// exactly by blend_mix.
__device__ __forceinline__ float abc_blend(float q, float t11, float t12, float t13, float p1a,
                                           float p1b, float p1c, float p0a, float p0b, float p0c,
                                           float p0d, float p0e, const BlendCoef &c, int fp32_ok)
{
    const float a2 = fm(2.0f, t11), b2 = fm(2.0f, t12), e2 = fm(2.0f, t13);
    float ext = fa(fa(fm(a2, p1a), fm(b2, p1b)), fm(e2, p1c));
    ext = fs(ext, fm(fm(t11, t11), p0a));
    ext = fs(ext, fm(fm(a2, t12), p0b));
    ext = fs(ext, fm(fa(fm(t12, t12), fm(a2, t13)), p0c));
    ext = fs(ext, fm(fm(b2, t13), p0d));
    ext = fs(ext, fm(fm(t13, t13), p0e));
    // The double mix by one FMA where blend_fma_ok proves it (fwi2d_exact.h),
    // the exact FP32 / FP64 evaluation otherwise.
    const float a = fm(c.w, ext);
    if (blend_fma_ok(a, q, c.khi, c.klo)) return __fmaf_rn(c.bh, q, a);
    return blend_mix(a, q, c, fp32_ok);
}

// Receiver index of padded column ix on the receiver row, or -1.
__device__ __forceinline__ int receiver_of(const Geom &g, int ix)
{
    const int off = ix - g.r_ix0;
    if (g.dr == 0) return off == 0 ? 0 : -1;
    if (off % g.dr) return -1;
    const int ir = off / g.dr;
    return (ir >= 0 && ir < g.nr) ? ir : -1;
}

// Inner velocity at padded cell (iz, ix): get_velp's edge replication
// (fdtd2D_modelling.c:1187-1238) is a clamp of both coordinates.
__device__ __forceinline__ float padded_velocity(const Geom &g, const float *vel, int iz, int ix)
{
    int jz = min(max(iz - g.pml, 0), g.nz - 1);
    int jx = min(max(ix - g.pml, 0), g.nx - 1);
    return vel[(long long)jz * g.nx + jx];
}

}  // namespace gbfwi
