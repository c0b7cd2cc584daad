// fwi2d_step.cuh -- the FD time step of the 2-D engine, forward and adjoint.
//
// One launch advances every (sample, shot) solve of a wave by one step: the
// 2*(Lc-1)-order Laplacian stencil (fdtd_2d_calculate_p, geopvi/forward/fwi2d/
// fdtd2D_modelling.c:756-780), the hybrid one-way absorbing boundary
// (abc_for_p, :833-900), Ricker source injection and receiver sampling
// (forward_IO, :902-939) or residual injection and the zero-lag imaging /
// gradient term (backward_IO, :941-978).  updata_p's copies (:1053-1066) become
// a rotation of three buffers, so no step copies a field.
//
// Data movement: a block is one warp and owns some rows of one solve, 64
// columns of the interior (two a lane, 8-byte accesses) or 32 columns.  An
// elected lane stages the previous level with its stencil halo by one TMA
// tensor load; the warp sweeps its rows with the z window in registers, reads
// the level before (p0) and v*dt coalesced, and writes whole 128-byte lines.
// Only cells that change are covered: tiles start at row Lc and skip rim-only
// columns, and the rim keeps the zeros the ring is cleared to (the reference
// never changes the rim from its initial zero: the stencil leaves it out and
// the boundary passes blend rim cells from rim cells only -- unless a source
// or a receiver lies in it, see Geom::tile_r0).
//
// A tile is of one class -- interior, top or bottom strip, left or right strip,
// corner -- so its rows run one of three loops without region tests:
// sweep_wide, sweep_z and sweep_x.  Corners, the source's and the receivers'
// rows, and leftover rows run sweep_edge, which tests everything.  All but
// sweep_wide go row by row inward from the grid's edge, so the top and the
// bottom strip's one-way extrapolation are the same code, the row step negated.
//
// Arithmetic: the forward pass is the reference's, operation by operation,
// with exact shortcuts for its divisions and its double boundary mix
// (fwi2d_exact.h).  The adjoint's result is a gradient that is compared at
// 1e-4: it takes the second differences in the same order and the boundary
// passes as they are, and rounds the update less often -- the grid constants
// 1/dx^2, 1/dz^2 in two words, one fused sum.  (Fusing the second
// differences' sums too saves 16 operations a cell and rounds less, yet its
// gradient is 1.6 times as far from 64 bits: with the forward pass's own
// rounding the two fields' errors cancel in part.  The boundary mix unproved
// and its factors without their range test are off by a rounding now and
// then, and are wrong for infinities.)
//
// Measured (200x400, 20 shots, 8 models, 800 steps of misfit + gradient; us per
// step of 18 M padded cells): 112 with 32x16 tiles in one class and inline exact
// fallbacks; 97 with the second differences' quotients in two operations and
// the strips' and interior rows' loops separate; 81 with straight-line tails
// and untouched tiles skipped; 76 with the tails out of line (no spills in order
// 8; the other orders' forward kernels spill 24 to 80 bytes under the cap of 72
// registers, k_step_multi up to 224); 70 with a shorter prologue; 71.6 -> 74.4 with
// the adjoint's boundary mix proved and its skipped tiles' stored field looked at.
// Two columns a lane: 115 -> 70 instructions per 32 interior cells (adjoint).
#pragma once

#include "fwi2d_step_launch.h"

namespace gbfwi {

__device__ __forceinline__ float ff(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// (x/y)/y of a divisor without the two-operation quotient, and s = v dt / dx
// outside it: out of line, so the sweeps keep one call each.
static __device__ __noinline__ float laplacian_rare(const Geom *g, float lx, float lz)
{
    const float x = g->fast_dx && in_fast_range(lx, kDiv2Lo, kDiv2Hi) ? div2_fast(lx, g->dx, -g->rdx)
                                                                      : div2_any(lx, g->dx, g->rdx, g->fast_dx);
    const float z = g->fast_dz && in_fast_range(lz, kDiv2Lo, kDiv2Hi) ? div2_fast(lz, g->dz, -g->rdz)
                                                                      : div2_any(lz, g->dz, g->rdz, g->fast_dz);
    return fa(x, z);
}

static __device__ __noinline__ float slowness_rare(const Geom *g, float vd)
{
    return div_const(vd, g->dx, g->rdx, g->fast_dx);
}

// lx/dx/dx + lz/dz/dz where the two-operation quotients hold; *ok says whether
// they do.
__device__ __forceinline__ float laplacian_two(float lx, float lz, const Geom &g, bool *ok)
{
    *ok = fminf(fabsf(lx), fabsf(lz)) >= g.lo2;
    return fa(div2_two(lx, g.rxh, g.rxl), div2_two(lz, g.rzh, g.rzl));
}

// ... and where they do not: the tails ahead of a wavefront, down to the
// subnormals.  Straight-line and called by the whole warp, so a warp of mixed
// magnitudes does not diverge; out of line, as inlined into the three sweeps it
// cost 180 bytes of spills.  A second difference of exactly zero is exact on
// the fast path.
static __device__ __noinline__ float laplacian_tail(float lx, float lz, const Geom *g)
{
    if (!g->two) return laplacian_rare(g, lx, lz);
    const float rxh = g->rxh, rxl = g->rxl, rzh = g->rzh, rzl = g->rzl, lo2 = g->lo2;
    const float x = div2_tiny(lx, g->dx, rxh, rxl), z = div2_tiny(lz, g->dz, rzh, rzl);
    return fa(fabsf(lx) < lo2 ? x : div2_two(lx, rxh, rxl), fabsf(lz) < lo2 ? z : div2_two(lz, rzh, rzl));
}

// The second differences of one cell: x[m], z[m] are its neighbours m cells
// away along each axis, m = -H..H.
template <int H, bool ADJ>
__device__ __forceinline__ void second_differences(const float *x, const float *z, float *lx, float *lz)
{
    float dx = fm(fd_weight<H>(0), z[0]);
    float dz = dx;
#pragma unroll
    for (int m = 1; m <= H; ++m) {
        const float sx = fa(x[m], x[-m]), sz = fa(z[m], z[-m]);
        dx = fa(dx, fm(fd_weight<H>(m), sx));
        dz = fa(dz, fm(fd_weight<H>(m), sz));
    }
    *lx = dx;
    *lz = dz;
}

// 2 p1 - p0 + (v dt)^2 (lx/dx^2 + lz/dz^2); forward: lap = laplacian_two's value.
__device__ __forceinline__ float update_forward(float p1c, float p0c, float vd, float lap)
{
    return fa(fs(fm(2.0f, p1c), p0c), fm(fm(vd, vd), lap));
}
__device__ __forceinline__ float update_adjoint(const Geom &g, float p1c, float p0c, float vd, float lx, float lz)
{
    const float lap = ff(lz, g.z2h, ff(lx, g.x2h, ff(lx, g.x2l, fm(lz, g.z2l))));
    return ff(fm(vd, vd), lap, ff(2.0f, p1c, -p0c));
}

// abc_for_p's extrapolation factors of a cell (fdtd2D_modelling.c:233-240):
// s = v dt / dx.
struct AbcCoef {
    float t11, t12, t13;
};

__device__ __forceinline__ AbcCoef abc_coef(const Geom &g, const Geom *gp, float vd)
{
    float s = div_two(vd, g.rxh, g.rxl);
    if (!(vd >= g.lo1 || vd == 0.0f)) s = slowness_rare(gp, vd);
    const float u = fs(2.0f, s);
    return AbcCoef{fm(fm(u, fs(1.0f, s)), 0.5f), fm(s, u), fm(fm(s, fs(s, 1.0f)), 0.5f)};
}

// One blend of abc_for_p (:843-849): a 2nd-order one-way extrapolation from
// the two previous levels along the inward direction, weighted by k.x = w
// against the current value q.  p1a..p1c = p1 at 0, 1, 2 steps inward;
// p0a..p0e = p0 at 0..4 steps inward.  `k` holds w, bh, khi2, klo2 of `c`, bl its bl.
// The adjoint, with its three terms in flight, has no registers to spare for the
// table's address: its rare path takes its arguments by value.  80 solves of
// 200x400, 3000 steps of both passes: 249 ms, 256 with the double formula inline
// in its place, 241 with the split evaluation taken unproved.
template <bool ADJ>
__device__ __forceinline__ float blend(float q, const AbcCoef &t, float p1a, float p1b, float p1c, float p0a,
                                       float p0b, float p0c, float p0d, float p0e, const float4 &k,
                                       float bl, const BlendCoef *c, int fp32_ok)
{
    const float a2 = fm(2.0f, t.t11), b2 = fm(2.0f, t.t12), e2 = fm(2.0f, t.t13);
    float ext = fa(fa(fm(a2, p1a), fm(b2, p1b)), fm(e2, p1c));
    ext = fs(ext, fm(fm(t.t11, t.t11), p0a));
    ext = fs(ext, fm(fm(a2, t.t12), p0b));
    ext = fs(ext, fm(fa(fm(t.t12, t.t12), fm(a2, t.t13)), p0c));
    ext = fs(ext, fm(fm(b2, t.t13), p0d));
    ext = fs(ext, fm(fm(t.t13, t.t13), p0e));
    const float a = fm(k.x, ext);
    if (ADJ) return blend_mix_values(a, q, k.y, bl, k.z, k.w, fp32_ok);
    // RN_f(RN_d(w ext + (1 - w) q)): one FMA, the split evaluation, or the
    // general one, each where it is proved (fwi2d_exact.h).
    float r = ff(k.y, q, a);
    if (!blend_one_fma(a, q, k.z, k.w)) {
        if (!(blend_mix_split(a, q, k.y, bl, &r) && fp32_ok)) r = blend_mix_at(a, q, c, fp32_ok);
    }
    return r;
}

__device__ __forceinline__ float4 blend_weights(const BlendCoef *c) { return __ldg(reinterpret_cast<const float4 *>(c)); }

// Per-warp view of one step.  Row 0 of the tile is its outermost row, rows go
// inward (dir = 1 down, -1 up).  Pointers are warp-uniform: row 0, the tile's
// first column (interior arrays: where that cell would lie); st and si lead
// one row inward.
struct WarpCtx {
    const float *s1;      // staged p1
    const float *p0, *vdt;
    float *p2;
    float *ps;                       // stored snapshot (forward), or null
    const float *a0, *a1, *a2;       // snapshots of the adjoint's terms (h0, h1, h2: which there are)
    float *G;                        // gradient accumulator, null when this step adds nothing
    bool h0, h1, h2;
    int iz0, ix0, dir;               // padded row and column of the tile's first cell
    int st, si;
    int lane;
    int inst, sample, shot;
};

// forward_IO's source injection (fdtd2D_modelling.c:910) on the source row, or
// backward_IO's residual injection (:949-959) on the receiver row.
template <bool ADJ>
__device__ __forceinline__ float inject(const Geom &g, const Batch &b, const StepArgs &sa, const WarpCtx &w, float q,
                                        int iz, int ix)
{
    float r;
    if (!ADJ) {
        if (ix != g.s_ix0 + w.shot * g.ds) return q;
        r = sa.rik;
    } else {
        const int ir = receiver_of(g, ix);
        if (ir < 0) return q;
        const float o = b.obs[((long long)w.shot * g.nt + sa.it) * g.nr + ir];
        r = b.imaging ? o : fs(b.syn[((long long)w.inst * g.nt + sa.it) * g.nr + ir], o);
    }
    const float v = padded_velocity(g, b.vel + (long long)w.sample * g.nx * g.nz, iz, ix);
    return fa(q, fm(fm(fm(fm(r, g.dt), g.dt), v), v));
}

// forward_IO's receiver sampling (:930-938).
__device__ __forceinline__ void sample_receiver(const Geom &g, const Batch &b, const StepArgs &sa, const WarpCtx &w,
                                                float q, int ix)
{
    const int ir = receiver_of(g, ix);
    if (ir >= 0) b.syn[((long long)w.inst * g.nt + sa.it) * g.nr + ir] = q;
}

// The stored field: p2 - 2 p1 + p0 (the 1/dt^2 of the reference's d2p/dt2 is
// applied once, in FP64, by the gradient reduction), or p2 when imaging.
__device__ __forceinline__ float snapshot(const Batch &b, float q, float p1c, float p0c)
{
    return b.imaging ? q : fa(fs(q, fm(2.0f, p1c)), p0c);
}

// The adjoint's pending terms, oldest first, added to the accumulator.
template <typename T>
struct Terms {
    T s0, s1, s2, g;
};
template <typename T>
__device__ __forceinline__ Terms<T> load_terms(const WarpCtx &w, int oi)
{
    Terms<T> t{};
    if (w.h0) t.s0 = __ldcs(reinterpret_cast<const T *>(w.a0 + oi));
    if (w.h1) t.s1 = __ldcs(reinterpret_cast<const T *>(w.a1 + oi));
    if (w.h2) t.s2 = __ldcs(reinterpret_cast<const T *>(w.a2 + oi));
    t.g = *reinterpret_cast<const T *>(w.G + oi);
    return t;
}
__device__ __forceinline__ float add_terms(const WarpCtx &w, float s0, float s1, float s2, float g, float p0c,
                                           float p1c, float q)
{
    if (w.h0) g = ff(s0, p0c, g);
    if (w.h1) g = ff(s1, p1c, g);
    if (w.h2) g = ff(s2, q, g);
    return g;
}

__device__ __forceinline__ float2 ldg2(const float *p) { return __ldg(reinterpret_cast<const float2 *>(p)); }

// Rows [ja, jb) of a wide tile, all interior: no strip, source or receiver; an
// even number of them.  Two adjacent columns a lane: the x taps are 2K aligned
// 8-byte loads, and every address, load and store serves two cells.  Two rows
// an iteration: half the register moves of the sliding window.  p0 and v*dt
// are fetched one row ahead.
template <int H, bool ADJ, int R>
__device__ __forceinline__ void sweep_wide(const Geom &g, const Geom *gp, const Batch &b, const WarpCtx &w, int ja,
                                           int jb)
{
    constexpr int BX = TileShape<H, R>::kWideX;
    constexpr int K = (H + 1) / 2;  // pairs on each side that hold the x taps
    constexpr int U = kWideUnroll;
    const float *scol = w.s1 + 2 * w.lane + ja * BX;
    float wa[2 * H + U], wb[2 * H + U];  // [u + H + m]: m rows from row j + u
#pragma unroll
    for (int m = 0; m < 2 * H; ++m) {
        const float2 v = *reinterpret_cast<const float2 *>(scol + (m - H) * BX);
        wa[m] = v.x;
        wb[m] = v.y;
    }
    const long long o = ja * (long long)g.pitch + 2 * w.lane;
    int oi = ja * g.ipitch + 2 * w.lane;
    const float *p0 = w.p0 + o, *vdt = w.vdt + o;
    float *p2 = w.p2 + o;
    float2 p0n = ldg2(p0), vdn = ldg2(vdt);
#pragma unroll 1
    for (int j = ja; j < jb; j += U) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float2 p0c = p0n, vd = vdn;
            p0 += g.pitch;
            vdt += g.pitch;
            if (u + 1 < U || j + U < jb) {
                p0n = ldg2(p0);
                vdn = ldg2(vdt);
            }
            Terms<float2> t{};
            if (ADJ && w.G) t = load_terms<float2>(w, oi);  // before the stencil work that hides their latency
            float x[4 * K + 2];  // x[2K + m]: m columns from the lane's first
#pragma unroll
            for (int k = -K; k <= K; ++k) {
                if (k == 0) continue;
                const float2 v = *reinterpret_cast<const float2 *>(scol + u * BX + 2 * k);
                x[2 * (K + k)] = v.x;
                x[2 * (K + k) + 1] = v.y;
            }
            x[2 * K] = wa[u + H];
            x[2 * K + 1] = wb[u + H];
            {
                const float2 v = *reinterpret_cast<const float2 *>(scol + (u + H) * BX);
                wa[u + 2 * H] = v.x;
                wb[u + 2 * H] = v.y;
            }
            const float p1a = wa[u + H], p1b = wb[u + H];
            float lxa, lza, lxb, lzb, qa, qb;
            second_differences<H, ADJ>(x + 2 * K, wa + u + H, &lxa, &lza);
            second_differences<H, ADJ>(x + 2 * K + 1, wb + u + H, &lxb, &lzb);
            if (ADJ) {
                qa = update_adjoint(g, p1a, p0c.x, vd.x, lxa, lza);
                qb = update_adjoint(g, p1b, p0c.y, vd.y, lxb, lzb);
            } else {
                bool oka, okb;
                float la = laplacian_two(lxa, lza, g, &oka), lb = laplacian_two(lxb, lzb, g, &okb);
                if (!__all_sync(0xffffffffu, oka && okb)) {
                    // a field the wave has not reached is zero, and exact as it is
                    const float any = fmaxf(fmaxf(fabsf(lxa), fabsf(lza)), fmaxf(fabsf(lxb), fabsf(lzb)));
                    if (__any_sync(0xffffffffu, any != 0.0f)) {
                        la = laplacian_tail(lxa, lza, gp);
                        lb = laplacian_tail(lxb, lzb, gp);
                    }
                }
                qa = update_forward(p1a, p0c.x, vd.x, la);
                qb = update_forward(p1b, p0c.y, vd.y, lb);
            }
            *reinterpret_cast<float2 *>(p2) = make_float2(qa, qb);
            p2 += g.pitch;
            if (ADJ) {
                if (w.G)
                    *reinterpret_cast<float2 *>(w.G + oi) =
                        make_float2(add_terms(w, t.s0.x, t.s1.x, t.s2.x, t.g.x, p0c.x, p1a, qa),
                                    add_terms(w, t.s0.y, t.s1.y, t.s2.y, t.g.y, p0c.y, p1b, qb));
            } else if (w.ps) {
                __stcs(reinterpret_cast<float2 *>(w.ps + oi),
                       make_float2(snapshot(b, qa, p1a, p0c.x), snapshot(b, qb, p1b, p0c.y)));
            }
            oi += g.ipitch;
        }
#pragma unroll
        for (int m = 0; m < 2 * H; ++m) {
            wa[m] = wa[m + U];
            wb[m] = wb[m + U];
        }
        scol += U * BX;
    }
}

// The update before the blends, for a converged warp of one column a lane.
// `idle` lanes discard the value.
template <int H, bool ADJ>
__device__ __forceinline__ float update(const Geom &g, const Geom *gp, const float *srow, const float *win, float p0c,
                                        float vd, bool idle)
{
    float lx, lz;
    second_differences<H, ADJ>(srow, win, &lx, &lz);
    if (ADJ) return update_adjoint(g, win[0], p0c, vd, lx, lz);
    bool ok;
    float lap = laplacian_two(lx, lz, g, &ok);
    ok |= idle | (lx == 0.0f && lz == 0.0f);
    if (__any_sync(0xffffffffu, !ok)) lap = laplacian_tail(lx, lz, gp);
    return update_forward(win[0], p0c, vd, lap);
}

// Rows [ja, jb) of a tile of interior columns in the top or bottom strip, no
// source or receiver among them (abc_for_p's top / bottom passes,
// fdtd2D_modelling.c:837-867).  The rows of p0 that the extrapolation reads
// slide through registers like the stencil's.
template <int H, bool ADJ, int R>
__device__ __forceinline__ void sweep_z(const Geom &g, const Geom *gp, const Batch &b, const WarpCtx &w, int ja, int jb)
{
    constexpr int BX = TileShape<H, R>::kNarrowX;
    const int sp = w.dir * BX;
    const float *scol = w.s1 + w.lane + ja * sp;
    float win[2 * H + 1];
#pragma unroll
    for (int m = 0; m < 2 * H; ++m) win[m] = scol[(m - H) * sp];
    const long long o = ja * (long long)w.st + w.lane, st = w.st;
    const float *p0 = w.p0 + o, *vdt = w.vdt + o;
    float *p2 = w.p2 + o;
    float z[5];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        z[m] = __ldg(p0);
        p0 += st;
    }
    float p0n = __ldg(p0), vdn = __ldg(vdt);
    const int iz = w.iz0 + w.dir * ja;
    const BlendCoef *cz = b.coef + (w.dir > 0 ? iz - g.Lc : g.ntz - g.Lc - 1 - iz);
#pragma unroll 1
    for (int j = ja; j < jb; ++j) {
        const float vd = vdn;
        z[4] = p0n;
        p0 += st;
        vdt += st;
        if (j + 1 < jb) {
            p0n = __ldg(p0);
            vdn = __ldg(vdt);
        }
        const float4 k = blend_weights(cz);
        const float bl = __ldg(&cz->bl);
        ++cz;
        win[2 * H] = scol[H * sp];
        float q = update<H, ADJ>(g, gp, scol, win + H, z[0], vd, false);
        q = blend<ADJ>(q, abc_coef(g, gp, vd), win[H], win[H + 1], win[H + 2], z[0], z[1], z[2], z[3], z[4], k,
                       bl, cz - 1, b.blend_fp32);
        *p2 = q;
        p2 += st;
#pragma unroll
        for (int m = 0; m < 2 * H; ++m) win[m] = win[m + 1];
#pragma unroll
        for (int m = 0; m < 4; ++m) z[m] = z[m + 1];
        scol += sp;
    }
}

// This lane's place among the columns of a narrow tile.
struct Column {
    int ix;
    bool live, sx, inner, xs, left;  // in the grid, updated, interior, in a strip, in the left half
    const BlendCoef *c;
    float4 k;
    float bl;
};
__device__ __forceinline__ Column column_of(const Geom &g, const Batch &b, int ix)
{
    Column c;
    c.ix = ix;
    c.live = ix >= 0 && ix < g.ntx;
    c.sx = ix >= g.Lc && ix < g.ntx - g.Lc;
    c.inner = ix >= g.pml && ix < g.ntx - g.pml;
    c.xs = c.sx && !c.inner;
    c.left = ix < g.pml;
    c.c = b.coef + (c.xs ? (c.left ? ix - g.Lc : g.ntx - g.Lc - ix - 1) : 0);
    c.k = blend_weights(c.c);
    c.bl = __ldg(&c.c->bl);
    return c;
}

// p0 at 1..4 columns inward of a strip's column: the same four loads for both
// strips, in opposite order.
struct Inward4 {
    float v1, v2, v3, v4;
};
__device__ __forceinline__ Inward4 inward4(const float *p, bool left)
{
    if (!left) p -= 5;
    const float l1 = __ldg(p + 1), l2 = __ldg(p + 2), l3 = __ldg(p + 3), l4 = __ldg(p + 4);
    return Inward4{left ? l1 : l4, left ? l2 : l3, left ? l3 : l2, left ? l4 : l1};
}

// The left / right pass of abc_for_p (:869-899) on a strip's cell.
template <bool ADJ>
__device__ __forceinline__ float blend_x(const Column &c, float q, const AbcCoef &t, const float *srow, float p1c,
                                         float p0c, const Inward4 &p, const Batch &b)
{
    const float *px = c.left ? srow : srow - 3;
    const float l1 = px[1], l2 = px[2];
    return blend<ADJ>(q, t, p1c, c.left ? l1 : l2, c.left ? l2 : l1, p0c, p.v1, p.v2, p.v3, p.v4, c.k, c.bl, c.c,
                      b.blend_fp32);
}

// Rows [ja, jb) of a narrow tile, all interior rows without source or receiver.
template <int H, bool ADJ, int R>
__device__ __forceinline__ void sweep_x(const Geom &g, const Geom *gp, const Batch &b, const WarpCtx &w, int ja, int jb)
{
    constexpr int BX = TileShape<H, R>::kNarrowX;
    const Column c = column_of(g, b, w.ix0 + w.lane);
    const float *scol = w.s1 + w.lane + ja * BX;
    float win[2 * H + 1];
#pragma unroll
    for (int m = 0; m < 2 * H; ++m) win[m] = scol[(m - H) * BX];
    const long long o = ja * (long long)g.pitch + w.lane;
    int oi = ja * g.ipitch + w.lane;
    const float *p0 = w.p0 + o, *vdt = w.vdt + o;
    float *p2 = w.p2 + o;
    float p0n = __ldg(p0), vdn = __ldg(vdt);
#pragma unroll 1
    for (int j = ja; j < jb; ++j) {
        const float p0c = p0n, vd = vdn;
        Inward4 pi{};
        if (c.xs) pi = inward4(p0, c.left);
        p0 += g.pitch;
        vdt += g.pitch;
        if (j + 1 < jb) {
            p0n = __ldg(p0);
            vdn = __ldg(vdt);
        }
        Terms<float> t{};
        if (ADJ && w.G && c.inner) t = load_terms<float>(w, oi);
        win[2 * H] = scol[H * BX];
        const float p1c = win[H];
        float q = update<H, ADJ>(g, gp, scol, win + H, p0c, vd, !c.sx);
        if (!c.sx) q = c.live ? p1c : 0.0f;  // the rim keeps the previous level, the row padding zero
        if (c.xs) q = blend_x<ADJ>(c, q, abc_coef(g, gp, vd), scol, p1c, p0c, pi, b);
        *p2 = q;
        p2 += g.pitch;
        if (c.inner) {
            if (ADJ) {
                if (w.G) w.G[oi] = add_terms(w, t.s0, t.s1, t.s2, t.g, p0c, p1c, q);
            } else if (w.ps) {
                __stcs(w.ps + oi, snapshot(b, q, p1c, p0c));
            }
        }
        oi += g.ipitch;
#pragma unroll
        for (int m = 0; m < 2 * H; ++m) win[m] = win[m + 1];
        scol += BX;
    }
}

// Rows [ja, jb) of 32 columns from the tile's column `col` on: strips, source,
// receivers, rim and row padding may be among them.  bx: columns of the staged
// tile.
template <int H, bool ADJ>
__device__ __forceinline__ void sweep_edge(const Geom &g, const Geom *gp, const Batch &b, const StepArgs &sa,
                                           const WarpCtx &w, int bx, int col, int ja, int jb)
{
    const int lc = col + w.lane;
    const Column c = column_of(g, b, w.ix0 + lc);
    const int sp = w.dir * bx;
    const float *scol = w.s1 + lc + ja * sp;
    float win[2 * H + 1];
#pragma unroll
    for (int m = 0; m < 2 * H; ++m) win[m] = scol[(m - H) * sp];
#pragma unroll 1
    for (int j = ja; j < jb; ++j) {
        const int iz = w.iz0 + w.dir * j;
        const float *p0 = w.p0 + (j * (long long)w.st + lc);
        const float p0c = __ldg(p0), vd = __ldg(w.vdt + (j * (long long)w.st + lc));
        const bool sz = iz >= g.Lc && iz < g.ntz - g.Lc;
        const bool inner_z = iz >= g.pml && iz < g.ntz - g.pml;
        const bool zb = sz && !inner_z;
        const bool image = c.inner && inner_z;
        const int oi = j * w.si + lc;
        win[2 * H] = scol[H * sp];
        const float p1c = win[H];
        float q = update<H, ADJ>(g, gp, scol, win + H, p0c, vd, !(c.sx && sz));
        if (!(c.sx && sz)) q = p1c;  // cells the stencil skips keep the previous level
        if (zb || c.xs) {
            const AbcCoef t = abc_coef(g, gp, vd);
            if (zb) {
                const BlendCoef *cz = b.coef + (w.dir > 0 ? iz - g.Lc : g.ntz - g.Lc - 1 - iz);
                const int st = w.st;
                q = blend<ADJ>(q, t, p1c, win[H + 1], win[H + 2], p0c, __ldg(p0 + st), __ldg(p0 + 2 * st),
                               __ldg(p0 + 3 * st), __ldg(p0 + 4 * st), blend_weights(cz), __ldg(&cz->bl), cz,
                               b.blend_fp32);
            }
            if (c.xs) q = blend_x<ADJ>(c, q, t, scol, p1c, p0c, inward4(p0, c.left), b);  // after top / bottom
        }
        if (iz == (ADJ ? g.r_iz : g.s_iz)) q = inject<ADJ>(g, b, sa, w, q, iz, c.ix);
        q = c.live ? q : 0.0f;  // the row padding stays zero
        w.p2[j * (long long)w.st + lc] = q;
        if (!ADJ && iz == g.r_iz) sample_receiver(g, b, sa, w, q, c.ix);
        if (image) {
            if (ADJ) {
                if (w.G) {
                    const Terms<float> t = load_terms<float>(w, oi);
                    w.G[oi] = add_terms(w, t.s0, t.s1, t.s2, t.g, p0c, p1c, q);
                }
            } else if (w.ps) {
                __stcs(w.ps + oi, snapshot(b, q, p1c, p0c));
            }
        }
#pragma unroll
        for (int m = 0; m < 2 * H; ++m) win[m] = win[m + 1];
        scol += sp;
    }
}

// Whether the staged p1 tile (n4 16-byte words) and the p0 values its rows read
// are all zero.  The middle row's values (at `mid`) settle it for nearly every
// live tile.
__device__ __forceinline__ bool tile_is_zero(const float *tile, int n4, int mid, const WarpCtx &w, int nrows, bool wide,
                                             const int *status)
{
    constexpr unsigned kAll = 0xffffffffu;
    if (__any_sync(kAll, tile[mid + w.lane] != 0.0f)) return false;
    unsigned bits = (unsigned)status[1];  // flagged: returns before p0 is read
    for (int i = w.lane; i < n4; i += 32) {
        const uint4 v = reinterpret_cast<const uint4 *>(tile)[i];
        bits |= (v.x | v.y | v.z | v.w) & 0x7fffffffu;
    }
    if (__any_sync(kAll, bits != 0u)) return false;
    // The blends read p0 up to 4 rows and columns inward; tiles lie at least
    // that far inside the field's memory, row padding included, but for grids with
    // tiles on the rim, where k_prepare's flag leaves none to look at.
    const float *p0 = w.p0 + w.lane;
    if (wide) {
        for (int j = 0; j < nrows; ++j, p0 += w.st) bits |= __float_as_uint(p0[0]) | __float_as_uint(p0[32]);
    } else {
        for (int j = 0; j < nrows + 4; ++j, p0 += w.st)
            bits |= __float_as_uint(p0[0]) | __float_as_uint(p0[-4]) | __float_as_uint(p0[4]);
    }
    return !__any_sync(kAll, (bits & 0x7fffffffu) != 0u);
}

// The new level of such a tile, and its stored field (interior tiles).
__device__ __forceinline__ void zero_tile(const Geom &g, const WarpCtx &w, int nrows, bool wide, bool interior)
{
    float *p2 = w.p2 + w.lane, *ps = w.ps + w.lane;
    const int ix = w.ix0 + w.lane;
    const bool store = w.ps && (interior || (w.iz0 >= g.pml && w.iz0 < g.ntz - g.pml && ix >= g.pml && ix < g.ntx - g.pml));
    for (int j = 0; j < nrows; ++j) {
        p2[0] = 0.0f;
        if (wide) p2[32] = 0.0f;
        if (store) {
            __stcs(ps, 0.0f);
            if (wide) __stcs(ps + 32, 0.0f);
        }
        p2 += w.st;
        ps += w.si;
    }
}

// The adjoint's terms of such a tile, rows of columns c0, c0 + 32, .. < c1: zeros,
// but NaN where a stored value is not finite (a forward pass that overflowed).
// s0, s1, s2: null where there is none.  Out of line, so its registers are not the
// sweeps' (inlined, order 8 spilled 20 bytes).  Reading the stored field here
// takes 0.6 % of 80 solves of 200x400; a look at the last forward level instead
// costs the forward kernel spills, 1.5 %.
static __device__ __noinline__ void zero_terms(const float *s0, const float *s1, const float *s2, float *G, int si,
                                               int nrows, int c0, int c1)
{
    for (int j = 0; j < nrows; ++j) {
        const int o = j * si;
        for (int c = c0; c < c1; c += 32) {
            float t = s0 ? fm(__ldcs(s0 + o + c), 0.0f) : 0.0f;
            if (s1) t = ff(__ldcs(s1 + o + c), 0.0f, t);
            if (s2) t = ff(__ldcs(s2 + o + c), 0.0f, t);
            if (!(t == 0.0f)) G[o + c] = t;
        }
    }
}

// One time step of every solve in the wave, one block per (resident slot,
// tile): blockIdx.x = solve, blockIdx.y = tile rank.  The maps view the ring
// as [levels * resident][ntz][pitch].
template <int H, bool ADJ, int R, int MINB>
__global__ void __launch_bounds__(kTileX, MINB)
    k_step(const __grid_constant__ StepMaps maps, const __grid_constant__ Geom g,
           const __grid_constant__ Batch b, const __grid_constant__ StepArgs sa)
{
    // Dynamic shared memory only (no static __shared__), so the tile starts
    // at the 1024-byte aligned base.
    extern __shared__ __align__(1024) float smem[];
    const StepMaps *tile_maps = &maps;
    const Geom *gp = &g;
    const int solve = blockIdx.x, rank = blockIdx.y;
#include "fwi2d_step_tile.inc"
}

// One time step k of the first `nact` pieces of a launch (sorted by nt,
// longest first, so the pieces still running at step k are a prefix):
// block -> piece by binary search of first[], then (solve, tile) as in
// k_step.  All of it comes from the parameter space, as k_step's geometry
// and buffers do: the grid's fields stay constant operands of the sweeps and
// a piece's are constant-bank loads, which nothing the kernel stores can
// alias.  Each piece's time index, snapshot index and Ricker value follow
// from its own nt and nt_interval.
template <int H, bool ADJ, int R, int MINB, int NP>
__global__ void __launch_bounds__(kTileX, MINB)
    k_step_multi(const __grid_constant__ MultiArgsN<NP> a, int nact, int k)
{
    extern __shared__ __align__(1024) float smem[];
    int lo = 0, hi = nact - 1;  // the last piece whose first block is <= blockIdx.x
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (a.first[mid] <= (int)blockIdx.x)
            lo = mid;
        else
            hi = mid - 1;
    }
    const PieceArgs &pc = a.piece[lo];
    Geom g = a.gc;
    g.s_iz = pc.s_iz;
    g.r_iz = pc.r_iz;
    g.r_ix0 = pc.r_ix0;
    g.dr = pc.dr;
    g.nr = pc.nr;
    g.ds = pc.ds;
    g.s_ix0 = pc.s_ix0;
    g.ns = pc.ns;
    g.nt = pc.nt;
    g.nti = pc.nti;
    g.nt_save = pc.nt_save;
    Batch b;
    b.vdt = pc.vdt;
    b.vel = pc.vel;
    b.obs = pc.obs;
    b.syn = pc.syn;
    b.ring = pc.ring;
    b.psave = pc.psave;
    b.gacc = pc.gacc;
    b.coef = a.coef;
    b.blend_fp32 = a.blend_fp32;
    b.status = a.status;
    b.inst0 = pc.inst0;
    b.slot0 = 0;
    b.levels = 3;
    b.tm_slot0 = pc.tm_slot0;
    b.imaging = a.imaging;
    b.store = a.store;
    b.spec = nullptr;
    b.kk = nullptr;
    b.spec_resident = 0;
    b.tl = a.tl;
    b.tl.by_ns = pc.by_ns;
    b.tl.stored = (long long)pc.nt_save * g.pstride;
    const int it = ADJ ? g.nt - 1 - k : k;
    StepArgs sa = ring_step(k, it, ADJ ? -1 : (it % g.nti) == 0 ? it / g.nti : -1, ADJ ? 0.0f : __ldg(pc.rik + it));
    if (ADJ) adjoint_terms(sa, g.nti, k, 0, g.nt - 1, 0);
    const int local = (int)blockIdx.x - pc.first_block;
    const int rank = local / pc.nres;
    const int solve = local - rank * pc.nres;
    const StepMaps *tile_maps = &a.tm;
    const Geom *gp = &a.gc;
#include "fwi2d_step_tile.inc"
}

}  // namespace gbfwi
