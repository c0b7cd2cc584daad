// fwi3d_engine.cu -- the 3-D acoustic FWI engine (C ABI in include/geopvi_fwi3d.h).
//
// The scheme is the 2-D reference solver's algorithm
// (geopvi/forward/fwi2d/fdtd2D_modelling.c) on three axes, stated step by
// step in the header; the CPU oracle (oracle/fwi3d_oracle.cpp) follows the
// same FP32 operations, and this engine reproduces them bit for bit.
//
// Per time step of a wave of resident (sample, shot) solves:
//   k3_step    stencil + the six absorbing passes for every updated cell, source
//              injection, and the stored d2p/dt2 (forward) or the imaging term
//              (adjoint) of the interior cells; blocks of its own sample the
//              receivers of the step before;
//   k3_io_adj  adjoint only: residual injection at the receivers (and their
//              imaging terms).
// k3_step: a block owns 64 x 16 columns -- eight warps, each lane two columns of
// two rows -- and marches along z through a chunk of planes.  These arrive by
// TMA in a ring of shared-memory stages, several planes ahead (mbarriers both
// ways; the warps take turns at issuing): p1 with its x and y halo, and p0 and
// v*dt.  The z windows slide in registers.  The z and y passes are uniform over
// a warp's row; the x pass, which few of a row's cells need, is done afterwards
// by as many lanes as there are strip cells, packed; the y and x passes take p0
// from the stages where its cells lie in the tile.  The rim (cells outside [L, n -
// L)), which the scheme never changes from zero, is not visited: the ring is
// cleared once.  A wave's solves run as two halves on two streams (streams.h).
// Fields are [z][y][x], the first updated column on a 32-byte boundary.  The
// adjoint runs the same operator backwards; its forward field is stored whole
// or, with GB_FWI3D_CHECKPOINT, as ceil(sqrt(nt))-step segments recomputed from
// checkpoints.
//
// What bounds it: instructions (425 / 510 per warp and plane of 128 cells,
// forward / adjoint, of which 68 are the stencil's, two columns at a time;
// schedulers issue on 57 % of their cycles with 16 warps an SM), DRAM at 3 TB/s.
// Measured on 160^3 cells, 4 shots, 200 steps of misfit + gradient: 104 ms with one
// column a thread reading its 16 x and y taps from global memory (219 instructions
// per 32 cells), 87 ms with the planes of p1 staged (two columns a lane, 8 rows),
// 93 ms with two rows a lane and the x pass in place, 79 ms with the x pass packed,
// 73 ms with tiles of interior columns compiled apart, 71.5 ms with packed
// arithmetic, 70.2 ms with p0 from the stages, 53.5 ms as two halves, 52.6 ms with
// chunks for halves.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "../../include/geopvi_fwi2d.h"
#include "../../include/geopvi_fwi3d.h"
#include "fd_weights.cuh"
#include "streams.h"
#include "tma.cuh"

namespace gbfwi3 {

using namespace gbfwi;

constexpr int kBX = 64;          // tile columns (x): one warp, two a lane
constexpr int kBlocksPerSM = 2;  // 128 registers a thread
constexpr int kMisfitBlocks = 64;

struct Geom3 {
    int ntx, nty, ntz, pitch;  // padded grid, x pitch in floats
    int nx, ny, nz;
    int L, pml, pml0;
    int nt, nti, ns, nr, nu;   // nu: distinct receiver cells
    int xoff, ioff, ipitch;    // memory column of x = 0, of interior x = 0, and the interior row pitch
    int tiles_x, tiles_y;
    long long sz;              // z stride (pitch * nty)
    long long fstride;         // floats per padded field
    long long istride;         // floats per interior field (ipitch * ny * nz)
    long long ncell;           // model cells
    float id[3], id2[3];       // 1/d and 1/d^2 for x, y, z
    float idt2, dt;
};

struct Batch3 {
    const float *vdt;   // [nsamples][fstride]  v*dt, padded
    const float *vel;   // [nsamples][ny*nx*nz] model order
    const float *obs;   // [ns][nt][nr]
    float *syn;         // [ninst][nt][nr]
    float *ring;        // [resident][3][fstride]
    float *snap;        // [resident][nsnap][istride]
    float *G;           // [ninst][istride]
    const float *w, *omw;       // [pml0]
    const int *src;             // [ns][3]
    const int *rec;             // [nr][3]
    const int *uoff;            // [nu + 1] receivers of each distinct cell, in receiver order
    const int *uidx;            // [nr]
    int nsnap;                  // stored steps per resident solve
    int inst0;                  // first solve of the wave
    int slot0;                  // resident slot of the launch's first solve
    int *status;                // nonzero: a bounded wait gave up, results are set to NaN
};

// One step: ring buffers (k, k+1, k+2) mod 3 = p0, p1, p2.
struct Step3 {
    int k;
    int snap;    // >= 0: the slot's stored-field index written (forward) or read (adjoint)
    float wav;   // source value (forward)
    int chunks, planes;   // z chunks and planes per chunk
    int sample_it;        // >= 0: sampling blocks record p1 as the data of this time index
    int sample_blocks;    // ... blocks per solve, after the tiles'
};

// Shape of a tile and what k3_step stages of it: kStages planes of p1 with their
// halo, and kPairs planes of p0 and v*dt.  A plane's p0 and v*dt travel with the
// p1 plane H ahead of it, under the same barrier.
template <int H>
struct Stage3 {
    static constexpr int kWarps = H <= 5 ? 8 : 6;  // two blocks' stages fit an SM
    static constexpr int kBY = 2 * kWarps;         // tile rows (y): two a warp
    static constexpr int kHaloX = H <= 4 ? 4 : 8;
    static constexpr int kX = kBX + 2 * kHaloX, kY = kBY + 2 * H;
    static constexpr int kBytes = 4 * kX * kY;
    static constexpr int kPitch = (kBytes + 127) / 128 * 32;  // floats from stage to stage
    static constexpr int kStages = H <= 4 ? H + 5 : 9;
    // A stage is free when the tap plane in it is done with; then so are p0 and
    // v*dt of that plane, kStages - H planes before those that go with the refill.
    static constexpr int kPairs = kStages - H;
    static constexpr int kOwn = kBX * kBY;  // the tile's own cells of a plane
    static constexpr int kPairBase = kStages * kPitch;
    static constexpr int kScratch = kPairBase + kPairs * 2 * kOwn;  // each warp's new values, for the x pass
    static constexpr int kBarriers = kScratch + kWarps * 2 * kBX;
    static constexpr int kSmem = 4 * kBarriers + 16 * kStages;
    static constexpr int kThreads = 32 * kWarps;
};

// Tensor maps: p1's planes with halo and the tile's own cells over a ring, and
// the own cells over v*dt.
struct Maps3 {
    CUtensorMap p1, p0, vdt;
};

__device__ __forceinline__ float fmaf_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// ((a * dt) * dt * v) * v: the injection factor of forward_IO / backward_IO.
__device__ __forceinline__ float inject(float a, float dt, float v)
{
    return __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(a, dt), dt), v), v);
}

// One absorbing blend along a face normal: p1a..p1c = p1 at 0, 1, 2 cells
// inward, p0a..p0e = p0 at 0..4 cells inward; s = v dt / d.
__device__ __forceinline__ float blend(float q, float s, float w, float omw, float p1a, float p1b, float p1c,
                                       float p0a, float p0b, float p0c, float p0d, float p0e)
{
    const float t11 = __fmul_rn(__fmul_rn(__fsub_rn(2.0f, s), __fsub_rn(1.0f, s)), 0.5f);
    const float t12 = __fmul_rn(s, __fsub_rn(2.0f, s));
    const float t13 = __fmul_rn(__fmul_rn(s, __fsub_rn(s, 1.0f)), 0.5f);
    const float k0 = __fmul_rn(2.0f, t11), k1 = __fmul_rn(2.0f, t12), k2 = __fmul_rn(2.0f, t13);
    const float k3 = __fmul_rn(t11, t11), k4 = __fmul_rn(k0, t12);
    const float k5 = fmaf_rn(t12, t12, __fmul_rn(k0, t13));
    const float k6 = __fmul_rn(k1, t13), k7 = __fmul_rn(t13, t13);
    float e = __fmul_rn(k0, p1a);
    e = fmaf_rn(k1, p1b, e);
    e = fmaf_rn(k2, p1c, e);
    e = fmaf_rn(-k3, p0a, e);
    e = fmaf_rn(-k4, p0b, e);
    e = fmaf_rn(-k5, p0c, e);
    e = fmaf_rn(-k6, p0d, e);
    e = fmaf_rn(-k7, p0e, e);
    return fmaf_rn(w, e, __fmul_rn(omw, q));
}

__device__ __forceinline__ long long padded_cell(const Geom3 &g, const int *xyz)
{
    return (long long)(xyz[2] + g.pml) * g.sz + (long long)(xyz[1] + g.pml) * g.pitch + (xyz[0] + g.pml + g.xoff);
}

__device__ __forceinline__ long long interior_cell(const Geom3 &g, const int *xyz)
{
    return ((long long)xyz[2] * g.ny + xyz[1]) * g.ipitch + xyz[0] + g.ioff;
}

__device__ __forceinline__ float model_velocity(const Geom3 &g, const float *vel, const int *xyz)
{
    return vel[((long long)xyz[1] * g.nx + xyz[0]) * g.nz + xyz[2]];
}

// Two neighbouring columns' values in one register pair, and the packed
// arithmetic on them: each half rounds as the scalar instruction does.
typedef unsigned long long Pair;

__device__ __forceinline__ Pair pair(float a, float b)
{
    Pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 split2(Pair p)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
    return r;
}
__device__ __forceinline__ Pair both(float a) { return pair(a, a); }
__device__ __forceinline__ Pair add2(Pair a, Pair b)
{
    Pair r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ Pair mul2(Pair a, Pair b)
{
    Pair r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c)
{
    Pair r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ Pair shared_pair(const float *p) { return *reinterpret_cast<const Pair *>(p); }

// The two cells' new level before the absorbing passes from their taps: y[m]
// and z[m] m cells away, x[k] the columns 2 k and 2 k + 1 from the first cell
// on; u = 2 p1 - p0.
template <int H>
__device__ __forceinline__ float2 update3(const Geom3 &g, const Pair *x, const Pair *y, const Pair *z, float2 p0c,
                                          Pair vd, float2 *u)
{
    const Pair pc = z[0];
    Pair lx = mul2(both(fd_weight<H>(0)), pc), ly = lx, lz = lx;
#pragma unroll
    for (int m = 1; m <= H; ++m) {
        const Pair w = both(fd_weight<H>(m));
        Pair sx;
        if (m % 2 == 0) {
            sx = add2(x[m / 2], x[-m / 2]);
        } else {
            const float2 r0 = split2(x[m / 2]), r1 = split2(x[m / 2 + 1]), l1 = split2(x[-m / 2 - 1]),
                         l0 = split2(x[-(m / 2)]);
            sx = pair(__fadd_rn(r0.y, l1.y), __fadd_rn(r1.x, l0.x));
        }
        lx = fma2(w, sx, lx);
        ly = fma2(w, add2(y[m], y[-m]), ly);
        lz = fma2(w, add2(z[m], z[-m]), lz);
    }
    Pair t = mul2(lz, both(g.id2[2]));
    t = fma2(ly, both(g.id2[1]), t);
    t = fma2(lx, both(g.id2[0]), t);
    const float2 c = split2(pc);
    *u = make_float2(fmaf_rn(2.0f, c.x, -p0c.x), fmaf_rn(2.0f, c.y, -p0c.y));
    return split2(fma2(mul2(vd, vd), t, pair(u->x, u->y)));
}

// p0 at 0 to 4 cells inward of a cell.
struct Inward {
    float p[5];
};
__device__ __forceinline__ Inward inward_global(const float *p0, float p0c, long long d)
{
    return Inward{{p0c, __ldg(p0 + d), __ldg(p0 + 2 * d), __ldg(p0 + 3 * d), __ldg(p0 + 4 * d)}};
}
__device__ __forceinline__ Inward inward_shared(const float *p0, int d)
{
    return Inward{{p0[0], p0[d], p0[2 * d], p0[3 * d], p0[4 * d]}};
}

// One face's blend of a cell along an axis: x1 and x2 are p1 at 1 and 2 cells
// inward, wi the weight index.
__device__ __forceinline__ float face(const Batch3 &b, float q, float s, int wi, float pc, float x1, float x2,
                                      const Inward &p0)
{
    return blend(q, s, __ldg(b.w + wi), __ldg(b.omw + wi), pc, x1, x2, p0.p[0], p0.p[1], p0.p[2], p0.p[3], p0.p[4]);
}

// Receivers of one resident solve: p1 (the level of time index it) into syn.  The
// launch before wrote that level, so its loads are coherent ones, after the wait.
__device__ __forceinline__ void sample3(const Geom3 &g, const Batch3 &b, const float *p, int inst, int it, int first,
                                        int stride)
{
    float *out = b.syn + ((long long)inst * g.nt + it) * g.nr;
    for (int r = first; r < g.nr; r += stride) out[r] = p[padded_cell(g, b.rec + 3 * r)];
}

__device__ __forceinline__ float2 shared2(const float *p) { return *reinterpret_cast<const float2 *>(p); }

// Two columns' store, whole or (EDGE) what is valid of it; STREAM: written once,
// read much later.
template <bool EDGE, bool STREAM>
__device__ __forceinline__ void store2(float *p, float u, float v, bool a, bool b)
{
    if (!EDGE) {
        const float2 t = make_float2(u, v);
        if (STREAM) __stcs(reinterpret_cast<float2 *>(p), t);
        else *reinterpret_cast<float2 *>(p) = t;
        return;
    }
    if (a) p[0] = u;
    if (b) p[1] = v;
}

// A tile of one step: planes z0..z1-1 of the rows and columns from y0, x0 on.
// Without EDGE its columns are all interior.
template <int H, bool ADJ, bool EDGE>
__device__ __forceinline__ void march3(const Maps3 &tm, const Geom3 &g, const Batch3 &b, const Step3 &sa, float *smem,
                                       int x0, int y0, int z0, int z1)
{
    using ST = Stage3<H>;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + ST::kBarriers), *empty = full + ST::kStages;
    const int slot = b.slot0 + blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int inst = b.inst0 + slot;
    const int sample = inst / g.ns, shot = inst - sample * g.ns;
    float *ring = b.ring + (long long)slot * 3 * g.fstride;
    const int L = g.L;
    if (threadIdx.x == 0) {
        for (int i = 0; i < ST::kStages; ++i) {
            mbar_init(full + i, 1);
            mbar_init(empty + i, ST::kWarps);
        }
        fence_barrier_init();
    }
    __syncthreads();

    // This lane's columns x, x + 1 of the rows y, y + 1.
    const int x = x0 + 2 * lane, y = y0 + 2 * warp;
    const bool ia = !EDGE || (x >= g.pml && x < g.ntx - g.pml);
    const bool ib = !EDGE || (x + 1 >= g.pml && x + 1 < g.ntx - g.pml);
    // Columns of the tile in the left and in the right strip: [L, pml) and
    // [ntx - pml, ntx - L) cut to it.
    const int xe = min(x0 + kBX, g.ntx - L), lx1 = min(xe, g.pml), rx0 = max(x0, g.ntx - g.pml);
    const int nl = max(0, lx1 - x0), nx = nl + max(0, xe - rx0);
    // Every p0 that the strips' cells read lies in the tile.
    const bool strips_in = (nl == 0 || lx1 + 4 <= x0 + kBX) && (xe <= rx0 || rx0 - 4 >= x0);
    float *scratch = smem + ST::kScratch + warp * 2 * kBX;
    bool row[2], yin[2];  // updated, interior
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        row[r] = y + r < g.nty - L;
        yin[r] = row[r] && y + r >= g.pml && y + r < g.nty - g.pml;
    }
    const bool yl = y < g.nty / 2;
    const int *src = b.src + 3 * shot;
    const int sy = ADJ ? -1 : __ldg(src + 1) + g.pml;
    const int sz = ADJ || (y != sy && y + 1 != sy) ? -1 : __ldg(src + 2) + g.pml;  // the source's plane, if in these rows

    // Everything above reads only what is constant through the call; the
    // previous step must be complete below.
    grid_dependency_wait();
    grid_launch_dependents();
    bool ok = true;  // no wait has given up
    // Plane i of the chunk, z0 - H + i, into its stage once every warp has
    // released the one before.
    const int nplanes = z1 - z0 + 2 * H;
    auto issue = [&](int i) {
        const int st = i % ST::kStages, use = i / ST::kStages;
        if (use > 0) ok = ok && mbar_wait_bounded(empty + st, (use - 1) & 1);
        if (!ok) return;
        mbar_arrive_expect_tx(full + st, ST::kBytes + (i >= 2 * H ? 8 * ST::kOwn : 0));
        tma_load_4d(smem + st * ST::kPitch, &tm.p1, full + st, x0 + g.xoff - ST::kHaloX, y0 - H, z0 - H + i,
                    slot * 3 + (sa.k + 1) % 3);
        if (i >= 2 * H) {  // the last p1 plane of plane z0 + i - 2H, which goes with it
            const int n = i - 2 * H;
            float *pair = smem + ST::kPairBase + n % ST::kPairs * 2 * ST::kOwn;
            tma_load_4d(pair, &tm.p0, full + st, x0 + g.xoff, y0, z0 + n, slot * 3 + sa.k % 3);
            tma_load_4d(pair + ST::kOwn, &tm.vdt, full + st, x0 + g.xoff, y0, z0 + n, sample);
        }
    };
    if (threadIdx.x == 0)
        for (int i = 0; i < min(ST::kStages, nplanes); ++i) issue(i);

    const long long col = z0 * g.sz + (long long)y * g.pitch + x + g.xoff;
    float *p2 = ring + (long long)((sa.k + 2) % 3) * g.fstride + col;
    const float *p0 = ring + (long long)(sa.k % 3) * g.fstride + col;
    const long long ps = (long long)g.ipitch * g.ny;  // interior plane stride
    float *sv = nullptr, *Gv = nullptr;
    if (sa.snap >= 0) {
        const long long j0 = ((long long)(z0 - g.pml) * g.ny + (y - g.pml)) * g.ipitch + (x - g.pml + g.ioff);
        sv = b.snap + ((long long)slot * b.nsnap + sa.snap) * g.istride + j0;
        if (ADJ) Gv = b.G + (long long)inst * g.istride + j0;
    }
    const int mine = (2 * warp + H) * ST::kX + ST::kHaloX + 2 * lane;  // this lane's place in a staged plane

    // The z windows: w[r][H + m] = plane z + m of row r's two columns.  The
    // chunk's first 2H planes only fill them; the first H of those are then free.
    Pair w[2][2 * H + 1];
#pragma unroll
    for (int i = 0; i < 2 * H; ++i) {
        // planes beyond the first kStages: one for every stage freed two steps ago
        if (i >= 2 && i < H + 2 && threadIdx.x == 0 && i - 2 + ST::kStages < nplanes) issue(i - 2 + ST::kStages);
        ok = __all_sync(0xffffffffu, ok && mbar_wait_bounded(full + i % ST::kStages, (i / ST::kStages) & 1));
#pragma unroll
        for (int r = 0; r < 2; ++r) w[r][i] = shared_pair(smem + i % ST::kStages * ST::kPitch + mine + r * ST::kX);
        if (i < H) {
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + i % ST::kStages);
        }
    }
    // Issued so far: kStages, and one for each i above.
    constexpr int kAhead = ST::kStages + (2 * H < H + 2 ? 2 * H : H + 2) - 2;
    int tap = H % ST::kStages, front = 2 * H % ST::kStages;  // stages of plane z and of plane z + H
    int front_phase = (2 * H / ST::kStages) & 1;
    int pair0 = ST::kPairBase;                               // p0 and v*dt of plane z
    // Adjoint stored step: the stored field and the accumulator, one plane ahead.
    float2 svn[2], gvn[2];
    auto load_terms = [&](int z, const float *s, const float *G) {
        if (ADJ && sv && (ia || ib) && z >= g.pml && z < g.ntz - g.pml) {
#pragma unroll
            for (int r = 0; r < 2; ++r)
                if (yin[r]) {
                    svn[r] = __ldcs(reinterpret_cast<const float2 *>(s + r * g.ipitch));
                    gvn[r] = *reinterpret_cast<const float2 *>(G + r * g.ipitch);
                }
        }
    };
    load_terms(z0, sv, Gv);
#pragma unroll 1
    for (int z = z0; z < z1 && ok; ++z) {
        // One more plane, into the stage that every warp released two planes ago.
        const int next = z - z0 + H - 2 + ST::kStages;
        if (lane == 0 && warp == (z - z0) % ST::kWarps && next >= kAhead && next < nplanes) issue(next);
        const bool zin = z >= g.pml && z < g.ntz - g.pml;
        const bool stored = sv && zin;
        float2 svc[2], gvc[2];
        if (ADJ) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                svc[r] = svn[r];
                gvc[r] = gvn[r];
            }
            if (z + 1 < z1) load_terms(z + 1, sv + ps, Gv + ps);
        }
        ok = ok && mbar_wait_bounded(full + front, front_phase);
        const float *pl = smem + tap * ST::kPitch + mine, *pf = smem + front * ST::kPitch + mine;
#pragma unroll
        for (int r = 0; r < 2; ++r) w[r][2 * H] = shared_pair(pf + r * ST::kX);
        // The columns' y neighbours: rows -H .. H + 1, the lane's own two at H, H + 1.
        Pair yt[2 * H + 2];
#pragma unroll
        for (int m = 0; m < 2 * H + 2; ++m)
            yt[m] = m == H || m == H + 1 ? w[m - H][H] : shared_pair(pl + (m - H) * ST::kX);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            constexpr int K = (H + 1) / 2;  // pairs on each side that hold the x taps
            Pair xt[2 * K + 1];
#pragma unroll
            for (int k = -K; k <= K; ++k) xt[K + k] = k == 0 ? w[r][H] : shared_pair(pl + r * ST::kX + 2 * k);
            const float *own = smem + pair0 + (2 * warp + r) * kBX + 2 * lane;
            const float2 p0c = shared2(own);
            const Pair vp = shared_pair(own + ST::kOwn);
            float2 u;
            const float2 q2 = update3<H>(g, xt + K, yt + H + r, w[r] + H, p0c, vp, &u);
            float qa = q2.x, qb = q2.y;
            if (row[r]) {
                // The absorbing passes: z, then y, then x (at most one face each)
                const float *p0r = p0 + r * g.pitch;
                const float2 pc = split2(w[r][H]), vd = split2(vp);
                if (!zin) {
                    const bool zl = z < g.pml;
                    const int wi = zl ? z - L : g.ntz - L - 1 - z;
                    const long long d = zl ? g.sz : -g.sz;
                    const float2 n1 = split2(zl ? w[r][H + 1] : w[r][H - 1]), n2 = split2(zl ? w[r][H + 2] : w[r][H - 2]);
                    qa = face(b, qa, __fmul_rn(vd.x, g.id[2]), wi, pc.x, n1.x, n2.x, inward_global(p0r, p0c.x, d));
                    qb = face(b, qb, __fmul_rn(vd.y, g.id[2]), wi, pc.y, n1.y, n2.y, inward_global(p0r + 1, p0c.y, d));
                }
                if (!yin[r]) {
                    const int wi = yl ? y + r - L : g.nty - L - 1 - y - r;
                    const int rr = 2 * warp + r, d = yl ? kBX : -kBX;
                    Inward ea, eb;
                    if (yl ? rr + 4 < ST::kBY : rr >= 4) {  // in the tile: staged
                        ea = inward_shared(own, d);
                        eb = inward_shared(own + 1, d);
                    } else {
                        const long long dg = yl ? g.pitch : -g.pitch;
                        ea = inward_global(p0r, p0c.x, dg);
                        eb = inward_global(p0r + 1, p0c.y, dg);
                    }
                    const float2 n1 = split2(yl ? yt[H + r + 1] : yt[H + r - 1]),
                                 n2 = split2(yl ? yt[H + r + 2] : yt[H + r - 2]);
                    qa = face(b, qa, __fmul_rn(vd.x, g.id[1]), wi, pc.x, n1.x, n2.x, ea);
                    qb = face(b, qb, __fmul_rn(vd.y, g.id[1]), wi, pc.y, n1.y, n2.y, eb);
                }
                if (!ADJ && z == sz && y + r == sy) {  // forward_IO's injection at the shot's cell
                    const int sx = __ldg(src) + g.pml;
                    const float inj = inject(sa.wav, g.dt, model_velocity(g, b.vel + (long long)sample * g.ncell, src));
                    if (x == sx) qa = __fadd_rn(qa, inj);
                    if (x + 1 == sx) qb = __fadd_rn(qb, inj);
                }
                store2<EDGE, false>(p2 + r * g.pitch, qa, qb, ia, ib);
                if (EDGE) *reinterpret_cast<float2 *>(scratch + r * kBX + 2 * lane) = make_float2(qa, qb);
                if (stored && yin[r]) {
                    if (ADJ)
                        store2<EDGE, false>(Gv + r * g.ipitch, fmaf_rn(svc[r].x, qa, gvc[r].x),
                                            fmaf_rn(svc[r].y, qb, gvc[r].y), ia, ib);
                    else
                        store2<EDGE, true>(sv + r * g.ipitch, __fmul_rn(__fsub_rn(qa, u.x), g.idt2),
                                           __fmul_rn(__fsub_rn(qb, u.y), g.idt2), ia, ib);
                }
            }
        }
        if (EDGE) {  // the x pass on the warp's strip cells, one a lane
            __syncwarp();
            for (int i = lane; i < 2 * nx; i += 32) {
                const int r = i >= nx, c = i - r * nx;
                const int xc = c < nl ? x0 + c : rx0 + c - nl, at = xc - x0, d = c < nl ? 1 : -1;
                if (y + r >= g.nty - L) break;
                const float *p1c = smem + tap * ST::kPitch + (2 * warp + r + H) * ST::kX + ST::kHaloX + at;
                const float *own = smem + pair0 + (2 * warp + r) * kBX + at;
                const float q = face(b, scratch[r * kBX + at], __fmul_rn(own[ST::kOwn], g.id[0]),
                                     c < nl ? xc - L : g.ntx - L - 1 - xc, p1c[0], p1c[d], p1c[2 * d],
                                     strips_in ? inward_shared(own, d)
                                               : inward_global(p0 + r * g.pitch + (xc - x), own[0], d));
                p2[r * g.pitch + (xc - x)] = q;
            }
        }
        ok = __all_sync(0xffffffffu, ok);
        // Every lane's reads of the stages, and of scratch, before lane 0's release
        // (and the next plane's scratch).
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + tap);
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int m = 0; m < 2 * H; ++m) w[r][m] = w[r][m + 1];
        pair0 += 2 * ST::kOwn;
        if (pair0 == ST::kScratch) pair0 = ST::kPairBase;
        p0 += g.sz;
        p2 += g.sz;
        if (sv) sv += ps;
        if (ADJ && Gv) Gv += ps;
        if (++tap == ST::kStages) tap = 0;
        if (++front == ST::kStages) {
            front = 0;
            front_phase ^= 1;
        }
    }
    if (!ok) {  // a wait gave up: record it, and let copies in flight land before the block retires
        if (lane == 0) atomicOr(b.status, 1);
        for (int i = 0; i < ST::kStages; ++i) mbar_wait_bounded(full + i, 0);
        for (int i = 0; i < ST::kStages; ++i) mbar_wait_bounded(full + i, 1);
    }
}

// One time step of every resident solve.  blockIdx.x = tile (x fastest, then
// y, then z chunk), then the sampling blocks; blockIdx.y = resident slot.  The
// maps view the ring as [3 * resident][z][y][x].
template <int H, bool ADJ>
__global__ void __launch_bounds__(Stage3<H>::kThreads, kBlocksPerSM)
    k3_step(const __grid_constant__ Maps3 tm, const __grid_constant__ Geom3 g, const __grid_constant__ Batch3 b,
            const __grid_constant__ Step3 sa)
{
    extern __shared__ __align__(1024) float smem[];
    const int tiles = g.tiles_x * g.tiles_y;
    int t = blockIdx.x;
    if (!ADJ && t >= tiles * sa.chunks) {
        grid_dependency_wait();
        grid_launch_dependents();
        const int slot = b.slot0 + blockIdx.y;
        sample3(g, b, b.ring + ((long long)slot * 3 + (sa.k + 1) % 3) * g.fstride, b.inst0 + slot, sa.sample_it,
                (t - tiles * sa.chunks) * blockDim.x + threadIdx.x, sa.sample_blocks * blockDim.x);
        return;
    }
    const int tx = t % g.tiles_x;
    t /= g.tiles_x;
    const int ty = t % g.tiles_y, cz = t / g.tiles_y;
    const int x0 = g.L + tx * kBX, y0 = g.L + ty * Stage3<H>::kBY;
    const int z0 = g.L + cz * sa.planes, z1 = min(z0 + sa.planes, g.ntz - g.L);
    if (x0 >= g.pml && x0 + kBX <= g.ntx - g.pml)
        march3<H, ADJ, false>(tm, g, b, sa, smem, x0, y0, z0, z1);
    else
        march3<H, ADJ, true>(tm, g, b, sa, smem, x0, y0, z0, z1);
}

// The receivers of the last step, time index it, in p (ring level `level`).
__global__ void k3_sample(const Geom3 g, const Batch3 b, int level, int it)
{
    const int slot = b.slot0 + blockIdx.y;
    grid_dependency_wait();
    sample3(g, b, b.ring + ((long long)slot * 3 + level) * g.fstride, b.inst0 + slot, it,
            blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// Adjoint IO of step k (time it): residual injection (syn - obs, the
// transpose of receiver sampling), receiver by receiver in receiver order per
// cell, with each injection's imaging term.
__global__ void k3_io_adj(const Geom3 g, const Batch3 b, int k, int it, int snap)
{
    const int slot = b.slot0 + blockIdx.y;
    const int inst = b.inst0 + slot;
    const int sample = inst / g.ns, shot = inst - sample * g.ns;
    grid_dependency_wait();
    grid_launch_dependents();
    float *p2 = b.ring + (long long)slot * 3 * g.fstride + (long long)((k + 2) % 3) * g.fstride;
    const float *syn = b.syn + ((long long)inst * g.nt + it) * g.nr;
    const float *obs = b.obs + ((long long)shot * g.nt + it) * g.nr;
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < g.nu; u += gridDim.x * blockDim.x) {
        const int r0 = b.uoff[u], r1 = b.uoff[u + 1];
        const int *xyz = b.rec + 3 * b.uidx[r0];
        const long long c = padded_cell(g, xyz);
        const long long j = interior_cell(g, xyz);
        float q = p2[c];
        float *Gc = b.G + (long long)inst * g.istride + j;
        const float sv = snap >= 0 ? b.snap[((long long)slot * b.nsnap + snap) * g.istride + j] : 0.0f;
        float gacc = snap >= 0 ? *Gc : 0.0f;
        for (int i = r0; i < r1; ++i) {
            const int r = b.uidx[i];
            const float inj = __fsub_rn(syn[r], obs[r]);
            q = __fadd_rn(q, inj);
            if (snap >= 0) gacc = fmaf_rn(sv, inj, gacc);
        }
        p2[c] = q;
        if (snap >= 0) *Gc = gacc;
    }
}

// Padded v*dt per sample (get_velp's edge replication is a clamp).
__global__ void k3_prepare(const Geom3 g, const float *__restrict__ vel, float *__restrict__ vdt, int nsamples)
{
    const long long total = (long long)nsamples * g.fstride;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int s = (int)(e / g.fstride);
        const long long r = e - (long long)s * g.fstride;
        const int z = (int)(r / g.sz);
        const long long rz = r - (long long)z * g.sz;
        const int y = (int)(rz / g.pitch), x = (int)(rz - (long long)y * g.pitch) - g.xoff;
        float v = 0.0f;
        if (x >= 0 && x < g.ntx) {
            const int jx = min(max(x - g.pml, 0), g.nx - 1);
            const int jy = min(max(y - g.pml, 0), g.ny - 1);
            const int jz = min(max(z - g.pml, 0), g.nz - 1);
            v = __fmul_rn(vel[(long long)s * g.ncell + ((long long)jy * g.nx + jx) * g.nz + jz], g.dt);
        }
        vdt[e] = v;
    }
}

// grad (model order) = 2 nt_interval dt^2 / v * sum over shots (in shot order,
// FP64): with P^{k+1} = 2P^k - P^{k-1} + v^2 dt^2 (lap P^k + f), dP^{k+1}/dv =
// (2/v)(P^{k+1} - 2P^k + P^{k-1}) = (2/v) dt^2 * (stored d2p/dt2).
__global__ void k3_reduce_grad(const Geom3 g, const float *__restrict__ G, const float *__restrict__ vel,
                               float *__restrict__ grad, int nsamples, const int *status)
{
    const long long cells = g.ncell;
    const long long total = (long long)nsamples * cells;
    const double coef = 2.0 * ((double)g.nti * (double)g.dt * (double)g.dt);
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int s = (int)(e / cells);
        const long long m = e - (long long)s * cells;
        const int iz = (int)(m % g.nz);
        const long long r = m / g.nz;
        const int ix = (int)(r % g.nx), iy = (int)(r / g.nx);
        const long long j = ((long long)iz * g.ny + iy) * g.ipitch + ix + g.ioff;
        double acc = 0.0;
        for (int shot = 0; shot < g.ns; ++shot) acc += (double)G[((long long)s * g.ns + shot) * g.istride + j];
        const double v = (double)vel[e];
        grad[e] = *status ? __int_as_float(0x7fffffff) : (float)(coef * acc / v);
    }
}

__global__ void k3_misfit_partial(const float *__restrict__ syn, const float *__restrict__ obs, long long per_sample,
                                  long long obs_len, double *__restrict__ part)
{
    const int s = blockIdx.y;
    double acc = 0.0;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < per_sample;
         e += (long long)gridDim.x * blockDim.x) {
        const double r = (double)syn[(long long)s * per_sample + e] - (double)obs[e % obs_len];
        acc += r * r;
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    __shared__ double red[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) red[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        part[(long long)s * gridDim.x + blockIdx.x] = t;
    }
}

__global__ void k3_misfit_final(const double *__restrict__ part, double *__restrict__ misfit, int nsamples,
                                const int *status)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsamples) return;
    double t = 0.0;
    for (int i = 0; i < kMisfitBlocks; ++i) t += part[(long long)s * kMisfitBlocks + i];
    misfit[s] = *status ? (double)__int_as_float(0x7fffffff) : 0.5 * t;
}

// The caller's data after a wait that gave up.
__global__ void k3_data_lost(float *__restrict__ syn, long long n, const int *status)
{
    if (*status == 0) return;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        syn[e] = __int_as_float(0x7fffffff);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

struct Host3 {
    Geom3 g;
    std::vector<float> w, omw;
    std::vector<int> uoff, uidx;
};

static int round_up(int v, int m) { return (v + m - 1) / m * m; }
static long long round_up64(long long v, long long m) { return (v + m - 1) / m * m; }

static int validate(const gb_fwi3d_params *p, const gb_fwi3d_acq *a)
{
    if (!p || !a || !a->src || !a->rec || !a->wavelet) return GB_FWI2D_EINVAL;
    if (p->nx < 1 || p->ny < 1 || p->nz < 1 || p->pml0 < 1 || p->Lc < 3 || p->Lc > 6 || p->ns < 1 ||
        p->nr < 1 || p->nt < 1 || p->nt_interval < 1)
        return GB_FWI2D_EINVAL;
    if (!(p->dx > 0) || !(p->dy > 0) || !(p->dz > 0) || !(p->dt > 0) || !std::isfinite(p->dx) ||
        !std::isfinite(p->dy) || !std::isfinite(p->dz) || !std::isfinite(p->dt))
        return GB_FWI2D_EINVAL;
    const long long pml = (long long)p->pml0 + p->Lc + 1;
    if (p->nx + 2 * pml > (1 << 20) || p->ny + 2 * pml > (1 << 20) || p->nz + 2 * pml > (1 << 20))
        return GB_FWI2D_EINVAL;
    for (int s = 0; s < p->ns; ++s) {
        const int *c = a->src + 3 * s;
        if (c[0] < 0 || c[0] >= p->nx || c[1] < 0 || c[1] >= p->ny || c[2] < 0 || c[2] >= p->nz)
            return GB_FWI2D_EINVAL;
    }
    for (int r = 0; r < p->nr; ++r) {
        const int *c = a->rec + 3 * r;
        if (c[0] < 0 || c[0] >= p->nx || c[1] < 0 || c[1] >= p->ny || c[2] < 0 || c[2] >= p->nz)
            return GB_FWI2D_EINVAL;
    }
    for (int it = 0; it < p->nt; ++it)
        if (!std::isfinite(a->wavelet[it])) return GB_FWI2D_EINVAL;
    return GB_FWI2D_OK;
}

static void derive(const gb_fwi3d_params &p, const gb_fwi3d_acq &a, Host3 &h)
{
    Geom3 &g = h.g;
    std::memset(&g, 0, sizeof g);
    g.L = p.Lc + 1;
    g.pml0 = p.pml0;
    g.pml = p.pml0 + g.L;
    g.nx = p.nx; g.ny = p.ny; g.nz = p.nz;
    g.ntx = p.nx + 2 * g.pml; g.nty = p.ny + 2 * g.pml; g.ntz = p.nz + 2 * g.pml;
    // Column L, where the tiles start, on a 32-byte boundary (a TMA box starts on
    // a 16-byte one); interior arrays share the alignment, so a lane's two
    // columns are one 8-byte access in both.
    g.xoff = round_up(g.L, 8) - g.L;
    g.pitch = round_up(g.xoff + g.ntx, 8);
    g.sz = (long long)g.pitch * g.nty;
    g.fstride = round_up64(g.sz * g.ntz, 64);
    g.ioff = (g.xoff + g.pml) % 8;
    g.ipitch = round_up(g.ioff + p.nx, 8);
    g.istride = (long long)g.ipitch * p.ny * p.nz;
    g.ncell = (long long)p.nx * p.ny * p.nz;
    g.nt = p.nt; g.nti = p.nt_interval; g.ns = p.ns; g.nr = p.nr;
    g.tiles_x = (g.ntx - 2 * g.L + kBX - 1) / kBX;
    const int by = g.L - 1 <= 5 ? 16 : 12;  // Stage3::kBY
    g.tiles_y = (g.nty - 2 * g.L + by - 1) / by;
    const double d[3] = {p.dx, p.dy, p.dz};
    for (int i = 0; i < 3; ++i) {
        g.id[i] = (float)(1.0 / d[i]);
        g.id2[i] = (float)(1.0 / (d[i] * d[i]));
    }
    g.idt2 = (float)(1.0 / ((double)p.dt * (double)p.dt));
    g.dt = p.dt;
    h.w.resize(p.pml0);
    h.omw.resize(p.pml0);
    for (int i = 0; i < p.pml0; ++i) {
        h.w[i] = (float)(1.0 - (double)i / p.pml0);
        h.omw[i] = (float)(1.0 - (double)h.w[i]);
    }
    // receivers grouped by cell, each group in receiver order
    std::vector<std::pair<long long, int>> rc(p.nr);
    for (int r = 0; r < p.nr; ++r) {
        const int *c = a.rec + 3 * r;
        rc[r] = {((long long)c[2] * p.ny + c[1]) * p.nx + c[0], r};
    }
    std::stable_sort(rc.begin(), rc.end(), [](const auto &u, const auto &v) { return u.first < v.first; });
    h.uoff.clear();
    h.uidx.resize(p.nr);
    for (int i = 0; i < p.nr; ++i) {
        if (i == 0 || rc[i].first != rc[i - 1].first) h.uoff.push_back(i);
        h.uidx[i] = rc[i].second;
    }
    h.uoff.push_back(p.nr);
    g.nu = (int)h.uoff.size() - 1;
}

struct Layout3 {
    size_t status, tab_src, tab_rec, tab_uoff, tab_uidx, tab_w, tab_omw;
    size_t vdt, ring, ring2, ckpt, snap, G, syn, part, total;
    int resident, K, nseg, nsnap;
};

static size_t a256(size_t v) { return (v + 255) & ~(size_t)255; }

static Layout3 plan(const Geom3 &g, int nsamples, int resident, bool fwd_only, bool ckpt, bool syn_in_work)
{
    Layout3 L{};
    const long long ninst = (long long)nsamples * g.ns;
    if (resident <= 0 || resident > ninst) resident = (int)ninst;
    resident = std::min(resident, 65535);
    L.resident = resident;
    if (fwd_only) {
        L.K = g.nt;
        L.nseg = 1;
        L.nsnap = 0;
    } else if (ckpt) {
        const int root = (int)std::ceil(std::sqrt((double)g.nt));
        L.K = (root + g.nti - 1) / g.nti * g.nti;
        L.nseg = (g.nt + L.K - 1) / L.K;
        L.nsnap = (L.K + g.nti - 1) / g.nti;
    } else {
        L.K = g.nt;
        L.nseg = 1;
        L.nsnap = (g.nt + g.nti - 1) / g.nti;
    }
    const size_t f = sizeof(float) * (size_t)g.fstride, fi = sizeof(float) * (size_t)g.istride;
    size_t off = 0;
    L.status = off;    off = a256(off + sizeof(int));
    L.tab_src = off;   off = a256(off + sizeof(int) * 3 * g.ns);
    L.tab_rec = off;   off = a256(off + sizeof(int) * 3 * g.nr);
    L.tab_uoff = off;  off = a256(off + sizeof(int) * (g.nr + 1));
    L.tab_uidx = off;  off = a256(off + sizeof(int) * g.nr);
    L.tab_w = off;     off = a256(off + sizeof(float) * g.pml0);
    L.tab_omw = off;   off = a256(off + sizeof(float) * g.pml0);
    L.vdt = off;       off = a256(off + f * nsamples);
    L.ring = off;      off = a256(off + f * 3 * resident);
    L.ring2 = L.ckpt = L.snap = L.G = off;
    if (!fwd_only) {
        L.ring2 = off; off = a256(off + f * 3 * resident);
        L.ckpt = off;
        if (L.nseg > 1) off = a256(off + f * 2 * (size_t)L.nseg * resident);
        L.snap = off;  off = a256(off + fi * (size_t)L.nsnap * resident);
        L.G = off;     off = a256(off + fi * (size_t)ninst);
    }
    L.syn = off;
    if (syn_in_work) off = a256(off + sizeof(float) * (size_t)ninst * g.nt * g.nr);
    L.part = off;      off = a256(off + sizeof(double) * kMisfitBlocks * nsamples);
    L.total = off;
    return L;
}

// A workspace may start anywhere: the layout does at its first multiple of
// kWorkAlign (the tensor maps need 16 bytes), for which its size has room.
constexpr size_t kWorkAlign = 256;
static size_t work_bytes_of(const Layout3 &L) { return L.total + kWorkAlign; }

static thread_local long long t_launches = 0;

static int grid_for(long long n, int block)
{
    return (int)std::min<long long>((n + block - 1) / block, 152LL * 32);
}


// Waves of at least two solves and this much work (tiles times planes of a step)
// run as two halves on two streams, so that one half's blocks fill the SMs that
// the other's last ones leave.  Misfit + gradient, ms, halves / one chain: 8 of
// 150^3 x 100 steps 44.6 / 51.3, 2 of 100^3 5.7 / 7.5, 3 of 60^3 (3000)
// with 12th order 6.7 / 6.1.
constexpr long long kSplitMinWork = 3500;
static bool split_wave(const Geom3 &g, int nres)
{
    return nres >= 2 && (long long)nres * g.tiles_x * g.tiles_y * (g.ntz - 2 * g.L) >= kSplitMinWork;
}

// z chunks of a launch of `nres` solves that has the device's 152 x kBlocksPerSM
// block slots, or half of them.  A chunk re-reads 2H planes and fills its
// pipeline, together worth 2H - 1 planes.  A launch's tiles cost unequal amounts:
// its last wave is about one whole wave too much, and what fits at once lasts as
// long as its slowest tile, 1.7 times the mean.  Misfit + gradient, ms, halves: 4
// of 160^3 x 200 steps in 2 / 4 / 6 / 8 chunks 71.5 / 53.5 / 51.4 / 52.0, 8 of
// 150^3 x 60 in 2 / 4 / 6 29.1 / 26.5 / 26.9, 8 of 60^3 in 2 / 4 / 6 / 8 9.5 / 6.0
// / 5.1 / 5.3; one chain: 8 of 150^3 in 1 / 4 / 6 44.0 / 32.2 / 30.8, one of 220^3
// x 100 in 5 / 12 25.7 / 19.5, 3 of 75 x 110 x 61, checkpointed, in 6 (288 blocks)
// / 7 28.4 / 32.9.
static void plan_chunks(const Geom3 &g, int nres, int H, bool half, Step3 &sa)
{
    const long long slots = 152LL * kBlocksPerSM / (half ? 2 : 1), cols = (long long)g.tiles_x * g.tiles_y * nres;
    const int planes = g.ntz - 2 * g.L;
    long long best = -1;
    for (int c = 1; c <= std::max(1, planes / 8); ++c) {
        const int per = (planes + c - 1) / c, chunks = (planes + per - 1) / per;
        const long long blocks = cols * chunks;
        const long long waves = half ? 20 * (blocks + slots) : blocks <= slots ? 34 * slots : 20 * blocks + 17 * slots;
        const long long cost = waves * (per + 2 * H - 1);
        if (best < 0 || cost < best) {
            best = cost;
            sa.chunks = chunks;
            sa.planes = per;
        }
    }
}

// Launches with programmatic dependent launch where the previous operation on
// the stream is a kernel of the same chain (they wait for it themselves).
template <typename... A>
static void launch(void (*kernel)(A...), dim3 grid, int threads, int smem, cudaStream_t st, bool overlap, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, args...);
    ++t_launches;
}

template <int H>
static void launch_step(bool adj, const Maps3 &tm, const Geom3 &g, const Batch3 &b, int nres, bool half,
                        Step3 sa, cudaStream_t st, bool overlap)
{
    using ST = Stage3<H>;
    static_assert(ST::kBY == (H <= 5 ? 16 : 12), "tiles_y of derive()");
    plan_chunks(g, nres, H, half, sa);
    const dim3 grid(g.tiles_x * g.tiles_y * sa.chunks + sa.sample_blocks, nres);
    if (adj)
        launch(k3_step<H, true>, grid, ST::kThreads, ST::kSmem, st, overlap, tm, g, b, sa);
    else
        launch(k3_step<H, false>, grid, ST::kThreads, ST::kSmem, st, overlap, tm, g, b, sa);
}

static void step(bool adj, const Maps3 &tm, const Geom3 &g, const Batch3 &b, int nres, bool half, const Step3 &sa,
                 cudaStream_t st, bool overlap)
{
    switch (g.L - 1) {
    case 3: launch_step<3>(adj, tm, g, b, nres, half, sa, st, overlap); break;
    case 4: launch_step<4>(adj, tm, g, b, nres, half, sa, st, overlap); break;
    case 5: launch_step<5>(adj, tm, g, b, nres, half, sa, st, overlap); break;
    default: launch_step<6>(adj, tm, g, b, nres, half, sa, st, overlap); break;
    }
}

// k3_step's stages may be more than the default 48 KB of shared memory.
template <int H>
static bool allow_smem()
{
    return cudaFuncSetAttribute(k3_step<H, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Stage3<H>::kSmem) ==
               cudaSuccess &&
           cudaFuncSetAttribute(k3_step<H, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Stage3<H>::kSmem) ==
               cudaSuccess;
}

static bool prepare_device(int H)
{
    switch (H) {
    case 3: return allow_smem<3>();
    case 4: return allow_smem<4>();
    case 5: return allow_smem<5>();
    default: return allow_smem<6>();
    }
}

// A 4-D fp32 tensor map over `depth` fields [depth][z][y][x] with a one-plane
// box; out-of-range elements read as zero.
static bool make_map3(CUtensorMap &m, void *base, const Geom3 &g, long long depth, int box_x, int box_y)
{
    auto enc = tensor_map_encoder();
    if (!enc || !ensure_context()) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)g.pitch, (cuuint64_t)g.nty, (cuuint64_t)g.ntz, (cuuint64_t)depth};
    const cuuint64_t strides[3] = {(cuuint64_t)g.pitch * 4, (cuuint64_t)g.sz * 4, (cuuint64_t)g.fstride * 4};
    const cuuint32_t box[4] = {(cuuint32_t)box_x, (cuuint32_t)box_y, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return enc(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
           CUDA_SUCCESS;
}

static bool make_maps3(Maps3 &m, void *ring, long long fields, void *vdt, int nsamples, const Geom3 &g)
{
    const int H = g.L - 1, halo = H <= 4 ? 4 : 8, by = H <= 5 ? 16 : 12;
    return make_map3(m.p1, ring, g, fields, kBX + 2 * halo, by + 2 * H) && make_map3(m.p0, ring, g, fields, kBX, by) &&
           make_map3(m.vdt, vdt, g, nsamples, kBX, by);
}

}  // namespace gbfwi3

using namespace gbfwi3;

extern "C" {

int gb_fwi3d_validate(const gb_fwi3d_params *p, const gb_fwi3d_acq *a) { return validate(p, a); }

int gb_fwi3d_workspace_size(const gb_fwi3d_params *p, const gb_fwi3d_acq *a, int nsamples, int max_resident,
                            unsigned flags, size_t *bytes)
{
    if (!bytes || nsamples < 1) return GB_FWI2D_EINVAL;
    const int st = validate(p, a);
    if (st) return st;
    Host3 h;
    derive(*p, *a, h);
    *bytes = work_bytes_of(plan(h.g, nsamples, max_resident, (flags & GB_FWI3D_FORWARD_ONLY) != 0,
                                (flags & GB_FWI3D_CHECKPOINT) != 0, true));
    return GB_FWI2D_OK;
}

int gb_fwi3d_max_resident(const gb_fwi3d_params *p, const gb_fwi3d_acq *a, int nsamples, unsigned flags,
                          size_t budget)
{
    if (nsamples < 1 || validate(p, a)) return 0;
    Host3 h;
    derive(*p, *a, h);
    const bool fo = (flags & GB_FWI3D_FORWARD_ONLY) != 0, ck = (flags & GB_FWI3D_CHECKPOINT) != 0;
    long long lo = 0, hi = std::min<long long>((long long)nsamples * p->ns, 65535);
    while (lo < hi) {
        const long long mid = (lo + hi + 1) / 2;
        if (work_bytes_of(plan(h.g, nsamples, (int)mid, fo, ck, true)) <= budget)
            lo = mid;
        else
            hi = mid - 1;
    }
    return (int)lo;
}

long long gb_fwi3d_last_launches(void) { return t_launches; }

int gb_fwi3d_run(const gb_fwi3d_params *p, const gb_fwi3d_acq *a, int nsamples, const float *vel, const float *obs,
                 float *syn, float *grad, double *misfit, void *work, size_t work_bytes, int max_resident,
                 unsigned flags, void *stream)
{
    t_launches = 0;
    if (nsamples < 1 || !vel || !work) return GB_FWI2D_EINVAL;
    int st0 = validate(p, a);
    if (st0) return st0;
    const bool fwd_only = (flags & GB_FWI3D_FORWARD_ONLY) != 0;
    const bool ckpt = (flags & GB_FWI3D_CHECKPOINT) != 0;
    if (!fwd_only && (!obs || !grad)) return GB_FWI2D_EINVAL;
    if (misfit && !obs) return GB_FWI2D_EINVAL;
    Host3 h;
    derive(*p, *a, h);
    const Geom3 &g = h.g;
    const Layout3 L = plan(g, nsamples, max_resident, fwd_only, ckpt, syn == nullptr);
    char *w = (char *)a256((size_t)work);
    if (L.total + (size_t)(w - (char *)work) > work_bytes) return GB_FWI2D_ENOMEM;
    cudaStream_t st = (cudaStream_t)stream;
    Maps3 tm, tm_adj;
    auto maps = [&](Maps3 &m, size_t ring) { return make_maps3(m, w + ring, 3LL * L.resident, w + L.vdt, nsamples, g); };
    if (!prepare_device(g.L - 1) || !maps(tm, L.ring)) return GB_FWI2D_ECUDA;
    if (!fwd_only && !maps(tm_adj, L.ring2)) return GB_FWI2D_ECUDA;
    cudaMemsetAsync(w + L.status, 0, sizeof(int), st);
    auto up = [&](size_t off, const void *src, size_t n) {
        if (n) cudaMemcpyAsync(w + off, src, n, cudaMemcpyHostToDevice, st);
    };
    up(L.tab_src, a->src, sizeof(int) * 3 * g.ns);
    up(L.tab_rec, a->rec, sizeof(int) * 3 * g.nr);
    up(L.tab_uoff, h.uoff.data(), sizeof(int) * h.uoff.size());
    up(L.tab_uidx, h.uidx.data(), sizeof(int) * h.uidx.size());
    up(L.tab_w, h.w.data(), sizeof(float) * h.w.size());
    up(L.tab_omw, h.omw.data(), sizeof(float) * h.omw.size());

    const long long ninst = (long long)nsamples * g.ns;
    Batch3 b{};
    b.vdt = (float *)(w + L.vdt);
    b.vel = vel;
    b.obs = obs;
    b.syn = syn ? syn : (float *)(w + L.syn);
    b.ring = (float *)(w + L.ring);
    b.snap = (float *)(w + L.snap);
    b.G = (float *)(w + L.G);
    b.w = (const float *)(w + L.tab_w);
    b.omw = (const float *)(w + L.tab_omw);
    b.src = (const int *)(w + L.tab_src);
    b.rec = (const int *)(w + L.tab_rec);
    b.uoff = (const int *)(w + L.tab_uoff);
    b.uidx = (const int *)(w + L.tab_uidx);
    b.nsnap = L.nsnap;
    b.status = (int *)(w + L.status);
    Batch3 ba = b;  // the adjoint's ring
    ba.ring = (float *)(w + L.ring2);

    k3_prepare<<<grid_for((long long)nsamples * g.fstride, 256), 256, 0, st>>>(g, vel, (float *)b.vdt, nsamples);
    ++t_launches;
    if (!fwd_only) cudaMemsetAsync(b.G, 0, sizeof(float) * (size_t)g.istride * ninst, st);
    const size_t fb = sizeof(float) * (size_t)g.fstride;
    float *ck = (float *)(w + L.ckpt);
    const size_t ck_pitch = 2 * (size_t)L.nseg * fb;
    const size_t ring_pitch = 3 * fb;
    const int io_threads = 256;
    const int sample_blocks = std::min(64, (g.nr + io_threads - 1) / io_threads);
    const int inject_blocks = std::min(64, (g.nu + io_threads - 1) / io_threads);
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(st, &cs);
    const SideStream *side = split_wave(g, L.resident) ? side_stream(st, cs == cudaStreamCaptureStatusNone) : nullptr;
    for (long long i0 = 0; i0 < ninst; i0 += L.resident) {
        const int nres = (int)std::min<long long>(L.resident, ninst - i0);
        b.inst0 = ba.inst0 = (int)i0;
        const Halves halves(split_wave(g, nres) ? side : nullptr, st, nres);
        bool chained = false;  // the last operation on the streams is a kernel of these chains
        // Forward steps: `record` samples the receivers, one step later (the
        // level of step k - 1 is p1 of step k).
        auto forward = [&](int k, int snap, bool record) {
            Step3 sa{};
            sa.k = k;
            sa.snap = snap;
            sa.wav = a->wavelet[k];
            sa.sample_it = k - 1;
            sa.sample_blocks = record && k > 0 ? sample_blocks : 0;
            halves.each([&](int first, int n, cudaStream_t on) {
                b.slot0 = first;
                step(false, tm, g, b, n, halves.side != nullptr, sa, on, chained);
            });
            chained = true;
        };
        // The pair (p0, p1) of step k between the ring and checkpoint s.
        auto copy_pair = [&](int k, int s, bool save) {
            halves.each([&](int first, int n, cudaStream_t on) {
                for (int hh = 0; hh < 2; ++hh) {
                    char *c0 = (char *)ck + first * ck_pitch + (size_t)(2 * s + hh) * fb;
                    char *r0 = (char *)b.ring + first * ring_pitch + (size_t)((k + hh) % 3) * fb;
                    cudaMemcpy2DAsync(save ? c0 : r0, save ? ck_pitch : ring_pitch, save ? r0 : c0,
                                      save ? ring_pitch : ck_pitch, fb, n, cudaMemcpyDeviceToDevice, on);
                }
            });
            chained = false;
        };
        // forward: data; the stored field (one segment) or the checkpoints
        cudaMemsetAsync(b.ring, 0, 3 * fb * (size_t)nres, st);
        if (!fwd_only) cudaMemsetAsync(ba.ring, 0, 3 * fb * (size_t)nres, st);
        halves.fork();
        for (int k = 0; k < g.nt; ++k) {
            if (!fwd_only && L.nseg > 1 && k % L.K == 0) copy_pair(k, k / L.K, true);
            forward(k, (!fwd_only && L.nseg == 1 && k % g.nti == 0) ? k / g.nti : -1, true);
        }
        halves.each([&](int first, int n, cudaStream_t on) {
            b.slot0 = first;
            launch(k3_sample, dim3(sample_blocks, n), io_threads, 0, on, true, g, b, (g.nt + 1) % 3, g.nt - 1);
        });
        // adjoint, segment by segment from the last
        for (int s = fwd_only ? -1 : L.nseg - 1; s >= 0; --s) {
            const int k0 = s * L.K, k1 = std::min(k0 + L.K, g.nt);
            if (L.nseg > 1) {
                copy_pair(k0, s, false);
                for (int k = k0; k < k1; ++k) forward(k, k % g.nti == 0 ? (k - k0) / g.nti : -1, false);
            }
            for (int it = k1 - 1; it >= k0; --it) {
                Step3 sa{};
                sa.k = g.nt - 1 - it;
                sa.snap = it % g.nti == 0 ? (L.nseg == 1 ? it / g.nti : (it - k0) / g.nti) : -1;
                halves.each([&](int first, int n, cudaStream_t on) {
                    ba.slot0 = first;
                    step(true, tm_adj, g, ba, n, halves.side != nullptr, sa, on, chained);
                    launch(k3_io_adj, dim3(inject_blocks, n), io_threads, 0, on, true, g, ba, sa.k, it, sa.snap);
                });
                chained = true;
            }
        }
        halves.join();
    }
    if (grad && !fwd_only) {
        k3_reduce_grad<<<grid_for((long long)nsamples * g.istride, 256), 256, 0, st>>>(g, b.G, vel, grad, nsamples, b.status);
        ++t_launches;
    }
    if (misfit) {
        double *part = (double *)(w + L.part);
        const long long per = (long long)g.ns * g.nt * g.nr;
        k3_misfit_partial<<<dim3(kMisfitBlocks, nsamples), 256, 0, st>>>(b.syn, obs, per, per, part);
        k3_misfit_final<<<(nsamples + 127) / 128, 128, 0, st>>>(part, misfit, nsamples, b.status);
        t_launches += 2;
    }
    if (syn) {  // after the misfit, which is NaN by the status itself
        const long long n = ninst * g.nt * g.nr;
        k3_data_lost<<<grid_for(n, 256), 256, 0, st>>>(syn, n, b.status);
        ++t_launches;
    }
    return cudaGetLastError() == cudaSuccess ? GB_FWI2D_OK : GB_FWI2D_ECUDA;
}

}  // extern "C"
