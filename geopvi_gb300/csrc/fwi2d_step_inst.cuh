// fwi2d_step_inst.cuh -- launchers of the step kernels for one FD half width.
#pragma once

#include "fwi2d_step.cuh"

namespace gbfwi {

static cudaLaunchConfig_t step_config(dim3 grid, int smem, cudaStream_t st, bool overlap, cudaLaunchAttribute *attr)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kTileX);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr->id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr->val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cfg;
}

template <int H, int V>
static cudaError_t launch_step_v(bool adj, const StepMaps &m, const Geom &g, const Batch &b, int nres,
                                 const StepArgs &sa, cudaStream_t st, bool overlap)
{
    constexpr StepVariant v = kStepVariants[V];
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg =
        step_config(dim3(nres, step_tiles(g, v.rows)), TileShape<H, v.rows>::kSmem, st, overlap, &attr);
    return adj ? cudaLaunchKernelEx(&cfg, k_step<H, true, v.rows, v.min_blocks>, m, g, b, sa)
               : cudaLaunchKernelEx(&cfg, k_step<H, false, v.rows, v.min_blocks>, m, g, b, sa);
}

template <int H>
cudaError_t launch_step_h(bool adj, const StepMaps &m, const Geom &g, const Batch &b, int nres, const StepArgs &sa,
                          cudaStream_t st, int variant, bool overlap)
{
    static_assert(kNumStepVariants == 4, "one case per entry of kStepVariants");
    switch (variant) {
    case 1: return launch_step_v<H, 1>(adj, m, g, b, nres, sa, st, overlap);
    case 2: return launch_step_v<H, 2>(adj, m, g, b, nres, sa, st, overlap);
    case 3: return launch_step_v<H, 3>(adj, m, g, b, nres, sa, st, overlap);
    default: return launch_step_v<H, 0>(adj, m, g, b, nres, sa, st, overlap);
    }
}

template <int H, int V, int NP>
static cudaError_t launch_multi_np(bool adj, const MultiArgs &full, int nact, int k, cudaStream_t st, bool overlap)
{
    constexpr StepVariant v = kStepVariants[V];
    MultiArgsN<NP> a;
    a.tm = full.tm;
    a.gc = full.gc;
    a.coef = full.coef;
    a.status = full.status;
    a.blend_fp32 = full.blend_fp32;
    a.imaging = full.imaging;
    a.store = full.store;
    a.npieces = full.npieces;
    a.tl = full.tl;
    for (int q = 0; q <= NP; ++q) a.first[q] = full.first[q];
    for (int q = 0; q < NP; ++q) a.piece[q] = full.piece[q];
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg =
        step_config(dim3((unsigned)full.first[nact]), TileShape<H, v.rows>::kSmem, st, overlap, &attr);
    return adj ? cudaLaunchKernelEx(&cfg, k_step_multi<H, true, v.rows, v.min_blocks, NP>, a, nact, k)
               : cudaLaunchKernelEx(&cfg, k_step_multi<H, false, v.rows, v.min_blocks, NP>, a, nact, k);
}

// The smallest parameter table that holds the launch's pieces.
template <int H, int V>
static cudaError_t launch_multi_v(bool adj, const MultiArgs &args, int nact, int k, cudaStream_t st, bool overlap)
{
    static_assert(kMaxPieces == 16, "tables of 1, 4 and 16 pieces");
    if (args.npieces <= 1) return launch_multi_np<H, V, 1>(adj, args, nact, k, st, overlap);
    if (args.npieces <= 4) return launch_multi_np<H, V, 4>(adj, args, nact, k, st, overlap);
    return launch_multi_np<H, V, 16>(adj, args, nact, k, st, overlap);
}

template <int H>
cudaError_t launch_multi_h(bool adj, const MultiArgs &args, int nact, int k, cudaStream_t st, int variant,
                           bool overlap)
{
    switch (variant) {
    case 1: return launch_multi_v<H, 1>(adj, args, nact, k, st, overlap);
    case 2: return launch_multi_v<H, 2>(adj, args, nact, k, st, overlap);
    case 3: return launch_multi_v<H, 3>(adj, args, nact, k, st, overlap);
    default: return launch_multi_v<H, 0>(adj, args, nact, k, st, overlap);
    }
}

}  // namespace gbfwi
