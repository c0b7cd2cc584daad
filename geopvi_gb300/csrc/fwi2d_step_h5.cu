// fwi2d_step_h5.cu -- the FD time step with half width 5 (order 10).
#include "fwi2d_step_inst.cuh"

namespace gbfwi {

template cudaError_t launch_step_h<5>(bool, const StepMaps &, const Geom &, const Batch &, int, const StepArgs &,
                                      cudaStream_t, int, bool);
template cudaError_t launch_multi_h<5>(bool, const MultiArgs &, int, int, cudaStream_t, int, bool);

}  // namespace gbfwi
