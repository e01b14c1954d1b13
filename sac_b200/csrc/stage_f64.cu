// stage_f64.cu -- the stage kernels instantiated for double storage; built with
// --fmad=false and IEEE division so that every expression rounds as the reference.
#include "sac_stage.cuh"
#include "sac_stage2d.cuh"
#include "sac_step1d.cuh"

namespace sacgpu {
template void launch_face<double>(const Stage2Args&, int, cudaStream_t);
template void launch_nu<double>(const Stage2Args&, cudaStream_t);
template void launch_update<double>(const Stage2Args&, cudaStream_t);
template void launch_cross<double>(const Stage2Args&, cudaStream_t);
template void launch_batch_face<double>(const BatchStageArgs&, double, cudaStream_t);
template void launch_batch_nu<double>(const BatchStageArgs&, cudaStream_t);
template void launch_batch_update<double>(const BatchStageArgs&, dim3, cudaStream_t);
template void launch_batch_courant<double>(const BatchStageArgs&, double, cudaStream_t);
template void launch_batch_ctot<double>(const BatchStageArgs&, cudaStream_t);
template cudaError_t launch_batch_stage2d<double>(const BatchStageArgs&, int, cudaStream_t);
template cudaError_t launch_step1d<double>(const Step1dArgs&, cudaStream_t);

void launch_count_divides(const Stage2Args& a, cudaStream_t st) {
  const Geom& g = a.g;
  const int n0 = g.hi[0] - g.lo[0] + 1, n1 = g.hi[1] - g.lo[1] + 1, n2 = g.hi[2] - g.lo[2] + 1;
  const dim3 blk(32, 8, 1), grd((n0 + 31) / 32, (n1 + 7) / 8, n2);
  if (g.ndim == 2)
    k_count_divides<2><<<grd, blk, 0, st>>>(a);
  else
    k_count_divides<3><<<grd, blk, 0, st>>>(a);
}
}  // namespace sacgpu
