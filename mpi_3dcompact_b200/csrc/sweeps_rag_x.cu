// Register-resident line solves of any line length along x (kernel in sweep_reg.cuh).
#include "sweep_reg.cuh"

namespace mc3d {
template int launch_sweep_rag<0, float>(const Grid3 &, const LineOpDev<float> &, const SweepBatch<float> &, int,
                                         const RhsFinalArgs<float> &, int, int, int, cudaStream_t);
template int launch_sweep_rag<0, double>(const Grid3 &, const LineOpDev<double> &, const SweepBatch<double> &, int,
                                          const RhsFinalArgs<double> &, int, int, int, cudaStream_t);
int wait_counter_rag_x(int **dev) {
    MC3D_CUDA_TRY(cudaGetSymbolAddress((void **)dev, g_bulk_wait_timeouts));
    return MC3D_OK;
}
}  // namespace mc3d
