// pf3d_marchsub.cu -- the z-marching passes that run one subroutine alone (FP64
// reference form, FP32 fast form).  Built without automatic multiply-add
// contraction, like every unit that inlines the per-cell arithmetic.
#include "pf3d_march.cuh"

namespace pf3d {
template cudaError_t launch_march_sweep<double>(const CUtensorMap&, const DomainDesc&, const StepArgs&, const void*, void*, void*, int, int*, cudaStream_t);
template cudaError_t launch_march_sweep<float>(const CUtensorMap&, const DomainDesc&, const StepArgs&, const void*, void*, void*, int, int*, cudaStream_t);
template cudaError_t launch_march_solute<double>(const CUtensorMap&, const DomainDesc&, const StepArgs&, const void*, void*, int, int*, cudaStream_t);
template cudaError_t launch_march_solute<float>(const CUtensorMap&, const DomainDesc&, const StepArgs&, const void*, void*, int, int*, cudaStream_t);
}  // namespace pf3d
