// plane_rx.cuh kernels for dim 3 in FP64.
#include "sweep_rx.inl"

namespace pscfg {

RX3_INSTANCES(double)
template int rx3_half<double>(const RxPlan &, cudaStream_t, const SweepField<double> *, int);   // (the adjoint: FP64 alone)

}  // namespace pscfg
